// What gemm.cu needs of the shared-memory tcgen05 kernel in gemm_tile.cu.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace atlas {

struct TileParams {
    const uint16_t *scales_t;   // [row/128][block][row%128]
    const int32_t *chunk_ptr;   // [strip][k_tiles + 1]
    const uint32_t *entries;    // row%16 << 24 | column, strip-major, column-sorted
    const uint16_t *ovals;      // values in the order of `entries`
    const uint16_t *bias;
    void *y;
    int64_t ldy;
    int m;
    int n_rows;
    int bs;
    int k_tiles;
    int blocks_per_row;
    int bs_tiles;    // k-tiles per scale block when block_size % 64 == 0 (scales staged by the producer), else 0
    int out_bf16;
    int x_bf16;      // the tensor map delivers bf16 rows: converted in the kernel
    int splits;      // K slices = CTAs of a cluster
    int *error_flag;
};

// Rows of x the kernel takes, and tokens per tile for m of them.
constexpr int TILE_MAX_TOKENS = 128;
int tile_tokens_for(int64_t m);

// How the kernel would run a shape, and about how long it would take.
struct TilePlan {
    int splits;      // K slices
    bool convert;    // bf16 rows are converted in the kernel, not by a copy kernel in front of it
    double us;
};
// A copy kernel in front of either kernel: one more launch in the chain, and its traffic.
inline double copy_us(int64_t m, int64_t k_tiles) { return 1. + 5.1e-5 * (double)m * (double)k_tiles; }
// can_convert: the rows are bf16 and a tensor map can take them as they are; needs_copy: a copy kernel makes them dense
// fp16 unless the kernel converts.
TilePlan plan_tile(int64_t m, int64_t n_rows, int k_tiles, bool can_convert, bool needs_copy, int sms);

// x_map: boxes of 64 columns x tile_tokens_for(m) rows, 128-byte swizzle; c_map: the code tiles as 64-byte rows, boxes
// of 128 rows, 64-byte swizzle.
int launch_tile(const CUtensorMap &x_map, const CUtensorMap &c_map, const TileParams &p, cudaStream_t st);

}  // namespace atlas
