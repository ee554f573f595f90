// Adaptive hybrid quantizer for sm_100a: one pass over the fp16 weights.
//
// Replaces quantize_tensor (atlasinfer_core/quant/adaptive_quantizer.py:51-148).
// The reference walks the blocks in a Python loop and concatenates four
// streams; here a persistent grid takes tiles of 8192 elements in order
// (dynamic tile ids), evaluates every block of a tile on chip, and
// finds where the tile's compacted codes and outliers start in the output
// through a decoupled look-back over per-tile outlier counts, so the input is
// read once and every output byte is written once.
//
// Bit-exactness contract (what PyTorch's CPU kernels compute for fp16 blocks):
//   mean  = fp16(S / n), S = fp32 sum in ATen's vectorised order: 8 lanes
//           (element i -> lane i % 8), four interleaved accumulators per lane
//           (8-wide chunk j -> accumulator j % 4), folded ((a0+a1)+a2)+a3,
//           lanes added 0..7                              (:46, torch.mean)
//   std   = fp16((float)sqrt(M2 / (n - 1))), M2 in fp64      (:47, torch.std)
//   z     = fp16(fp16(x - mean) / fp16(std + fp16(1e-6)))    (:49)
//   outlier iff |z| > fp16(z_threshold)                      (:107)
//   scale = max(fp16(max|non-outlier| / 127), fp16(1e-6)); 1.0 if none (:121-130)
//   code  = int8(clamp(rint(fp16(x / scale)), -127, 127))    (:125-126)
// The fp64 second moment is a two-pass sum here and a Welford recurrence in
// ATen; both carry ~1e-16 relative error, far below the fp16 rounding step.
#include <cmath>
#include <mutex>

#include "common.cuh"

namespace atlas {
namespace {

constexpr int QT_THREADS = 256;
constexpr int QT_TILE = 8192;             // elements per tile
constexpr int QT_WORDS = QT_TILE / 32;    // outlier-mask words per tile
constexpr int QT_MAX_BLOCKS = QT_TILE / 32;
constexpr int QT_SPIN_LIMIT = 1 << 20;    // bounded look-back wait (~0.1 s)

constexpr unsigned long long ST_AGG = 1ull << 62;     // tile's own outlier count is known
constexpr unsigned long long ST_PREFIX = 2ull << 62;  // inclusive count up to this tile is known
constexpr unsigned long long ST_VALUE = (1ull << 62) - 1;

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_u64(unsigned long long *p, unsigned long long v) {
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ float h2f_bits(uint16_t b) { return __half2float(__ushort_as_half(b)); }
__device__ __forceinline__ uint16_t f2h_bits(float f) { return __half_as_ushort(__float2half_rn(f)); }

// int8 code of one value given the block's fp32 scale: adaptive_quantizer.py:125-126.
__device__ __forceinline__ int quant_code(float xf, float scale_f) {
    float q = h2f_bits(f2h_bits(__fdiv_rn(xf, scale_f)));  // quotient rounded to fp16 first
    float r = rintf(q);                                     // half to even, as torch.round
    r = fminf(fmaxf(r, -127.0f), 127.0f);
    return (int)r;
}

struct QuantParams {
    const uint16_t *x;
    int64_t numel;
    int64_t padded;
    int64_t n_blocks;
    int64_t num_tiles;
    int bs;
    uint16_t thr_h;
    int8_t *codes;
    uint16_t *ovals;
    int64_t *oidx;
    int64_t ocap;
    uint16_t *scales;
    int64_t *counts;
    unsigned int *tile_counter;
    unsigned long long *status;
    int in_aligned;   // x is 16-byte aligned
    int out_aligned;  // codes is 16-byte aligned
    int tile;         // elements per tile: the largest multiple of the block size <= QT_TILE
};

__global__ void __launch_bounds__(QT_THREADS) quantize_kernel(QuantParams p) {
    __shared__ __align__(16) uint16_t s_x[QT_TILE];
    __shared__ __align__(16) uint8_t s_codes[QT_TILE + 32];
    __shared__ uint32_t s_mask[QT_WORDS];
    __shared__ uint32_t s_wordpre[QT_WORDS];
    __shared__ uint16_t s_scale[QT_MAX_BLOCKS];
    __shared__ uint32_t s_warp_tot[QT_THREADS / 32];
    __shared__ long long s_tile_prefix;
    __shared__ int s_tile_total;
    __shared__ unsigned int s_tile;

    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int bs = p.bs;
    const uint16_t eps_h = f2h_bits(1e-6f);
    const float eps_f = h2f_bits(eps_h);
    const float thr_f = h2f_bits(p.thr_h);

    for (;;) {
        __syncthreads();  // previous tile's shared state is no longer read
        if (tid == 0) s_tile = atomicAdd(p.tile_counter, 1u);
        __syncthreads();
        const int64_t tile = s_tile;
        if (tile >= p.num_tiles) break;
        const int64_t tile_base = tile * p.tile;   // tiles hold whole blocks
        const int tile_elems = (int)min((int64_t)p.tile, p.padded - tile_base);
        const int tile_real = (int)max((int64_t)0, min((int64_t)tile_elems, p.numel - tile_base));
        const int tile_blocks = tile_elems / bs;

        // ---- stage the tile (zero padding included) -------------------------------
        if (p.in_aligned) {
            const uint4 *src = reinterpret_cast<const uint4 *>(p.x + tile_base);
            for (int v = tid; v < QT_TILE / 8; v += QT_THREADS) {
                int e0 = v * 8;
                if (e0 + 8 <= tile_real) {
                    reinterpret_cast<uint4 *>(s_x)[v] = __ldg(src + v);
                } else if (e0 < tile_elems) {
                    for (int e = e0; e < e0 + 8; ++e) s_x[e] = (e < tile_real) ? p.x[tile_base + e] : (uint16_t)0;
                }
            }
        } else {
            for (int e = tid; e < tile_elems; e += QT_THREADS)
                s_x[e] = (e < tile_real) ? p.x[tile_base + e] : (uint16_t)0;
        }
        for (int w = tid; w < QT_WORDS; w += QT_THREADS) s_mask[w] = 0u;
        __syncthreads();

        // ---- phase A: per-block statistics, 8 threads per block ----------------------
        {
            const int l = tid & 7;    // ATen SIMD lane this thread plays
            const int grp = tid >> 3;
            const unsigned gmask = 0xffu << (lane & 24);
            const int nv = bs >> 3;   // 8-wide chunks per block (multiple of 4)
            for (int b = grp; b < tile_blocks; b += QT_THREADS / 8) {
                const uint16_t *xb = s_x + b * bs;
                // fp32 sum in ATen's order + exact fp64 sum
                float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
                double dsum = 0.0;
                for (int j = 0; j < nv; j += 4) {
                    float f0 = h2f_bits(xb[(j + 0) * 8 + l]);
                    float f1 = h2f_bits(xb[(j + 1) * 8 + l]);
                    float f2 = h2f_bits(xb[(j + 2) * 8 + l]);
                    float f3 = h2f_bits(xb[(j + 3) * 8 + l]);
                    a0 = __fadd_rn(a0, f0);
                    a1 = __fadd_rn(a1, f1);
                    a2 = __fadd_rn(a2, f2);
                    a3 = __fadd_rn(a3, f3);
                    dsum += ((double)f0 + (double)f1) + ((double)f2 + (double)f3);  // exact
                }
                float lane_sum = __fadd_rn(__fadd_rn(__fadd_rn(a0, a1), a2), a3);
                float fin = 0.f;
#pragma unroll
                for (int s = 0; s < 8; ++s) fin = __fadd_rn(fin, __shfl_sync(gmask, lane_sum, s, 8));
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) dsum += __shfl_xor_sync(gmask, dsum, o, 8);
                const float mean_f = h2f_bits(f2h_bits(__fdiv_rn(fin, (float)bs)));
                const double mean_d = dsum / (double)bs;
                // second moment in fp64
                double m2 = 0.0;
                for (int j = 0; j < nv; ++j) {
                    double d = (double)h2f_bits(xb[j * 8 + l]) - mean_d;
                    m2 = fma(d, d, m2);
                }
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) m2 += __shfl_xor_sync(gmask, m2, o, 8);
                const double var = m2 / (double)(bs - 1);
                const float std_f = h2f_bits(f2h_bits(__double2float_rn(sqrt(var))));
                const float den_f = h2f_bits(f2h_bits(__fadd_rn(std_f, eps_f)));
                // z test, outlier mask, absmax of the rest
                int cnt = 0;
                unsigned int maxabs = 0;  // fp16 magnitude bits order like the values
                for (int j = 0; j < nv; ++j) {
                    const int e = j * 8 + l;
                    const uint16_t xbits = xb[e];
                    const float xf = h2f_bits(xbits);
                    const float d = h2f_bits(f2h_bits(__fsub_rn(xf, mean_f)));
                    const float z = h2f_bits(f2h_bits(__fdiv_rn(d, den_f)));
                    if (fabsf(z) > thr_f) {
                        const int pos = b * bs + e;
                        atomicOr(&s_mask[pos >> 5], 1u << (pos & 31));
                        cnt++;
                    } else {
                        maxabs = max(maxabs, (unsigned int)(xbits & 0x7fffu));
                    }
                }
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) {
                    cnt += __shfl_xor_sync(gmask, cnt, o, 8);
                    maxabs = max(maxabs, __shfl_xor_sync(gmask, maxabs, o, 8));
                }
                if (l == 0) {
                    uint16_t sc = 0x3c00u;  // 1.0 when the block has no non-outliers
                    if (cnt < bs) {
                        sc = f2h_bits(__fdiv_rn(h2f_bits((uint16_t)maxabs), 127.0f));
                        if (h2f_bits(sc) < eps_f) sc = eps_h;
                    }
                    s_scale[b] = sc;
                }
            }
        }
        __syncthreads();

        // ---- exclusive scan of outliers per mask word --------------------------------
        {
            const uint32_t c = __popc(s_mask[tid]);  // QT_WORDS == QT_THREADS
            uint32_t inc = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                uint32_t n = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += n;
            }
            if (lane == 31) s_warp_tot[warp] = inc;
            __syncthreads();
            uint32_t wbase = 0;
            for (int w = 0; w < warp; ++w) wbase += s_warp_tot[w];
            s_wordpre[tid] = wbase + inc - c;
            if (tid == QT_THREADS - 1) s_tile_total = (int)(wbase + inc);
        }
        __syncthreads();

        // ---- decoupled look-back over tiles (warp 0) -------------------------------------
        if (warp == 0) {
            const unsigned long long agg = (unsigned long long)s_tile_total;
            long long prefix = 0;
            if (tile == 0) {
                if (lane == 0) st_release_u64(p.status, ST_PREFIX | agg);
            } else {
                if (lane == 0) st_release_u64(p.status + tile, ST_AGG | agg);
                int64_t look = tile - 1;
                bool done = false;
                while (!done) {
                    const int64_t idx = look - lane;
                    unsigned long long v = ST_PREFIX;  // tiles before the first count as prefix 0
                    int spins = 0;
                    bool gave_up = false;
                    for (;;) {
                        if (idx >= 0) v = ld_acquire_u64(p.status + idx);
                        const bool ready = (v >> 62) != 0;
                        if (__all_sync(0xffffffffu, ready)) break;
                        if (++spins > QT_SPIN_LIMIT) { gave_up = true; break; }
                        __nanosleep(64);
                    }
                    if (gave_up) {  // record and leave; the host reports ATLAS_ERR_TIMEOUT
                        if (lane == 0) atomicExch((unsigned long long *)&p.counts[2], 1ull);
                        break;
                    }
                    const unsigned pm = __ballot_sync(0xffffffffu, (v >> 62) == 2);
                    const int first = pm ? (__ffs(pm) - 1) : 32;
                    long long contrib = (lane <= first) ? (long long)(v & ST_VALUE) : 0;
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) contrib += __shfl_xor_sync(0xffffffffu, contrib, o);
                    prefix += contrib;
                    if (pm) done = true; else look -= 32;
                }
                if (lane == 0) st_release_u64(p.status + tile, ST_PREFIX | (unsigned long long)(prefix + (long long)agg));
            }
            if (lane == 0) {
                s_tile_prefix = prefix;
                if (tile == p.num_tiles - 1) {
                    const long long total_out = prefix + (long long)agg;
                    p.counts[0] = p.padded - total_out;
                    p.counts[1] = total_out;
                }
            }
        }
        __syncthreads();

        // ---- phase B: codes into a shared staging buffer, outliers straight out --------
        const long long tile_prefix = s_tile_prefix;
        const int64_t code_base = tile_base - tile_prefix;  // where this tile's codes start
        const int shift = p.out_aligned ? (int)(code_base & 15) : 0;
        for (int i = tid * 4; i < tile_elems; i += QT_THREADS * 4) {
            const float sc_f = h2f_bits(s_scale[i / bs]);
            const uint32_t word = s_mask[i >> 5];
            const uint32_t m4 = (word >> (i & 31)) & 0xfu;
            int before = (int)s_wordpre[i >> 5] + __popc(word & ((1u << (i & 31)) - 1u));
            const uint2 raw = *reinterpret_cast<const uint2 *>(s_x + i);
            const uint16_t xs[4] = {(uint16_t)(raw.x & 0xffffu), (uint16_t)(raw.x >> 16),
                                    (uint16_t)(raw.y & 0xffffu), (uint16_t)(raw.y >> 16)};
            const int dst = shift + i - before;
            if (m4 == 0u && (dst & 3) == 0) {
                uint32_t packed = 0;
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    packed |= (uint32_t)(quant_code(h2f_bits(xs[e]), sc_f) & 0xff) << (8 * e);
                *reinterpret_cast<uint32_t *>(s_codes + dst) = packed;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    if ((m4 >> e) & 1u) {
                        const long long pos = tile_prefix + before;
                        if (pos < p.ocap) {
                            p.ovals[pos] = xs[e];
                            p.oidx[pos] = tile_base + i + e;
                        }
                        before++;
                    } else {
                        s_codes[shift + i + e - before] = (uint8_t)quant_code(h2f_bits(xs[e]), sc_f);
                    }
                }
            }
        }
        __syncthreads();

        // ---- copy the compacted codes out: 16-byte stores inside, bytes at the ragged ends --
        {
            const int total = tile_elems - s_tile_total;  // code bytes of this tile
            const int end = shift + total;
            int8_t *gdst = p.codes + (code_base - shift);  // 16-byte aligned when out_aligned
            const int nchunks = (end + 15) >> 4;
            for (int c = tid; c < nchunks; c += QT_THREADS) {
                const int lo = c << 4;
                if (p.out_aligned && lo >= shift && lo + 16 <= end) {
                    *reinterpret_cast<uint4 *>(gdst + lo) = *reinterpret_cast<const uint4 *>(s_codes + lo);
                } else {
                    const int a = max(lo, shift), z = min(lo + 16, end);
                    for (int q = a; q < z; ++q) gdst[q] = (int8_t)s_codes[q];
                }
            }
            const int64_t block0 = tile_base / bs;
            for (int b = tid; b < tile_blocks; b += QT_THREADS) p.scales[block0 + b] = s_scale[b];
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Fast variant for block sizes 32 / 64 / 128 / 256, up to 16 tensors per launch.  Same results as quantize_kernel above, bit
// for bit.  11008 x 4096 in blocks of 128: 120 us, 54 M warp instructions, 43 % of the issue slots used; the seven weights of
// a 7B-shaped layer in one launch instead of seven, with their outliers copied by one kernel instead of fourteen copies:
// 777 -> 600 us through quantize_tensors.
//
// Eight warps of a CTA hold a tile's elements in registers, a ninth numbers the tiles and looks back.  A tile's codes and
// outlier mask stay in shared memory while the next tile is worked on, and are written out after it: by then its place in
// the streams is known, and the elements of the tile after that are on their way.  A tile so costs one CTA barrier.  What
// the warps wait for is that barrier (8 of 20 cycles per instruction) and the loads (5 of 20).
//
// Four threads work on a block (eight on one of 256); thread t holds the 8-wide chunks t, t + 4, ..., that is ATen's
// accumulator t of all eight SIMD lanes, so that a chunk is one 16-byte load; the accumulators change hands through 1 KB of
// shared memory per warp.  Values stay packed two to a register and most steps cost one instruction per pair (fp32 pairs:
// add, mul and fma.rn.f32x2).  What replaces the IEEE divisions and the fp64 moment, and why the results are the same:
//   * code.  x and the scale have 11-bit significands, so a quotient x / scale is never the midpoint of two fp16 numbers
//     (scale times a midpoint's odd 12-bit significand needs more than 11 bits) and is more than 2^-23 away from one,
//     relatively: |a 2^k - m b| >= 1 with m < 2^12, b < 2^11.  x * (1 / scale), two roundings to fp32, is within 2^-23:
//     it rounds to the same fp16 number.  (Quotients below the fp16 normal range give code 0 either way.)  Adding 1536
//     in fp16, where the spacing is 1, rounds half to even and leaves the two's-complement code in the low byte.
//   * scale.  maxabs * (1 / 127) instead of maxabs / 127 by the same argument.
//   * z test.  fp16(|d| / den) > thr iff |d| lies above T * den, T the midpoint between thr and the next fp16 number:
//     12 by 11 bits, exact in fp32.  |d| is an fp16 number, so it is compared in fp16 with the largest one that does not
//     exceed T * den.  A tie (only possible for subnormal thresholds) goes to the even neighbour: if thr is odd, |d| =
//     T * den is an outlier too.
//   * d = fp16(x - mean) is one fp16 subtraction.
//   * standard deviation.  fp32 sum of squares minus the squared sum, if the mean takes less than a fifth of it away, else a
//     second pass about the mean; only if rounding it to fp16 could go either way within 4e-6 is it recomputed in fp64
//     (about 1 % of blocks).  The bound, with u = 2^-24, Q the sum of squares, M = Q - F^2 / n the second moment and blocks
//     of 256, the longest sums: Q carries at most 31 additions of a thread and 3 across threads, 34 u Q.  F carries 7 + 3 in a lane
//     and 7 over the lanes, 17 u sum|x| <= 17 u sqrt(n Q), and |F| <= sqrt(0.2 n Q) here, so F^2 / n is off by
//     2 * 0.45 * 17 u Q = 15 u Q.  With Q <= 1.25 M that is 62 u of M, 31 u of its root, and 4 u for the product, the root
//     and the rounding of M: 35 u = 2.1e-6.  The second pass adds at most 64 times (66 u with the shuffles, 2 u for the squared
//     differences), 34 u of the root, and 4 u as above: 2.3e-6; the mean it is taken about enters only through r1^2 / n,
//     which is small because values that round in F make the block spread by a thirtieth of the largest at least.  (The
//     largest error in an emulation over 4.8 M blocks of six kinds, offsets and wide exponents among them: 6.5e-7.)
// The dense codes of a tile go to shared memory once; the compaction is driven by the output: a thread finds where its 16
// bytes of the code stream start in the tile, takes them with one unaligned read, and squeezes out the places of outliers.
struct FastConsts {
    float T;         // |z| decision boundary
    int tie_out;     // an exact tie is an outlier
};

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_u64(unsigned long long *p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// One tensor of a launch.
struct QuantItem {
    const uint16_t *x;
    int8_t *codes;
    uint16_t *ovals;
    int64_t *oidx;
    uint16_t *scales;
    int64_t *counts;
    int64_t numel, padded, ocap;
    int64_t first_tile;   // of this tensor, among the tiles of the launch
    int in_aligned;       // x is 16-byte aligned
    int out_aligned;      // codes is 16-byte aligned
};
constexpr int QF_MAX_ITEMS = 16;
struct QuantBatch {
    QuantItem item[QF_MAX_ITEMS];
    int n;
    unsigned int num_tiles;
    unsigned int *tile_counter;
    unsigned long long *status;   // one word per tile
};

constexpr int QF_WORKERS = 8;                        // warps that work on elements: 1024 of a tile each
constexpr int QF_THREADS = (QF_WORKERS + 1) * 32;    // and one for the tile numbers and the look-back
constexpr int QF_CTAS = 4;                           // per SM: 56 registers
constexpr int QF_BUFS = 3;                           // tiles a CTA holds codes of
static_assert(QF_WORKERS * 1024 == QT_TILE && QT_WORDS == QF_WORKERS * 32, "a warp's elements are its 32 mask words");

// Outliers of the launch's tiles [first, tile) (whole warp).  A status word holds all that is passed on, so relaxed
// accesses do; a round trip covers 256 tiles.
__device__ __forceinline__ long long look_back(const unsigned long long *status, int64_t first, int64_t tile, int lane, int64_t *counts) {
    long long prefix = 0;
    int64_t look = tile - 1;
    for (int spins = 0; spins <= QT_SPIN_LIMIT; ++spins) {
        unsigned long long v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int64_t idx = look - k * 32 - lane;
            v[k] = idx >= first ? ld_relaxed_u64(status + idx) : ST_PREFIX;   // tiles before the tensor's first count as prefix 0
        }
        int taken = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (taken != k) continue;
            const unsigned pm = __ballot_sync(0xffffffffu, (v[k] >> 62) == 2), none = __ballot_sync(0xffffffffu, (v[k] >> 62) == 0);
            const int first_pm = pm ? __ffs(pm) - 1 : 31;
            if (none & (0xffffffffu >> (31 - first_pm))) continue;       // not there yet
            unsigned int contrib = lane < first_pm || (!pm && lane == first_pm) ? (unsigned int)(v[k] & ST_VALUE) : 0u;   // a tile's own count
            prefix += (long long)__reduce_add_sync(0xffffffffu, contrib);
            if (pm) return prefix + (long long)(__shfl_sync(0xffffffffu, v[k], first_pm) & ST_VALUE);
            ++taken;
        }
        look -= taken * 32;
        if (taken == 0) __nanosleep(32);
    }
    if (lane == 0) atomicExch((unsigned long long *)&counts[2], 1ull);   // record and leave; the host reports ATLAS_ERR_TIMEOUT
    return prefix;
}

// Byte offset of element e's code in the dense tile: 32-byte pieces permuted so that the four 128-element runs a
// half-warp stores to fall on different banks.
__device__ __forceinline__ int dense_byte(int e) { return e ^ (((e >> 7) & 3) << 5); }

// Two fp32 values in one register pair: one instruction works on both.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float2 h2f2(uint32_t v) { return __half22float2(*reinterpret_cast<const __half2 *>(&v)); }

// Values held packed are converted anew in every pass: the compiler must not keep 32 floats for the next one.
__device__ __forceinline__ void forget(uint4 (&x)[4]) {
#pragma unroll
    for (int c = 0; c < 4; ++c) asm volatile("" : "+r"(x[c].x), "+r"(x[c].y), "+r"(x[c].z), "+r"(x[c].w));
}

struct FastShared {
    __align__(16) uint8_t dense[QF_BUFS][QT_TILE + 128];
    __align__(16) float fold[QF_WORKERS][256];       // accumulators of a warp, on their way to the threads that add them
    __align__(16) uint32_t mask[QF_BUFS][QT_WORDS + 4];   // bit e & 31 of word e >> 5: element e is an outlier
    uint32_t word_before[QF_BUFS][QT_WORDS];         // outliers before the word, counted in its warp's elements
    uint32_t warp_total[QF_BUFS][QF_WORKERS];
    uint32_t warp_base[QF_BUFS][QF_WORKERS + 1];     // outliers of the tile before the warp's elements; the last: of the tile
    long long prefix[2];                             // outliers of the tensor before the tile
    unsigned int tile[4];
    int item[4];
};

// The 32 elements (four runs of eight) of this thread in a tile; zeros beyond the tensor's end.
template <class At>
__device__ __forceinline__ void load_elements(const QuantItem &q, int64_t tile_base, const At &at, uint4 (&x)[4]) {
    const uint16_t *src = q.x + tile_base;
    const int real = (int)min((int64_t)QT_TILE, q.numel - tile_base);
    if (q.in_aligned && real == QT_TILE) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
            asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                         : "=r"(x[c].x), "=r"(x[c].y), "=r"(x[c].z), "=r"(x[c].w) : "l"(src + at(c)));
        return;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int e = at(c);
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            w[i] = e + 2 * i < real ? __ldg(src + e + 2 * i) : 0u;
            if (e + 2 * i + 1 < real) w[i] |= (uint32_t)__ldg(src + e + 2 * i + 1) << 16;
        }
        x[c] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// Second moment of a block about its mean as fp32 has it, the first moment about that taken out again, so that the
// rounding of the mean itself only enters to second order (whole warp; x0 ... x3: the thread's runs of the block, the
// first four, two or one of them for blocks of 128 and more, 64 and 32).  Rare, so it is a call: inlined, its registers
// would spill the others'.
template <int BS>
__device__ __noinline__ float moment_about(uint4 x0, uint4 x1, uint4 x2, uint4 x3, float mean) {
    constexpr int NW = BS < 128 ? BS / 8 : 16, GROUP = BS == 256 ? 8 : 4;
    const uint32_t xw[16] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w, x2.x, x2.y, x2.z, x2.w, x3.x, x3.y, x3.z, x3.w};
    float r1 = 0.f, m2 = 0.f;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        const float2 f = h2f2(xw[w]);
        const float d0 = f.x - mean, d1 = f.y - mean;
        r1 += d0 + d1;
        m2 = fmaf(d0, d0, fmaf(d1, d1, m2));
    }
#pragma unroll
    for (int o = 1; o < GROUP; o <<= 1) {
        m2 += __shfl_xor_sync(0xffffffffu, m2, o);
        r1 += __shfl_xor_sync(0xffffffffu, r1, o);
    }
    return fmaxf(fmaf(-r1, r1 * (1.f / (float)BS), m2), 0.f);
}

// fp16 standard deviation of a block from fp64 moments (as above).
template <int BS>
__device__ __noinline__ uint16_t std_in_fp64(uint4 x0, uint4 x1, uint4 x2, uint4 x3) {
    constexpr int NW = BS < 128 ? BS / 8 : 16, GROUP = BS == 256 ? 8 : 4;
    const uint32_t xw[16] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w, x2.x, x2.y, x2.z, x2.w, x3.x, x3.y, x3.z, x3.w};
    double dsum = 0.0;
#pragma unroll
    for (int w = 0; w < NW; ++w) { const float2 f = h2f2(xw[w]); dsum += (double)f.x + (double)f.y; }
#pragma unroll
    for (int o = 1; o < GROUP; o <<= 1) dsum += __shfl_xor_sync(0xffffffffu, dsum, o);
    const double mean = dsum / (double)BS;
    double m2 = 0.0;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        const float2 f = h2f2(xw[w]);
        const double d0 = (double)f.x - mean, d1 = (double)f.y - mean;
        m2 = fma(d0, d0, fma(d1, d1, m2));
    }
#pragma unroll
    for (int o = 1; o < GROUP; o <<= 1) m2 += __shfl_xor_sync(0xffffffffu, m2, o);
    return f2h_bits(__double2float_rn(sqrt(m2 / (double)(BS - 1))));
}

template <int BS>
__global__ void __launch_bounds__(QF_THREADS, QF_CTAS) quantize_fast_kernel(const __grid_constant__ QuantBatch p, FastConsts fc) {
    constexpr int NB = BS < 128 ? 128 / BS : 1;   // blocks a thread has a part of
    constexpr int CK = 4 / NB;                    // its runs of eight in each
    __shared__ FastShared s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr unsigned ALL = 0xffffffffu, NO_TILE = 0xffffffffu;

    if (warp == QF_WORKERS) {
        // ---- the warp that numbers the tiles and looks back -------------------------------------------
        const int64_t item_first = lane < p.n ? p.item[lane].first_tile : INT64_MAX;
        auto fetch = [&](int slot) {
            unsigned int t = 0;
            if (lane == 0) t = atomicAdd(p.tile_counter, 1u);
            t = __shfl_sync(ALL, t, 0);
            const int it = __popc(__ballot_sync(ALL, item_first <= (int64_t)t)) - 1;
            if (lane == 0) {
                s.tile[slot] = t < p.num_tiles ? t : NO_TILE;
                s.item[slot] = it;
            }
        };
        if (lane < QF_BUFS) s.mask[lane][QT_WORDS] = 0u;
        fetch(0);
        __syncthreads();
        unsigned int prev = NO_TILE;
        int prev_item = 0;
        long long prev_total = 0;
        for (int i = 0, buf = 0;; ++i, buf = buf == QF_BUFS - 1 ? 0 : buf + 1) {
            const unsigned int cur = s.tile[i & 3];
            const int cur_item = s.item[i & 3];
            if (cur != NO_TILE) fetch((i + 1) & 3);
            if (prev != NO_TILE) {
                const QuantItem &q = p.item[prev_item];
                long long prefix = 0;
                if (prev != q.first_tile) {
                    prefix = look_back(p.status, q.first_tile, prev, lane, q.counts);
                    if (lane == 0) st_relaxed_u64(p.status + prev, ST_PREFIX | (unsigned long long)(prefix + prev_total));
                }
                if (lane == 0) {
                    s.prefix[(i - 1) & 1] = prefix;
                    if (((int64_t)prev - q.first_tile + 1) * QT_TILE >= q.padded) {   // the tensor's last tile
                        q.counts[0] = q.padded - (prefix + prev_total);
                        q.counts[1] = prefix + prev_total;
                    }
                }
            }
            __syncthreads();
            if (cur == NO_TILE) break;
            const uint32_t own = lane < QF_WORKERS ? s.warp_total[buf][lane] : 0u;
            uint32_t inc = own;
#pragma unroll
            for (int o = 1; o < QF_WORKERS; o <<= 1) {
                const uint32_t n = __shfl_up_sync(ALL, inc, o);
                if (lane >= o) inc += n;
            }
            prev_total = __shfl_sync(ALL, inc, QF_WORKERS - 1);
            if (lane < QF_WORKERS) s.warp_base[buf][lane] = inc - own;
            if (lane == QF_WORKERS) s.warp_base[buf][lane] = (uint32_t)prev_total;
            if (lane == 0)
                st_relaxed_u64(p.status + cur, (cur == p.item[cur_item].first_tile ? ST_PREFIX : ST_AGG) | (unsigned long long)prev_total);
            prev = cur;
            prev_item = cur_item;
        }
        return;
    }

    // ---- workers -------------------------------------------------------------------------------------
    const int t = lane & 3, grp = lane >> 2;
    const int run0 = warp * 1024 + grp * (BS < 128 ? BS : 128) + t * 8;
    auto at = [&](int c) { return run0 + (c / CK) * 8 * BS + (c % CK) * 32; };   // first element of run c in the tile
    const uint16_t eps_h = f2h_bits(1e-6f);
    const float eps_f = h2f_bits(eps_h);
    const unsigned gmask = BS == 256 ? 0xffu << (lane & 24) : 0xfu << (lane & 28);   // the threads of a block
    float *fold = s.fold[warp];

    __syncthreads();
    uint4 x[4];
    unsigned int cur = s.tile[0], prev = NO_TILE;
    int cur_item = s.item[0], prev_item = 0;
    if (cur != NO_TILE) load_elements(p.item[cur_item], ((int64_t)cur - p.item[cur_item].first_tile) * QT_TILE, at, x);

    for (int i = 0, buf = 0, prev_buf = 0;; ++i, prev_buf = buf, buf = buf == QF_BUFS - 1 ? 0 : buf + 1) {
        // ---- statistics, codes and outlier mask of this thread's elements ---------------------------
        if (cur != NO_TILE) {
            const QuantItem &q = p.item[cur_item];
            const int64_t tile_base = ((int64_t)cur - q.first_tile) * QT_TILE;
            const int tile_elems = (int)min((int64_t)QT_TILE, q.padded - tile_base);
            uint16_t *scales = q.scales + tile_base / BS;
            uint32_t mask16[2] = {0u, 0u};   // outlier bits of runs 0, 1 and 2, 3
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                const uint32_t *xw = reinterpret_cast<const uint32_t *>(x) + b * CK * 4;
                // fp32 sum in ATen's order, and the sum of squares.  This thread holds accumulator t of all eight lanes.
                uint64_t a[4], sq2[2];
#pragma unroll
                for (int w = 0; w < CK * 4; ++w) {
                    const float2 f = h2f2(xw[w]);
                    const uint64_t f2 = pack2(f.x, f.y);
                    a[w & 3] = w < 4 ? f2 : add2(a[w & 3], f2);
                    sq2[w & 1] = w < 2 ? mul2(f2, f2) : fma2(f2, f2, sq2[w & 1]);
                }
                forget(x);
                float *slot = fold + grp * 32 + (t ^ (grp & 3)) * 8;   // permuted against bank conflicts
                auto store_fold = [&]() {
                    const float2 a0 = unpack2(a[0]), a1 = unpack2(a[1]), a2 = unpack2(a[2]), a3 = unpack2(a[3]);
                    *reinterpret_cast<float4 *>(slot + (grp & 1) * 4) = make_float4(a0.x, a0.y, a1.x, a1.y);
                    *reinterpret_cast<float4 *>(slot + (~grp & 1) * 4) = make_float4(a2.x, a2.y, a3.x, a3.y);
                };
                __syncwarp();
                store_fold();
                __syncwarp();
                if (BS == 256) {
                    // the block's second half goes on from the first half's accumulators
                    const int pg = grp & 6;
                    const float *ps = fold + pg * 32 + (t ^ (pg & 3)) * 8;
                    const float4 p0 = *reinterpret_cast<const float4 *>(ps), p1 = *reinterpret_cast<const float4 *>(ps + 4);
                    a[0] = pack2(p0.x, p0.y); a[1] = pack2(p0.z, p0.w); a[2] = pack2(p1.x, p1.y); a[3] = pack2(p1.z, p1.w);
#pragma unroll
                    for (int w = 0; w < CK * 4; ++w) {
                        const float2 f = h2f2(xw[w]);
                        a[w & 3] = add2(a[w & 3], pack2(f.x, f.y));
                    }
                    __syncwarp();
                    if (grp & 1) store_fold();
                    __syncwarp();
                }
                float fin;
                {
                    // this thread adds lanes 2t and 2t + 1: accumulators in order, then the lanes in order
                    const int g = BS == 256 ? grp | 1 : grp;
                    const float *src = fold + g * 32 + ((t >> 1) ^ (g & 1)) * 4 + (t & 1) * 2;
                    uint64_t l = *reinterpret_cast<const uint64_t *>(src + (0 ^ (g & 3)) * 8);
#pragma unroll
                    for (int j = 1; j < 4; ++j) l = add2(l, *reinterpret_cast<const uint64_t *>(src + (j ^ (g & 3)) * 8));
                    const float2 lv = unpack2(l);
                    fin = __fadd_rn(__fadd_rn(0.f, lv.x), lv.y);
#pragma unroll
                    for (int j = 1; j < 4; ++j) fin = __fadd_rn(__fadd_rn(__shfl_sync(ALL, fin, j - 1, 4), lv.x), lv.y);
                    fin = __shfl_sync(ALL, fin, 3, 4);
                }
                const float mean32 = fin * (1.f / (float)BS);   // a power of two: exact
                const uint16_t mean_h = f2h_bits(mean32);
                constexpr int GROUP = BS == 256 ? 8 : 4;
                const float2 sv = unpack2(add2(sq2[0], sq2[1]));
                float sq = sv.x + sv.y;
#pragma unroll
                for (int o = 1; o < GROUP; o <<= 1) sq += __shfl_xor_sync(ALL, sq, o);
                float m2f = fmaf(-fin, mean32, sq);
                forget(x);
                const bool about_mean = !(sq <= 1.25f * m2f);   // (the same decision in all threads of a block)
                if (__any_sync(ALL, about_mean)) {
                    const float m2 = moment_about<BS>(x[b * CK], x[b * CK + (CK > 1)], x[b * CK + (CK > 2) * 2], x[b * CK + (CK > 2) * 3], mean32);
                    if (about_mean) m2f = m2;
                }
                forget(x);
                float std32;
                asm("sqrt.approx.f32 %0, %1;" : "=f"(std32) : "f"(m2f * (1.f / (float)(BS - 1))));
                uint16_t std_h = f2h_bits(std32 * (1.f - 4e-6f));
                const bool unsure = std_h != f2h_bits(std32 * (1.f + 4e-6f));   // the fp16 rounding is within reach of the fp32 error
                if (__any_sync(ALL, unsure)) {
                    const uint16_t exact = std_in_fp64<BS>(x[b * CK], x[b * CK + (CK > 1)], x[b * CK + (CK > 2) * 2], x[b * CK + (CK > 2) * 3]);
                    if (unsure) std_h = exact;
                }
                forget(x);
                const float den_f = h2f_bits(f2h_bits(__fadd_rn(h2f_bits(std_h), eps_f)));
                // the largest |d| that is not an outlier
                const float bound = fc.T * den_f;
                uint16_t cut = __half_as_ushort(__float2half_rd(bound));
                if (fc.tie_out && h2f_bits(cut) == bound) --cut;
                const __half2 cut2 = __half2half2(__ushort_as_half(cut)), mean2 = __half2half2(__ushort_as_half(mean_h));
                // z test, outlier bits (low half: even elements, high half: odd ones), absmax of the rest
                uint32_t bits2[2] = {0u, 0u}, maxabs = 0u;
#pragma unroll
                for (int w = 0; w < CK * 4; ++w) {
                    const int c = b * CK + (w >> 2);   // run
                    const __half2 d = __hsub2(*reinterpret_cast<const __half2 *>(&xw[w]), mean2);
                    const uint32_t out = __hgt2_mask(__habs2(d), cut2);
                    bits2[c >> 1] |= out & (0x00020001u << ((c & 1) * 8 + (w & 3) * 2));
                    maxabs = __vmaxu2(maxabs, xw[w] & 0x7fff7fffu & ~out);   // fp16 magnitude bits order like the values
                }
                bool kept;
                if (CK == 4) {
                    const uint32_t m0 = (bits2[0] | bits2[0] >> 16) & 0xffffu, m1 = (bits2[1] | bits2[1] >> 16) & 0xffffu;
                    kept = (m0 & m1) != 0xffffu;
                    mask16[0] = m0;
                    mask16[1] = m1;
                } else {
                    const int h = (b * CK) >> 1, sh = ((b * CK) & 1) * 8;
                    constexpr uint32_t full = CK == 2 ? 0xffffu : 0xffu;
                    const uint32_t m = (bits2[h] | bits2[h] >> 16) & (full << sh);
                    kept = m != full << sh;
                    mask16[h] |= m;
                }
                const bool any_kept = (__ballot_sync(ALL, kept) & gmask) != 0u;
#pragma unroll
                for (int o = 1; o < GROUP; o <<= 1) maxabs = __vmaxu2(maxabs, __shfl_xor_sync(ALL, maxabs, o));
                maxabs = max(maxabs & 0xffffu, maxabs >> 16);
                uint16_t sc = 0x3c00u;  // 1.0 when the block has no non-outliers
                if (any_kept) sc = max(f2h_bits(h2f_bits((uint16_t)maxabs) * (1.0f / 127.0f)), eps_h);
                if (t == 0 && (BS < 256 || !(grp & 1)) && at(b * CK) < tile_elems) scales[at(b * CK) / BS] = sc;
                const float rsc = __frcp_rn(h2f_bits(sc));
                const uint64_t rsc2 = pack2(rsc, rsc);
                const __half2 magic = __float2half2_rn(1536.f);
                uint8_t *db = s.dense[buf];
                // A kept value is at most 127 (1 + 2^-11) scales, 127.06, which the sum rounds to 127, unless the scale
                // is subnormal (its rounding is coarser) or not finite: such blocks take the second form.
                if (!__any_sync(ALL, (uint16_t)(sc - 0x400u) >= 0x7800u)) {
#pragma unroll
                    for (int k = 0; k < CK; ++k) {
                        uint32_t h[4];
#pragma unroll
                        for (int w = 0; w < 4; ++w) {
                            const float2 f = h2f2(xw[k * 4 + w]);
                            const float2 qf = unpack2(mul2(pack2(f.x, f.y), rsc2));
                            const __half2 v = __hadd2(__floats2half2_rn(qf.x, qf.y), magic);
                            h[w] = *reinterpret_cast<const uint32_t *>(&v);
                        }
                        *reinterpret_cast<uint2 *>(db + dense_byte(at(b * CK + k))) =
                            make_uint2(__byte_perm(h[0], h[1], 0x6420), __byte_perm(h[2], h[3], 0x6420));
                    }
                } else {
                    // A NaN quotient is code 0.  It takes an infinity or a NaN among the values kept, which makes the scale
                    // infinite or NaN and every other quotient of the block 0 or NaN: such a block gets zero bytes.
                    const uint32_t finite = sc < 0x7c00u ? 0xffffffffu : 0u;
                    const __half2 lim = __float2half2_rn(127.f), nlim = __float2half2_rn(-127.f);
#pragma unroll
                    for (int k = 0; k < CK; ++k) {
                        uint32_t h[4];
#pragma unroll
                        for (int w = 0; w < 4; ++w) {
                            const float2 f = h2f2(xw[k * 4 + w]);
                            __half2 v = __floats2half2_rn(f.x * rsc, f.y * rsc);
                            v = __hadd2(__hmax2(__hmin2(v, lim), nlim), magic);
                            h[w] = *reinterpret_cast<const uint32_t *>(&v);
                        }
                        *reinterpret_cast<uint2 *>(db + dense_byte(at(b * CK + k))) =
                            make_uint2(__byte_perm(h[0], h[1], 0x6420) & finite, __byte_perm(h[2], h[3], 0x6420) & finite);
                    }
                }
            }
            uint8_t *mb = reinterpret_cast<uint8_t *>(s.mask[buf]);
#pragma unroll
            for (int c = 0; c < 4; ++c)   // (blocks beyond the end of the tensor have no outliers)
                mb[at(c) >> 3] = at(c) < tile_elems ? (uint8_t)(mask16[c >> 1] >> ((c & 1) * 8)) : (uint8_t)0;
            __syncwarp();
            const uint32_t own = __popc(s.mask[buf][tid]);
            uint32_t inc = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t n = __shfl_up_sync(ALL, inc, o);
                if (lane >= o) inc += n;
            }
            s.word_before[buf][tid] = inc - own;
            if (lane == 31) s.warp_total[buf][warp] = inc;
        }
        __syncthreads();
        const unsigned int next = cur != NO_TILE ? s.tile[(i + 1) & 3] : NO_TILE;
        const int next_item = next != NO_TILE ? s.item[(i + 1) & 3] : 0;
        // the next tile's elements travel while the previous one is written out
        if (next != NO_TILE) load_elements(p.item[next_item], ((int64_t)next - p.item[next_item].first_tile) * QT_TILE, at, x);

        // ---- the previous tile, whose place in the streams is known by now -------------------------------
        if (prev != NO_TILE) {
            const QuantItem &q = p.item[prev_item];
            const int64_t tile_base = ((int64_t)prev - q.first_tile) * QT_TILE;
            const int tile_elems = (int)min((int64_t)QT_TILE, q.padded - tile_base);
            const uint32_t *mask = s.mask[prev_buf], *base = s.warp_base[prev_buf], *word_before = s.word_before[prev_buf];
            const uint8_t *dense = s.dense[prev_buf];
            auto before = [&](int w) { return (int)(word_before[w] + base[w >> 5]); };
            const long long tile_prefix = s.prefix[(i - 1) & 1];
            const int64_t code_base = tile_base - tile_prefix;  // where this tile's codes start
            const int shift = q.out_aligned ? (int)(code_base & 15) : 0;
            // outliers, one mask word per thread; their values are read again
            {
                uint32_t word = mask[tid];
                long long pos = tile_prefix + before(tid);
                while (word) {
                    const int64_t e = tile_base + tid * 32 + __ffs(word) - 1;
                    word &= word - 1;
                    if (pos < q.ocap) {
                        q.ovals[pos] = e < q.numel ? __ldg(q.x + e) : (uint16_t)0;
                        q.oidx[pos] = e;
                    }
                    ++pos;
                }
            }
            // the compacted codes, 16 bytes to an aligned global address per thread and step
            const int total = tile_elems - (int)base[QF_WORKERS];  // code bytes of this tile
            const int end = shift + total;
            int8_t *gdst = q.codes + (code_base - shift);  // 16-byte aligned when out_aligned
            const int nchunks = (end + 15) >> 4;
            const uint32_t *s32 = reinterpret_cast<const uint32_t *>(dense);
            for (int c = tid; c < nchunks; c += QF_WORKERS * 32) {
                const int lo = c << 4, a = max(lo, shift), z = min(lo + 16, end);
                const int o0 = a - shift;                    // first code of the piece, counted in the tile
                int w = o0 >> 5;                             // the mask word it lies in
                while (w < QT_WORDS - 1 && (w + 1) * 32 - before(w + 1) <= o0) ++w;
                const int skip = o0 - (w * 32 - before(w));  // codes of that word in front of it
                const uint32_t word = mask[w];
                int in_word = skip;
                if (word) {                                  // position of code number `skip` among the word's codes
                    for (int k = 0; k < 32; ++k) {
                        const int next_at = skip + __popc(word & (0xffffffffu >> (31 - min(in_word, 31))));
                        if (next_at == in_word) break;
                        in_word = next_at;
                    }
                }
                const int pos = w * 32 + in_word;
                // 20 dense codes from there and their outlier bits
                uint32_t m = __funnelshift_r(mask[pos >> 5], mask[min((pos >> 5) + 1, QT_WORDS)], pos & 31) & 0xfffffu;
                uint32_t v[5];
                {
                    const int wi = pos >> 2, r = (pos & 3) * 8;
                    uint32_t raw[6];
#pragma unroll
                    for (int k = 0; k < 6; ++k) raw[k] = s32[(wi + k) ^ ((((wi + k) >> 5) & 3) << 3)];
#pragma unroll
                    for (int k = 0; k < 5; ++k) v[k] = __funnelshift_r(raw[k], raw[k + 1], r);
                }
                if (__popc(m) <= 4) {
                    while (m & 0xffffu) {                    // squeeze out the first outlier's place
                        const int j = __ffs(m) - 1, jw = j >> 2;
                        const uint32_t low = (1u << (8 * (j & 3))) - 1u;
#pragma unroll
                        for (int k = 0; k < 5; ++k) {
                            const uint32_t down = __funnelshift_r(v[k], k < 4 ? v[k < 4 ? k + 1 : 4] : 0u, 8);
                            v[k] = k < jw ? v[k] : (k == jw ? ((v[k] & low) | (down & ~low)) : down);
                        }
                        m = (m >> 1) & ~((1u << j) - 1u);
                    }
                } else {                                     // dense outliers: code by code
#pragma unroll
                    for (int k = 0; k < 4; ++k) v[k] = 0u;
                    int at_e = pos;
#pragma unroll
                    for (int k = 0; k < 16; ++k) {
                        if (a + k < z) {
                            while ((mask[at_e >> 5] >> (at_e & 31)) & 1u) ++at_e;
                            v[k >> 2] |= (uint32_t)dense[dense_byte(at_e)] << (8 * (k & 3));
                            ++at_e;
                        }
                    }
                }
                if (q.out_aligned && z - a == 16) {
                    *reinterpret_cast<uint4 *>(gdst + lo) = make_uint4(v[0], v[1], v[2], v[3]);
                } else {
#pragma unroll
                    for (int k = 0; k < 16; ++k)
                        if (a + k < z) gdst[a + k] = (int8_t)(v[k >> 2] >> (8 * (k & 3)));
                }
            }
        }
        if (cur == NO_TILE) break;
        prev = cur;
        prev_item = cur_item;
        cur = next;
        cur_item = next_item;
    }
}

// |fp16(q)| > thr_h  <=>  |q| beyond T, the midpoint between thr_h and the next fp16 number above it
// (a tie goes to the even neighbour).
FastConsts make_fast_consts(uint16_t thr_h) {
    FastConsts fc;
    const float thr = __half2float(__ushort_as_half(thr_h));
    fc.tie_out = 0;
    if ((thr_h & 0x7fffu) > 0x7c00u) fc.T = INFINITY;          // NaN threshold: nothing compares greater
    else if (thr_h == 0x7c00u) fc.T = INFINITY;                 // +inf
    else if (thr_h > 0x8000u) fc.T = -1.f;                      // negative: every |z| is greater
    else if (thr_h == 0x8000u) fc.T = 0x1p-25f;                 // as +0
    else if (thr_h == 0x7bffu) fc.T = 65520.f;                  // next above the largest finite is inf
    else fc.T = 0.5f * (thr + __half2float(__ushort_as_half((uint16_t)(thr_h + 1))));
    if (!(thr_h & 0x8000u) && fc.T != INFINITY) fc.tie_out = thr_h & 1;
    return fc;
}

// ---- several copies in one launch ------------------------------------------------------------
// A layer's fourteen outlier streams are 20 KB to 1 MB each: a copy's launch (4 us of host time) costs more than the copy.
constexpr int CP_THREADS = 256;
constexpr int CP_MAX_ITEMS = 32;
struct CopyBatch {
    AtlasCopyItem item[CP_MAX_ITEMS];
    int n;
};
__global__ void __launch_bounds__(CP_THREADS) copy_many_kernel(const __grid_constant__ CopyBatch p) {
    const AtlasCopyItem it = p.item[blockIdx.y];
    const int64_t first = (int64_t)blockIdx.x * CP_THREADS + threadIdx.x, step = (int64_t)gridDim.x * CP_THREADS;
    const bool vec = ((((uintptr_t)it.dst) | ((uintptr_t)it.src)) & 15) == 0;
    const int64_t pieces = vec ? it.bytes >> 4 : 0;
    for (int64_t i = first; i < pieces; i += step) reinterpret_cast<uint4 *>(it.dst)[i] = __ldg(reinterpret_cast<const uint4 *>(it.src) + i);
    for (int64_t i = pieces * 16 + first; i < it.bytes; i += step)
        reinterpret_cast<uint8_t *>(it.dst)[i] = __ldg(reinterpret_cast<const uint8_t *>(it.src) + i);
}

struct DeviceInfo {
    int dev = -1;
    int sms = 0;
    int quant_ctas_per_sm = 0;
};

int device_info(DeviceInfo &out) {
    static thread_local DeviceInfo cache;
    int dev = 0;
    int rc = check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
    if (rc) return rc;
    if (cache.dev != dev) {
        DeviceInfo d;
        d.dev = dev;
        rc = check_cuda(cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev), "sm count");
        if (rc) return rc;
        rc = check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&d.quant_ctas_per_sm, quantize_kernel,
                                                                      QT_THREADS, 0),
                        "occupancy(quantize_kernel)");
        if (rc) return rc;
        if (d.quant_ctas_per_sm < 1) d.quant_ctas_per_sm = 1;
        cache = d;
    }
    out = cache;
    return ATLAS_OK;
}

}  // namespace
}  // namespace atlas

extern "C" {

size_t atlas_quantize_workspace_bytes(int64_t numel, int block_size) {
    if (numel <= 0 || block_size <= 0 || block_size > atlas::QT_TILE) return 16;
    const int64_t padded = atlas::ceil_div_i64(numel, block_size) * block_size;
    const int64_t tile = (atlas::QT_TILE / block_size) * block_size;   // a tile holds whole blocks
    const int64_t tiles = atlas::ceil_div_i64(padded, tile);
    return (size_t)(16 + 8 * tiles);
}

size_t atlas_quantize_many_workspace_bytes(int count, const AtlasQuantizeItem *items, int block_size) {
    size_t bytes = 0;
    for (int i = 0; items && i < count; ++i) bytes += atlas_quantize_workspace_bytes(items[i].numel, block_size);
    return bytes;
}

int atlas_quantize_many(int count, const AtlasQuantizeItem *items, int block_size, double z_threshold,
                        void *workspace, size_t workspace_bytes, void *stream) {
    using namespace atlas;
    clear_error();
    ATLAS_RETURN_IF(count < 1 || !items, ATLAS_ERR_BAD_ARGUMENT, "atlas_quantize: no tensors");
    for (int i = 0; i < count; ++i)
        ATLAS_RETURN_IF(items[i].numel < 0 || items[i].counts == nullptr || items[i].outlier_capacity < 0, ATLAS_ERR_BAD_ARGUMENT,
                        "atlas_quantize: negative size or null counts");
    ATLAS_RETURN_IF(block_size < 32 || block_size > 512 || block_size % 32 != 0, ATLAS_ERR_UNSUPPORTED,
                    "atlas_quantize: block_size %d is not a multiple of 32 in [32, 512]", block_size);
    int rc = check_device();
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    size_t need = 0;   // (an empty tensor has no tiles)
    bool counts_in_a_row = true;
    for (int i = 0; i < count; ++i) {
        const AtlasQuantizeItem &a = items[i];
        if (i > 0) counts_in_a_row = counts_in_a_row && a.counts == items[i - 1].counts + 4;
        if (a.numel == 0) continue;
        ATLAS_RETURN_IF(!a.w || !a.codes || !a.scales || !workspace || (a.outlier_capacity > 0 && (!a.outlier_vals || !a.outlier_idx)),
                        ATLAS_ERR_BAD_ARGUMENT, "atlas_quantize: null buffer");
        need += atlas_quantize_workspace_bytes(a.numel, block_size);
        ATLAS_RETURN_IF(workspace_bytes < need, ATLAS_ERR_CAPACITY,
                        "atlas_quantize: workspace holds %zu bytes, %zu needed", workspace_bytes, need);
        ATLAS_RETURN_IF(((uintptr_t)workspace & 15) != 0 || ((uintptr_t)a.w & 1) != 0 ||
                            ((uintptr_t)a.outlier_idx & 7) != 0 || ((uintptr_t)a.counts & 7) != 0,
                        ATLAS_ERR_BAD_ARGUMENT, "atlas_quantize: misaligned buffer");
    }
    const size_t counts_bytes = 4 * sizeof(int64_t);
    if (counts_in_a_row && need && (char *)items[0].counts + count * counts_bytes == (char *)workspace) {
        rc = check_cuda(cudaMemsetAsync(items[0].counts, 0, count * counts_bytes + need, st), "memset(counts, workspace)");
        if (rc) return rc;
    } else {
        if (counts_in_a_row) {
            rc = check_cuda(cudaMemsetAsync(items[0].counts, 0, count * counts_bytes, st), "memset(counts)");
        } else {
            for (int i = 0; i < count && !rc; ++i) rc = check_cuda(cudaMemsetAsync(items[i].counts, 0, counts_bytes, st), "memset(counts)");
        }
        if (rc) return rc;
        if (need) rc = check_cuda(cudaMemsetAsync(workspace, 0, need, st), "memset(workspace)");
        if (rc) return rc;
    }
    if (!need) return ATLAS_OK;
    DeviceInfo di;
    rc = device_info(di);
    if (rc) return rc;
    const uint16_t thr_h = __half_as_ushort(__float2half_rn((float)z_threshold));
    const bool fast = block_size == 32 || block_size == 64 || block_size == 128 || block_size == 256;
    const int64_t tile = (QT_TILE / block_size) * block_size;
    char *ws = (char *)workspace;
    if (!fast) {
        for (int i = 0; i < count; ++i) {
            const AtlasQuantizeItem &a = items[i];
            if (a.numel == 0) continue;
            QuantParams p;
            p.x = (const uint16_t *)a.w;
            p.numel = a.numel;
            p.n_blocks = ceil_div_i64(a.numel, block_size);
            p.padded = p.n_blocks * block_size;
            p.tile = (int)tile;
            p.num_tiles = ceil_div_i64(p.padded, tile);
            p.bs = block_size;
            p.thr_h = thr_h;
            p.codes = a.codes;
            p.ovals = (uint16_t *)a.outlier_vals;
            p.oidx = a.outlier_idx;
            p.ocap = a.outlier_capacity;
            p.scales = (uint16_t *)a.scales;
            p.counts = a.counts;
            p.tile_counter = (unsigned int *)ws;
            p.status = (unsigned long long *)(ws + 16);
            p.in_aligned = ((uintptr_t)a.w & 15) == 0;
            p.out_aligned = ((uintptr_t)a.codes & 15) == 0;
            ws += atlas_quantize_workspace_bytes(a.numel, block_size);
            const int64_t max_ctas = (int64_t)di.sms * di.quant_ctas_per_sm;
            quantize_kernel<<<(int)(p.num_tiles < max_ctas ? p.num_tiles : max_ctas), QT_THREADS, 0, st>>>(p);
            rc = check_cuda(cudaGetLastError(), "quantize_kernel launch");
            if (rc) return rc;
        }
        return ATLAS_OK;
    }
    const FastConsts fc = make_fast_consts(thr_h);
    for (int i = 0; i < count;) {
        QuantBatch b = {};
        int64_t tiles = 0;
        for (; i < count && b.n < QF_MAX_ITEMS; ++i) {
            const AtlasQuantizeItem &a = items[i];
            if (a.numel == 0) continue;
            const int64_t padded = ceil_div_i64(a.numel, block_size) * block_size, own = ceil_div_i64(padded, tile);
            if (b.n && tiles + own > 0x7fffffff) break;
            b.item[b.n++] = {(const uint16_t *)a.w, a.codes, (uint16_t *)a.outlier_vals, a.outlier_idx, (uint16_t *)a.scales,
                             a.counts, a.numel, padded, a.outlier_capacity, tiles, ((uintptr_t)a.w & 15) == 0, ((uintptr_t)a.codes & 15) == 0};
            tiles += own;
        }
        if (b.n == 0) break;
        ATLAS_RETURN_IF(tiles > 0x7fffffff, ATLAS_ERR_UNSUPPORTED, "atlas_quantize: tensor too large");
        b.num_tiles = (unsigned int)tiles;
        b.tile_counter = (unsigned int *)ws;
        b.status = (unsigned long long *)(ws + 16);
        ws += 16 + 8 * tiles;
        const int64_t max_ctas = (int64_t)di.sms * QF_CTAS;
        const int grid = (int)(tiles < max_ctas ? tiles : max_ctas);
        switch (block_size) {
            case 32: quantize_fast_kernel<32><<<grid, QF_THREADS, 0, st>>>(b, fc); break;
            case 64: quantize_fast_kernel<64><<<grid, QF_THREADS, 0, st>>>(b, fc); break;
            case 128: quantize_fast_kernel<128><<<grid, QF_THREADS, 0, st>>>(b, fc); break;
            default: quantize_fast_kernel<256><<<grid, QF_THREADS, 0, st>>>(b, fc); break;
        }
        rc = check_cuda(cudaGetLastError(), "quantize_fast_kernel launch");
        if (rc) return rc;
    }
    return ATLAS_OK;
}

int atlas_quantize(const void *w, int64_t numel, int block_size, double z_threshold, int8_t *codes,
                   void *outlier_vals, int64_t *outlier_idx, int64_t outlier_capacity, void *scales,
                   int64_t *counts, void *workspace, size_t workspace_bytes, void *stream) {
    const AtlasQuantizeItem item = {w, numel, codes, outlier_vals, outlier_idx, outlier_capacity, scales, counts};
    return atlas_quantize_many(1, &item, block_size, z_threshold, workspace, workspace_bytes, stream);
}

int atlas_copy_many(int count, const AtlasCopyItem *items, void *stream) {
    using namespace atlas;
    clear_error();
    ATLAS_RETURN_IF(count < 0 || (count && !items), ATLAS_ERR_BAD_ARGUMENT, "atlas_copy_many: bad count");
    for (int i = 0; i < count; ++i)
        ATLAS_RETURN_IF(items[i].bytes < 0 || (items[i].bytes && (!items[i].dst || !items[i].src)), ATLAS_ERR_BAD_ARGUMENT,
                        "atlas_copy_many: null buffer or negative length");
    int rc = check_device();
    if (rc) return rc;
    for (int i = 0; i < count;) {
        CopyBatch b = {};
        int64_t longest = 0;
        for (; i < count && b.n < CP_MAX_ITEMS; ++i) {
            if (!items[i].bytes) continue;
            b.item[b.n++] = items[i];
            if (items[i].bytes > longest) longest = items[i].bytes;
        }
        if (b.n == 0) break;
        const int64_t want = ceil_div_i64(longest, CP_THREADS * 16);
        copy_many_kernel<<<dim3((unsigned)(want < 64 ? want : 64), (unsigned)b.n), CP_THREADS, 0, (cudaStream_t)stream>>>(b);
        rc = check_cuda(cudaGetLastError(), "copy_many_kernel launch");
        if (rc) return rc;
    }
    return ATLAS_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------
// Quantize without any allocation by anyone: scratch in a file-scope device array.
//
// The look-back needs a tile counter and one status word per tile.  atlas_quantize takes them
// from a caller-provided workspace; callers that are not allowed to allocate device memory at
// the point of the call (a pre-allocated arena they may not grow, a fixed-memory serving loop
// where every cudaMalloc is a synchronisation and a fragmentation risk, a plug-in host that
// owns the allocator) cannot provide one.  For them the same kernel runs against the static
// array below, sized for ATLAS_QUANTIZE_NOALLOC_MAX_ELEMENTS padded elements (64 Mi: 8192 tiles,
// 64 KB + 16 B).  The array lives in every context that loads this library until it exits.
constexpr int64_t NOALLOC_MAX_TILES = ATLAS_QUANTIZE_NOALLOC_MAX_ELEMENTS / atlas::QT_TILE;
static __device__ __align__(256) unsigned char g_quantize_scratch[16 + 8 * NOALLOC_MAX_TILES];

namespace {
// In host code `g_quantize_scratch` is only a handle for the symbol, not a device address: the
// address is looked up once per device, with that device current, and cached.
int noalloc_scratch_ptr(void **out) {
    constexpr int kMaxDevices = 64;
    static void *cache[kMaxDevices] = {nullptr};
    static std::mutex mu;
    int dev = -1;
    int rc = atlas::check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
    if (rc) return rc;
    if (dev < 0 || dev >= kMaxDevices) {
        atlas::set_error("atlas_quantize_noalloc: device ordinal %d outside [0, %d)", dev, kMaxDevices);
        return ATLAS_ERR_UNSUPPORTED;
    }
    std::lock_guard<std::mutex> lock(mu);
    if (cache[dev] == nullptr) {
        void *ptr = nullptr;
        rc = atlas::check_cuda(cudaGetSymbolAddress(&ptr, g_quantize_scratch),
                               "cudaGetSymbolAddress(g_quantize_scratch)");
        if (rc) return rc;
        cache[dev] = ptr;
    }
    *out = cache[dev];
    return ATLAS_OK;
}
}  // namespace

extern "C" int atlas_quantize_noalloc(const void *w, int64_t numel, int block_size, double z_threshold,
                                      int8_t *codes, void *outlier_vals, int64_t *outlier_idx,
                                      int64_t outlier_capacity, void *scales, int64_t *counts, void *stream) {
    using namespace atlas;
    clear_error();
    ATLAS_RETURN_IF(numel < 0 || block_size <= 0, ATLAS_ERR_BAD_ARGUMENT,
                    "atlas_quantize_noalloc: negative size or block size");
    const int64_t padded = ceil_div_i64(numel, block_size) * block_size;
    ATLAS_RETURN_IF(padded > ATLAS_QUANTIZE_NOALLOC_MAX_ELEMENTS, ATLAS_ERR_CAPACITY,
                    "atlas_quantize_noalloc: %lld padded elements exceed the static scratch limit of %lld; "
                    "use atlas_quantize with a caller-provided workspace",
                    (long long)padded, (long long)ATLAS_QUANTIZE_NOALLOC_MAX_ELEMENTS);
    // block sizes that do not divide the 8192-element tile use slightly smaller tiles, hence more status words
    ATLAS_RETURN_IF(block_size <= QT_TILE && atlas_quantize_workspace_bytes(numel, block_size) > sizeof(g_quantize_scratch),
                    ATLAS_ERR_CAPACITY,
                    "atlas_quantize_noalloc: %lld elements in blocks of %d exceed the static scratch limit; "
                    "use atlas_quantize with a caller-provided workspace", (long long)numel, block_size);
    void *scratch = nullptr;
    int rc = check_device();
    if (rc) return rc;
    rc = noalloc_scratch_ptr(&scratch);
    if (rc) return rc;
    // atlas_quantize zeroes the scratch it is given on the stream before the kernel runs
    return atlas_quantize(w, numel, block_size, z_threshold, codes, outlier_vals, outlier_idx, outlier_capacity,
                          scales, counts, scratch, sizeof(g_quantize_scratch), stream);
}
