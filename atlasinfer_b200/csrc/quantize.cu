// Adaptive hybrid quantizer for sm_100a: one pass over the fp16 weights.
//
// Replaces quantize_tensor (atlasinfer_core/quant/adaptive_quantizer.py:51-148).
// The reference walks the blocks in a Python loop and concatenates four
// streams; here a persistent grid takes tiles of 8192 elements in order
// (dynamic tile ids), evaluates every block of a tile in shared memory, and
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
// Fast variant for block sizes 32 / 64 / 128 / 256.  Same results as quantize_kernel above, bit for bit, at a quarter of
// its instructions: 121 us for 11008 x 4096 in blocks of 128 back to back, 128 with L2 flushed before (165 back to back with
// guard bands around the roundings and byte-wise compaction), 46 % of the issue slots used, the rest mostly the barriers around the look-back.
//
// Four threads work on a block; thread t plays ATen's SIMD lanes 2t and 2t + 1, whose elements are neighbours, so the
// values stay packed two to a register and most steps cost one instruction per pair.  What replaces the IEEE divisions
// and the fp64 moment, and why the results are the same:
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
//     of 256, the longest sums: Q carries 31 additions of a thread and 3 across threads, 34 u Q.  F carries 7 + 3 in a lane
//     and 7 over the lanes, 17 u sum|x| <= 17 u sqrt(n Q), and |F| <= sqrt(0.2 n Q) here, so F^2 / n is off by
//     2 * 0.45 * 17 u Q = 15 u Q.  With Q <= 1.25 M that is 62 u of M, 31 u of its root, and 4 u for the product, the root
//     and the rounding of M: 35 u = 2.1e-6.  The second pass adds 64 times (66 u with the shuffles, 2 u for the squared
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

// Outliers of all tiles before `tile` (whole warp).  All resident CTAs finish a tile at about the same time and find only
// counts, no prefixes, among each other's, so the walk back covers 256 tiles per round trip.  A status word holds all
// that is passed on, so relaxed accesses do.
__device__ __forceinline__ long long look_back(const unsigned long long *status, int64_t tile, int lane, int64_t *counts) {
    long long prefix = 0;
    int64_t look = tile - 1;
    for (int spins = 0; spins <= QT_SPIN_LIMIT; ++spins) {
        unsigned long long v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int64_t idx = look - k * 32 - lane;
            v[k] = idx >= 0 ? ld_relaxed_u64(status + idx) : ST_PREFIX;   // tiles before the first count as prefix 0
        }
        int taken = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (taken != k) continue;
            const unsigned pm = __ballot_sync(0xffffffffu, (v[k] >> 62) == 2), none = __ballot_sync(0xffffffffu, (v[k] >> 62) == 0);
            const int first = pm ? __ffs(pm) - 1 : 31;
            if (none & (0xffffffffu >> (31 - first))) continue;          // not there yet
            unsigned int contrib = lane < first || (!pm && lane == first) ? (unsigned int)(v[k] & ST_VALUE) : 0u;   // a tile's own count
            prefix += (long long)__reduce_add_sync(0xffffffffu, contrib);
            if (pm) return prefix + (long long)(__shfl_sync(0xffffffffu, v[k], first) & ST_VALUE);
            ++taken;
        }
        look -= taken * 32;
        if (taken == 0) __nanosleep(32);
    }
    if (lane == 0) atomicExch((unsigned long long *)&counts[2], 1ull);   // record and leave; the host reports ATLAS_ERR_TIMEOUT
    return prefix;
}

// Byte offset of element e's code in the dense tile: 16-byte pieces permuted so that the eight blocks a warp works on
// fall on different banks.
__device__ __forceinline__ int dense_byte(int e) { return e ^ (((e >> 7) & 7) << 4); }

template <int BS>
__global__ void __launch_bounds__(QT_THREADS, 5) quantize_fast_kernel(QuantParams p, FastConsts fc) {
    constexpr int NP = BS / 8;                // pairs per thread
    constexpr int TILE_BLOCKS = QT_TILE / BS;
    // blocks are padded by 16 bytes so that the eight blocks a warp works on at a time fall on different banks
    constexpr int XSTRIDE = BS * 2 + 16;      // bytes
    __shared__ __align__(16) uint8_t s_xb[TILE_BLOCKS * XSTRIDE];
    __shared__ __align__(16) uint8_t s_dense[QT_TILE + 128];
    auto xref = [&](int e) -> uint16_t & {
        return *reinterpret_cast<uint16_t *>(s_xb + (e / BS) * XSTRIDE + (e % BS) * 2);
    };
    __shared__ uint32_t s_mask[QT_WORDS + 1];
    __shared__ uint32_t s_wordpre[QT_WORDS];
    __shared__ uint16_t s_scale[TILE_BLOCKS];
    __shared__ uint32_t s_warp_tot[QT_THREADS / 32];
    __shared__ long long s_tile_prefix;
    __shared__ int s_tile_total;
    __shared__ unsigned int s_tile;

    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const uint16_t eps_h = f2h_bits(1e-6f);
    const float eps_f = h2f_bits(eps_h);
    if (tid == 0) s_mask[QT_WORDS] = 0u;

    for (;;) {
        __syncthreads();  // previous tile's shared state is no longer read
        if (tid == 0) s_tile = atomicAdd(p.tile_counter, 1u);
        __syncthreads();
        const int64_t tile = s_tile;
        if (tile >= p.num_tiles) break;
        const int64_t tile_base = tile * QT_TILE;
        const int tile_elems = (int)min((int64_t)QT_TILE, p.padded - tile_base);
        const int tile_real = (int)max((int64_t)0, min((int64_t)tile_elems, p.numel - tile_base));
        const int tile_blocks = tile_elems / BS;

        // ---- stage the tile (zero padding included) -------------------------------
        if (p.in_aligned) {
            const uint4 *src = reinterpret_cast<const uint4 *>(p.x + tile_base);
#pragma unroll
            for (int i = 0; i < QT_TILE / 8 / QT_THREADS; ++i) {
                const int v = tid + i * QT_THREADS, e0 = v * 8;
                if (e0 + 8 <= tile_real) {
                    *reinterpret_cast<uint4 *>(s_xb + (e0 / BS) * XSTRIDE + (e0 % BS) * 2) = __ldg(src + v);
                } else if (e0 < tile_elems) {
                    for (int e = e0; e < e0 + 8; ++e) xref(e) = (e < tile_real) ? p.x[tile_base + e] : (uint16_t)0;
                }
            }
        } else {
            for (int e = tid; e < tile_elems; e += QT_THREADS)
                xref(e) = (e < tile_real) ? p.x[tile_base + e] : (uint16_t)0;
        }
        s_mask[tid] = 0u;   // QT_WORDS == QT_THREADS
        __syncthreads();

        // ---- statistics and codes of whole blocks, 4 threads per block ----------
        {
            const int t = tid & 3;
            const unsigned gmask = 0xfu << (lane & 28);
            for (int b = tid >> 2; b < tile_blocks; b += QT_THREADS / 4) {
                const uint32_t *xb = reinterpret_cast<const uint32_t *>(s_xb + b * XSTRIDE) + t;
                // (read from shared memory again in every pass: keeping 32 floats costs the fifth CTA of an SM)
                auto pair = [&](int j) { return __half22float2(*reinterpret_cast<const __half2 *>(xb + j * 4)); };
                // fp32 sum in ATen's order, and the sum of squares
                float lo4[4] = {0.f, 0.f, 0.f, 0.f}, hi4[4] = {0.f, 0.f, 0.f, 0.f}, sq = 0.f, sq_hi = 0.f;
#pragma unroll
                for (int j = 0; j < NP; ++j) {
                    const float2 f = pair(j);
                    lo4[j & 3] = __fadd_rn(lo4[j & 3], f.x);
                    hi4[j & 3] = __fadd_rn(hi4[j & 3], f.y);
                    sq = fmaf(f.x, f.x, sq);
                    sq_hi = fmaf(f.y, f.y, sq_hi);
                }
                asm volatile("" ::: "memory");
                const float lo_sum = __fadd_rn(__fadd_rn(__fadd_rn(lo4[0], lo4[1]), lo4[2]), lo4[3]);
                const float hi_sum = __fadd_rn(__fadd_rn(__fadd_rn(hi4[0], hi4[1]), hi4[2]), hi4[3]);
                float fin = 0.f;
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    fin = __fadd_rn(fin, __shfl_sync(gmask, lo_sum, s, 4));
                    fin = __fadd_rn(fin, __shfl_sync(gmask, hi_sum, s, 4));
                }
                const float mean32 = fin * (1.f / (float)BS);   // a power of two: exact
                const uint16_t mean_h = f2h_bits(mean32);
                sq += sq_hi;
                sq += __shfl_xor_sync(gmask, sq, 1, 4);
                sq += __shfl_xor_sync(gmask, sq, 2, 4);
                float m2f = fmaf(-fin, mean32, sq);
                if (!(sq <= 1.25f * m2f)) {   // (the same decision in all four threads)
                    // about mean32, with the first moment about it taken out again, so that the rounding of mean32
                    // itself only enters to second order
                    float r1 = 0.f;
                    m2f = 0.f;
#pragma unroll 1
                    for (int j = 0; j < NP; ++j) {
                        const float2 f = pair(j);
                        const float d0 = f.x - mean32, d1 = f.y - mean32;
                        r1 += d0 + d1;
                        m2f = fmaf(d0, d0, fmaf(d1, d1, m2f));
                    }
#pragma unroll
                    for (int o = 1; o < 4; o <<= 1) {
                        m2f += __shfl_xor_sync(gmask, m2f, o, 4);
                        r1 += __shfl_xor_sync(gmask, r1, o, 4);
                    }
                    m2f = fmaxf(fmaf(-r1, r1 * (1.f / (float)BS), m2f), 0.f);
                }
                float std32;
                asm("sqrt.approx.f32 %0, %1;" : "=f"(std32) : "f"(m2f * (1.f / (float)(BS - 1))));
                uint16_t std_h = f2h_bits(std32 * (1.f - 4e-6f));
                if (std_h != f2h_bits(std32 * (1.f + 4e-6f))) {
                    // the fp16 rounding is within reach of the fp32 error: redo it in fp64
                    double dsum = 0.0;
#pragma unroll 1
                    for (int j = 0; j < NP; ++j) { const float2 f = pair(j); dsum += (double)f.x + (double)f.y; }
#pragma unroll
                    for (int o = 1; o < 4; o <<= 1) dsum += __shfl_xor_sync(gmask, dsum, o, 4);
                    const double mean_d = dsum / (double)BS;
                    double m2 = 0.0;
#pragma unroll 1
                    for (int j = 0; j < NP; ++j) {
                        const float2 f = pair(j);
                        const double d0 = (double)f.x - mean_d, d1 = (double)f.y - mean_d;
                        m2 = fma(d0, d0, fma(d1, d1, m2));
                    }
#pragma unroll
                    for (int o = 1; o < 4; o <<= 1) m2 += __shfl_xor_sync(gmask, m2, o, 4);
                    std_h = f2h_bits(__double2float_rn(sqrt(m2 / (double)(BS - 1))));
                }
                const float den_f = h2f_bits(f2h_bits(__fadd_rn(h2f_bits(std_h), eps_f)));
                // the largest |d| that is not an outlier
                const float bound = fc.T * den_f;
                uint16_t cut = __half_as_ushort(__float2half_rd(bound));
                if (fc.tie_out && h2f_bits(cut) == bound) --cut;
                const __half2 cut2 = __half2half2(__ushort_as_half(cut)), mean2 = __half2half2(__ushort_as_half(mean_h));
                // z test, outlier mask (low half: even elements, high half: odd ones), absmax of the rest
                constexpr int NM = (NP + 15) / 16;
                uint32_t omask[NM], maxabs = 0u;
#pragma unroll
                for (int i = 0; i < NM; ++i) omask[i] = 0u;
#pragma unroll
                for (int j = 0; j < NP; ++j) {
                    const uint32_t x2 = xb[j * 4];
                    const __half2 d = __hsub2(*reinterpret_cast<const __half2 *>(&x2), mean2);
                    const uint32_t out = __hgt2_mask(__habs2(d), cut2);
                    omask[j >> 4] |= out & (0x00010001u << (j & 15));
                    maxabs = __vmaxu2(maxabs, x2 & 0x7fff7fffu & ~out);   // fp16 magnitude bits order like the values
                }
                asm volatile("" ::: "memory");
                int cnt = 0;
#pragma unroll
                for (int i = 0; i < NM; ++i) cnt += __popc(omask[i]);
                const bool any_out = cnt != 0;
#pragma unroll
                for (int o = 1; o < 4; o <<= 1) {
                    cnt += __shfl_xor_sync(gmask, cnt, o, 4);
                    maxabs = __vmaxu2(maxabs, __shfl_xor_sync(gmask, maxabs, o, 4));
                }
                maxabs = max(maxabs & 0xffffu, maxabs >> 16);
                uint16_t sc = 0x3c00u;  // 1.0 when the block has no non-outliers
                if (cnt < BS) sc = max(f2h_bits(h2f_bits((uint16_t)maxabs) * (1.0f / 127.0f)), eps_h);
                if (t == 0) s_scale[b] = sc;
                const float rsc = __frcp_rn(h2f_bits(sc));
                // A NaN quotient is code 0.  It takes an infinity or a NaN among the values kept, which makes the scale
                // infinite or NaN and every other quotient of the block 0 or NaN: such a block selects zero bytes
                // instead of the low bytes of its (min/max-cleaned) sums, which costs the others nothing.
                const uint32_t low_bytes = sc < 0x7c00u ? 0x4420u : 0x4444u;
                uint8_t *db = s_dense;
                const int e0 = b * BS + 2 * t;
                const __half2 lim = __float2half2_rn(127.f), nlim = __float2half2_rn(-127.f), magic = __float2half2_rn(1536.f);
#pragma unroll
                for (int j = 0; j < NP; ++j) {
                    const float2 f = pair(j);
                    __half2 q = __floats2half2_rn(f.x * rsc, f.y * rsc);
                    q = __hmax2(__hmin2(q, lim), nlim);
                    q = __hadd2(q, magic);
                    const uint32_t bits = *reinterpret_cast<uint32_t *>(&q);
                    *reinterpret_cast<uint16_t *>(db + dense_byte(e0 + j * 8)) = (uint16_t)__byte_perm(bits, 0u, low_bytes);
                }
                if (any_out) {
#pragma unroll
                    for (int i = 0; i < NM; ++i)
                        for (uint32_t m = omask[i]; m; m &= m - 1) {
                            const int bit = __ffs(m) - 1;
                            const int pos = e0 + ((bit & 15) + i * 16) * 8 + (bit >> 4);
                            atomicOr(&s_mask[pos >> 5], 1u << (pos & 31));
                        }
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
                if (lane == 0) st_relaxed_u64(p.status, ST_PREFIX | agg);
            } else {
                if (lane == 0) st_relaxed_u64(p.status + tile, ST_AGG | agg);
                prefix = look_back(p.status, tile, lane, p.counts);
                if (lane == 0) st_relaxed_u64(p.status + tile, ST_PREFIX | (unsigned long long)(prefix + (long long)agg));
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

        // ---- with the prefix: outliers straight out, one mask word per thread ------------------------
        const long long tile_prefix = s_tile_prefix;
        const int64_t code_base = tile_base - tile_prefix;  // where this tile's codes start
        const int shift = p.out_aligned ? (int)(code_base & 15) : 0;
        {
            uint32_t word = s_mask[tid];   // QT_WORDS == QT_THREADS
            long long pos = tile_prefix + s_wordpre[tid];
            while (word) {
                const int e = tid * 32 + __ffs(word) - 1;
                word &= word - 1;
                if (pos < p.ocap) {
                    p.ovals[pos] = xref(e);
                    p.oidx[pos] = tile_base + e;
                }
                ++pos;
            }
        }

        // ---- the compacted codes, 16 bytes to an aligned global address per thread and step ------------------------
        {
            const int total = tile_elems - s_tile_total;  // code bytes of this tile
            const int end = shift + total;
            int8_t *gdst = p.codes + (code_base - shift);  // 16-byte aligned when out_aligned
            const int nchunks = (end + 15) >> 4;
            const uint32_t *s32 = reinterpret_cast<const uint32_t *>(s_dense);
            for (int c = tid; c < nchunks; c += QT_THREADS) {
                const int lo = c << 4, a = max(lo, shift), z = min(lo + 16, end);
                const int o0 = a - shift;                    // first code of the piece, counted in the tile
                int w = o0 >> 5;                             // the mask word it lies in
                while (w < QT_WORDS - 1 && (w + 1) * 32 - (int)s_wordpre[w + 1] <= o0) ++w;
                const int skip = o0 - (w * 32 - (int)s_wordpre[w]);   // codes of that word in front of it
                const uint32_t word = s_mask[w];
                int in_word = skip;
                if (word) {                                  // position of code number `skip` among the word's codes
                    for (int i = 0; i < 32; ++i) {
                        const int next = skip + __popc(word & (0xffffffffu >> (31 - min(in_word, 31))));
                        if (next == in_word) break;
                        in_word = next;
                    }
                }
                const int pos = w * 32 + in_word;
                // 20 dense codes from there and their outlier bits
                uint32_t m = __funnelshift_r(s_mask[pos >> 5], s_mask[min((pos >> 5) + 1, QT_WORDS)], pos & 31) & 0xfffffu;
                uint32_t v[5];
                {
                    const int wi = pos >> 2, r = (pos & 3) * 8;
                    uint32_t raw[6];
#pragma unroll
                    for (int i = 0; i < 6; ++i) raw[i] = s32[(wi + i) ^ ((((wi + i) >> 5) & 7) << 2)];
#pragma unroll
                    for (int i = 0; i < 5; ++i) v[i] = __funnelshift_r(raw[i], raw[i + 1], r);
                }
                if (__popc(m) <= 4) {
                    while (m & 0xffffu) {                    // squeeze out the first outlier's place
                        const int j = __ffs(m) - 1, jw = j >> 2;
                        const uint32_t low = (1u << (8 * (j & 3))) - 1u;
#pragma unroll
                        for (int i = 0; i < 5; ++i) {
                            const uint32_t down = __funnelshift_r(v[i], i < 4 ? v[i < 4 ? i + 1 : 4] : 0u, 8);
                            v[i] = i < jw ? v[i] : (i == jw ? ((v[i] & low) | (down & ~low)) : down);
                        }
                        m = (m >> 1) & ~((1u << j) - 1u);
                    }
                } else {                                     // dense outliers: code by code
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[i] = 0u;
                    int q = pos;
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        if (a + i < z) {
                            while ((s_mask[q >> 5] >> (q & 31)) & 1u) ++q;
                            v[i >> 2] |= (uint32_t)s_dense[dense_byte(q)] << (8 * (i & 3));
                            ++q;
                        }
                    }
                }
                if (p.out_aligned && z - a == 16) {
                    *reinterpret_cast<uint4 *>(gdst + lo) = make_uint4(v[0], v[1], v[2], v[3]);
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        if (a + i < z) gdst[a + i] = (int8_t)(v[i >> 2] >> (8 * (i & 3)));
                }
            }
            const int64_t block0 = tile_base / BS;
            for (int b = tid; b < tile_blocks; b += QT_THREADS) p.scales[block0 + b] = s_scale[b];
        }
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

int atlas_quantize(const void *w, int64_t numel, int block_size, double z_threshold, int8_t *codes,
                   void *outlier_vals, int64_t *outlier_idx, int64_t outlier_capacity, void *scales,
                   int64_t *counts, void *workspace, size_t workspace_bytes, void *stream) {
    using namespace atlas;
    clear_error();
    ATLAS_RETURN_IF(numel < 0 || counts == nullptr || outlier_capacity < 0, ATLAS_ERR_BAD_ARGUMENT,
                    "atlas_quantize: negative size or null counts");
    ATLAS_RETURN_IF(block_size < 32 || block_size > 512 || block_size % 32 != 0, ATLAS_ERR_UNSUPPORTED,
                    "atlas_quantize: block_size %d is not a multiple of 32 in [32, 512]", block_size);
    int rc = check_device();
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    rc = check_cuda(cudaMemsetAsync(counts, 0, 4 * sizeof(int64_t), st), "memset(counts)");
    if (rc) return rc;
    if (numel == 0) return ATLAS_OK;
    ATLAS_RETURN_IF(!w || !codes || !scales || !workspace ||
                        (outlier_capacity > 0 && (!outlier_vals || !outlier_idx)),
                    ATLAS_ERR_BAD_ARGUMENT, "atlas_quantize: null buffer");
    const size_t need = atlas_quantize_workspace_bytes(numel, block_size);
    ATLAS_RETURN_IF(workspace_bytes < need, ATLAS_ERR_CAPACITY,
                    "atlas_quantize: workspace holds %zu bytes, %zu needed", workspace_bytes, need);
    ATLAS_RETURN_IF(((uintptr_t)workspace & 15) != 0 || ((uintptr_t)w & 1) != 0 ||
                        ((uintptr_t)outlier_idx & 7) != 0 || ((uintptr_t)counts & 7) != 0,
                    ATLAS_ERR_BAD_ARGUMENT, "atlas_quantize: misaligned buffer");

    QuantParams p;
    p.x = (const uint16_t *)w;
    p.numel = numel;
    p.n_blocks = ceil_div_i64(numel, block_size);
    p.padded = p.n_blocks * block_size;
    p.tile = (QT_TILE / block_size) * block_size;
    p.num_tiles = ceil_div_i64(p.padded, p.tile);
    p.bs = block_size;
    p.thr_h = __half_as_ushort(__float2half_rn((float)z_threshold));
    p.codes = codes;
    p.ovals = (uint16_t *)outlier_vals;
    p.oidx = outlier_idx;
    p.ocap = outlier_capacity;
    p.scales = (uint16_t *)scales;
    p.counts = counts;
    p.tile_counter = (unsigned int *)workspace;
    p.status = (unsigned long long *)((char *)workspace + 16);
    p.in_aligned = ((uintptr_t)w & 15) == 0;
    p.out_aligned = ((uintptr_t)codes & 15) == 0;

    rc = check_cuda(cudaMemsetAsync(workspace, 0, need, st), "memset(workspace)");
    if (rc) return rc;
    DeviceInfo di;
    rc = device_info(di);
    if (rc) return rc;
    const bool fast = block_size == 32 || block_size == 64 || block_size == 128 || block_size == 256;
    const int per_sm = fast ? 5 : di.quant_ctas_per_sm;   // resident CTAs of the fast kernels
    const int64_t max_ctas = (int64_t)di.sms * per_sm;
    const int grid = (int)(p.num_tiles < max_ctas ? p.num_tiles : max_ctas);
    if (fast) {
        const FastConsts fc = make_fast_consts(p.thr_h);
        switch (block_size) {
            case 32: quantize_fast_kernel<32><<<grid, QT_THREADS, 0, st>>>(p, fc); break;
            case 64: quantize_fast_kernel<64><<<grid, QT_THREADS, 0, st>>>(p, fc); break;
            case 128: quantize_fast_kernel<128><<<grid, QT_THREADS, 0, st>>>(p, fc); break;
            default: quantize_fast_kernel<256><<<grid, QT_THREADS, 0, st>>>(p, fc); break;
        }
        return check_cuda(cudaGetLastError(), "quantize_fast_kernel launch");
    }
    quantize_kernel<<<grid, QT_THREADS, 0, st>>>(p);
    return check_cuda(cudaGetLastError(), "quantize_kernel launch");
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
