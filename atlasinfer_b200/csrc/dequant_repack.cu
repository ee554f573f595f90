// Inverse of the quantizer, and expansion of the compacted code stream into
// the tile-major kernel layout.
//
// Replaces dequantize_tensor (atlasinfer_core/quant/adaptive_quantizer.py:156-251).
// The reference keeps a running offset into the code stream and, per block,
// masks the whole outlier index list (:194-196, O(blocks x outliers)).  Here the
// sorted outlier index list is searched once per span of 16384 elements: the
// number of outliers before the span both locates the span's outliers and
// gives the span's offset into the compacted code stream (position minus
// outliers before it), so every span is independent.
//
// Both directions only move bytes: HBM is the bound (1.04 bytes read per element, 2 or 1 written).  A span's outlier
// positions become a bit mask with a prefix count per word, its codes are staged with 16-byte loads, and a thread
// builds 16 bytes of output at a time: one unaligned read of the staged codes, a zero byte slipped in per set bit
// (an outlier sits in every 20th such unit), one 16-byte store.
#include "common.cuh"

namespace atlas {
namespace {

constexpr int DQ_THREADS = 256;
constexpr int DQ_SPAN = 16384;                // padded elements per CTA
constexpr int DQ_WORDS = DQ_SPAN / 32;        // outlier-mask words: two per thread
static_assert(DQ_WORDS == 2 * DQ_THREADS, "two mask words per thread");
constexpr int DQ_MAX_REPACK = 8;              // tensors one repack launch takes
constexpr int RP_STRIP_CAP = 2560;            // outliers of a strip kept in shared memory (16 x 4096 weights: 200 at 0.3 %)
constexpr int RP_SCALE_KB = 16;               // scale blocks per CTA of the scale transposition (one 32-byte sector a row)

// First i in [0, n) with idx[i] >= key, found by a whole warp: 32 probes a step, so 135 k outliers take four
// dependent loads instead of eighteen.
__device__ __forceinline__ int64_t warp_lower_bound(const int64_t *idx, int64_t n, int64_t key, int lane) {
    int64_t lo = 0, hi = n;
    while (hi - lo > 32) {
        const int64_t step = (hi - lo + 32) / 33;
        const int64_t pos = lo + step * (lane + 1) - 1;
        const int c = __popc(__ballot_sync(0xffffffffu, pos < hi && __ldg(idx + pos) < key));
        if (c < 32) hi = min(hi, lo + step * (c + 1) - 1);
        lo = lo + step * c;
    }
    return lo + __popc(__ballot_sync(0xffffffffu, lo + lane < hi && __ldg(idx + lo + lane) < key));
}

struct Span {
    __align__(16) uint32_t mask[DQ_WORDS];                  // bit p: position p of the span is an outlier
    __align__(16) uint32_t before[DQ_WORDS];                // outliers of the span before the word
    uint32_t warp_total[DQ_THREADS / 32];
    int64_t lo, hi;                           // the span's outliers in the outlier streams
    __align__(16) uint8_t codes[DQ_SPAN + 48];
    int shift;                                // where the span's first code sits in `codes` (the misalignment of its address)
};

// Stages the span [span0, span1): mask, prefix counts and codes.  Nothing outside codes[0, n_codes) and oidx[0, n_out)
// is read, whatever oidx holds; if it is not ascending (a damaged file) the values are arbitrary, but hi >= lo keeps the
// staged length within the span and, as every bit of the mask stands for an index in [lo, hi), the outliers read within
// [lo, hi) too.
__device__ __forceinline__ void stage_span(Span &s, const int8_t *codes, int64_t n_codes, const int64_t *oidx,
                                           int64_t n_out, int64_t span0, int64_t span1) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    *reinterpret_cast<uint2 *>(s.mask + 2 * tid) = make_uint2(0u, 0u);
    if (warp < 2) {
        const int64_t r = warp_lower_bound(oidx, n_out, warp == 0 ? span0 : span1, lane);
        if (lane == 0) (warp == 0 ? s.lo : s.hi) = r;
    }
    __syncthreads();
    const int64_t lo = s.lo, hi = max(lo, s.hi);
    for (int64_t i = lo + tid; i < hi; i += DQ_THREADS) {
        const int64_t p = __ldg(oidx + i) - span0;
        if (p >= 0 && p < DQ_SPAN) atomicOr(&s.mask[p >> 5], 1u << (p & 31));
    }
    const int64_t c0 = span0 - lo;            // the span's first code
    const int len = (int)max((int64_t)0, span1 - span0 - (hi - lo));
    const int shift = (int)((uintptr_t)(codes + c0) & 15);
    if (tid == 0) s.shift = shift;
    for (int c = tid; c * 16 < shift + len; c += DQ_THREADS) {
        const int64_t g = c0 - shift + c * 16;
        uint4 v;
        if (g >= 0 && g + 16 <= n_codes) {
            v = __ldg(reinterpret_cast<const uint4 *>(codes + g));
        } else {
            uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int e = 0; e < 16; ++e)
                if (g + e >= 0 && g + e < n_codes) w[e >> 2] |= (uint32_t)(uint8_t)codes[g + e] << (8 * (e & 3));
            v = make_uint4(w[0], w[1], w[2], w[3]);
        }
        *reinterpret_cast<uint4 *>(s.codes + c * 16) = v;
    }
    __syncthreads();
    const uint2 words = *reinterpret_cast<const uint2 *>(s.mask + 2 * tid);
    const uint32_t own = __popc(words.x) + __popc(words.y);
    uint32_t inc = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t n = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += n;
    }
    if (lane == 31) s.warp_total[warp] = inc;
    __syncthreads();
    uint32_t base = 0;
    for (int w = 0; w < warp; ++w) base += s.warp_total[w];
    *reinterpret_cast<uint2 *>(s.before + 2 * tid) = make_uint2(base + inc - own, base + inc - __popc(words.y));
    __syncthreads();
}

// The 4 * W codes of the unit that starts at position p of the span (p a multiple of 4 * W, W = 2 or 4), biased by 128;
// an outlier's place holds code 0.  `bits` are its outliers, `before` the span's outliers in front of it.
template <int W>
__device__ __forceinline__ void span_unit(const Span &s, int p, uint32_t (&w)[W], uint32_t &bits, int &before) {
    const uint32_t word = s.mask[p >> 5];
    bits = (word >> (p & 31)) & ((1u << (4 * W)) - 1u);
    before = (int)s.before[p >> 5] + __popc(word & ((1u << (p & 31)) - 1u));
    const int o = s.shift + p - before, r = (o & 3) * 8;
    const uint32_t *src = reinterpret_cast<const uint32_t *>(s.codes) + (o >> 2);
    uint32_t raw[W + 1];
#pragma unroll
    for (int i = 0; i <= W; ++i) raw[i] = src[i];
#pragma unroll
    for (int i = 0; i < W; ++i) w[i] = __funnelshift_r(raw[i], raw[i + 1], r);
    for (uint32_t m = bits; m; m &= m - 1) {   // a zero byte in the outlier's place, the later codes move up by one
        const int j = __ffs(m) - 1, jw = j >> 2;
        const uint32_t low = (1u << (8 * (j & 3))) - 1u;
#pragma unroll
        for (int i = W - 1; i >= 0; --i) {
            const uint32_t up = i > 0 ? __funnelshift_l(w[i > 0 ? i - 1 : 0], w[i], 8) : w[i] << 8;
            const uint32_t here = (w[i] & low) | ((w[i] & ~low) << 8);
            w[i] = i > jw ? up : (i == jw ? here : w[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < W; ++i) w[i] ^= 0x80808080u;
}

// Two biased codes of a word (bytes 0, 1 or 2, 3) as fp16(code), exact.
template <uint32_t SEL>
__device__ __forceinline__ __half2 code_pair(uint32_t w) {
    const uint32_t h = __byte_perm(w, 0x64646464u, SEL);   // halves 1024 + u
    const __half2 bias = __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480));  // 1152
    return __hsub2(*reinterpret_cast<const __half2 *>(&h), bias);
}

// 8 elements (16 bytes of output) per thread and step.  The product of the code and the scale is rounded to fp16 once
// (adaptive_quantizer.py:216).  11008 x 4096 in blocks of 128:
// 50 us (2.7 TB/s).  With one binary search per element and 2-byte stores the seven weights of a 7B-shaped layer took
// 1316 us through the API, now 275.
__global__ void __launch_bounds__(DQ_THREADS)
dequantize_kernel(const int8_t *codes, int64_t n_codes, const uint16_t *ovals, const int64_t *oidx,
                  int64_t n_out, const uint16_t *scales, int64_t numel, int64_t padded, int bs, int bs_shift,
                  int w_aligned, uint16_t *w) {
    __shared__ Span s;
    const int64_t span0 = (int64_t)blockIdx.x * DQ_SPAN;
    const int64_t span1 = min(span0 + DQ_SPAN, padded);
    stage_span(s, codes, n_codes, oidx, n_out, span0, span1);
    const int64_t out_lo = s.lo;
#pragma unroll 1
    for (int p = threadIdx.x * 8; p < DQ_SPAN; p += DQ_THREADS * 8) {
        const int64_t gp = span0 + p;
        if (gp >= numel) break;
        uint32_t c[2], bits;
        int before;
        span_unit<2>(s, p, c, bits, before);
        __half2 h[4] = {code_pair<0x5140>(c[0]), code_pair<0x5342>(c[0]), code_pair<0x5140>(c[1]), code_pair<0x5342>(c[1])};
        if ((bs & 7) == 0) {                   // the unit lies in one block
            const int64_t b = bs_shift >= 0 ? gp >> bs_shift : gp / bs;
            const __half2 sc = __half2half2(__ushort_as_half(__ldg(scales + b)));
#pragma unroll
            for (int i = 0; i < 4; ++i) h[i] = __hmul2(h[i], sc);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int64_t b0 = min((gp + 2 * i) / bs, (padded - 1) / bs), b1 = min((gp + 2 * i + 1) / bs, (padded - 1) / bs);
                h[i] = __hmul2(h[i], __halves2half2(__ushort_as_half(__ldg(scales + b0)), __ushort_as_half(__ldg(scales + b1))));
            }
        }
        uint32_t o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) o[i] = *reinterpret_cast<uint32_t *>(&h[i]);
        int64_t k = out_lo + before;
        for (uint32_t m = bits; m; m &= m - 1, ++k) {
            const int j = __ffs(m) - 1;
            const uint32_t v = __ldg(ovals + k);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i == j >> 1) o[i] = (j & 1) ? __byte_perm(o[i], v, 0x5410) : __byte_perm(o[i], v, 0x3254);
        }
        if (w_aligned && gp + 8 <= numel) {
            *reinterpret_cast<uint4 *>(w + gp) = make_uint4(o[0], o[1], o[2], o[3]);
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (gp + e < numel) w[gp + e] = (uint16_t)(o[e >> 1] >> (16 * (e & 1)));
        }
    }
}

// Byte offset of weight (row, col) inside the tile-major layout.
__device__ __forceinline__ int64_t tile_offset(int64_t row, int64_t col, int64_t k_tiles) {
    const int64_t rt = row >> 7, kt = col >> 6;
    const int strip = (int)(row & 127) >> 4, h = (int)(row & 15) >> 3, g = (int)(row & 7);
    const int tig = (int)(col & 63) >> 4, byte = (int)(col & 15);
    return ((((rt * k_tiles + kt) * 8 + strip) * 2 + h) * 32 + (g * 4 + tig)) * 16 + byte;
}

struct RepackTensor {
    const int8_t *codes;
    const int64_t *oidx;
    const uint16_t *ovals;
    const uint16_t *scales;
    int64_t n_codes, n_out, n_rows, n_cols, rows_padded;
    uint8_t *tiles;
    uint16_t *scales_t;
    int32_t *row_ptr;          // null: not wanted
    int32_t *chunk_ptr;
    uint32_t *entries;         // this tensor's part of the entry list, which starts entry_base entries into the whole
    uint16_t *vals_sorted;
    int32_t entry_base;
    int32_t blocks_per_row;
    uint32_t strip_end, scale_end, block_end;   // this tensor's CTAs: strips, then scales, then codes; ends in the grid
};
struct RepackParams {
    RepackTensor t[DQ_MAX_REPACK];
    int n;
};

struct StripScratch {
    int64_t row_at[17];                       // first outlier of the strip's rows in the streams
    uint32_t col[RP_STRIP_CAP];
};
union RepackShared {
    Span span;
    StripScratch strip;
    uint16_t scale[RP_SCALE_KB][128 + 2];
};

// entries of [lo, hi) (offsets into the strip's list, one row, ascending columns) with column < key
template <class ColAt>
__device__ __forceinline__ int count_below(const ColAt &col_at, int lo, int hi, uint32_t key) {
    const int base = lo;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (col_at(mid) < key) lo = mid + 1; else hi = mid;
    }
    return lo - base;
}

// The outlier lists of one 16-row strip: row_ptr, chunk_ptr[c] = first entry with column >= 64 * c, and the entries
// (row%16 << 24 | column) sorted by column, rows in order within a column.  The position of an entry is found by
// counting, over the 16 row lists (each sorted by column already), the entries that precede it: deterministic, no atomics.
template <class ColAt>
__device__ __forceinline__ void write_strip(const RepackTensor &t, int64_t strip, const StripScratch &s, const ColAt &col_at) {
    const int total = (int)(s.row_at[16] - s.row_at[0]);
    const int64_t first = s.row_at[0];
    const int n_chunks = (int)(t.n_cols >> 6);
    for (int i = threadIdx.x; i < total; i += DQ_THREADS) {
        int row = 0;
#pragma unroll
        for (int r = 1; r < 16; ++r) row += s.row_at[r] - first <= i;
        const uint32_t col = col_at(i);
        int rank = 0;
        for (int r = 0; r < 16; ++r)   // rows above: columns up to and with this one; this row and below: columns before it
            rank += count_below(col_at, (int)(s.row_at[r] - first), (int)(s.row_at[r + 1] - first), col + (r < row ? 1u : 0u));
        t.entries[first + rank] = (uint32_t)row << 24 | col;
        t.vals_sorted[first + rank] = __ldg(t.ovals + first + i);
    }
    for (int c = threadIdx.x; c <= n_chunks; c += DQ_THREADS) {
        int count = 0;
        for (int r = 0; r < 16; ++r)
            count += count_below(col_at, (int)(s.row_at[r] - first), (int)(s.row_at[r + 1] - first), (uint32_t)c * 64u);
        t.chunk_ptr[strip * (n_chunks + 1) + c] = (int32_t)(t.entry_base + first + count);
    }
}

// One launch expands up to DQ_MAX_REPACK tensors; a CTA does one of three jobs: the outlier lists of a strip (first in
// the grid: the longest chain of dependent loads), a 128-row x 16-block piece of the scale transposition, or 16384
// positions of the code tiles, 16 codes (one unit of the layout; n_cols is a multiple of 64, so a unit never straddles
// rows) per thread and step.  Rows beyond n_rows in the last 128-row tile get code 0 and scale 0.
__global__ void __launch_bounds__(DQ_THREADS) repack_kernel(const __grid_constant__ RepackParams p) {
    __shared__ RepackShared sh;
    int ti = 0;
    while (ti + 1 < p.n && blockIdx.x >= p.t[ti].block_end) ++ti;
    const RepackTensor &t = p.t[ti];
    const uint32_t begin = ti ? p.t[ti - 1].block_end : 0u;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    if (blockIdx.x < t.strip_end) {
        const int64_t strip = blockIdx.x - begin;
        for (int r = warp; r < 17; r += DQ_THREADS / 32) {
            const int64_t row = min(strip * 16 + r, t.n_rows);
            const int64_t at = warp_lower_bound(t.oidx, t.n_out, row * t.n_cols, lane);
            if (lane == 0) sh.strip.row_at[r] = at;
        }
        __syncthreads();
        const int64_t first = sh.strip.row_at[0];
        const int total = (int)(sh.strip.row_at[16] - first);
        if (t.row_ptr && tid < 17 && strip * 16 + tid <= t.n_rows && (tid < 16 || strip * 16 + 16 == t.n_rows))
            t.row_ptr[strip * 16 + tid] = (int32_t)sh.strip.row_at[tid];
        // The ranks below are a permutation, and what the linear kernels index with the entries lies in the strip, only if
        // the strip's positions ascend and its rows begin where the searches say.  A strip of which that is not true (a
        // damaged file) gets an empty list.
        const int64_t strip0 = strip * 16 * t.n_cols, strip1 = min(strip * 16 + 16, t.n_rows) * t.n_cols;
        const uint32_t n_cols = (uint32_t)t.n_cols;   // (a strip has at most 2^28 positions)
        int bad = 0;
        if (tid < 17) {
            const int64_t at = sh.strip.row_at[tid], end = sh.strip.row_at[16], key = min(strip0 + tid * t.n_cols, strip1);
            bad = at < first || at > end || (tid < 16 && sh.strip.row_at[tid + 1] < at);
            if (!bad) bad = (at > first && __ldg(t.oidx + at - 1) >= key) || (at < end && __ldg(t.oidx + at) < key);
        }
        for (int i = tid; i < total; i += DQ_THREADS) {
            const int64_t *at = t.oidx + first + i;
            bad |= i > 0 && __ldg(at - 1) >= __ldg(at);
            if (i < RP_STRIP_CAP) sh.strip.col[i] = (uint32_t)(__ldg(at) - strip0) % n_cols;
        }
        if (__syncthreads_or(bad)) {
            const int n_chunks = (int)(n_cols >> 6);
            for (int c = tid; c <= n_chunks; c += DQ_THREADS) t.chunk_ptr[strip * (n_chunks + 1) + c] = (int32_t)(t.entry_base + first);
        } else if (total <= RP_STRIP_CAP) {
            write_strip(t, strip, sh.strip, [&](int i) { return sh.strip.col[i]; });
        } else {
            write_strip(t, strip, sh.strip, [&](int i) { return (uint32_t)(__ldg(t.oidx + first + i) - strip0) % n_cols; });
        }
        return;
    }
    if (blockIdx.x < t.scale_end) {
        const int bpr = t.blocks_per_row;
        const int pieces = (bpr + RP_SCALE_KB - 1) / RP_SCALE_KB;
        const int64_t piece = blockIdx.x - t.strip_end, rt = piece / pieces;
        const int kb0 = (int)(piece - rt * pieces) * RP_SCALE_KB, nkb = min(RP_SCALE_KB, bpr - kb0);
        for (int i = tid; i < 128 * RP_SCALE_KB; i += DQ_THREADS) {
            const int r = i / RP_SCALE_KB, kb = i % RP_SCALE_KB;
            const int64_t row = rt * 128 + r;
            if (kb < nkb) sh.scale[kb][r] = row < t.n_rows ? __ldg(t.scales + row * bpr + kb0 + kb) : (uint16_t)0;
        }
        __syncthreads();
        uint16_t *dst = t.scales_t + (rt * bpr + kb0) * 128;
        for (int i = tid; i < 128 * nkb; i += DQ_THREADS) dst[i] = sh.scale[i >> 7][i & 127];
        return;
    }
    const int64_t numel = t.n_rows * t.n_cols, padded = t.rows_padded * t.n_cols;
    const int64_t span0 = (int64_t)(blockIdx.x - t.scale_end) * DQ_SPAN;
    const int64_t span1 = min(span0 + DQ_SPAN, numel);
    const int64_t row0 = span0 / t.n_cols;
    const uint32_t col0 = (uint32_t)(span0 - row0 * t.n_cols), n_cols = (uint32_t)t.n_cols;
    if (span0 < numel) stage_span(sh.span, t.codes, t.n_codes, t.oidx, t.n_out, span0, span1);
#pragma unroll 1
    for (int q = tid * 16; q < DQ_SPAN; q += DQ_THREADS * 16) {
        if (span0 + q >= padded) break;
        uint32_t w[4] = {0x80808080u, 0x80808080u, 0x80808080u, 0x80808080u}, bits;
        int before;
        if (span0 + q < numel) span_unit<4>(sh.span, q, w, bits, before);
        const uint32_t c = col0 + (uint32_t)q, dr = c / n_cols;
        *reinterpret_cast<uint4 *>(t.tiles + tile_offset(row0 + dr, c - dr * n_cols, n_cols >> 6)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

}  // namespace
}  // namespace atlas

extern "C" {

int atlas_dequantize(const int8_t *codes, int64_t n_codes, const void *outlier_vals,
                     const int64_t *outlier_idx, int64_t n_outliers, const void *scales, int64_t numel,
                     int block_size, void *w_out, void *stream) {
    using namespace atlas;
    clear_error();
    ATLAS_RETURN_IF(numel < 0 || n_codes < 0 || n_outliers < 0 || block_size < 1, ATLAS_ERR_BAD_ARGUMENT,
                    "atlas_dequantize: negative size or block_size < 1");
    if (numel == 0) return ATLAS_OK;
    const int64_t padded = ceil_div_i64(numel, block_size) * block_size;
    ATLAS_RETURN_IF(n_codes + n_outliers != padded, ATLAS_ERR_BAD_ARGUMENT,
                    "atlas_dequantize: %lld codes + %lld outliers do not cover %lld padded elements",
                    (long long)n_codes, (long long)n_outliers, (long long)padded);
    ATLAS_RETURN_IF(!w_out || !scales || (n_codes && !codes) || (n_outliers && (!outlier_vals || !outlier_idx)),
                    ATLAS_ERR_BAD_ARGUMENT, "atlas_dequantize: null buffer");
    int rc = check_device();
    if (rc) return rc;
    const int64_t grid = ceil_div_i64(padded, DQ_SPAN);
    ATLAS_RETURN_IF(grid > 0x7fffffff, ATLAS_ERR_UNSUPPORTED, "atlas_dequantize: tensor too large");
    const int bs_shift = (block_size & (block_size - 1)) == 0 ? __builtin_ctz((unsigned)block_size) : -1;
    dequantize_kernel<<<(unsigned)grid, DQ_THREADS, 0, (cudaStream_t)stream>>>(
        codes, n_codes, (const uint16_t *)outlier_vals, outlier_idx, n_outliers, (const uint16_t *)scales,
        numel, padded, block_size, bs_shift, ((uintptr_t)w_out & 15) == 0, (uint16_t *)w_out);
    return check_cuda(cudaGetLastError(), "dequantize_kernel launch");
}

size_t atlas_tiles_bytes(int64_t n_rows, int64_t n_cols) {
    if (n_rows <= 0 || n_cols <= 0) return 0;
    return (size_t)(atlas::ceil_div_i64(n_rows, 128) * 128 * n_cols);
}

int atlas_repack_many(int count, const AtlasRepackItem *items, void *stream) {
    using namespace atlas;
    clear_error();
    ATLAS_RETURN_IF(count < 1 || !items, ATLAS_ERR_BAD_ARGUMENT, "atlas_repack: no tensors");
    for (int i = 0; i < count; ++i) {
        const AtlasRepackItem &a = items[i];
        ATLAS_RETURN_IF(a.n_rows <= 0 || a.n_cols <= 0 || a.n_codes < 0 || a.n_outliers < 0 || a.block_size < 1 || a.block_size > 0x7fffffff || a.entry_base < 0,
                        ATLAS_ERR_BAD_ARGUMENT, "atlas_repack: bad size");
        ATLAS_RETURN_IF(a.n_cols % 64 != 0 || a.block_size % 16 != 0 || a.n_cols % a.block_size != 0,
                        ATLAS_ERR_UNSUPPORTED,
                        "atlas_repack: needs n_cols %% 64 == 0, block_size %% 16 == 0 and n_cols %% block_size == 0 "
                        "(got n_cols=%lld block_size=%d)", (long long)a.n_cols, (int)a.block_size);
        ATLAS_RETURN_IF(a.n_cols >= (1 << 24) || a.n_outliers > 0x7fffffff || a.entry_base + a.n_outliers > 0x7fffffff,
                        ATLAS_ERR_UNSUPPORTED, "atlas_repack: n_cols >= 2^24 or more than 2^31 outliers");
        ATLAS_RETURN_IF(a.n_codes + a.n_outliers != a.n_rows * a.n_cols, ATLAS_ERR_BAD_ARGUMENT,
                        "atlas_repack: %lld codes + %lld outliers do not cover %lld x %lld",
                        (long long)a.n_codes, (long long)a.n_outliers, (long long)a.n_rows, (long long)a.n_cols);
        ATLAS_RETURN_IF(!a.tiles || !a.scales || !a.scales_tiled || !a.outlier_chunk_ptr || (a.n_codes && !a.codes) ||
                            (a.n_outliers && (!a.outlier_idx || !a.outlier_vals || !a.outlier_entries || !a.outlier_vals_sorted)),
                        ATLAS_ERR_BAD_ARGUMENT, "atlas_repack: null buffer");
        ATLAS_RETURN_IF(((uintptr_t)a.tiles & 15) != 0, ATLAS_ERR_BAD_ARGUMENT, "atlas_repack: tiles must be 16-byte aligned");
    }
    int rc = check_device();
    if (rc) return rc;
    for (int i0 = 0; i0 < count; i0 += DQ_MAX_REPACK) {
        RepackParams p;
        p.n = count - i0 < DQ_MAX_REPACK ? count - i0 : DQ_MAX_REPACK;
        int64_t end = 0;
        for (int i = 0; i < p.n; ++i) {
            const AtlasRepackItem &a = items[i0 + i];
            RepackTensor &t = p.t[i];
            t.codes = a.codes;
            t.oidx = a.outlier_idx;
            t.ovals = (const uint16_t *)a.outlier_vals;
            t.scales = (const uint16_t *)a.scales;
            t.n_codes = a.n_codes;
            t.n_out = a.n_outliers;
            t.n_rows = a.n_rows;
            t.n_cols = a.n_cols;
            t.rows_padded = ceil_div_i64(a.n_rows, 128) * 128;
            t.tiles = a.tiles;
            t.scales_t = (uint16_t *)a.scales_tiled;
            t.row_ptr = a.outlier_row_ptr;
            t.chunk_ptr = a.outlier_chunk_ptr;
            t.entries = a.outlier_entries;
            t.vals_sorted = (uint16_t *)a.outlier_vals_sorted;
            t.entry_base = (int32_t)a.entry_base;
            t.blocks_per_row = (int32_t)(a.n_cols / a.block_size);
            const int64_t strips = t.rows_padded / 16;
            const int64_t scale_ctas = t.rows_padded / 128 * ceil_div_i64(t.blocks_per_row, RP_SCALE_KB);
            const int64_t code_ctas = ceil_div_i64(t.rows_padded * t.n_cols, DQ_SPAN);
            ATLAS_RETURN_IF(end + strips + scale_ctas + code_ctas > 0x7fffffff, ATLAS_ERR_UNSUPPORTED, "atlas_repack: tensor too large");
            t.strip_end = (uint32_t)(end + strips);
            t.scale_end = (uint32_t)(end + strips + scale_ctas);
            end += strips + scale_ctas + code_ctas;
            t.block_end = (uint32_t)end;
        }
        repack_kernel<<<(unsigned)end, DQ_THREADS, 0, (cudaStream_t)stream>>>(p);
        rc = check_cuda(cudaGetLastError(), "repack_kernel launch");
        if (rc) return rc;
    }
    return ATLAS_OK;
}

int atlas_repack(const int8_t *codes, int64_t n_codes, const void *outlier_vals, const int64_t *outlier_idx,
                 int64_t n_outliers, const void *scales, int64_t n_rows, int64_t n_cols, int block_size,
                 uint8_t *tiles, void *scales_tiled, int32_t *outlier_row_ptr, int32_t *outlier_chunk_ptr,
                 uint32_t *outlier_entries, void *outlier_vals_sorted, void *stream) {
    using namespace atlas;
    AtlasRepackItem a = {};
    a.codes = codes;
    a.n_codes = n_codes;
    a.outlier_vals = outlier_vals;
    a.outlier_idx = outlier_idx;
    a.n_outliers = n_outliers;
    a.scales = scales;
    a.n_rows = n_rows;
    a.n_cols = n_cols;
    a.block_size = block_size;
    a.tiles = tiles;
    a.scales_tiled = scales_tiled;
    a.outlier_row_ptr = outlier_row_ptr;
    a.outlier_chunk_ptr = outlier_chunk_ptr;
    a.outlier_entries = outlier_entries;
    a.outlier_vals_sorted = outlier_vals_sorted;
    if (n_rows > 0 && n_cols > 0 && block_size > 0 && tiles && scales && scales_tiled)
        ATLAS_RETURN_IF(!outlier_row_ptr, ATLAS_ERR_BAD_ARGUMENT, "atlas_repack: null buffer");
    return atlas_repack_many(1, &a, stream);
}

}  // extern "C"
