// Inverse of the quantizer, and expansion of the compacted code stream into
// the tile-major kernel layout.
//
// Replaces dequantize_tensor (atlasinfer_core/quant/adaptive_quantizer.py:156-251).
// The reference keeps a running offset into the code stream and, per block,
// masks the whole outlier index list (:194-196, O(blocks x outliers)).  Here
// every span of 8192 elements finds where its outliers begin and end in the
// sorted index list, by a search or, dequantizing, from a first kernel's one pass
// over the list for all spans; the number of outliers before the span gives its
// offset into the compacted code stream (position minus outliers before it), so
// every span is independent.
//
// Both directions only move bytes: HBM is the bound in principle (1.04 bytes read per element, 2 or 1 written), memory latency
// and instructions in practice.  A span's outlier positions become a bit mask with a code offset per word, its codes are
// staged with 16-byte copies, and a thread builds 16 bytes of output at a time from one unaligned read of the staged codes;
// units that hold outliers (every 20th to 40th) are left out of that and built afterwards, one per thread.
// 11008 x 4096 in blocks of 128: dequantize 52.7 -> 34.9 us (3.9 TB/s; 4096 x 4096 27.2 -> 18.5, 512 x 512 9.3 -> 6.3) against a
// search of four dependent round trips per span of 16384 and zero bytes slipped in per outlier under divergence; in blocks of 96
// or 160 55 -> 35, of 100 101 -> 70, to an output on no 16-byte boundary 84 -> 72; repack
// 43.2 -> 39.9 (4096 x 4096 18.6 -> 18.6, 4096 x 11008 43.1 -> 40.4; with the spans marked beforehand 45.2, 20.6 and 44.2, and
// with ten times the outliers 4096 x 4096 343 instead of 234): its strips' lists take as long.  Spans of 4096 and CTAs of 128
// threads: 33.6 for the dequantizer, but 62 for the repack of 4096 x 11008, whose strips hold 530 outliers.
#include "common.cuh"

namespace atlas {
namespace {

constexpr int DQ_THREADS = 256;
constexpr int DQ_SPAN = 8192;                 // padded elements per CTA
constexpr int DQ_WORDS = DQ_SPAN / 32;        // outlier-mask words
static_assert(DQ_WORDS == DQ_THREADS, "a mask word per thread");
constexpr int64_t DQ_SEARCHED = 1024;         // up to as many outliers a CTA searches for its own: two round trips
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

// Where a span's outliers are in the outlier list is found beforehand, by one pass over the list in a kernel of its own:
// every thread compares two neighbours, which is one round trip to memory (2 to 3 us here) for all spans together, where a
// search is four for each.  Both ends go to the first 16 bytes of the span's own output, which the span's CTA reads and
// overwrites; no other memory is needed.
struct Ends {
    int64_t lo, hi;
};
// Thread i's part of it: the spans that begin after outlier i - 1 and not after outlier i.  `put(span)` is where a span's
// ends go.  A whole warp calls it: long runs of spans without outliers are shared out.
template <class Put>
__device__ __forceinline__ void mark_spans(const int64_t *oidx, int64_t n_out, int64_t spans, int64_t i, int lane, const Put &put) {
    int64_t first = 1, last = 0;
    if (i <= n_out) {
        first = i > 0 ? max((int64_t)0, __ldg(oidx + i - 1) / DQ_SPAN + 1) : 0;
        last = i < n_out ? min(__ldg(oidx + i) / DQ_SPAN, spans) : spans;
    }
    auto mark = [&](int64_t s, int64_t at) {
        if (s < spans) put(s)->lo = at;
        if (s > 0) put(s - 1)->hi = at;
    };
    const bool many = last - first >= 8;
    if (!many)
        for (int64_t s = first; s <= last; ++s) mark(s, i);
    for (unsigned m = __ballot_sync(0xffffffffu, many); m; m &= m - 1) {
        const int from = __ffs(m) - 1;
        const int64_t f = __shfl_sync(0xffffffffu, first, from), l = __shfl_sync(0xffffffffu, last, from), at = __shfl_sync(0xffffffffu, i, from);
        for (int64_t s = f + lane; s <= l; s += 32) mark(s, at);
    }
}

struct Span {
    uint32_t mask[DQ_WORDS];                  // bit p: position p of the span is an outlier
    uint32_t start[DQ_WORDS];                 // where the word's first code lies in `codes`
    uint32_t warp_total[DQ_THREADS / 32];
    int64_t lo, hi;                           // the span's outliers in the outlier streams
    __align__(16) uint8_t codes[DQ_SPAN + 48];
};

// The ends of the span [span0, span1) in the outlier list, searched for by two warps of the CTA.
__device__ __forceinline__ Ends search_span(Span &s, const int64_t *oidx, int64_t n_out, int64_t span0, int64_t span1) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < 2) {
        const int64_t r = warp_lower_bound(oidx, n_out, warp == 0 ? span0 : span1, lane);
        if (lane == 0) (warp == 0 ? s.lo : s.hi) = r;
    }
    __syncthreads();
    const Ends ends = {s.lo, s.hi};
    __syncthreads();
    return ends;
}

// Stages the span [span0, span1), whose outliers are [lo, hi): mask, code offsets and codes.  Nothing outside
// codes[0, n_codes) and oidx[0, n_out) is read, whatever oidx and the ends hold; if oidx is not ascending (a damaged file) the
// values are arbitrary and need not repeat (a marked span may have no ends of its own, nor all of its codes be staged), but
// hi >= lo keeps the staged length within the span and, as every bit of the mask stands for an index in [lo, hi), the
// outliers read within [lo, hi) too.
__device__ __forceinline__ void stage_span(Span &s, const int8_t *codes, int64_t n_codes, const int64_t *oidx, int64_t n_out, Ends ends,
                                           int64_t span0, int64_t span1) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t lo = max((int64_t)0, min(ends.lo, n_out)), hi = max(lo, min(ends.hi, n_out));
    const int64_t first = lo + tid < hi ? __ldg(oidx + lo + tid) - span0 : -1;   // (a span has 12 at 0.3 %)
    s.mask[tid] = 0u;
    if (tid == 0) {
        s.lo = lo;
        s.hi = hi;
    }
    const int64_t c0 = span0 - lo;            // the span's first code
    const int len = (int)max((int64_t)0, span1 - span0 - (hi - lo));
    const int shift = (int)((uintptr_t)(codes + c0) & 15);
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s.codes);
    for (int c = tid; c * 16 < shift + len; c += DQ_THREADS) {
        const int64_t g = c0 - shift + c * 16;
        if (g >= 0 && g + 16 <= n_codes) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + c * 16), "l"(codes + g) : "memory");
        } else {
            uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int e = 0; e < 16; ++e)
                if (g + e >= 0 && g + e < n_codes) w[e >> 2] |= (uint32_t)(uint8_t)codes[g + e] << (8 * (e & 3));
            *reinterpret_cast<uint4 *>(s.codes + c * 16) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
    __syncthreads();
    if (first >= 0 && first < DQ_SPAN) atomicOr(&s.mask[first >> 5], 1u << (first & 31));
    for (int64_t i = lo + tid + DQ_THREADS; i < hi; i += DQ_THREADS) {
        const int64_t p = __ldg(oidx + i) - span0;
        if (p >= 0 && p < DQ_SPAN) atomicOr(&s.mask[p >> 5], 1u << (p & 31));
    }
    __syncthreads();
    const uint32_t own = __popc(s.mask[tid]);
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
    s.start[tid] = (uint32_t)(shift + tid * 32) - (base + inc - own);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
}

// Byte of the staged codes where position p's code lies, or would, and the outliers of the 32 positions p is among.
__device__ __forceinline__ uint32_t code_at(const Span &s, int p, uint32_t &word) {
    word = s.mask[p >> 5];
    return s.start[p >> 5] + (uint32_t)(p & 31) - (uint32_t)__popc(word & ((1u << (p & 31)) - 1u));
}
// The 4 * W codes from byte `o` of the staged codes on, biased by 128.
template <int W>
__device__ __forceinline__ void codes_at(const Span &s, uint32_t o, uint32_t (&w)[W]) {
    const uint32_t *src = reinterpret_cast<const uint32_t *>(s.codes) + (o >> 2);
    const uint32_t r = (o & 3u) * 8u;
    uint32_t raw[W + 1];
#pragma unroll
    for (int i = 0; i <= W; ++i) raw[i] = src[i];
#pragma unroll
    for (int i = 0; i < W; ++i) w[i] = __funnelshift_r(raw[i], raw[i + 1], r) ^ 0x80808080u;
}
// The same for positions with outliers (`bits`) among them: code 0 in their places.
template <int W>
__device__ __forceinline__ void codes_around(const Span &s, uint32_t o, uint32_t bits, uint32_t (&w)[W]) {
#pragma unroll
    for (int i = 0; i < W; ++i) w[i] = 0u;
#pragma unroll
    for (int e = 0; e < 4 * W; ++e) {
        const bool out = (bits >> e) & 1u;
        const uint32_t code = out ? 0x80u : (uint32_t)s.codes[o] ^ 0x80u;
        o += out ? 0u : 1u;
        w[e >> 2] |= code << (8 * (e & 3));
    }
}
// Calls f(unit) in one thread for every unit (2^SHIFT positions) of the span that holds outliers.  Work per element is what
// bounds these kernels beside latency, and most warps have some outlier: so units without are written first, without a
// branch, and those with afterwards, one per thread.
template <int SHIFT, class F>
__device__ __forceinline__ void for_units_with_outliers(const Span &s, const int64_t *oidx, int64_t span0, const F &f) {
    for (int64_t i = s.lo + threadIdx.x; i < s.hi; i += DQ_THREADS) {
        const int64_t p = __ldg(oidx + i) - span0, before = i > s.lo ? __ldg(oidx + i - 1) - span0 : -1;
        if (p >= 0 && p < DQ_SPAN && (before < 0 || before >> SHIFT != p >> SHIFT)) f((int)(p >> SHIFT));
    }
}

// Two biased codes of a word (bytes 0, 1 or 2, 3) as fp16(code), exact.
template <uint32_t SEL>
__device__ __forceinline__ __half2 code_pair(uint32_t w) {
    const uint32_t h = __byte_perm(w, 0x64646464u, SEL);   // halves 1024 + u
    const __half2 bias = __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480));  // 1152
    return __hsub2(*reinterpret_cast<const __half2 *>(&h), bias);
}

__device__ __forceinline__ void scale_unit(const uint32_t (&c)[2], uint16_t scale, uint32_t (&o)[4]) {
    const __half2 s2 = __half2half2(__ushort_as_half(scale));
    __half2 h[4] = {code_pair<0x5140>(c[0]), code_pair<0x5342>(c[0]), code_pair<0x5140>(c[1]), code_pair<0x5342>(c[1])};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        h[i] = __hmul2(h[i], s2);
        o[i] = *reinterpret_cast<uint32_t *>(&h[i]);
    }
}

struct DequantParams {
    const int8_t *codes;
    int64_t n_codes;
    const uint16_t *ovals;
    const int64_t *oidx;
    int64_t n_out;
    const uint16_t *scales;
    int64_t numel, padded, spans;
    int bs, bs_shift, w_aligned;
    int marked;                               // the spans' ends are where mark_dequant_kernel puts them
    uint16_t *w;
};
__global__ void __launch_bounds__(256) mark_dequant_kernel(DequantParams p) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    mark_spans(p.oidx, p.n_out, p.spans, (int64_t)blockIdx.x * 256 + threadIdx.x, threadIdx.x & 31,
               [&](int64_t span) { return reinterpret_cast<Ends *>(p.w + span * DQ_SPAN); });
}

// One unit (8 elements, 16 bytes of output) per thread and step.  The product of the code and the scale is rounded to fp16
// once (adaptive_quantizer.py:216).  POW2: the block size is a power of two; others divide, 32 bits wide, once per unit.
// Both in one kernel cost the powers of two 1 us of 34 at 11008 x 4096.
template <bool POW2>
__global__ void __launch_bounds__(DQ_THREADS) dequantize_kernel(DequantParams p) {
    __shared__ Span s;
    const int tid = threadIdx.x;
    const int64_t span0 = (int64_t)blockIdx.x * DQ_SPAN, span1 = min(span0 + DQ_SPAN, p.padded);
    const bool in_one_block = (p.bs & 7) == 0;   // blocks are whole units
    const bool whole = span0 + DQ_SPAN <= p.numel && p.w_aligned && in_one_block;
    constexpr int STEPS = DQ_SPAN / (DQ_THREADS * 8);
    uint16_t sc[STEPS];
    // the span's first block, and the place of its first element in it: below, 32 bits do
    const int64_t block0 = POW2 ? span0 >> p.bs_shift : span0 / p.bs;
    const uint32_t in_block = POW2 ? (uint32_t)(span0 & (p.bs - 1)) : (uint32_t)(span0 - block0 * p.bs);
    const uint16_t *scales = p.scales + block0;
    auto block_of = [&](uint32_t e) { return POW2 ? (in_block + e) >> p.bs_shift : (in_block + e) / (uint32_t)p.bs; };
    auto scale_of = [&](int unit) { return __ldg(scales + block_of((uint32_t)unit * 8u)); };
#pragma unroll
    for (int k = 0; k < STEPS; ++k) sc[k] = whole ? scale_of(tid + k * DQ_THREADS) : (uint16_t)0;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    uint16_t *w = p.w + span0;
    Ends ends;
    if (p.marked && span0 + 8 <= p.numel) {
        const volatile Ends *at = reinterpret_cast<const volatile Ends *>(w);   // (all threads, before any of them writes)
        ends = {at->lo, at->hi};
    } else {
        ends = search_span(s, p.oidx, p.n_out, span0, span1);
    }
    stage_span(s, p.codes, p.n_codes, p.oidx, p.n_out, ends, span0, span1);
    // the outliers of a unit (`bits`), the first of which is the span's outlier number `before`, into its output
    auto put_outliers = [&](uint32_t (&o)[4], uint32_t bits, uint32_t before) {
        const uint16_t *val = p.ovals + s.lo + before;
        for (uint32_t m = bits; m; m &= m - 1, ++val) {
            const int j = __ffs(m) - 1;
            const uint32_t v = __ldg(val);
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (q == j >> 1) o[q] = (j & 1) ? __byte_perm(o[q], v, 0x5410) : __byte_perm(o[q], v, 0x3254);
        }
    };
    const uint32_t shift = (uint32_t)((uintptr_t)(p.codes + (span0 - s.lo)) & 15);   // where stage_span put the first code
    if (whole) {
#pragma unroll
        for (int k = 0; k < STEPS; ++k) {
            const int unit = tid + k * DQ_THREADS;
            uint32_t word, c[2], o[4];
            const uint32_t at = code_at(s, unit * 8, word);
            codes_at<2>(s, at, c);
            scale_unit(c, sc[k], o);
            if (!((word >> ((unit & 3) * 8)) & 0xffu)) *reinterpret_cast<uint4 *>(w + unit * 8) = make_uint4(o[0], o[1], o[2], o[3]);
        }
        for_units_with_outliers<3>(s, p.oidx, span0, [&](int unit) {
            uint32_t word, c[2], o[4];
            const uint32_t at = code_at(s, unit * 8, word), bits = (word >> ((unit & 3) * 8)) & 0xffu;
            codes_around<2>(s, at, bits, c);
            scale_unit(c, scale_of(unit), o);
            put_outliers(o, bits, shift + (uint32_t)unit * 8u - at);
            *reinterpret_cast<uint4 *>(w + unit * 8) = make_uint4(o[0], o[1], o[2], o[3]);
        });
        return;
    }
    const int real = (int)min((int64_t)DQ_SPAN, p.numel - span0);   // (none or less: blocks of padding alone)
    if (!p.w_aligned) {
        // an output on no 16-byte boundary: element by element, so that a warp's 2-byte stores are neighbours (eight of a
        // thread's own in a row are 10 % slower)
        const uint32_t bs = (uint32_t)p.bs, blocks_on = POW2 ? 0u : DQ_THREADS / bs, in_block_on = POW2 ? 0u : DQ_THREADS % bs;
        uint32_t block = block_of(tid), place = POW2 ? 0u : in_block + tid - block * bs;
        for (int e = tid; e < real; e += DQ_THREADS) {
            if (POW2) block = block_of(e);
            const uint16_t scale = __ldg(scales + block);
            if (!POW2) {   // the next element's block, without another division
                block += blocks_on;
                place += in_block_on;
                if (place >= bs) {
                    place -= bs;
                    ++block;
                }
            }
            uint32_t word;
            const uint32_t at = code_at(s, e, word);
            if ((word >> (e & 31)) & 1u) {
                w[e] = __ldg(p.ovals + s.lo + (shift + (uint32_t)e - at));
            } else {
                const __half code = __short2half_rn((short)(int8_t)s.codes[at]);
                w[e] = __half_as_ushort(__hmul(code, __ushort_as_half(scale)));
            }
        }
        return;
    }
    // the last span, and blocks that end inside a unit
#pragma unroll 1
    for (int unit = tid; unit * 8 < real; unit += DQ_THREADS) {
        uint32_t word, c[2], o[4];
        const uint32_t at = code_at(s, unit * 8, word), bits = (word >> ((unit & 3) * 8)) & 0xffu;
        if (bits) codes_around<2>(s, at, bits, c);
        else codes_at<2>(s, at, c);
        if (in_one_block) {
            scale_unit(c, scale_of(unit), o);
        } else {
            // (at most every place has a block of its own, and places beyond the padded end have none)
            __half2 h[4] = {code_pair<0x5140>(c[0]), code_pair<0x5342>(c[0]), code_pair<0x5140>(c[1]), code_pair<0x5342>(c[1])};
            const int last = real - 1;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint16_t a = __ldg(scales + block_of((uint32_t)min(unit * 8 + 2 * i, last)));
                const uint16_t b = __ldg(scales + block_of((uint32_t)min(unit * 8 + 2 * i + 1, last)));
                h[i] = __hmul2(h[i], __halves2half2(__ushort_as_half(a), __ushort_as_half(b)));
                o[i] = *reinterpret_cast<uint32_t *>(&h[i]);
            }
        }
        put_outliers(o, bits, shift + (uint32_t)unit * 8u - at);
        if (unit * 8 + 8 <= real) {
            *reinterpret_cast<uint4 *>(w + unit * 8) = make_uint4(o[0], o[1], o[2], o[3]);
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (unit * 8 + e < real) w[unit * 8 + e] = (uint16_t)(o[e >> 1] >> (16 * (e & 1)));
        }
    }
}

// Byte offset of weight (row, col) inside the tile-major layout: 128-row x 64-column tiles, row by row.
__device__ __forceinline__ int64_t tile_offset(int64_t row, int64_t col, int64_t k_tiles) {
    return ((row >> 7) * k_tiles + (col >> 6)) * 8192 + (row & 127) * 64 + (col & 63);
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
// the grid: the longest chain of dependent loads), a 128-row x 16-block piece of the scale transposition, or 8192
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
        const int64_t strip0 = strip * 16 * t.n_cols, strip1 = max(strip0, min(strip * 16 + 16, t.n_rows) * t.n_cols);
        const uint32_t n_cols = (uint32_t)t.n_cols;   // (a strip has at most 2^28 positions)
        StripScratch &s = sh.strip;
        if (warp < 2) {
            const int64_t at = warp_lower_bound(t.oidx, t.n_out, warp == 0 ? strip0 : strip1, lane);
            if (lane == 0) s.row_at[warp * 16] = at;
        }
        __syncthreads();
        const int64_t first = s.row_at[0], end = max(first, s.row_at[16]);
        const int total = (int)(end - first);
        __syncthreads();
        // The ranks below are a permutation, and what the linear kernels index with the entries lies in the strip, only if
        // the strip's positions ascend and lie in it; then its rows begin where the rows of two neighbours differ (which takes
        // one more round trip to memory, where a search per row took four, three times over).
        int bad = 0;
        for (int i = tid; i < total && total <= RP_STRIP_CAP; i += DQ_THREADS) {
            const int64_t at = __ldg(t.oidx + first + i) - strip0, before = i > 0 ? __ldg(t.oidx + first + i - 1) - strip0 : -1;
            if (before >= at || at < 0 || at >= strip1 - strip0) {
                bad = 1;
            } else {
                const int row = (int)((uint32_t)at / n_cols), above = before >= 0 ? (int)((uint32_t)before / n_cols) : -1;
                s.col[i] = (uint32_t)at - (uint32_t)row * n_cols;
                for (int r = above + 1; r <= row; ++r) s.row_at[r] = first + i;
                if (i == total - 1)
                    for (int r = row + 1; r <= 16; ++r) s.row_at[r] = end;
            }
        }
        if (total == 0 && tid < 17) s.row_at[tid] = first;
        bad = __syncthreads_or(bad);
        if (bad || total > RP_STRIP_CAP) {
            // Many outliers, or a damaged file: a search per row.  A strip whose positions do not ascend or whose rows do not
            // begin where the searches say gets an empty list.
            for (int r = warp; r < 17; r += DQ_THREADS / 32) {
                const int64_t at = warp_lower_bound(t.oidx, t.n_out, min(strip * 16 + r, t.n_rows) * t.n_cols, lane);
                if (lane == 0) s.row_at[r] = at;
            }
            __syncthreads();
            if (!bad) {
                if (tid < 17) {
                    const int64_t at = s.row_at[tid], key = min(strip0 + tid * t.n_cols, strip1);
                    bad = at < first || at > end || (tid < 16 && s.row_at[tid + 1] < at);
                    if (!bad) bad = (at > first && __ldg(t.oidx + at - 1) >= key) || (at < end && __ldg(t.oidx + at) < key);
                }
                for (int i = tid + 1; i < total; i += DQ_THREADS) bad |= __ldg(t.oidx + first + i - 1) >= __ldg(t.oidx + first + i);
            }
            bad = __syncthreads_or(bad);
        }
        if (t.row_ptr && tid < 17 && strip * 16 + tid <= t.n_rows && (tid < 16 || strip * 16 + 16 == t.n_rows))
            t.row_ptr[strip * 16 + tid] = (int32_t)s.row_at[tid];
        if (bad) {
            const int n_chunks = (int)(n_cols >> 6);
            for (int c = tid; c <= n_chunks; c += DQ_THREADS) t.chunk_ptr[strip * (n_chunks + 1) + c] = (int32_t)(t.entry_base + first);
        } else if (total <= RP_STRIP_CAP) {
            write_strip(t, strip, s, [&](int i) { return s.col[i]; });
        } else {
            write_strip(t, strip, s, [&](int i) { return (uint32_t)(__ldg(t.oidx + first + i) - strip0) % n_cols; });
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
    const uint32_t k_tiles = n_cols >> 6, in_tile = (uint32_t)row0 & 127u;
    uint8_t *tiles = t.tiles + (row0 >> 7) * (int64_t)k_tiles * 8192;
    auto place = [&](uint32_t q) -> uint8_t * {
        const uint32_t c = col0 + q, dr = c / n_cols, col = c - dr * n_cols, row = in_tile + dr;
        return tiles + ((uint64_t)((row >> 7) * k_tiles + (col >> 6)) * 8192u + (row & 127u) * 64u + (col & 63u));
    };
    if (span0 < numel) {
        // (a search in every CTA: they begin while the strips are at work, and marking the spans beforehand, as the
        // dequantizer does, only held them up: 11008 x 4096 45 us, so 40)
        const Ends ends = search_span(sh.span, t.oidx, t.n_out, span0, span1);
        stage_span(sh.span, t.codes, t.n_codes, t.oidx, t.n_out, ends, span0, span1);
    }
#pragma unroll
    for (int k = 0; k < DQ_SPAN / (DQ_THREADS * 16); ++k) {
        const int q = tid * 16 + k * DQ_THREADS * 16;
        if (span0 + q >= padded) break;
        uint32_t w[4] = {0x80808080u, 0x80808080u, 0x80808080u, 0x80808080u}, word = 0u;
        if (span0 + q < numel) codes_at<4>(sh.span, code_at(sh.span, q, word), w);
        if (!((word >> (q & 31)) & 0xffffu)) *reinterpret_cast<uint4 *>(place(q)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    if (span0 < numel)
        for_units_with_outliers<4>(sh.span, t.oidx, span0, [&](int unit) {
            uint32_t word, w[4];
            const uint32_t at = code_at(sh.span, unit * 16, word);
            codes_around<4>(sh.span, at, (word >> ((unit & 1) * 16)) & 0xffffu, w);
            *reinterpret_cast<uint4 *>(place(unit * 16)) = make_uint4(w[0], w[1], w[2], w[3]);
        });
}

// Launches the dequantizer, whose CTAs may start while the marking kernel in front of it still runs (`beside`).
int launch_dequantize(unsigned grid, bool beside, cudaStream_t st, const DequantParams &p) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(DQ_THREADS);
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = beside ? 1 : 0;
    return check_cuda(cudaLaunchKernelEx(&cfg, p.bs_shift >= 0 ? dequantize_kernel<true> : dequantize_kernel<false>, p), "dequantize_kernel launch");
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
    const int64_t spans = ceil_div_i64(padded, DQ_SPAN);
    ATLAS_RETURN_IF(spans > 0x7fffffff, ATLAS_ERR_UNSUPPORTED, "atlas_dequantize: tensor too large");
    DequantParams p;
    p.codes = codes;
    p.n_codes = n_codes;
    p.ovals = (const uint16_t *)outlier_vals;
    p.oidx = outlier_idx;
    p.n_out = n_outliers;
    p.scales = (const uint16_t *)scales;
    p.numel = numel;
    p.padded = padded;
    p.spans = ceil_div_i64(numel, DQ_SPAN) - (numel % DQ_SPAN > 0 && numel % DQ_SPAN < 8 ? 1 : 0);   // those with room for their ends
    p.bs = block_size;
    p.bs_shift = (block_size & (block_size - 1)) == 0 ? __builtin_ctz((unsigned)block_size) : -1;
    p.w_aligned = ((uintptr_t)w_out & 15) == 0;
    p.marked = p.w_aligned && n_outliers > DQ_SEARCHED;
    p.w = (uint16_t *)w_out;
    if (p.marked) {
        mark_dequant_kernel<<<(unsigned)ceil_div_i64(n_outliers + 1, 256), 256, 0, (cudaStream_t)stream>>>(p);
        rc = check_cuda(cudaGetLastError(), "mark_dequant_kernel launch");
        if (rc) return rc;
    }
    return launch_dequantize((unsigned)spans, p.marked, (cudaStream_t)stream, p);
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
