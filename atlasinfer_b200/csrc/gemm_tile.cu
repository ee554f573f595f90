// Quantized linear for up to 128 rows of x: y[m][n] = sum_k x[m][k] * W[n][k] + bias[n] on tcgen05, two CTAs per SM.
//
// Replaces the dequantize-then-F.linear of QuantizedLinear.forward (integration/atlas_wrappers.py:56,67) between single
// rows (gemv.cu) and prompts (gemm.cu).  The bound is HBM (1.03 bytes per weight); what competes with it is the
// instruction stream that rebuilds the fp16 weights.
//
// One CTA computes 128 (output features) x BN (tokens) over a slice of K; the slices of a tile are the CTAs of one
// cluster.  A pipeline step is one k-tile (64 columns of K).
//   warp 0       activation producer: TMA of the BN x 64 tile (128-byte swizzle)
//   warp 3       bf16 rows, where the tensor map delivers them: converted to fp16 in place, 16 bytes at a time (the
//                swizzle only permutes 16-byte pieces)
//   warp 2       code producer: TMA of the 8 KB code tile (64-byte swizzle) and 256 B of scales
//   warps 4-11   dequantizers, thread = row: warp (q, ph) rebuilds rows 32q .. 32q+31 of every second k-tile as
//                fp16(fp16(code) * scale) and stores them into a 16 KB K-major A tile in shared memory.  The outliers
//                of the warp's two strips are then written over their zero-coded slots, one 2-byte store per outlier
//                and lane: with the operand in shared memory a weight is addressable, while patching it in registers
//                (as the prompt kernel must, whose operand goes to tensor memory) costs a select per register.
//   warp 1       one thread issues four tcgen05.mma (M 128, N = BN, K 16, fp32 accumulators in TMEM) per k-tile
// Shared memory holds half of an SM's: two CTAs are resident, so one's prologue, epilogue and barrier round trips are
// covered by the other's stream, and the first CTAs of the next launch (programmatic dependent launch) fetch their
// codes while the last ones of this launch finish.
//
// The K slices of a tile add up through distributed shared memory: every CTA leaves its fp32 tile in its own shared
// memory, and after a cluster barrier each one adds its share of the elements over all slices, in slice order
// (deterministic), adds the bias and writes y.  No partial sums in global memory, no second kernel.
//
// Measured (us, launch chain, against gemm.cu's kernel that served these sizes before): 57344 x 8192 at 32 rows 201 -> 156,
// 64 rows 207 -> 163; 8192 x 28672 at 32 rows 95 -> 76; 22016 x 4096 at 32 rows 52 -> 37, 128 rows 58 -> 48; 4096 x 11008
// at 128 rows 66 -> 27 (where gemm.cu's kernel is the faster one, route_for in gemm.cu leaves it the call).  Issue slots are 45 % used (ncu, 22016 x 4096 at 32
// rows); the rest is the chain of a k-tile through one A tile (rebuild, fence, MMA, commit), of which four are in flight
// per SM.  Up to 16 rows (BN = 16) this is reached on request only: the per-strip kernel serves them.
//
// Every mbarrier wait is bounded; when one runs out the CTA sets the caller's status word, the producers and the MMA
// thread wait (bounded) for what they have issued, and the CTA takes part in the cluster barriers, frees its TMEM and
// returns with nothing in flight.
#include <cuda_bf16.h>

#include "common.cuh"
#include "gemm_tile.cuh"
#include "tensor_core.cuh"

namespace atlas {
namespace {

constexpr int TL_BM = 128, TL_BK = 64;
constexpr int TL_DQ_WARPS = 8;                        // 4 row quarters x 2 k-tile phases
constexpr int TL_CTRL_WARPS = 4;
constexpr int TL_THREADS = (TL_CTRL_WARPS + TL_DQ_WARPS) * 32;
constexpr int TL_DONE = 8;                            // `done` barriers; a ring that waits on them has at most 8 slots
constexpr int TL_AS = 2;                              // A tiles: one per phase
constexpr uint32_t TL_A_BYTES = TL_BM * TL_BK * 2;    // 16 KB rebuilt weights
constexpr uint32_t TL_C_BYTES = TL_BM * TL_BK;        // 8 KB codes
constexpr uint32_t TL_S_BYTES = 256;                  // scales of 128 rows
constexpr int TL_RED = TL_BM + 4;                     // floats per token of the fp32 tile: the pad keeps banks apart

template <int BN>
struct TileSmem {
    static constexpr uint32_t X_BYTES = BN * TL_BK * 2;
    // Slots of the activation and of the code ring: what is left of half an SM's shared memory.  A load takes 2 to 3 us
    // under this traffic whether it comes from HBM or, as the activations, from L2, so both rings must be deep.
    static constexpr int XS = BN <= 16 ? 8 : (BN == 32 ? 7 : (BN == 64 ? 5 : (BN == 96 ? 3 : 2)));
    static constexpr int CS = BN <= 16 ? 7 : (BN == 32 ? 6 : (BN == 64 ? 4 : 5));
    // A dequantizer takes every second k-tile, so with an odd ring it comes back to a slot two rounds later, when a
    // parity can no longer tell the rounds apart.  It is never that far ahead: before k-tile kt - 2 it has waited for the
    // MMAs of kt - 4, so k-tile kt - CS, the round in between, has landed.
    static_assert(CS % 2 == 0 || CS >= 4, "code ring parity");
    static constexpr uint32_t OFF_A = 0;
    static constexpr uint32_t OFF_X = OFF_A + TL_AS * TL_A_BYTES;
    static constexpr uint32_t OFF_C = OFF_X + XS * X_BYTES;
    static constexpr uint32_t OFF_S = OFF_C + CS * TL_C_BYTES;
    static constexpr uint32_t OFF_BAR = OFF_S + CS * TL_S_BYTES;
    static constexpr uint32_t TOTAL = OFF_BAR + 512 + 1024 /*alignment slack*/;
    static constexpr uint32_t TMEM_COLS = BN <= 32 ? 32 : (BN <= 64 ? 64 : 128);
    static_assert(BN * TL_RED * 4 <= OFF_S, "the fp32 tile goes over the idle rings");
    static_assert(TOTAL + 1024 <= 228 * 1024 / 2, "two CTAs per SM");
};

template <int BN>
constexpr uint32_t tl_idesc() { return (1u << 4) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(TL_BM >> 4) << 24); }

__device__ __forceinline__ void cluster_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr, uint32_t rank) {
    float4 v;
    asm volatile(
        "{\n\t.reg .b32 a;\n\t"
        "mapa.shared::cluster.u32 a, %4, %5;\n\t"
        "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr), "r"(rank) : "memory");
    return v;
}

template <int BN>
__global__ void __launch_bounds__(TL_THREADS, 2)
tile_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap c_map, TileParams p) {
    using SM = TileSmem<BN>;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    constexpr int CS = SM::CS, XS = SM::XS;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;          // operand tiles need 1024-byte alignment
    unsigned char *base_ptr = smem_raw + (base - raw);
    const uint32_t bars = base + SM::OFF_BAR;
    auto done_bar = [&](int kt) { return bars + 8u * (kt % TL_DONE); };               // MMAs of k-tile kt have finished
    auto done_par = [&](int kt) { return (uint32_t)((kt / TL_DONE) & 1); };
    auto ready_bar = [&](int kt) { return bars + 8u * (TL_DONE + (kt & 1)); };        // A tile stored: 4 warps
    auto x_full = [&](int s) { return bars + 8u * (TL_DONE + 2 + s); };               // fp16 activations in the slot
    auto x_land = [&](int s) { return bars + 8u * (TL_DONE + 2 + XS + s); };          // bf16 activations in the slot
    auto full_c = [&](int s) { return bars + 8u * (TL_DONE + 2 + 2 * XS + s); };
    auto empty_c = [&](int s) { return bars + 8u * (TL_DONE + 2 + 2 * XS + CS + s); };
    constexpr int N_BARS = TL_DONE + 2 + 2 * XS + 2 * CS;
    static_assert(N_BARS * 8 + 16 <= 512 && XS <= TL_DONE, "barrier area");
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(base_ptr + SM::OFF_BAR + 8 * N_BARS);
    volatile int *s_abort = reinterpret_cast<volatile int *>(base_ptr + SM::OFF_BAR + 8 * N_BARS + 8);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n0 = blockIdx.x * TL_BM;
    const int slice = blockIdx.y;
    const int rows = p.m;   // tokens, at most BN
    const int kt_begin = (int)((long long)p.k_tiles * slice / p.splits);
    const int KT = (int)((long long)p.k_tiles * (slice + 1) / p.splits) - kt_begin;

    if (tid == 1 || tid == 32 * 2 + 1)
        asm volatile("prefetch.tensormap [%0];" ::"l"(tid < 32 ? (const void *)&x_map : (const void *)&c_map) : "memory");
    if (tid == 0) {
        for (int s = 0; s < TL_DONE; ++s) mbar_init(done_bar(s), 1);
        for (int s = 0; s < TL_AS; ++s) mbar_init(ready_bar(s), 4);
        for (int s = 0; s < XS; ++s) { mbar_init(x_full(s), 1); mbar_init(x_land(s), 1); }
        for (int s = 0; s < CS; ++s) { mbar_init(full_c(s), 1); mbar_init(empty_c(s), 4); }
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32((const void *)tmem_slot)), "r"(SM::TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    int issued = 0;   // k-tiles that this thread (either producer, the MMA thread) has asked for

    if (warp == 0) {
        // ------------------------------ activations ------------------------------
        asm volatile("griddepcontrol.wait;" ::: "memory");   // x comes from earlier kernels of the stream
        if (lane == 0) {
            for (int kt = 0; kt < KT && !*s_abort; ++kt) {
                if (kt >= XS && !mbar_wait<20>(done_bar(kt - XS), done_par(kt - XS))) { *s_abort = 1; break; }
                const uint32_t bar = p.x_bf16 ? x_land(kt % XS) : x_full(kt % XS);
                mbar_arrive_expect_tx(bar, SM::X_BYTES);
                tma_load_2d(base + SM::OFF_X + (kt % XS) * SM::X_BYTES, &x_map, (kt_begin + kt) * TL_BK, 0, bar);
                issued = kt + 1;
            }
        }
    } else if (warp == 3) {
        // ------------------------------ bf16 -> fp16 in place ------------------------------
        // rows in 16-byte pieces, whatever their swizzle
        if (p.x_bf16) {
            const int pieces = rows * 8;
            for (int kt = 0; kt < KT; ++kt) {
                if (!mbar_wait_warp<0>(x_land(kt % XS), (uint32_t)((kt / XS) & 1), s_abort)) { *s_abort = 1; break; }
                uint4 *tile = reinterpret_cast<uint4 *>(base_ptr + SM::OFF_X + (kt % XS) * SM::X_BYTES);
                for (int i0 = lane; i0 < pieces; i0 += 128) {   // four pieces at a time: their loads overlap
                    uint4 v[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (i0 + u * 32 < pieces) v[u] = tile[i0 + u * 32];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (i0 + u * 32 < pieces)
                            tile[i0 + u * 32] = make_uint4(bf16x2_to_f16x2(v[u].x), bf16x2_to_f16x2(v[u].y),
                                                           bf16x2_to_f16x2(v[u].z), bf16x2_to_f16x2(v[u].w));
                }
                fence_async_smem();   // the tensor core reads the tile through the async proxy
                __syncwarp();
                if (lane == 0) mbar_arrive(x_full(kt % XS));
            }
        }
    } else if (warp == 2) {
        // ------------------------------ codes and scales ------------------------------
        if (lane == 0) {
            const int64_t crow0 = (int64_t)blockIdx.x * p.k_tiles + kt_begin;   // code tiles are runs of 128 rows of the map
            for (int kt = 0; kt < KT; ++kt) {
                const int slot = kt % CS, round = kt / CS;
                if (round > 0 && !mbar_wait<40>(empty_c(slot), (uint32_t)((round - 1) & 1))) { *s_abort = 1; break; }
                if (*s_abort) break;
                mbar_arrive_expect_tx(full_c(slot), TL_C_BYTES + (p.bs_tiles ? TL_S_BYTES : 0u));
                tma_load_2d(base + SM::OFF_C + slot * TL_C_BYTES, &c_map, 0, (int)((crow0 + kt) * TL_BM), full_c(slot));
                if (p.bs_tiles)
                    bulk_load_1d(base + SM::OFF_S + slot * TL_S_BYTES,
                                 p.scales_t + ((size_t)blockIdx.x * p.blocks_per_row + (kt_begin + kt) / p.bs_tiles) * 128, TL_S_BYTES, full_c(slot));
                issued = kt + 1;
            }
        }
    } else if (warp == 1) {
        // ------------------------------ MMA ------------------------------
        if (lane == 0) {
            const uint64_t da0 = make_smem_desc(base + SM::OFF_A), db0 = make_smem_desc(base + SM::OFF_X);
            bool ok = true;
            for (int kt = 0; kt < KT && ok; ++kt) {
                ok = mbar_wait(x_full(kt % XS), (uint32_t)((kt / XS) & 1)) && mbar_wait(ready_bar(kt), (uint32_t)((kt >> 1) & 1));
                if (!ok || ((kt & 7) == 7 && *s_abort)) { ok = false; break; }
                tcgen05_fence_after();
                const uint64_t da = da0 + (uint64_t)(((kt & 1) * TL_A_BYTES) >> 4);   // the address field counts 16-byte units
                const uint64_t db = db0 + (uint64_t)(((kt % XS) * SM::X_BYTES) >> 4);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    umma_f16_ss(tmem_base, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), tl_idesc<BN>(), (kt | k) != 0);
                umma_commit(done_bar(kt));   // frees the A tile and the activation slot
                issued = kt + 1;
            }
            if (!ok) *s_abort = 1;
        }
    } else {
        // ------------------------------ dequantizers ------------------------------
        const int q = warp & 3, ph = (warp - TL_CTRL_WARPS) >> 2;   // TMEM lane quarter = row quarter, k-tile phase
        const int rl = q * 32 + lane;
        const uint32_t code_off = (uint32_t)rl * 64u, swz = (uint32_t)((rl >> 1) & 3);
        unsigned char *a_row = base_ptr + SM::OFF_A + ph * TL_A_BYTES + rl * 128;
        const uint32_t a_swz = (uint32_t)(rl & 7);
        // Side-table: a half-warp serves its own strip.  The entry range of a k-tile is requested three of the warp's k-tiles
        // ahead, its first 16 entries two ahead: they come from HBM like the codes.  (Four ahead through an unrolled
        // loop was slower, 43 against 39 us at 22016 x 4096 and 32 tokens: the loop then misses the instruction cache.)
        const int half = lane >> 4, ej = lane & 15;
        const int64_t strip = (int64_t)blockIdx.x * 8 + 2 * q + half;
        const int32_t *cp = p.chunk_ptr + strip * (p.k_tiles + 1) + kt_begin;
        unsigned char *a_strip = base_ptr + SM::OFF_A + ph * TL_A_BYTES + (q * 32 + half * 16) * 128;
        const uint16_t *sc_tile = p.scales_t + (size_t)blockIdx.x * p.blocks_per_row * 128;
        auto range = [&](int kt, int &b, int &e) {
            b = e = 0;
            if (kt < KT) { b = __ldg(cp + kt); e = __ldg(cp + kt + 1); }
        };
        auto entry = [&](int b, int e, uint32_t &ent, uint32_t &val) {
            ent = val = 0u;
            if (b + ej < e) { ent = __ldg(p.entries + b + ej); val = __ldg(p.ovals + b + ej); }
        };
        int b0, e0, b1, e1, b2, e2;
        uint32_t ent0, val0, ent1, val1;
        range(ph, b0, e0);
        range(ph + 2, b1, e1);
        range(ph + 4, b2, e2);
        entry(b0, e0, ent0, val0);
        entry(b1, e1, ent1, val1);
        bool ok = true;
#pragma unroll 1
        for (int kt = ph; kt < KT; kt += 2) {
            int b3, e3;
            uint32_t ent2, val2;
            range(kt + 6, b3, e3);
            entry(b2, e2, ent2, val2);
            const int slot = kt % CS;
            if (!mbar_wait_warp<20>(full_c(slot), (uint32_t)((kt / CS) & 1), s_abort)) { ok = false; break; }
            const unsigned char *codes = base_ptr + SM::OFF_C + slot * TL_C_BYTES + code_off;
            uint4 L[4];   // chunk c sits at c ^ ((row >> 1) & 3) under the 64-byte swizzle
#pragma unroll
            for (int c = 0; c < 4; ++c) L[c] = *reinterpret_cast<const uint4 *>(codes + ((c ^ swz) << 4));
            __half sh[4];
            const int col0 = (kt_begin + kt) * TL_BK;
            if (p.bs_tiles) {
                sh[0] = sh[1] = sh[2] = sh[3] = __ushort_as_half(reinterpret_cast<const uint16_t *>(base_ptr + SM::OFF_S + slot * TL_S_BYTES)[rl]);
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c) sh[c] = __ushort_as_half(__ldg(sc_tile + (int64_t)((col0 + c * 16) / p.bs) * 128 + rl));
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty_c(slot));
            // the A tile must have been read by the MMAs of its previous use
            if (kt >= TL_AS && !mbar_wait_warp<20>(done_bar(kt - TL_AS), done_par(kt - TL_AS), s_abort)) { ok = false; break; }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const __half2 s2 = __half2half2(sh[c]);
                uint4 lo, hi;
                dequant4(L[c].x, s2, lo.x, lo.y);
                dequant4(L[c].y, s2, lo.z, lo.w);
                dequant4(L[c].z, s2, hi.x, hi.y);
                dequant4(L[c].w, s2, hi.z, hi.w);
                *reinterpret_cast<uint4 *>(a_row + (((2 * c) ^ a_swz) << 4)) = lo;
                *reinterpret_cast<uint4 *>(a_row + (((2 * c + 1) ^ a_swz) << 4)) = hi;
            }
            __syncwarp();   // the outliers go over codes that other lanes have stored
            auto put = [&](uint32_t e, uint32_t v) {
                const uint32_t row = e >> 24, col = (e & 0xffffffu) - (uint32_t)col0;
                *reinterpret_cast<uint16_t *>(a_strip + row * 128 + (((col >> 3) ^ (row & 7)) << 4) + (col & 7) * 2) = (uint16_t)v;
            };
            if (b0 + ej < e0) put(ent0, val0);
            for (int i = b0 + 16 + ej; i < e0; i += 16) put(__ldg(p.entries + i), __ldg(p.ovals + i));
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(ready_bar(kt));
            b0 = b1; e0 = e1; b1 = b2; e1 = e2; b2 = b3; e2 = e3;
            ent0 = ent1; val0 = val1; ent1 = ent2; val1 = val2;
        }
        // ------------------------------ accumulators -> fp32 tile in shared memory ------------------------------
        // (the rings are idle once the last MMAs have finished)
        ok = ok && mbar_wait_warp<20>(done_bar(KT - 1), done_par(KT - 1), s_abort);
        if (__all_sync(0xffffffffu, ok)) {
            tcgen05_fence_after();
            float *red = reinterpret_cast<float *>(base_ptr);
#pragma unroll 1
            for (int c = ph; c < (BN + 31) / 32; c += 2) {
                if (c * 32 >= rows) break;
                uint32_t v[32];
                tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(c * 32), v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < (BN < 32 ? BN : 32); ++j) red[(c * 32 + j) * TL_RED + rl] = __uint_as_float(v[j]);
            }
            tcgen05_fence_before();
        } else {
            *s_abort = 1;
        }
    }

    __syncthreads();
    if (*s_abort) {
        // a wait ran out somewhere: no copy may land, and no MMA run, once this CTA has gone, however far their issuers were
        if (tid == 0)
            for (int i = max(0, issued - XS); i < issued; ++i) mbar_wait<100>(p.x_bf16 ? x_land(i % XS) : x_full(i % XS), (uint32_t)((i / XS) & 1));
        if (tid == 2 * 32)
            for (int i = max(0, issued - CS); i < issued; ++i) mbar_wait<100>(full_c(i % CS), (uint32_t)((i / CS) & 1));
        if (tid == 1 * 32 && issued > 0) mbar_wait<100>(done_bar(issued - 1), done_par(issued - 1));
        __syncthreads();
    }
    tcgen05_fence_after();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(SM::TMEM_COLS) : "memory");
    if (tid == 0 && *s_abort && p.error_flag) atomicExch(p.error_flag, 1);
    if (p.splits > 1) cluster_sync();
    // ------------------------------ sum of the slices, bias, y ------------------------------
    {
        const uint32_t red = base;
        const bool vec = (p.ldy % 4 == 0) && (((uintptr_t)p.y & 7) == 0);
        for (int idx = slice * TL_THREADS + tid; idx < rows * (TL_BM / 4); idx += p.splits * TL_THREADS) {
            const int t = idx >> 5, n = n0 + (idx & 31) * 4;
            if (n >= p.n_rows) continue;
            const uint32_t at = red + (uint32_t)(t * TL_RED + (idx & 31) * 4) * 4u;
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
            if (p.splits == 1) {
                a = *reinterpret_cast<const float4 *>(base_ptr + (at - base));
            } else {
                for (int s = 0; s < p.splits; ++s) {
                    const float4 b = ld_cluster_f4(at, (uint32_t)s);
                    a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
                }
            }
            float f[4] = {a.x, a.y, a.z, a.w};
            uint16_t o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (p.bias && n + e < p.n_rows) f[e] += __half2float(__ushort_as_half(__ldg(p.bias + n + e)));
                o[e] = p.out_bf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(f[e])) : __half_as_ushort(__float2half_rn(f[e]));
            }
            uint16_t *dst = reinterpret_cast<uint16_t *>(p.y) + (int64_t)t * p.ldy + n;
            if (vec && n + 4 <= p.n_rows) {
                *reinterpret_cast<uint2 *>(dst) = make_uint2(o[0] | (uint32_t)o[1] << 16, o[2] | (uint32_t)o[3] << 16);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (n + e < p.n_rows) dst[e] = o[e];
            }
        }
    }
    if (p.splits > 1) cluster_sync();   // nobody leaves while its tile is still being read
}

template <int BN>
int launch_tile_bn(const CUtensorMap &x_map, const CUtensorMap &c_map, const TileParams &p, cudaStream_t st) {
    static thread_local int configured_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (configured_dev != dev) {
        int rc = check_cuda(cudaFuncSetAttribute(tile_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TileSmem<BN>::TOTAL),
                            "cudaFuncSetAttribute(tile smem)");
        if (rc) return rc;
        configured_dev = dev;
    }
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1;
    attr[1].val.clusterDim.y = (unsigned)p.splits;
    attr[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ceil_div_i64(p.n_rows, TL_BM), (unsigned)p.splits, 1);
    cfg.blockDim = dim3(TL_THREADS);
    cfg.dynamicSmemBytes = TileSmem<BN>::TOTAL;
    cfg.stream = st;
    const bool early = early_start();
    cfg.attrs = attr + (early ? 0 : 1);
    cfg.numAttrs = (early ? 1 : 0) + (p.splits > 1 ? 1 : 0);
    return check_cuda(cudaLaunchKernelEx(&cfg, tile_kernel<BN>, x_map, c_map, p), "tile_kernel launch");
}

// Clusters of s CTAs that are resident at once, two CTAs per SM.  A cluster lies within one GPC, so the sizes that do not
// divide a GPC's places leave some empty, and one cluster too many costs a whole second wave (K 2048 at 32 rows in four
// slices: 71 row tiles 11.1 us, 72 tiles 16.4).  The occupancy query counts one CTA per SM for this kernel.  Two CTAs of a
// cluster share an SM, so an even s takes the count of s / 2; an odd one lies between its neighbours.  Measured by stepping
// the number of tiles on one B200: 92, 71, 56, 45, 37, 33 clusters of 3 .. 8; this gives 92, 71, 53, 45, 36, 33.  (Four
// CTAs on two SMs lose a little of their count to placements on three.)
struct Clusters {
    int dev = -1;
    int resident[9];
};
const int *resident_clusters(int sms) {
    static thread_local Clusters cache;
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && dev == cache.dev) return cache.resident;
    int raw[9];
    bool ok = cudaFuncSetAttribute(tile_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TileSmem<128>::TOTAL) == cudaSuccess;
    for (int s = 1; s <= 8 && ok; ++s) {
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = 1;
        attr.val.clusterDim.y = (unsigned)s;
        attr.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(512, (unsigned)s, 1);
        cfg.blockDim = dim3(TL_THREADS);
        cfg.dynamicSmemBytes = TileSmem<128>::TOTAL;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        ok = cudaOccupancyMaxActiveClusters(&raw[s], tile_kernel<128>, &cfg) == cudaSuccess && raw[s] > 0;
    }
    if (!ok) cudaGetLastError();   // (the launch that follows reports what is wrong)
    int *n = cache.resident;
    for (int s = 1; s <= 8; ++s) n[s] = !ok ? (s <= 2 ? 2 * sms / s : 2 * sms * 8 / (10 * s)) : (raw[1] > sms ? raw[s] : (s == 1 ? 2 * raw[1] : raw[s / 2]));
    if (ok && raw[1] <= sms) {
        n[4] = raw[2] * 24 / 25;
        for (int s = 3; s <= 7; s += 2) n[s] = (n[s - 1] * (s - 1) + n[s + 1] * (s + 1)) * 48 / (100 * s);
    }
    for (int s = 1; s <= 8; ++s) n[s] = n[s] > 1 ? n[s] : 1;
    cache.dev = ok ? dev : -1;
    return cache.resident;
}

// us per k-tile and per CTA, for a CTA that has an SM to itself and for one of two that share it, by token tile.  Fitted
// to 3760 shapes (1 to 448 row tiles, K 1024 to 28672, 17 to 128 rows, fp16 and bf16, each with 1 to 8 slices): what is
// chosen by it takes 1.3 % longer than the best choice of kernel and slices, geometric mean.
struct TileCost { int tokens; double alone_kt, alone, shared_kt, shared, convert_kt; };
constexpr TileCost TILE_COST[] = {{16, .38, 3.1, .58, 4.4, .12}, {32, .405, 3.3, .60, 4.75, .16}, {64, .495, 3.2, .625, 5.7, .335},
                                  {96, .47, 5.3, .61, 6.55, 0.}, {128, .485, 5.95, .68, 7.4, 0.}};

double tile_us(const TileCost &c, int64_t tiles, int k_tiles, int s, bool convert, const int *resident, int sms) {
    const int64_t ctas = tiles * s, places = (int64_t)resident[s] * s;
    const int64_t full = ctas / places, rest = ctas % places;
    const double kt = (double)ceil_div_i64(k_tiles, s), extra = convert ? c.convert_kt : 0.;
    // f: how much of the last wave runs two to an SM.  CTAs of one slice spread over the SMs before they share.  Those of
    // a cluster share while others stand empty, the more the fuller the chip is; clusters of two and four fit beside
    // each other best; the longer they run the more it shows (the next launch has less of its work under this one's).
    const double at = (double)rest / sms;
    double f = s == 1 ? (at > 1. ? 1. : 0.) : (at - .213) / (s == 2 || s == 4 ? 1.5 : 1.);
    if (s > 1 && kt > 16.) f *= 1. + (kt - 16.) / 80.;
    f = f < 0. ? 0. : (f > 1. ? 1. : f);
    const double sum = s > 2 ? 1.8e-5 * c.tokens * c.tokens * (s - 2) : 0.;   // the sum over the slices' tiles
    const double shared = (c.shared_kt + extra) * kt + c.shared + sum, alone = (c.alone_kt + extra) * kt + c.alone;
    // (without clusters a place is taken again as soon as one CTA ends, under the work of the other CTA of the SM)
    const double us = (double)full * (s == 1 ? shared - c.shared : shared) + (rest ? f * shared + (1. - f) * alone : 0.);
    // (clusters of seven never share their SMs evenly; clusters of a further wave wait for all the places they need)
    return s == 7 || (s > 1 && full > 0) ? 1.04 * us : us;
}

}  // namespace

int tile_tokens_for(int64_t m) { return m <= 16 ? 16 : (m <= 32 ? 32 : (m <= 64 ? 64 : (m <= 96 ? 96 : 128))); }

// The slices (at most the portable cluster size) that take the least time by the model above.  What it corrects against
// counting waves of 2 x 148 CTAs: 74 row tiles in four slices do not fit one wave (9472 x 2048, 32 fp16 rows: 16.7 us, in
// two slices 11.0); many short CTAs share SMs (4096 x 1024, 64 fp16 rows: in eight slices 8.7 us, in four 6.9); one warp
// converts bf16 slower than the rest of a CTA works (1024 x 8192, 64 rows: 19.4 us, with a copy kernel in front 13.4).
TilePlan plan_tile(int64_t m, int64_t n_rows, int k_tiles, bool can_convert, bool needs_copy, int sms) {
    const int bn = tile_tokens_for(m);
    const TileCost *c = TILE_COST;
    while (c->tokens != bn) ++c;
    const int *resident = resident_clusters(sms);
    const int64_t tiles = ceil_div_i64(n_rows, TL_BM);
    TilePlan best = {1, false, 1e300};
    for (int s = 1; s <= 8 && s <= k_tiles; ++s) {
        if (can_convert && bn <= 64) {
            const double us = tile_us(*c, tiles, k_tiles, s, true, resident, sms);
            if (us < best.us) best = {s, true, us};
        }
        const double us = tile_us(*c, tiles, k_tiles, s, false, resident, sms) + (needs_copy ? copy_us(m, k_tiles) : 0.);
        if (us < best.us) best = {s, false, us};
    }
    return best;
}

int launch_tile(const CUtensorMap &x_map, const CUtensorMap &c_map, const TileParams &p, cudaStream_t st) {
    switch (tile_tokens_for(p.m)) {
        case 16: return launch_tile_bn<16>(x_map, c_map, p, st);
        case 32: return launch_tile_bn<32>(x_map, c_map, p, st);
        case 64: return launch_tile_bn<64>(x_map, c_map, p, st);
        case 96: return launch_tile_bn<96>(x_map, c_map, p, st);
        default: return launch_tile_bn<128>(x_map, c_map, p, st);
    }
}

}  // namespace atlas
