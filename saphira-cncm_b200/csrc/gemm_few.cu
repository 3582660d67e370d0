// Products of a weight matrix with 2 to 640 rows, and what stands between them in a block.
//
// A decode step of a batch (and the first levels of a generate) multiplies every weight matrix with few rows, so it is bound
// by streaming the weights. The fp16-pair engine (gemm_h3.cu) makes the rows of x the 128-row side of its tiles: with 27 rows
// most of every x tile is padding that still passes through shared memory, and N = 896 gives 28 CTAs. Here the weights are the
// 128-row side: a CTA takes 128 weight rows and a slice of K, its tokens are the columns of the MMA (32 to 128; more rows take a second
// CTA), and nothing is read twice but the small x. Raw sums of the K slices go to a partial buffer and the kernel that follows in the block adds
// them while it does its own work: rotation and cache write after QKV, residual and the next norm after the other two.
//
// The products are those of the fp16-pair engine: x1 W1 + x2 W1 (+ x1 W2 where the second halves are not all zero), one fp32
// accumulator. Weights are requested before the kernel waits for its predecessor (nothing in a step writes them).
//
// Up to 16 rows the products are fp32 multiply-adds on fp32 operands (k_few_f32): 22 bits of x, the dropped x2 W2 and the accumulator's
// truncation put the pair products 1.2 to 2 times as far from 64 bits as fp32 ones (logits of decode steps of 2 to 16 rows), and the pair
// format ends at +-4094, which the inner activations of a trained MLP can pass.
#include "gemm_few.cuh"
#include "tc_common.cuh"
#include "tc_epilogue.cuh"

#include <algorithm>

namespace ncmb {

constexpr int FW_WTILE = 128 * 64 * 2;
constexpr int fw_xtile(int NT) { return NT * 64 * 2; }
constexpr int fw_stage(int NT, bool W2) { return FW_WTILE * (W2 ? 2 : 1) + 2 * fw_xtile(NT); }
// stages that leave room for a second CTA on the SM (the next kernel's, whose first weights are then on their way), up to four
constexpr int fw_stages(int NT, bool W2) {
    int s = (110 * 1024) / fw_stage(NT, W2);
    return s > 4 ? 4 : (s < 2 ? 2 : s);
}
constexpr int FW_THREADS = 320;          // producer warp, MMA warp, eight epilogue warps (two per TMEM quadrant)
constexpr size_t fw_smem(int NT, bool W2) { return 1024 + (size_t)fw_stages(NT, W2) * fw_stage(NT, W2) + (2 * fw_stages(NT, W2) + 1) * 8 + 16; }

struct FewDev {
    int M, N, num_kb, kb_per, act, glu;
    float acc_scale;
    const float *bias;
    float *y, *y_lo; int64_t ldy;
    float *part;
    int *err;
};

// eight columns each of two accumulators
__device__ __forceinline__ void tmem_ld8x2(uint32_t ta, uint32_t tb, uint32_t *a, uint32_t *b) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%16];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%17];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]), "=r"(a[4]), "=r"(a[5]), "=r"(a[6]), "=r"(a[7]),
                   "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]), "=r"(b[4]), "=r"(b[5]), "=r"(b[6]), "=r"(b[7])
                 : "r"(ta), "r"(tb) : "memory");
}
// silu through ex2.approx / rcp.approx, as in the fp16-pair engine's gated epilogue; the other activations as everywhere
__device__ __forceinline__ float fw_act(float v, int act) { return act == ACT_SILU ? __fdividef(v, 1.0f + __expf(-v)) : tc_act(v, act); }

template <int NT, bool W2>
__global__ void __launch_bounds__(FW_THREADS) k_gemm_few(const __grid_constant__ CUtensorMap tmW1, const __grid_constant__ CUtensorMap tmW2,
                                                            const __grid_constant__ CUtensorMap tmX1, const __grid_constant__ CUtensorMap tmX2, FewDev a) {
    constexpr int ST = fw_stages(NT, W2), STAGE = fw_stage(NT, W2), WB = FW_WTILE * (W2 ? 2 : 1), XT = fw_xtile(NT);
    constexpr int COLS = 2 * NT;                             // W1 x1 (+ W2 x1) in the first NT columns, W1 x2 in the rest
    extern __shared__ unsigned char fw_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)fw_raw + 1023) & ~(uintptr_t)1023);
    uint64_t *bars = (uint64_t *)(smem + ST * STAGE);
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 * ST + 1);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + ST), done = smem_u32(bars + 2 * ST);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * 128, kb0 = blockIdx.y * a.kb_per, nkb = min(a.num_kb - kb0, a.kb_per);
    const int m0 = blockIdx.z * NT, rows = min(a.M - m0, NT);                 // this CTA's tokens
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; s++) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // only now may the successor start: it allocates tensor memory of its own, which must not come between this CTA and its share
    pdl_launch_dependents();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            auto load_w = [&](int i) {
                const int s = i % ST;
                const uint32_t dst = smem_u32(smem + s * STAGE), bar = full0 + 8 * s;
                mbar_expect_tx(bar, STAGE);
                tma_load_2d(dst, &tmW1, (kb0 + i) * 64, n0, bar);
                if (W2) tma_load_2d(dst + FW_WTILE, &tmW2, (kb0 + i) * 64, n0, bar);
            };
            auto load_x = [&](int i) {
                const int s = i % ST;
                const uint32_t dst = smem_u32(smem + s * STAGE) + WB, bar = full0 + 8 * s;
                tma_load_2d(dst, &tmX1, (kb0 + i) * 64, m0, bar);
                tma_load_2d(dst + XT, &tmX2, (kb0 + i) * 64, m0, bar);
            };
            const int first = min(ST, nkb);
            for (int i = 0; i < first; i++) load_w(i);
            pdl_wait();
            for (int i = 0; i < first; i++) load_x(i);
            int armed = first;
            bool ok = true;
            for (int i = first; i < nkb; i++) {
                ok = mbar_wait(empty0 + 8 * (i % ST), (uint32_t)((i / ST) & 1) ^ 1u, a.err, 51);
                if (!ok) break;
                load_w(i);
                load_x(i);
                armed = i + 1;
            }
            if (!ok)
                for (int k = armed - ST < 0 ? 0 : armed - ST; k < armed; k++) mbar_wait(full0 + 8 * (k % ST), (uint32_t)((k / ST) & 1), a.err, 52);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // x1 and x2 are one operand of 2 NT rows: W1 is fetched once for both products (short MMAs are paced by the fetch of
            // their 128-row operand, not by their columns)
            constexpr uint32_t idesc = umma_idesc_f16(128, NT), idesc2 = umma_idesc_f16(128, 2 * NT);
            for (int i = 0; i < nkb; i++) {
                const int s = i % ST;
                if (!mbar_wait(full0 + 8 * s, (uint32_t)((i / ST) & 1), a.err, 53)) break;
                tc_fence_after();
                const uint32_t base = smem_u32(smem + s * STAGE);
                const uint64_t w1 = umma_desc_sw128(base), w2 = umma_desc_sw128(base + FW_WTILE);
                const uint64_t x = umma_desc_sw128(base + WB);
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const uint64_t o = (uint64_t)(k * 2);
                    umma_f16(tmem, w1 + o, x + o, idesc2, (i | k) ? 1u : 0u);
                    if (W2) umma_f16(tmem, w2 + o, x + o, idesc, 1u);
                }
                umma_commit(empty0 + 8 * s);
            }
            umma_commit(done);
        }
    } else {
        const int q = warp & 3, t_half = (warp - 2) >> 2;    // two warps share a quadrant's columns, eight tokens at a time
        const int n = n0 + q * 32 + lane;                    // this thread's weight row = output column
        const float b = (a.bias && n < a.N) ? a.bias[n] : 0.f;
        pdl_wait();                                          // earlier readers of y / part have finished
        const bool ok = mbar_wait(done, 0, a.err, 54);
        tc_fence_after();
        const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16);
        for (int t0 = t_half * 8; ok && t0 < rows; t0 += 16) {
            uint32_t r[8], r2[8];
            tmem_ld8x2(trow + (uint32_t)t0, trow + (uint32_t)(NT + t0), r, r2);
            float v[8];
#pragma unroll
            for (int t = 0; t < 8; t++) v[t] = (__uint_as_float(r[t]) + __uint_as_float(r2[t])) * a.acc_scale + b;
            if (a.part) {
                float *p = a.part + ((int64_t)blockIdx.y * a.M + m0 + t0) * a.N + n;
#pragma unroll
                for (int t = 0; t < 8; t++)
                    if (t0 + t < rows && n < a.N) p[(int64_t)t * a.N] = v[t];
            } else if (a.glu) {
                // even lanes hold a unit's gate, odd lanes its up row: the pair exchanges so that each has both of one of two tokens
                const bool odd = lane & 1;
                const int64_t at = (int64_t)(m0 + t0 + (odd ? 1 : 0)) * a.ldy + (n >> 1);
#pragma unroll
                for (int t = 0; t < 8; t += 2) {
                    const float got = __shfl_xor_sync(0xffffffffu, odd ? v[t] : v[t + 1], 1);
                    const float o = __fmul_rn(fw_act(odd ? got : v[t], a.act), odd ? v[t + 1] : got);
                    if (t0 + t + (odd ? 1 : 0) < rows && n < a.N) {
                        if (a.y_lo) store_split1(a.y, a.y_lo, at + t * a.ldy, o, SPLIT_H16);
                        else a.y[at + t * a.ldy] = o;
                    }
                }
            } else {
                const int64_t at = (int64_t)(m0 + t0) * a.ldy + n;
#pragma unroll
                for (int t = 0; t < 8; t++)
                    if (t0 + t < rows && n < a.N) {
                        const float o = fw_act(v[t], a.act);
                        if (a.y_lo) store_split1(a.y, a.y_lo, at + t * a.ldy, o, SPLIT_H16);
                        else a.y[at + t * a.ldy] = o;
                    }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS) : "memory");
    }
}

// ---- 2 to 16 rows: the same products in fp32 ----
// A CTA takes 64 weight rows (32 from nine tokens on: the sums of 64 would leave an SM room for one CTA) and a slice of K. The
// weights come by TMA in chunks of 128 bytes a row (32 floats or 64 bf16 values) with the rows of x that go with them; each of eight warps
// takes 16 bytes of every row of a chunk. A lane of it holds a block of rows x tokens (2 x 2, 2 x 4 or 4 x 4), so that a 16-byte read of
// shared memory feeds enough multiply-adds, free of bank conflicts (128-byte swizzle) or as a broadcast; they are issued two at a time
// (even and odd positions of K). Sums run over at most 16 products each, then in pairs over the warps and in order over the slices.
//
// Bound by issue: at 16 tokens and bf16 weights a chunk takes 64 two-wide multiply-adds, 12 shared-memory reads and 32 conversions a warp,
// and moves of registers besides (4 to 7% fewer with the compiler's own two-wide multiply-add than with inline PTX). A step of the Qwen2
// shape in bf16 with 2 / 4 / 8 / 16 rows takes 0.62 / 0.73 / 0.95 / 1.28 ms (on fp16 pairs 0.70 / 0.71 / 0.73 / 0.74, on the GEMV kernels
// 1.05 / 1.55 / 2.87 / 4.66), of the GPT-2 shape in fp32 0.30 / 0.33 / 0.40 / 0.47 (0.34 / 0.35 / 0.36 / 0.35; 0.43 / 0.64 / 0.91 / 1.59).
// Error of a step's logits against 64 bits: that of the GEMV kernels or less (2.9e-7 relative for GPT-2, 5.2e-7 for Qwen2; pairs
// 2.2e-6 and more).
constexpr int FF_WARPS = 8, FF_ST = 8, FF_RUN = 32, FF_THREADS = FF_WARPS * 32 + 32;
constexpr int ff_tile(int MT) { return MT > 8 ? 32 : 64; }
constexpr int ff_tgroups(int MT) { return MT > 8 ? 4 : (MT > 4 ? 2 : 1); }       // groups of tokens a warp's lanes are dealt to
constexpr int ff_wt(int MT) { return ff_tile(MT) * 128; }
constexpr int ff_xtile(int MT) { return MT * 128 < 1024 ? 1024 : MT * 128; }
constexpr int ff_stage(int MT, bool W16) { return ff_wt(MT) + (W16 ? 2 : 1) * ff_xtile(MT); }
constexpr size_t ff_smem(int MT, bool W16) { return 1024 + (size_t)FF_ST * ff_stage(MT, W16) + 2 * FF_ST * 8; }
struct FewF32Dev {
    int M, N, K, k_per, act, glu;            // glu: rows n and N / 2 + n of W are a unit's gate and up row
    const float *bias;
    float *y; int64_t ldy;
    float *part;
    int *err;
};

template <int MT, bool W16>
__global__ void __launch_bounds__(FF_THREADS, 2) k_few_f32(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, FewF32Dev a) {
    constexpr int KC = W16 ? 64 : 32, XN = W16 ? 2 : 1, TILE = ff_tile(MT), WT = ff_wt(MT), XT = ff_xtile(MT), STAGE = ff_stage(MT, W16);
    constexpr int TG = ff_tgroups(MT), TL = MT / TG, RG = 32 / TG, RL = TILE / RG;       // a lane: RL weight rows x TL tokens
    constexpr int XO = TL < 8 / TG ? TL : 8 / TG;                                        // the swizzle repeats after eight tokens
    static_assert(FF_WARPS * MT * TILE * 4 <= FF_ST * STAGE, "the warps' sums are exchanged in the ring");
    static_assert(RG % 8 == 0 && (FF_ST & (FF_ST - 1)) == 0, "");
    extern __shared__ unsigned char fw_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)fw_raw + 1023) & ~(uintptr_t)1023);
    uint64_t *bars = (uint64_t *)(smem + FF_ST * STAGE);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + FF_ST);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int k0 = blockIdx.y * a.k_per, nst = (min(a.K - k0, a.k_per) + KC - 1) / KC;
    const int r0 = blockIdx.x * (a.glu ? TILE / 2 : TILE), r1 = (a.glu ? a.N >> 1 : TILE / 2) + r0;      // the tile's two runs of weight rows
    if (tid == 0) {
        for (int s = 0; s < FF_ST; s++) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, FF_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_launch_dependents();

    if (warp == FF_WARPS) {
        if (lane == 0) {
            auto load_w = [&](int i) {
                const int s = i % FF_ST;
                const uint32_t dst = smem_u32(smem + s * STAGE), bar = full0 + 8 * s;
                mbar_expect_tx(bar, WT + XN * MT * 128);
                tma_load_2d(dst, &tmW, k0 + i * KC, r0, bar);
                tma_load_2d(dst + WT / 2, &tmW, k0 + i * KC, r1, bar);
            };
            auto load_x = [&](int i) {
                const int s = i % FF_ST;
                const uint32_t dst = smem_u32(smem + s * STAGE) + WT, bar = full0 + 8 * s;
#pragma unroll
                for (int h = 0; h < XN; h++) tma_load_2d(dst + h * XT, &tmX, k0 + i * KC + h * 32, 0, bar);
            };
            const int first = min(FF_ST, nst);
            for (int i = 0; i < first; i++) load_w(i);
            pdl_wait();
            for (int i = 0; i < first; i++) load_x(i);
            int armed = first;
            for (; armed < nst; armed++) {
                if (!mbar_wait(empty0 + 8 * (armed % FF_ST), (uint32_t)((armed / FF_ST) & 1) ^ 1u, a.err, 56)) break;
                load_w(armed);
                load_x(armed);
            }
            for (int k = armed - FF_ST < 0 ? 0 : armed - FF_ST; k < armed; k++)        // every copy has landed before the CTA may end
                mbar_wait(full0 + 8 * (k % FF_ST), (uint32_t)((k / FF_ST) & 1), a.err, 57);
        }
        return;
    }
    const int rg = lane & (RG - 1), tg = lane / RG;
    float2 acc[RL][TL];                                    // two sums: over even and over odd positions of K
    float sum[RL][TL];
#pragma unroll
    for (int r = 0; r < RL; r++)
#pragma unroll
        for (int t = 0; t < TL; t++) { acc[r][t] = make_float2(0.f, 0.f); sum[r][t] = 0.f; }
    auto put_aside = [&] {
#pragma unroll
        for (int r = 0; r < RL; r++)
#pragma unroll
            for (int t = 0; t < TL; t++) { sum[r][t] += acc[r][t].x + acc[r][t].y; acc[r][t] = make_float2(0.f, 0.f); }
    };
    bool ok = true;
    const unsigned char *wl = smem + rg * 128 + ((warp ^ (rg & 7)) << 4);        // (row rg + RG r has the same place in its swizzle group)
    const unsigned char *xl = smem + WT + (W16 ? (warp >> 2) * XT : 0) + tg * 128;
    int xo[XO][XN];                                          // this warp's 16-byte pieces of the tokens' rows
#pragma unroll
    for (int t = 0; t < XO; t++)
#pragma unroll
        for (int h = 0; h < XN; h++) xo[t][h] = TG * t * 128 + (((W16 ? (warp & 3) * 2 + h : warp) ^ ((tg + TG * t) & 7)) << 4);
    for (int i = 0; i < nst; i++) {
        const int s = i & (FF_ST - 1);
        ok = mbar_wait(full0 + 8 * s, (uint32_t)((i / FF_ST) & 1), a.err, 58);
        if (!ok) break;
        uint4 w[RL];                                         // 16 bytes of row rg + RG r
#pragma unroll
        for (int r = 0; r < RL; r++) w[r] = *(const uint4 *)(wl + s * STAGE + RG * r * 128);
#pragma unroll
        for (int h = 0; h < XN; h++) {                       // four positions of K
            float4 x[TL];
#pragma unroll
            for (int t = 0; t < TL; t++) x[t] = *(const float4 *)(xl + s * STAGE + xo[t % XO][h] + TG * (t / XO * XO) * 128);
#pragma unroll
            for (int r = 0; r < RL; r++) {
                float2 w0, w1;
                if (W16) {
                    const uint32_t u0 = h ? w[r].z : w[r].x, u1 = h ? w[r].w : w[r].y;
                    w0 = make_float2(__uint_as_float(u0 << 16), __uint_as_float(u0 & 0xffff0000u)); w1 = make_float2(__uint_as_float(u1 << 16), __uint_as_float(u1 & 0xffff0000u));
                } else { w0 = make_float2(__uint_as_float(w[r].x), __uint_as_float(w[r].y)); w1 = make_float2(__uint_as_float(w[r].z), __uint_as_float(w[r].w)); }
#pragma unroll
                for (int t = 0; t < TL; t++) { acc[r][t] = __ffma2_rn(w0, make_float2(x[t].x, x[t].y), acc[r][t]); acc[r][t] = __ffma2_rn(w1, make_float2(x[t].z, x[t].w), acc[r][t]); }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty0 + 8 * s);
        if ((i + 1) % (FF_RUN / (KC / FF_WARPS)) == 0) put_aside();
    }
    put_aside();
    auto bar_warps = [] { asm volatile("bar.sync 1, %0;" ::"n"(FF_WARPS * 32) : "memory"); };
    bar_warps();                                             // every chunk has been read: the ring is free
    float *red = (float *)smem;                              // [warp][token][TILE]
#pragma unroll
    for (int r = 0; r < RL; r++)
#pragma unroll
        for (int t = 0; t < TL; t++) red[(warp * MT + tg + TG * t) * TILE + rg + RG * r] = sum[r][t];
    pdl_wait();                                              // earlier readers of y / part have finished
    bar_warps();
    if (!ok) return;
    auto total = [&](int t, int r) {
        float v[FF_WARPS];
#pragma unroll
        for (int w = 0; w < FF_WARPS; w++) v[w] = red[(w * MT + t) * TILE + r];
        return ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
    };
    if (a.glu) {
        constexpr int UT = TILE / 2;
        const int u = r0 + tid % UT, half = a.N >> 1;        // a unit: gate row u, up row half + u
        const float bg = a.bias && u < half ? a.bias[u] : 0.f, bu = a.bias && u < half ? a.bias[half + u] : 0.f;
        if (u < half)
            for (int t = tid / UT; t < a.M; t += FF_WARPS * 32 / UT) {
                const float g = total(t, tid % UT), p = total(t, UT + tid % UT);
                if (a.part) *(float2 *)(a.part + ((int64_t)blockIdx.y * a.M + t) * a.N + 2 * u) = make_float2(g, p);
                else a.y[t * a.ldy + u] = __fmul_rn(tc_act(g + bg, a.act), p + bu);
            }
    } else {
        const int n = r0 + tid % TILE;
        const float b = a.bias && n < a.N ? a.bias[n] : 0.f;
        if (n < a.N)
            for (int t = tid / TILE; t < a.M; t += FF_WARPS * 32 / TILE) {
                const float v = total(t, tid % TILE);
                if (a.part) a.part[((int64_t)blockIdx.y * a.M + t) * a.N + n] = v;
                else a.y[t * a.ldy + n] = tc_act(v + b, a.act);
            }
    }
}

// ---- what follows a sliced product in a block ----
// t[0] = t[0] + ... + t[N - 1], in pairs: the error grows with the logarithm of their number
template <int N>
__device__ __forceinline__ void add_pairs(float4 (&t)[N]) {
#pragma unroll
    for (int w = 1; w < N; w *= 2)
#pragma unroll
        for (int u = 0; u + w < N; u += 2 * w) { t[u].x += t[u + w].x; t[u].y += t[u + w].y; t[u].z += t[u + w].z; t[u].w += t[u + w].w; }
}
// One CTA per row: the slices' sums, bias and residual, then the norm of the row as an fp16 pair (y2 null: in fp32) for the next product.
// The row stays in registers between the two (C up to 4096).
constexpr int FR_T = 256, FR_V = 4, FR_IN = 12;
__global__ void __launch_bounds__(FR_T) k_few_reduce_norm(float *__restrict__ x, const float *__restrict__ part, int S, const float *__restrict__ bias, int rows, int C,
                                                         int ln_kind, const float *__restrict__ ln_w, const float *__restrict__ ln_b, float eps,
                                                         unsigned short *__restrict__ y1, unsigned short *__restrict__ y2) {
    __shared__ float red[2][FR_T / 32];
    const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, c4n = C >> 2;
    // the successor may start only once everything before this kernel is complete: attention reads the cache and the step
    // counter before it waits for the product that follows here
    // (the norm's gains and the bias are weights: requested before the wait)
    float4 w4[FR_V], b4[FR_V], bias4[FR_V];
#pragma unroll
    for (int i = 0; i < FR_V; i++) {
        const int c = (tid + i * FR_T) * 4;
        const bool on = tid + i * FR_T < c4n;
        w4[i] = on && ln_w ? __ldg((const float4 *)(ln_w + c)) : make_float4(1.f, 1.f, 1.f, 1.f);
        b4[i] = on && ln_b ? __ldg((const float4 *)(ln_b + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
        bias4[i] = on && bias ? __ldg((const float4 *)(bias + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    pdl_wait();
    pdl_launch_dependents();
    float4 v[FR_V];
#pragma unroll
    for (int i = 0; i < FR_V; i++) {
        v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        const int c = tid + i * FR_T;
        if (c >= c4n) continue;
        const float4 r = *(const float4 *)(x + (int64_t)row * C + c * 4);
        if (S > 0) {
            const float *p = part + (int64_t)row * C + c * 4;
            const int64_t step = (int64_t)rows * C;
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int s = 0; s < S; s += FR_IN) {                     // FR_IN slices in flight, added in pairs
                float4 t[FR_IN];
#pragma unroll
                for (int u = 0; u < FR_IN; u++) t[u] = s + u < S ? __ldcg((const float4 *)(p + (s + u) * step)) : make_float4(0.f, 0.f, 0.f, 0.f);
                add_pairs<FR_IN>(t);
                a.x += t[0].x; a.y += t[0].y; a.z += t[0].z; a.w += t[0].w;
            }
            a.x += bias4[i].x; a.y += bias4[i].y; a.z += bias4[i].z; a.w += bias4[i].w;
            v[i] = make_float4(a.x + r.x, a.y + r.y, a.z + r.z, a.w + r.w);
            *(float4 *)(x + (int64_t)row * C + c * 4) = v[i];
        } else v[i] = r;
    }
    if (!ln_kind) return;
    auto block_sum = [&](float s, int k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) red[k][warp] = s;
        __syncthreads();
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < FR_T / 32; w++) t += red[k][w];
        return t;
    };
    float mean = 0.f;
    if (ln_kind == 1) {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < FR_V; i++) s += (v[i].x + v[i].y) + (v[i].z + v[i].w);
        mean = block_sum(s, 0) / (float)C;
    }
    float q = 0.f;
#pragma unroll
    for (int i = 0; i < FR_V; i++)
        if (tid + i * FR_T < c4n) {
            const float d0 = v[i].x - mean, d1 = v[i].y - mean, d2 = v[i].z - mean, d3 = v[i].w - mean;
            q += (d0 * d0 + d1 * d1) + (d2 * d2 + d3 * d3);
        }
    const float inv = 1.0f / sqrtf(block_sum(q, 1) / (float)C + eps);
#pragma unroll
    for (int i = 0; i < FR_V; i++) {
        const int c = (tid + i * FR_T) * 4;
        if (tid + i * FR_T >= c4n) continue;
        const float4 w = w4[i], b = b4[i];
        const float4 o = make_float4(__fadd_rn(__fmul_rn(__fmul_rn(v[i].x - mean, inv), w.x), b.x), __fadd_rn(__fmul_rn(__fmul_rn(v[i].y - mean, inv), w.y), b.y),
                                     __fadd_rn(__fmul_rn(__fmul_rn(v[i].z - mean, inv), w.z), b.z), __fadd_rn(__fmul_rn(__fmul_rn(v[i].w - mean, inv), w.w), b.w));
        if (y2) store_split4((float *)y1, (float *)y2, (int64_t)row * C + c, o, SPLIT_H16);
        else *(float4 *)((float *)y1 + (int64_t)row * C + c) = o;
    }
}

// The sums of an up-projection that was cut into slices, through bias and activation to an fp16 pair (y2 null: to fp32); glu: columns
// are interleaved gate / up pairs and the result has N / 2 of them. Four columns per thread.
__global__ void __launch_bounds__(256) k_few_reduce_act(const float *__restrict__ part, int S, int64_t rows, int N, const float *__restrict__ bias, int act, int glu,
                                                       unsigned short *__restrict__ y1, unsigned short *__restrict__ y2) {
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    const int n4 = N >> 2;
    if (i >= rows * n4) return;
    const int64_t row = i / n4; const int c = (int)(i - row * n4) * 4;
    const float *p = part + row * N + c;
    const int64_t step = rows * N;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = 0; s < S; s += 8) {
        float4 t[8];
#pragma unroll
        for (int u = 0; u < 8; u++) t[u] = s + u < S ? __ldcg((const float4 *)(p + (s + u) * step)) : make_float4(0.f, 0.f, 0.f, 0.f);
        add_pairs<8>(t);
        a.x += t[0].x; a.y += t[0].y; a.z += t[0].z; a.w += t[0].w;
    }
    if (bias) { const float4 b = __ldg((const float4 *)(bias + c)); a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }
    if (!y2) {
        float *y = (float *)y1;
        if (glu) *(float2 *)(y + row * (N / 2) + c / 2) = make_float2(__fmul_rn(tc_act(a.x, act), a.y), __fmul_rn(tc_act(a.z, act), a.w));
        else *(float4 *)(y + row * N + c) = make_float4(tc_act(a.x, act), tc_act(a.y, act), tc_act(a.z, act), tc_act(a.w, act));
    } else if (glu) {
        uint32_t hi, lo;
        h16_pair2(__fmul_rn(fw_act(a.x, act), a.y), __fmul_rn(fw_act(a.z, act), a.w), hi, lo);
        *(uint32_t *)(y1 + row * (N / 2) + c / 2) = hi;
        *(uint32_t *)(y2 + row * (N / 2) + c / 2) = lo;
    } else {
        store_split4((float *)y1, (float *)y2, row * N + c, make_float4(fw_act(a.x, act), fw_act(a.y, act), fw_act(a.z, act), fw_act(a.w, act)), SPLIT_H16);
    }
}

// One thread per pair (d, d + hd / 2) of a head of a row: slice sums and bias, rotation of query / key heads, q to its buffer,
// k | v to the buffer and / or the cache.
__global__ void __launch_bounds__(256) k_few_reduce_qkv(FewQkv a) {
    const int half = a.hd >> 1, heads = a.H + 2 * a.Hkv, row = blockIdx.x;
    const int i = blockIdx.y * 256 + threadIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    if (i >= heads * half) return;
    const int h = i / half, d = i - h * half, Wq = heads * a.hd;
    const float *p = a.part + (int64_t)row * Wq + h * a.hd + d;
    const int64_t step = (int64_t)a.rows * Wq;
    float v0 = 0.f, v1 = 0.f;
    int s = 0;
    for (; s + 4 <= a.S; s += 4) {
        float t0[4], t1[4];
#pragma unroll
        for (int u = 0; u < 4; u++) { t0[u] = __ldcg(p + (s + u) * step); t1[u] = __ldcg(p + (s + u) * step + half); }
#pragma unroll
        for (int u = 0; u < 4; u++) { v0 += t0[u]; v1 += t1[u]; }
    }
    for (; s < a.S; s++) { v0 += __ldcg(p + s * step); v1 += __ldcg(p + s * step + half); }
    if (a.bias) { v0 += __ldg(a.bias + h * a.hd + d); v1 += __ldg(a.bias + h * a.hd + d + half); }
    const int64_t st = a.step_d ? (int64_t)*a.step_d : 0;
    if (a.cos_t && h < a.H + a.Hkv) {
        const int64_t at = (int64_t)a.pos[st * a.pos_step + row] * a.hd + d;
        const float y0 = __fadd_rn(__fmul_rn(v0, a.cos_t[at]), __fmul_rn(-v1, a.sin_t[at]));
        const float y1 = __fadd_rn(__fmul_rn(v1, a.cos_t[at + half]), __fmul_rn(v0, a.sin_t[at + half]));
        v0 = y0; v1 = y1;
    }
    if (h < a.H || a.kv_self) { float *q = a.q + (int64_t)row * a.ldq + h * a.hd + d; q[0] = v0; q[half] = v1; }
    if (h >= a.H && a.kv) {
        const int rps = a.rps > 0 ? a.rps : 1;
        float *k = a.kv + (int64_t)(row / rps) * a.seq_pitch + (int64_t)(row % rps) * a.pitch + st * a.step + (h - a.H) * a.hd + d;
        k[0] = v0; k[half] = v1;
    }
}

// ---- host side ----
bool gemm_few_supported(int64_t M, int N, int K, const void *W) {
    return ctx().gemm_mode >= 3 && M >= 2 && M <= FEW_MAX_ROWS && N >= 32 && K >= 32 && (K & 7) == 0 && (M > FEW_F32_ROWS || ((uintptr_t)W & 15) == 0);
}
static int few_tile(int M) { return M <= FEW_F32_ROWS ? ff_tile(M) : 128; }      // weight rows of a CTA
// Slices of K: as many as give every SM one CTA (two of the fp32 kernel's), each at least two 64-wide steps; a slice more costs another read of the rows in
// the kernel that adds them, so a long row count takes fewer.
int gemm_few_slices(int M, int N, int K, int max_slices) {
    const int tiles = (int)(cdiv(N, few_tile(M)) * cdiv(M, 128)), nkb = (int)cdiv(K, 64);
    int s = std::max(1, (M <= FEW_F32_ROWS ? 2 : 1) * ctx().sm_count / tiles);
    s = std::min(std::min(s, std::max(1, nkb / 2)), max_slices);
    const int kb_per = (int)cdiv(nkb, s);
    return (int)cdiv(nkb, kb_per);
}

template <int NT, bool W2>
static void launch_few(const FewGemm &g, const FewDev &d, const H3Weights &w, int slices) {
    static bool set = false;
    if (!set) { CUDA_CHECK(cudaFuncSetAttribute((k_gemm_few<NT, W2>), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fw_smem(NT, W2))); set = true; }
    const CUtensorMap mw1 = tc_get_map_h16(w.v1, g.N, g.K, g.K, 128), mw2 = tc_get_map_h16(w.v2, g.N, g.K, g.K, 128);
    const CUtensorMap mx1 = tc_get_map_h16(g.x1, g.M, g.K, g.ldx, NT), mx2 = tc_get_map_h16(g.x2, g.M, g.K, g.ldx, NT);
    LAUNCH_PDL((k_gemm_few<NT, W2>), dim3((unsigned)cdiv(g.N, 128), (unsigned)slices, (unsigned)cdiv(g.M, NT)), FW_THREADS, fw_smem(NT, W2), mw1, mw2, mx1, mx2, d);
}

template <int MT, bool W16>
static void launch_f32(const FewGemm &g, const FewF32Dev &d, int slices) {
    static bool set = false;
    if (!set) { CUDA_CHECK(cudaFuncSetAttribute((k_few_f32<MT, W16>), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ff_smem(MT, W16))); set = true; }
    const CUtensorMap mw = W16 ? tc_get_map_h16(g.W16, g.N, g.K, g.K, ff_tile(MT) / 2) : tc_get_map(g.W, g.N, g.K, g.K, ff_tile(MT) / 2, false);
    const CUtensorMap mx = tc_get_map((const float *)g.x1, g.M, g.K, g.ldx, MT, false);
    const int64_t tiles = g.glu ? cdiv(g.N / 2, ff_tile(MT) / 2) : cdiv(g.N, ff_tile(MT));
    LAUNCH_PDL((k_few_f32<MT, W16>), dim3((unsigned)tiles, (unsigned)slices), FF_THREADS, ff_smem(MT, W16), mw, mx, d);
}
static void gemm_few_f32(const FewGemm &g) {
    FewF32Dev d{};
    const int slices = g.part ? gemm_few_slices(g.M, g.N, g.K, g.max_slices) : 1;
    d.M = g.M; d.N = g.N; d.K = g.K; d.k_per = (int)cdiv(cdiv(g.K, 64), slices) * 64; d.act = g.act; d.glu = g.glu;
    d.bias = g.part ? nullptr : g.bias; d.y = g.y; d.ldy = g.ldy; d.part = g.part; d.err = tc_err_flag();
    ProfScope ps(NCMB_K_GEMM, 2.0 * (double)g.M * g.N * g.K, (g.W16 ? 2.0 : 4.0) * (double)g.N * g.K);
#define FF_CASE(MT_) do { if (g.W16) launch_f32<MT_, true>(g, d, slices); else launch_f32<MT_, false>(g, d, slices); } while (0)
    if (g.M <= 2) FF_CASE(2);
    else if (g.M <= 4) FF_CASE(4);
    else if (g.M <= 8) FF_CASE(8);
    else FF_CASE(16);
#undef FF_CASE
}

void gemm_few(const FewGemm &g) {
    if (g.M <= FEW_F32_ROWS) { gemm_few_f32(g); return; }
    const H3Weights w = gemm_h3_weights(g.W, (int64_t)g.N * g.K);
    FewDev d{};
    const int nkb = (int)cdiv(g.K, 64);
    const int slices = g.part ? gemm_few_slices(g.M, g.N, g.K, g.max_slices) : 1;
    d.M = g.M; d.N = g.N; d.num_kb = nkb; d.kb_per = (int)cdiv(nkb, slices); d.act = g.act; d.glu = g.glu;
    d.acc_scale = H16_X_UNSCALE / w.scale;
    d.bias = g.part ? nullptr : g.bias; d.y = g.y; d.y_lo = g.y_lo; d.ldy = g.ldy; d.part = g.part; d.err = tc_err_flag();
    ProfScope ps(NCMB_K_GEMM, 2.0 * (double)g.M * g.N * g.K, (w.v2_zero ? 2.0 : 4.0) * (double)g.N * g.K);
#define FEW_CASE(NT_) do { if (w.v2_zero) launch_few<NT_, false>(g, d, w, slices); else launch_few<NT_, true>(g, d, w, slices); } while (0)
    if (g.M <= 32) FEW_CASE(32);
    else if (g.M <= 64) FEW_CASE(64);
    else FEW_CASE(128);
#undef FEW_CASE
}

void few_head(const void *x1, const void *x2, int rows, const float *W, const unsigned short *W16, const float *bias, int N, int K, float *y) {
    if (rows <= 64) {
        FewGemm g{x1, x2, K, W, rows, N, K};
        g.W16 = W16; g.bias = bias; g.y = y; g.ldy = N;
        gemm_few(g);
        return;
    }
    GemmArgs g;
    g.x = (const float *)x1; g.x_lo = (const float *)x2; g.x_fmt = SPLIT_H16; g.ldx = K; g.W = W; g.bias = bias; g.y = y; g.ldy = N; g.M = rows; g.N = N; g.K = K;
    gemm(g);
}
void few_reduce_norm(float *x, const float *part, int S, const float *bias, int rows, int C, int ln_kind, const float *ln_w, const float *ln_b,
                     float eps, void *y1, void *y2) {
    if (C % 4 || C > FR_T * FR_V * 4) fatal("few_reduce_norm: width %d", C);
    ProfScope ps(NCMB_K_NORM, 0, (double)rows * C * 4 * (S + 3));
    LAUNCH_PDL(k_few_reduce_norm, (unsigned)rows, FR_T, 0, x, part, S, bias, rows, C, ln_kind, ln_w, ln_b, eps, (unsigned short *)y1, (unsigned short *)y2);
}
int few_up_slices(int M, int N, int K, int max_slices) {
    const int64_t tiles = cdiv(N, few_tile(M)) * cdiv(M, 128);
    return tiles * 3 > ctx().sm_count || N % 8 ? 1 : gemm_few_slices(M, N, K, max_slices);
}
void few_reduce_act(const float *part, int S, int rows, int N, const float *bias, int act, int glu, void *y1, void *y2) {
    const int64_t n = (int64_t)rows * (N / 4);
    ProfScope ps(NCMB_K_ELEM, 0, (double)rows * N * 4 * (S + 1));
    LAUNCH_PDL(k_few_reduce_act, grid1d(n, 256), 256, 0, part, S, (int64_t)rows, N, bias, act, glu, (unsigned short *)y1, (unsigned short *)y2);
}
void few_reduce_qkv(const FewQkv &a) {
    const int items = (a.H + 2 * a.Hkv) * a.hd / 2;
    ProfScope ps(NCMB_K_ELEM, 0, (double)a.rows * items * 8 * (a.S + 1));
    LAUNCH_PDL(k_few_reduce_qkv, dim3((unsigned)a.rows, (unsigned)cdiv(items, 256)), 256, 0, a);
}

} // namespace ncmb
