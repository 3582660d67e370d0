// Products of a weight matrix with 2 to 640 rows, and what stands between them in a block.
//
// A decode step of a batch (and the first levels of a generate) multiplies every weight matrix with few rows, so it is bound
// by streaming the weights. The fp16-pair engine (gemm_h3.cu) makes the rows of x the 128-row side of its tiles: with 27 rows
// most of every x tile is padding that still passes through shared memory, and N = 896 gives 28 CTAs. Here the weights are the
// 128-row side: a CTA takes 128 weight rows and a slice of K, its tokens are the columns of the MMA (16 to 128; more rows take a second
// CTA), and nothing is
// read twice but the small x. Raw sums of the K slices go to a partial buffer and the kernel that follows in the block adds
// them while it does its own work: rotation and cache write after QKV, residual and the next norm after the other two.
//
// The products are those of the fp16-pair engine: x1 W1 + x2 W1 (+ x1 W2 where the second halves are not all zero), one fp32
// accumulator. Weights are requested before the kernel waits for its predecessor (nothing in a step writes them).
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

// ---- what follows a sliced product in a block ----
// One CTA per row: the slices' sums, bias and residual, then the norm of the row as an fp16 pair for the next product. The row
// stays in registers between the two (C up to 4096).
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
            int s = 0;
            for (; s < S; s += FR_IN) {                          // FR_IN slices in flight (absent ones are not added)
                float4 t[FR_IN];
#pragma unroll
                for (int u = 0; u < FR_IN; u++)
                    if (s + u < S) t[u] = __ldcg((const float4 *)(p + (s + u) * step));
#pragma unroll
                for (int u = 0; u < FR_IN; u++)
                    if (s + u < S) { a.x += t[u].x; a.y += t[u].y; a.z += t[u].z; a.w += t[u].w; }
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
        store_split4((float *)y1, (float *)y2, (int64_t)row * C + c, o, SPLIT_H16);
    }
}

// The sums of an up-projection that was cut into slices, through bias and activation to an fp16 pair; glu: columns are
// interleaved gate / up pairs and the result has N / 2 of them. Four columns per thread.
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
        for (int u = 0; u < 8; u++)
            if (s + u < S) t[u] = __ldcg((const float4 *)(p + (s + u) * step));
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (s + u < S) { a.x += t[u].x; a.y += t[u].y; a.z += t[u].z; a.w += t[u].w; }
    }
    if (bias) { const float4 b = __ldg((const float4 *)(bias + c)); a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }
    if (glu) {
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
bool gemm_few_supported(int64_t M, int N, int K) {
    return ctx().gemm_mode >= 3 && M >= 2 && M <= FEW_MAX_ROWS && N >= 32 && K >= 32 && (K & 7) == 0;
}
// Slices of K: as many as give every SM one CTA, each at least two 64-wide steps; a slice more costs another read of the rows in
// the kernel that adds them, so a long row count takes fewer.
int gemm_few_slices(int M, int N, int K, int max_slices) {
    const int tiles = (int)(cdiv(N, 128) * cdiv(M, 128)), nkb = (int)cdiv(K, 64);
    int s = std::max(1, ctx().sm_count / tiles);
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

void gemm_few(const FewGemm &g) {
    const H3Weights w = gemm_h3_weights(g.W, (int64_t)g.N * g.K);
    FewDev d{};
    const int nkb = (int)cdiv(g.K, 64);
    const int slices = g.part ? gemm_few_slices(g.M, g.N, g.K, g.max_slices) : 1;
    d.M = g.M; d.N = g.N; d.num_kb = nkb; d.kb_per = (int)cdiv(nkb, slices); d.act = g.act; d.glu = g.glu;
    d.acc_scale = H16_X_UNSCALE / w.scale;
    d.bias = g.part ? nullptr : g.bias; d.y = g.y; d.y_lo = g.y_lo; d.ldy = g.ldy; d.part = g.part; d.err = tc_err_flag();
    ProfScope ps(NCMB_K_GEMM, 2.0 * (double)g.M * g.N * g.K, (w.v2_zero ? 2.0 : 4.0) * (double)g.N * g.K);
#define FEW_CASE(NT_) do { if (w.v2_zero) launch_few<NT_, false>(g, d, w, slices); else launch_few<NT_, true>(g, d, w, slices); } while (0)
    if (g.M <= 16) FEW_CASE(16);
    else if (g.M <= 32) FEW_CASE(32);
    else if (g.M <= 64) FEW_CASE(64);
    else FEW_CASE(128);
#undef FEW_CASE
}

void few_head(const void *x1, const void *x2, int rows, const float *W, const float *bias, int N, int K, float *y) {
    if (rows <= 64) {
        FewGemm g{x1, x2, K, W, rows, N, K};
        g.bias = bias; g.y = y; g.ldy = N;
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
    const int64_t tiles = cdiv(N, 128) * cdiv(M, 128);
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
