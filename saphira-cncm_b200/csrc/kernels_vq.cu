// Small strided kernels behind the quantizer's resampling path: conv1d /
// conv-transpose1d / GroupNorm / area and linear resampling. Every kernel takes
// explicit (batch, channel, time) strides, so the same code serves the reference
// kernel API's channel-major [N][C][T] tensors (src/ncm.h:172-180) and the
// token-major [N][T][C] tensors the generate path keeps (no transposes on the path).
#include "common.cuh"

#include <algorithm>

namespace ncmb {

// mode 0: y = conv; 1: y = add + conv; 2: y = (1-r)*add + r*conv (r = alpha), add read with y's strides
__global__ void k_conv1d(const float *__restrict__ x, NCT xs, const float *__restrict__ W,
                         const float *__restrict__ b, float *__restrict__ y, NCT ys,
                         int N, int Cin, int Cout, int T, int Tout, int K, int stride, int pad,
                         const float *__restrict__ add, float alpha, int mode) {
    int64_t total = (int64_t)N * Cout * Tout;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        int co = (int)(i % Cout); int t = (int)((i / Cout) % Tout); int n = (int)(i / ((int64_t)Cout * Tout));
        float acc = b ? b[co] : 0.f;
        const float *wr = W + (int64_t)co * Cin * K;
        for (int ci = 0; ci < Cin; ci++) {
            const float *xc = x + n * xs.sn + ci * xs.sc;
            for (int kk = 0; kk < K; kk++) {
                int ti = t * stride + kk - pad;
                if (ti < 0 || ti >= T) continue;
                acc = fmaf(xc[ti * xs.st], wr[ci * K + kk], acc);
            }
        }
        int64_t o = n * ys.sn + co * ys.sc + t * ys.st;
        if (mode == 1) acc = __fadd_rn(add[o], acc);
        else if (mode == 2) acc = __fadd_rn(__fmul_rn(1.0f - alpha, add[o]), __fmul_rn(alpha, acc));
        y[o] = acc;
    }
}

// weight layout [Cin][Cout][K] (torch ConvTranspose1d), no padding
__global__ void k_convT1d(const float *__restrict__ x, NCT xs, const float *__restrict__ W,
                          const float *__restrict__ b, float *__restrict__ y, NCT ys,
                          int N, int Cin, int Cout, int T, int Tout, int K, int stride) {
    int64_t total = (int64_t)N * Cout * Tout;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        int co = (int)(i % Cout); int t = (int)((i / Cout) % Tout); int n = (int)(i / ((int64_t)Cout * Tout));
        float acc = b ? b[co] : 0.f;
        if (K == stride) {                    // non-overlapping taps (the up-cascade): exactly one (input step, tap) per output step
            const int ti = t / stride, kk = t - ti * stride;
            if (ti < T) {
                const float *xc = x + n * xs.sn + ti * xs.st;
                const float *wc = W + (int64_t)co * K + kk;
                for (int ci = 0; ci < Cin; ci++) acc = fmaf(xc[ci * xs.sc], wc[(int64_t)ci * Cout * K], acc);
            }
            y[n * ys.sn + co * ys.sc + t * ys.st] = acc;
            continue;
        }
        for (int ci = 0; ci < Cin; ci++) {
            const float *xc = x + n * xs.sn + ci * xs.sc;
            for (int kk = 0; kk < K; kk++) {
                int num = t - kk;
                if (num < 0 || num % stride != 0) continue;
                int ti = num / stride;
                if (ti >= T) continue;
                acc = fmaf(xc[ti * xs.st], W[((int64_t)ci * Cout + co) * K + kk], acc);
            }
        }
        y[n * ys.sn + co * ys.sc + t * ys.st] = acc;
    }
}

// ---- convolutions whose taps do not overlap (K == stride), token-major tensors: a matrix product over patches ----
// conv:  y[n][t][co]          = b[co] + sum_{kk, ci} x[n][t * s + kk][ci] W[co][ci][kk]   (a patch is s * Cin consecutive floats)
// convT: y[n][t * s + kk][co] = b[co] + sum_ci       x[n][t][ci] W[ci][co][kk]            (s * Cout consecutive floats per input step)
// 64 patches x 64 columns per CTA step, 4 x 4 per thread; the weights of the 64 columns sit in shared memory (read through
// their own layout once per CTA), CTAs are persistent over the patches.
constexpr int PG_T = 64, PG_LD = 68, PG_MAXK = 256;
__global__ void __launch_bounds__(256) k_patch_gemm(const float *__restrict__ x, const float *__restrict__ W, const float *__restrict__ b,
                                                    float *__restrict__ y, int64_t rows, int T, int patches, int Cin, int Cout, int K, int KC, int ncols, int trans) {
    extern __shared__ __align__(16) float pg_sm[];
    const int ldw = KC + 4;
    float *Ws = pg_sm, *Xs = pg_sm + PG_T * ldw;                        // [64 columns][KC + 4], [64 patches][64 + 4]
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, n0 = blockIdx.y * PG_T;
    for (int i = tid; i < PG_T * KC; i += 256) {
        const int c = i / KC, k = i - c * KC, n = n0 + c;
        float w = 0.f;
        if (n < ncols) w = trans ? W[((int64_t)k * Cout + n % Cout) * K + n / Cout] : W[((int64_t)n * Cin + k % Cin) * K + k / Cin];
        Ws[c * ldw + k] = w;
    }
    const int64_t tiles = (rows + PG_T - 1) / PG_T;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t r0 = tile * PG_T;
        float acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
        for (int k0 = 0; k0 < KC; k0 += PG_T) {
            __syncthreads();
#pragma unroll
            for (int i = tid; i < PG_T * PG_T / 4; i += 256) {
                const int rr = i >> 4, k = k0 + (i & 15) * 4;
                const int64_t r = r0 + rr;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (r < rows && k < KC) {
                    const int64_t n = r / patches; const int t = (int)(r - n * patches);
                    v = *(const float4 *)(x + (n * T + (int64_t)t * (trans ? 1 : K)) * Cin + k);
                }
                *(float4 *)(Xs + rr * PG_LD + (i & 15) * 4) = v;
            }
            __syncthreads();
            const int kn = min(PG_T, KC - k0);
            for (int k = 0; k < kn; k += 4) {
                float4 a[4], w[4];
#pragma unroll
                for (int i = 0; i < 4; i++) a[i] = *(const float4 *)(Xs + (ty + 16 * i) * PG_LD + k);
#pragma unroll
                for (int j = 0; j < 4; j++) w[j] = *(const float4 *)(Ws + (tx + 16 * j) * ldw + k0 + k);
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        acc[i][j] = fmaf(a[i].x, w[j].x, acc[i][j]); acc[i][j] = fmaf(a[i].y, w[j].y, acc[i][j]);
                        acc[i][j] = fmaf(a[i].z, w[j].z, acc[i][j]); acc[i][j] = fmaf(a[i].w, w[j].w, acc[i][j]);
                    }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int64_t r = r0 + ty + 16 * i;
            if (r >= rows) continue;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int n = n0 + tx + 16 * j;
                if (n < ncols) y[r * ncols + n] = (b ? b[n % Cout] : 0.f) + acc[i][j];
            }
        }
    }
}
static bool same_layout(const NCT &a, const NCT &b) { return a.sn == b.sn && a.sc == b.sc && a.st == b.st; }
// patches of at least this many rows go to k_patch_gemm: below, the weights' trip through shared memory is the longer part
constexpr int64_t PG_MIN_ROWS = 64;
static bool patch_gemm(const float *x, NCT xs, const float *W, const float *b, float *y, NCT ys, int N, int Cin, int Cout, int T, int Tout, int K, int trans) {
    const int KC = trans ? Cin : Cin * K, ncols = trans ? Cout * K : Cout, patches = trans ? T : Tout;
    const int64_t rows = (int64_t)N * patches;
    if (rows < PG_MIN_ROWS || KC > PG_MAXK || (Cin & 3) || ((uintptr_t)x & 15) || !same_layout(xs, nlc(Cin, T)) || !same_layout(ys, nlc(Cout, Tout))) return false;
    const size_t smem = (size_t)(PG_T * (KC + 4) + PG_T * PG_LD) * 4;
    static bool set = false;
    if (!set) { CUDA_CHECK(cudaFuncSetAttribute(k_patch_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (PG_T * (PG_MAXK + 4) + PG_T * PG_LD) * 4)); set = true; }
    const int64_t cap = (int64_t)ctx().sm_count * 2;
    dim3 grid((unsigned)std::min<int64_t>(cdiv(rows, PG_T), cap), (unsigned)cdiv(ncols, PG_T));
    LAUNCH(k_patch_gemm, grid, 256, smem, x, W, b, y, rows, T, patches, Cin, Cout, K, KC, ncols, trans);
    return true;
}

// affine-free GroupNorm, eps 1e-5: one CTA per (n, group), statistics over Cg x T
__global__ void __launch_bounds__(128) k_groupnorm(const float *__restrict__ x, NCT xs, float *__restrict__ y, NCT ys,
                                                   int G, int C, int T) {
    int n = blockIdx.x / G, g = blockIdx.x % G;
    int Cg = C / G, cnt = Cg * T;
    __shared__ float red[128];
    __shared__ float stat[2];
    float s = 0.f;
    for (int i = threadIdx.x; i < cnt; i += 128) {
        int c = g * Cg + i / T, t = i % T;
        s += x[n * xs.sn + c * xs.sc + t * xs.st];
    }
    red[threadIdx.x] = s; __syncthreads();
    for (int o = 64; o > 0; o >>= 1) { if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o]; __syncthreads(); }
    if (threadIdx.x == 0) stat[0] = red[0] / (float)cnt;
    __syncthreads();
    float mean = stat[0], q = 0.f;
    for (int i = threadIdx.x; i < cnt; i += 128) {
        int c = g * Cg + i / T, t = i % T;
        float d = x[n * xs.sn + c * xs.sc + t * xs.st] - mean;
        q += d * d;
    }
    __syncthreads();
    red[threadIdx.x] = q; __syncthreads();
    for (int o = 64; o > 0; o >>= 1) { if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o]; __syncthreads(); }
    if (threadIdx.x == 0) stat[1] = 1.0f / sqrtf(red[0] / (float)cnt + 1e-5f);
    __syncthreads();
    float inv = stat[1];
    for (int i = threadIdx.x; i < cnt; i += 128) {
        int c = g * Cg + i / T, t = i % T;
        y[n * ys.sn + c * ys.sc + t * ys.st] = (x[n * xs.sn + c * xs.sc + t * xs.st] - mean) * inv;
    }
}

// Token-major tensors: one warp per sequence takes all groups. A lane holds four channels, 128 / C time steps go by at once,
// and the lanes of a group meet by shuffles (the kernel above reads a few channels of a row at a time from a CTA per group).
__global__ void __launch_bounds__(256) k_groupnorm_nlc(const float *__restrict__ x, float *__restrict__ y, int N, int lpg, int C, int T) {
    const int n = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (n >= N) return;
    const int lpr = C >> 2, tp = 32 / lpr, c4 = lane % lpr, t0 = lane / lpr;            // lanes per row, rows per pass
    const float4 *xr = (const float4 *)(x + (int64_t)n * T * C) + c4;
    float4 *yr = (float4 *)(y + (int64_t)n * T * C) + c4;
    const float cnt = (float)(lpg * 4 * T);
    auto group_sum = [&](float v) {
        for (int o = 1; o < lpg; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        for (int o = lpr; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    };
    float s = 0.f;
    for (int t = t0; t < T; t += tp) { const float4 v = xr[t * lpr]; s += (v.x + v.y) + (v.z + v.w); }
    const float mean = group_sum(s) / cnt;
    float q = 0.f;
    for (int t = t0; t < T; t += tp) {
        const float4 v = xr[t * lpr];
        const float d0 = v.x - mean, d1 = v.y - mean, d2 = v.z - mean, d3 = v.w - mean;
        q += (d0 * d0 + d1 * d1) + (d2 * d2 + d3 * d3);
    }
    const float inv = 1.0f / sqrtf(group_sum(q) / cnt + 1e-5f);
    for (int t = t0; t < T; t += tp) {
        const float4 v = xr[t * lpr];
        yr[t * lpr] = make_float4((v.x - mean) * inv, (v.y - mean) * inv, (v.z - mean) * inv, (v.w - mean) * inv);
    }
}

// ATen "area": equal-weight mean over [floor(t*Tin/Tout), ceil((t+1)*Tin/Tout))
__global__ void k_interp_area(const float *__restrict__ x, NCT xs, float *__restrict__ y, NCT ys,
                              int N, int C, int Tin, int Tout) {
    int64_t total = (int64_t)N * C * Tout;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        int c = (int)(i % C); int t = (int)((i / C) % Tout); int n = (int)(i / ((int64_t)C * Tout));
        int s = (int)(((int64_t)t * Tin) / Tout);
        int e = (int)(((int64_t)(t + 1) * Tin + Tout - 1) / Tout);
        if (e <= s) e = s + 1;
        if (e > Tin) e = Tin;
        const float *xc = x + n * xs.sn + c * xs.sc;
        float acc = 0.f;
        for (int k = s; k < e; k++) acc += xc[k * xs.st];
        y[n * ys.sn + c * ys.sc + t * ys.st] = acc / (float)(e - s);
    }
}

// ATen "linear", align_corners=False; mean when either length is 1
__global__ void k_interp_linear(const float *__restrict__ x, NCT xs, float *__restrict__ y, NCT ys,
                                int N, int C, int Tin, int Tout) {
    int64_t total = (int64_t)N * C * Tout;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        int c = (int)(i % C); int t = (int)((i / C) % Tout); int n = (int)(i / ((int64_t)C * Tout));
        const float *xc = x + n * xs.sn + c * xs.sc;
        float out;
        if (Tout == 1 || Tin == 1) {
            float acc = 0.f;
            for (int k = 0; k < Tin; k++) acc += xc[k * xs.st];
            out = acc / (float)Tin;
        } else {
            double scale = (double)Tin / Tout;
            double src = (t + 0.5) * scale - 0.5;
            int s0 = (int)floor(src);
            double w1 = src - s0, w0 = 1.0 - w1;
            int i0 = s0 < 0 ? 0 : (s0 >= Tin ? Tin - 1 : s0);
            int s1 = s0 + 1;
            int i1 = s1 < 0 ? 0 : (s1 >= Tin ? Tin - 1 : s1);
            out = (float)(w0 * (double)xc[i0 * xs.st] + w1 * (double)xc[i1 * xs.st]);
        }
        y[n * ys.sn + c * ys.sc + t * ys.st] = out;
    }
}

__global__ void k_l2sq(const float *__restrict__ a, const float *__restrict__ b, float *__restrict__ d2,
                       int64_t rows, int64_t cols, int C) {
    int64_t total = rows * cols;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        int64_t r = i / cols, j = i % cols;
        float s = 0.f;
        for (int c = 0; c < C; c++) { float d = a[r * C + c] - b[j * C + c]; s = fmaf(d, d, s); }
        d2[i] = s;
    }
}

static unsigned vq_grid(int64_t n) {
    int64_t g = cdiv(n, 128);
    int64_t cap = (int64_t)ctx().sm_count * 32;
    if (g > cap) g = cap;
    return (unsigned)(g < 1 ? 1 : g);
}

void conv1d(const float *x, NCT xs, const float *W, const float *b, float *y, NCT ys,
            int N, int Cin, int Cout, int T, int K, int stride, int pad, const float *add, float alpha) {
    int Tout = (T + 2 * pad - K) / stride + 1;
    int64_t n = (int64_t)N * Cout * Tout;
    if (n <= 0) return;
    int mode = !add ? 0 : (alpha == 0.f ? 1 : 2);
    ProfScope ps(NCMB_K_VQ, 2.0 * n * Cin * K, 0);
    if (mode == 0 && stride == K && pad == 0 && patch_gemm(x, xs, W, b, y, ys, N, Cin, Cout, T, Tout, K, 0)) return;
    LAUNCH(k_conv1d, vq_grid(n), 128, 0, x, xs, W, b, y, ys, N, Cin, Cout, T, Tout, K, stride, pad, add, alpha, mode);
}
void convT1d(const float *x, NCT xs, const float *W, const float *b, float *y, NCT ys,
             int N, int Cin, int Cout, int T, int K, int stride) {
    int Tout = (T - 1) * stride + K;
    int64_t n = (int64_t)N * Cout * Tout;
    if (n <= 0) return;
    ProfScope ps(NCMB_K_VQ, 2.0 * n * Cin, 0);
    if (stride == K && patch_gemm(x, xs, W, b, y, ys, N, Cin, Cout, T, Tout, K, 1)) return;
    LAUNCH(k_convT1d, vq_grid(n), 128, 0, x, xs, W, b, y, ys, N, Cin, Cout, T, Tout, K, stride);
}
void groupnorm(const float *x, NCT xs, float *y, NCT ys, int N, int G, int C, int T) {
    if (N <= 0) return;
    ProfScope ps(NCMB_K_VQ);
    const int lpr = C / 4, lpg = G > 0 ? C / G / 4 : 0;
    auto pow2 = [](int v) { return v > 0 && (v & (v - 1)) == 0; };
    if (C % 4 == 0 && C % G == 0 && (C / G) % 4 == 0 && pow2(lpr) && lpr <= 32 && pow2(lpg) && same_layout(xs, nlc(C, T)) && same_layout(ys, nlc(C, T)) &&
        (((uintptr_t)x | (uintptr_t)y) & 15) == 0) {
        LAUNCH(k_groupnorm_nlc, grid1d((int64_t)N * 32, 256), 256, 0, x, y, N, lpg, C, T);
        return;
    }
    LAUNCH(k_groupnorm, (unsigned)(N * G), 128, 0, x, xs, y, ys, G, C, T);
}
void interp_area(const float *x, NCT xs, float *y, NCT ys, int N, int C, int Tin, int Tout) {
    int64_t n = (int64_t)N * C * Tout;
    if (n <= 0) return;
    ProfScope ps(NCMB_K_VQ);
    LAUNCH(k_interp_area, vq_grid(n), 128, 0, x, xs, y, ys, N, C, Tin, Tout);
}
void interp_linear(const float *x, NCT xs, float *y, NCT ys, int N, int C, int Tin, int Tout) {
    int64_t n = (int64_t)N * C * Tout;
    if (n <= 0) return;
    ProfScope ps(NCMB_K_VQ);
    LAUNCH(k_interp_linear, vq_grid(n), 128, 0, x, xs, y, ys, N, C, Tin, Tout);
}

} // namespace ncmb

using namespace ncmb;

extern "C" {

void conv1d_fwd(const float *x, const float *W, const float *b, float *y, int N, int Cin, int Cout, int T, int K, int stride, int pad) {
    ensure_device();
    int Tout = (T + 2 * pad - K) / stride + 1;
    conv1d(x, ncl(Cin, T), W, b, y, ncl(Cout, Tout), N, Cin, Cout, T, K, stride, pad, nullptr, 0.f);
}
void convtranspose1d_fwd(const float *x, const float *W, const float *b, float *y, int N, int Cin, int Cout, int T, int K, int stride) {
    ensure_device();
    int Tout = (T - 1) * stride + K;
    convT1d(x, ncl(Cin, T), W, b, y, ncl(Cout, Tout), N, Cin, Cout, T, K, stride);
}
void groupnorm_fwd(const float *x, float *y, int N, int G, int C, int T) {
    ensure_device();
    groupnorm(x, ncl(C, T), y, ncl(C, T), N, G, C, T);
}
void interpolate_area_fwd(const float *x, float *y, int N, int C, int Tin, int Tout) {
    ensure_device();
    interp_area(x, ncl(C, Tin), y, ncl(C, Tout), N, C, Tin, Tout);
}
void interpolate_linear_fwd(const float *x, float *y, int N, int C, int Tin, int Tout) {
    ensure_device();
    interp_linear(x, ncl(C, Tin), y, ncl(C, Tout), N, C, Tin, Tout);
}
void rowwise_l2sq(const float *a, const float *b, float *d2, int64_t rows, int64_t colsA, int C) {
    ensure_device();
    int64_t n = rows * colsA;
    if (n <= 0) return;
    ProfScope ps(NCMB_K_VQ, 3.0 * n * C, 4.0 * n);
    LAUNCH(k_l2sq, vq_grid(n), 128, 0, a, b, d2, rows, colsA, C);
}

} // extern "C"
