// The VQ-VAE's transformer stacks (reference vae_block, src/vqvae.c:44-225) at embedding width 64 as ONE kernel: the tokens
// of a few boards stay in shared memory from the embedding to the last norm, and only ids (or latents) come in and latents
// (or token ids) go out. Layer by layer, each of the twelve 64 x 64 weight blocks of a layer is staged in turn and applied to
// all rows of the CTA (fp32 multiply-adds, 4 columns x RI row groups per thread); attention takes one warp per (board, head,
// 32 queries) with a query per lane.
//
// Bound: fp32 multiply-adds (49 K per token and layer, two shared-memory reads per sixteen) for large batches, the chain of
// weight blocks (about a microsecond each) for small ones. The separate kernels it stands in for moved the hidden layer
// (256 wide, as pairs) and every other intermediate through HBM, about fourteen launches per stack.
#include "vae_fused.cuh"

namespace ncmb {

constexpr int VF_D = 64, VF_LD = 68, VF_QLD = 196, VF_MAXL = 8;

struct VaeStack {
    struct Layer { const float *ln1w, *ln1b, *qkvw, *qkvb, *ow, *ob, *ln2w, *ln2b, *fcw, *fcb, *pw, *pb; } l[VF_MAXL];
    int nl, heads, T, nb, B; float eps;
    const int *ids; const float *wte, *wpe, *x;              // input: wte[ids] (+ wpe) or x (+ wpe)
    const float *lnf; float *y;                              // output: norm(x) * lnf (lnf null: x itself), or ...
    const float *out_w; int V; int *tok;                     // ... V <= 64 output rows: the first-index argmax of each token's logits
};

// weight block rows [n0, n0 + 64) x columns [k0, k0 + 64) of W [N][ldw]; rows from N on are zero
struct WBlock { float4 v[4]; };
__device__ __forceinline__ void vf_fetch(WBlock &b, const float *__restrict__ W, int ldw, int n0, int k0, int N = 1 << 30) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int e = threadIdx.x + 256 * i, n = n0 + (e >> 4);
        b.v[i] = n < N ? __ldg((const float4 *)(W + (int64_t)n * ldw + k0 + (e & 15) * 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}
__device__ __forceinline__ void vf_stage(const WBlock &b, float *Ws) {
#pragma unroll
    for (int i = 0; i < 4; i++) { const int e = threadIdx.x + 256 * i; *(float4 *)(Ws + (e >> 4) * VF_LD + (e & 15) * 4) = b.v[i]; }
}
// acc[i][j] += A[ty + 16 i][:] . Ws[tx + 16 j][:]
template <int RI>
__device__ __forceinline__ void vf_mac(const float *A, int lda, const float *Ws, float (&acc)[RI][4]) {
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll 4
    for (int k = 0; k < VF_D; k += 4) {
        float4 a[RI], w[4];
#pragma unroll
        for (int i = 0; i < RI; i++) a[i] = *(const float4 *)(A + (ty + 16 * i) * lda + k);
#pragma unroll
        for (int j = 0; j < 4; j++) w[j] = *(const float4 *)(Ws + (tx + 16 * j) * VF_LD + k);
#pragma unroll
        for (int i = 0; i < RI; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                acc[i][j] = fmaf(a[i].x, w[j].x, acc[i][j]); acc[i][j] = fmaf(a[i].y, w[j].y, acc[i][j]);
                acc[i][j] = fmaf(a[i].z, w[j].z, acc[i][j]); acc[i][j] = fmaf(a[i].w, w[j].w, acc[i][j]);
            }
    }
}
template <int RI>
__device__ __forceinline__ void vf_zero(float (&acc)[RI][4]) {
#pragma unroll
    for (int i = 0; i < RI; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
}
// rows of src normalised (LayerNorm, the arithmetic of k_layernorm) into dst: four threads per row
template <int RI>
__device__ __forceinline__ void vf_norm(const float *src, float *dst, const float *__restrict__ w, const float *__restrict__ b, float eps) {
    const int part = threadIdx.x & 3;
    for (int r = threadIdx.x >> 2; r < RI * 16; r += 64) {
        const float *xr = src + r * VF_LD + part * 16;
        float4 v[4];
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < 4; i++) { v[i] = *(const float4 *)(xr + 4 * i); s += (v[i].x + v[i].y) + (v[i].z + v[i].w); }
        s += __shfl_xor_sync(0xffffffffu, s, 1); s += __shfl_xor_sync(0xffffffffu, s, 2);
        const float mean = s / (float)VF_D;
        float q = 0.f;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            v[i].x -= mean; v[i].y -= mean; v[i].z -= mean; v[i].w -= mean;
            q += (v[i].x * v[i].x + v[i].y * v[i].y) + (v[i].z * v[i].z + v[i].w * v[i].w);
        }
        q += __shfl_xor_sync(0xffffffffu, q, 1); q += __shfl_xor_sync(0xffffffffu, q, 2);
        const float inv = 1.0f / sqrtf(q / (float)VF_D + eps);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int c = part * 16 + 4 * i;
            const float4 ww = w ? __ldg((const float4 *)(w + c)) : make_float4(1.f, 1.f, 1.f, 1.f);
            const float4 bb = b ? __ldg((const float4 *)(b + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
            *(float4 *)(dst + r * VF_LD + c) = make_float4(__fadd_rn(__fmul_rn(__fmul_rn(v[i].x, inv), ww.x), bb.x), __fadd_rn(__fmul_rn(__fmul_rn(v[i].y, inv), ww.y), bb.y),
                                                           __fadd_rn(__fmul_rn(__fmul_rn(v[i].z, inv), ww.z), bb.z), __fadd_rn(__fmul_rn(__fmul_rn(v[i].w, inv), ww.w), bb.w));
        }
    }
}
// bidirectional attention of one (board, head, 32-query block): the lane owns a query; the context replaces the query
template <int HD>
__device__ __forceinline__ void vf_attend(float *QKV, int row0, int T, int h, int q0, int lane) {
    const int qi = q0 + lane;
    const bool on = qi < T;
    float *qp = QKV + (row0 + (on ? qi : 0)) * VF_QLD + h * HD;
    float q[HD], o[HD];
#pragma unroll
    for (int d = 0; d < HD; d += 4) {
        const float4 v = *(const float4 *)(qp + d);
        q[d] = v.x; q[d + 1] = v.y; q[d + 2] = v.z; q[d + 3] = v.w;
        o[d] = o[d + 1] = o[d + 2] = o[d + 3] = 0.f;
    }
    __syncwarp();
    const float scale = 1.0f / sqrtf((float)HD);
    float m = -INFINITY, l = 0.f;
    for (int j0 = 0; j0 < T; j0 += 8) {
        float s[8], mx = m;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            s[j] = -INFINITY;
            if (j0 + j < T) {
                const float *kp = QKV + (row0 + j0 + j) * VF_QLD + VF_D + h * HD;
                float d0 = 0.f;
#pragma unroll
                for (int d = 0; d < HD; d += 4) {
                    const float4 v = *(const float4 *)(kp + d);
                    d0 = fmaf(q[d], v.x, d0); d0 = fmaf(q[d + 1], v.y, d0); d0 = fmaf(q[d + 2], v.z, d0); d0 = fmaf(q[d + 3], v.w, d0);
                }
                s[j] = d0 * scale;
                mx = fmaxf(mx, s[j]);
            }
        }
        const float al = m == -INFINITY ? 0.f : expf(m - mx);
        l *= al; m = mx;
#pragma unroll
        for (int d = 0; d < HD; d++) o[d] *= al;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (j0 + j < T) {
                const float p = expf(s[j] - m);
                l += p;
                const float *vp = QKV + (row0 + j0 + j) * VF_QLD + 2 * VF_D + h * HD;
#pragma unroll
                for (int d = 0; d < HD; d += 4) {
                    const float4 v = *(const float4 *)(vp + d);
                    o[d] = fmaf(p, v.x, o[d]); o[d + 1] = fmaf(p, v.y, o[d + 1]); o[d + 2] = fmaf(p, v.z, o[d + 2]); o[d + 3] = fmaf(p, v.w, o[d + 3]);
                }
            }
        }
    }
    const float inv = 1.0f / l;
    if (on) {
#pragma unroll
        for (int d = 0; d < HD; d += 4) *(float4 *)(qp + d) = make_float4(o[d] * inv, o[d + 1] * inv, o[d + 2] * inv, o[d + 3] * inv);
    }
}

template <int RI, int HD>
__global__ void __launch_bounds__(256) k_vae_stack(const __grid_constant__ VaeStack a) {
    extern __shared__ __align__(16) float vf_sm[];
    constexpr int R = RI * 16;
    float *X = vf_sm, *N = X + R * VF_LD, *QKV = N + R * VF_LD, *Ws = QKV + R * VF_QLD;
    float *H = QKV;                                          // the hidden block: q, k, v are dead by then
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, warp = tid >> 5, lane = tid & 31;
    const int T = a.T, b0 = blockIdx.x * a.nb, nboard = min(a.nb, a.B - b0), rows = nboard * T;
    const int64_t g0 = (int64_t)b0 * T;                      // first token of the CTA
    WBlock wb;
    vf_fetch(wb, a.l[0].qkvw, VF_D, 0, 0);
    for (int e = tid; e < R * 16; e += 256) {
        const int r = e >> 4, c = (e & 15) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows) {
            v = a.ids ? *(const float4 *)(a.wte + (int64_t)a.ids[g0 + r] * VF_D + c) : *(const float4 *)(a.x + (g0 + r) * VF_D + c);
            if (a.wpe) { const float4 p = *(const float4 *)(a.wpe + (r % T) * VF_D + c); v.x = __fadd_rn(v.x, p.x); v.y = __fadd_rn(v.y, p.y); v.z = __fadd_rn(v.z, p.z); v.w = __fadd_rn(v.w, p.w); }
        }
        *(float4 *)(X + r * VF_LD + c) = v;
    }
    __syncthreads();
    float acc[RI][4];
    for (int li = 0; li < a.nl; li++) {
        const VaeStack::Layer &L = a.l[li];
        vf_norm<RI>(X, N, L.ln1w, L.ln1b, a.eps);
#pragma unroll 1
        for (int blk = 0; blk < 3; blk++) {                  // q, k, v
            __syncthreads();
            vf_stage(wb, Ws);
            __syncthreads();
            if (blk < 2) vf_fetch(wb, L.qkvw, VF_D, (blk + 1) * 64, 0); else vf_fetch(wb, L.ow, VF_D, 0, 0);
            vf_zero<RI>(acc);
            vf_mac<RI>(N, VF_LD, Ws, acc);
#pragma unroll
            for (int i = 0; i < RI; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int c = blk * 64 + tx + 16 * j;
                    QKV[(ty + 16 * i) * VF_QLD + c] = acc[i][j] + (L.qkvb ? __ldg(L.qkvb + c) : 0.f);
                }
        }
        __syncthreads();
        vf_stage(wb, Ws);                                    // the output projection's block, while the warps attend
        const int qb = (T + 31) >> 5, items = nboard * a.heads * qb;
        for (int it = warp; it < items; it += 8) {
            const int bd = it / (a.heads * qb), rem = it - bd * a.heads * qb;
            vf_attend<HD>(QKV, bd * T, T, rem / qb, (rem % qb) * 32, lane);
        }
        __syncthreads();
        vf_fetch(wb, L.fcw, VF_D, 0, 0);
        vf_zero<RI>(acc);
        vf_mac<RI>(QKV, VF_QLD, Ws, acc);
#pragma unroll
        for (int i = 0; i < RI; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) { const int c = tx + 16 * j; X[(ty + 16 * i) * VF_LD + c] += acc[i][j] + (L.ob ? __ldg(L.ob + c) : 0.f); }
        __syncthreads();
        vf_norm<RI>(X, N, L.ln2w, L.ln2b, a.eps);
        float out[RI][4];
        vf_zero<RI>(out);
#pragma unroll 1
        for (int hc = 0; hc < 4; hc++) {                     // 64 hidden units at a time
            __syncthreads();
            vf_stage(wb, Ws);
            __syncthreads();
            vf_fetch(wb, L.pw, 4 * VF_D, 0, hc * 64);
            vf_zero<RI>(acc);
            vf_mac<RI>(N, VF_LD, Ws, acc);
#pragma unroll
            for (int i = 0; i < RI; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int c = tx + 16 * j;
                    const float v = acc[i][j] + (L.fcb ? __ldg(L.fcb + hc * 64 + c) : 0.f);
                    H[(ty + 16 * i) * VF_LD + c] = 0.5f * v * (1.0f + erff(v * 0.7071067811865475f));
                }
            __syncthreads();
            vf_stage(wb, Ws);
            __syncthreads();
            if (hc < 3) vf_fetch(wb, L.fcw, VF_D, (hc + 1) * 64, 0);
            else if (li + 1 < a.nl) vf_fetch(wb, a.l[li + 1].qkvw, VF_D, 0, 0);
            else if (a.tok) vf_fetch(wb, a.out_w, VF_D, 0, 0, a.V);
            vf_mac<RI>(H, VF_LD, Ws, out);
        }
#pragma unroll
        for (int i = 0; i < RI; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) { const int c = tx + 16 * j; X[(ty + 16 * i) * VF_LD + c] += out[i][j] + (L.pb ? __ldg(L.pb + c) : 0.f); }
        __syncthreads();
    }
    const float *fin = X;
    if (a.lnf) { vf_norm<RI>(X, N, a.lnf, nullptr, a.eps); fin = N; }
    if (a.tok) vf_stage(wb, Ws);
    __syncthreads();
    if (a.y) {
        for (int e = tid; e < rows * 16; e += 256) {
            const int r = e >> 4, c = (e & 15) * 4;
            *(float4 *)(a.y + (g0 + r) * VF_D + c) = *(const float4 *)(fin + r * VF_LD + c);
        }
    }
    if (a.tok) {
        vf_zero<RI>(acc);
        vf_mac<RI>(fin, VF_LD, Ws, acc);
#pragma unroll
        for (int i = 0; i < RI; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) H[(ty + 16 * i) * VF_LD + tx + 16 * j] = acc[i][j];
        __syncthreads();
        for (int r = tid; r < rows; r += 256) {
            int best = 0;
            for (int v = 1; v < a.V; v++) if (H[r * VF_LD + v] > H[r * VF_LD + best]) best = v;
            a.tok[g0 + r] = best;
        }
    }
}

bool vae_stack_supported(const std::vector<BlockWeights> &layers, int D, int heads, int T, int window) {
    if (ctx().gemm_mode == 1 || layers.empty() || layers.size() > VF_MAXL || D != VF_D || T > 96 || window > 0) return false;
    if (heads != 1 && heads != 2 && heads != 4 && heads != 8) return false;
    for (auto &w : layers)
        if (w.norm != NORM_LAYER || w.gated || w.act != ACT_GELU || w.Hh != 4 * VF_D || w.qnw || w.knw || !w.ln1w || !w.ln2w || w.eps != layers[0].eps) return false;
    return true;
}

template <int RI, int HD>
static void launch_stack(const VaeStack &a) {
    constexpr size_t smem = sizeof(float) * (RI * 16 * (2 * VF_LD + VF_QLD) + 64 * VF_LD);
    static bool set = false;
    if (!set) { CUDA_CHECK(cudaFuncSetAttribute((k_vae_stack<RI, HD>), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); set = true; }
    LAUNCH((k_vae_stack<RI, HD>), (unsigned)cdiv(a.B, a.nb), 256, smem, a);
}
template <int RI>
static void launch_stack_hd(const VaeStack &a) {
    switch (a.heads) {
        case 1: launch_stack<RI, 64>(a); break;
        case 2: launch_stack<RI, 32>(a); break;
        case 4: launch_stack<RI, 16>(a); break;
        default: launch_stack<RI, 8>(a);
    }
}

void vae_stack(const std::vector<BlockWeights> &layers, int heads, int B, int T, const VaeStackIO &io) {
    if (B <= 0) return;
    VaeStack a{};
    a.nl = (int)layers.size(); a.heads = heads; a.T = T; a.B = B; a.eps = layers[0].eps;
    for (int i = 0; i < a.nl; i++) {
        const BlockWeights &w = layers[i];
        a.l[i] = VaeStack::Layer{w.ln1w, w.ln1b, w.qkvw, w.qkvb, w.ow, w.ob, w.ln2w, w.ln2b, w.fcw, w.fcb, w.pw, w.pb};
    }
    a.ids = io.ids; a.wte = io.wte; a.x = io.x; a.wpe = io.wpe; a.lnf = io.lnf; a.y = io.y; a.out_w = io.out_w; a.V = io.V; a.tok = io.tok;
    // boards per CTA: 64 rows (a weight block's reads are shared by all of them) once that still gives every SM two CTAs,
    // one board before
    int nb = T >= 64 ? 1 : 64 / T;
    while (nb > 1 && cdiv(B, nb) < 2 * (int64_t)ctx().sm_count) nb--;
    a.nb = nb;
    const int ri = (int)cdiv((int64_t)nb * T, 16);
    ProfScope ps(NCMB_K_GEMM, 2.0 * (double)B * T * a.nl * (12.0 * VF_D * VF_D + 2.0 * T * VF_D), 4.0 * (double)B * T * 2 * VF_D);
    if (ri <= 1) launch_stack_hd<1>(a);
    else if (ri <= 2) launch_stack_hd<2>(a);
    else if (ri <= 4) launch_stack_hd<4>(a);
    else launch_stack_hd<6>(a);
}

} // namespace ncmb
