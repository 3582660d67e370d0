// Multiscale residual quantizer on the device (reference src/vq.c).
//
// The reference walks every level through host memory (code gather, z_hat += up,
// Phi blend, argmin over a materialised [rows][V] distance matrix). Here every
// tensor stays token-major [B][L][D] in HBM: the resampling kernels take strides,
// so no [B][L][D] <-> [B][D][L] transposes are issued, and the nearest-code search
// (nearest.cu) keeps running minima instead of writing distances out.
#include "common.cuh"
#include "vq.cuh"
#include "nearest.cuh"

namespace ncmb {

// rowmod > 0: row b reads the codes of row b % rowmod (the CFG half shares the sampled codes)
__global__ void k_gather_codes(const float *__restrict__ E, const int *__restrict__ codes, int stride, int rowmod, int tlen,
                               int D, int V, int64_t n, float *__restrict__ out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        int d = (int)(i % D); int64_t r = i / D; int t = (int)(r % tlen); int64_t b = r / tlen;
        if (rowmod > 0) b %= rowmod;
        int code = codes[b * stride + t];
        code = code < 0 ? 0 : (code >= V ? V - 1 : code);
        out[i] = E[(int64_t)code * D + d];
    }
}
__global__ void k_axpy_inplace(float *__restrict__ y, const float *__restrict__ x, float a, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) y[i] = __fadd_rn(y[i], a * x[i]);
}

// One level's contribution in one pass over z: dst = src + sign * up, and next = the mean of dst over the L / tnext positions of
// each step of the next level (its quantizer input), where up is the level's codes brought to length L by linear interpolation
// (align_corners = False; constant when the level has one step), or read from `up_in`. Four channels per thread; src == null is
// zero. One read and one write of z (memory bound) where gather, interpolation, update and mean were passes of their own.
struct LevelStep {
    const float *E; const int *codes; int stride, rowmod, tlen, V;
    const float *up_in, *src; float *dst, *next;
    float sign; int L, D, tnext; int64_t n4;                 // n4 = B * tnext * D / 4 threads
};
__global__ void __launch_bounds__(256) k_level_step(LevelStep a) {
    extern __shared__ double ls_tab[];                       // [L] weights of the lower step, then [L] lower and upper steps
    int *i0 = (int *)(ls_tab + a.L), *i1 = i0 + a.L;
    const bool flat = a.tlen == 1 || a.L == 1;               // the mean of the level's steps, at every position
    if (!a.up_in && !flat) {
        for (int t = threadIdx.x; t < a.L; t += blockDim.x) {
            const double src = (t + 0.5) * ((double)a.tlen / a.L) - 0.5;
            const int s0 = (int)floor(src);
            ls_tab[t] = src - s0;
            i0[t] = s0 < 0 ? 0 : (s0 >= a.tlen ? a.tlen - 1 : s0);
            i1[t] = s0 + 1 < 0 ? 0 : (s0 + 1 >= a.tlen ? a.tlen - 1 : s0 + 1);
        }
        __syncthreads();
    }
    const int D4 = a.D >> 2, w = a.L / a.tnext;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.n4; i += (int64_t)gridDim.x * blockDim.x) {
        const int d = (int)(i % D4) * 4; const int64_t bt = i / D4; const int tn = (int)(bt % a.tnext); const int64_t b = bt / a.tnext;
        const int *cb = a.codes + (a.rowmod > 0 ? b % a.rowmod : b) * a.stride;
        auto code_row = [&](int j) {
            int c = cb[j];
            c = c < 0 ? 0 : (c >= a.V ? a.V - 1 : c);
            return *(const float4 *)(a.E + (int64_t)c * a.D + d);
        };
        float4 one = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!a.up_in && flat) {
            for (int j = 0; j < a.tlen; j++) { const float4 v = code_row(j); one.x += v.x; one.y += v.y; one.z += v.z; one.w += v.w; }
            const float c = (float)a.tlen;
            one = make_float4(one.x / c, one.y / c, one.z / c, one.w / c);
        }
        float4 m = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int t = tn * w; t < (tn + 1) * w; t++) {
            const int64_t at = (b * a.L + t) * a.D + d;
            float4 u = one;
            if (a.up_in) u = *(const float4 *)(a.up_in + at);
            else if (!flat) {
                const double w1 = ls_tab[t], w0 = 1.0 - w1;
                const float4 p = code_row(i0[t]), q = code_row(i1[t]);
                u.x = (float)(w0 * (double)p.x + w1 * (double)q.x); u.y = (float)(w0 * (double)p.y + w1 * (double)q.y);
                u.z = (float)(w0 * (double)p.z + w1 * (double)q.z); u.w = (float)(w0 * (double)p.w + w1 * (double)q.w);
            }
            float4 z = a.src ? *(const float4 *)(a.src + at) : make_float4(0.f, 0.f, 0.f, 0.f);
            z.x = __fadd_rn(z.x, a.sign * u.x); z.y = __fadd_rn(z.y, a.sign * u.y); z.z = __fadd_rn(z.z, a.sign * u.z); z.w = __fadd_rn(z.w, a.sign * u.w);
            *(float4 *)(a.dst + at) = z;
            m.x += z.x; m.y += z.y; m.z += z.z; m.w += z.w;
        }
        if (a.next) {
            const float c = (float)w;
            *(float4 *)(a.next + (b * a.tnext + tn) * a.D + d) = make_float4(m.x / c, m.y / c, m.z / c, m.w / c);
        }
    }
}

static unsigned ew(int64_t n) {
    int64_t g = cdiv(n, 256), cap = (int64_t)ctx().sm_count * 16;
    return (unsigned)(g < 1 ? 1 : (g > cap ? cap : g));
}

// q [B][tlen][D] -> out [B][L][D]  (reference up_to_full, src/vq.c:327-376). tmp1/tmp2: [B][L][D] scratch.
static void up_to_full_dev(VQState *v, const float *q, int B, int tlen, int level, float *out, float *tmp1, float *tmp2) {
    int D = v->D, L = v->L;
    if (level == 0 && v->has_l1) {
        const float *cur = q;
        int Tc = tlen;
        float *bufs[2] = {tmp1, tmp2};
        int flip = 0;
        for (int i = 0; i < v->n_up; i++) {
            int s = v->upK[i], To = (Tc - 1) * s + s;
            if (v->l1_norm && i > 0) {
                float *gn = bufs[flip]; flip ^= 1;
                groupnorm(cur, nlc(D, Tc), gn, nlc(D, Tc), B, 8, D, Tc);
                cur = gn;
            }
            bool last = (i == v->n_up - 1) && !v->l1_norm_final;
            float *nx = last ? out : bufs[flip];
            if (!last) flip ^= 1;
            convT1d(cur, nlc(D, Tc), v->upW[i], v->upB[i], nx, nlc(D, To), B, D, D, Tc, s, s);
            cur = nx; Tc = To;
        }
        if (Tc != L) fatal("learned up cascade yields length %d, expected %d", Tc, L);
        if (v->l1_norm_final) groupnorm(cur, nlc(D, Tc), out, nlc(D, Tc), B, 8, D, Tc);
        else if (cur != out) CUDA_CHECK(cudaMemcpyAsync(out, cur, (size_t)B * L * D * 4, cudaMemcpyDeviceToDevice, stream()));
    } else {
        interp_linear(q, nlc(D, tlen), out, nlc(D, L), B, D, tlen, L);
    }
    if (v->has_all && level >= 1 && level <= v->n_levels - 2 && v->urefW[level]) {
        conv1d(out, nlc(D, L), v->urefW[level], v->urefB[level], tmp1, nlc(D, L), B, D, D, L, 3, 1, 1, out, 0.f);
        CUDA_CHECK(cudaMemcpyAsync(out, tmp1, (size_t)B * L * D * 4, cudaMemcpyDeviceToDevice, stream()));
    }
}

// z [B][Lin][D] -> out [B][levels[level]][D]  (reference down_for_quant, src/vq.c:271-324)
static void down_for_quant_dev(VQState *v, const float *z, int B, int Lin, int level, float *out, float *tmp1, float *tmp2) {
    int D = v->D, tlen = v->levels[level];
    if (level == 0 && v->has_l1) {
        const float *cur = z;
        int Tc = Lin;
        float *bufs[2] = {tmp1, tmp2};
        int flip = 0;
        for (int i = 0; i < v->n_down; i++) {
            int s = v->downK[i], To = Tc / s;
            if (v->l1_norm && i > 0) {
                float *gn = bufs[flip]; flip ^= 1;
                groupnorm(cur, nlc(D, Tc), gn, nlc(D, Tc), B, 8, D, Tc);
                cur = gn;
            }
            bool last = (i == v->n_down - 1) && !v->l1_norm_final;
            float *nx = last ? out : bufs[flip];
            if (!last) flip ^= 1;
            conv1d(cur, nlc(D, Tc), v->downW[i], v->downB[i], nx, nlc(D, To), B, D, D, Tc, s, s, 0, nullptr, 0.f);
            cur = nx; Tc = To;
        }
        if (v->l1_norm_final) groupnorm(cur, nlc(D, Tc), out, nlc(D, Tc), B, 8, D, Tc);
        else if (cur != out) CUDA_CHECK(cudaMemcpyAsync(out, cur, (size_t)B * Tc * D * 4, cudaMemcpyDeviceToDevice, stream()));
    } else {
        interp_area(z, nlc(D, Lin), out, nlc(D, tlen), B, D, Lin, tlen);
    }
}
// the refining convolution of an inner level's quantizer input
static void down_refine_dev(VQState *v, int level, int B, float *out, float *tmp1) {
    int D = v->D, tlen = v->levels[level];
    conv1d(out, nlc(D, tlen), v->drefW[level], v->drefB[level], tmp1, nlc(D, tlen), B, D, D, tlen, 3, 1, 1, out, 0.f);
    CUDA_CHECK(cudaMemcpyAsync(out, tmp1, (size_t)B * tlen * D * 4, cudaMemcpyDeviceToDevice, stream()));
}

static int phi_index(const VQState *v, int level) {       // reference src/vq.c:212-221
    if (v->n_phi == 1) return 0;
    double at = (double)level / (v->n_levels - 1);
    int best = 0; double bd = 1e300;
    for (int j = 0; j < v->n_phi; j++) {
        double d = fabs(v->ticks[j] - at);
        if (d < bd) { bd = d; best = j; }
    }
    return best;
}

void vq_increment_dev(VQState *v, const int *codes_dev, int stride, int rowmod, int level, int B, float *up, float *scratch) {
    int D = v->D, L = v->L, tlen = v->levels[level];
    size_t n = (size_t)B * L * D;
    float *q = scratch, *t1 = scratch + n, *t2 = scratch + 2 * n, *t3 = scratch + 3 * n;
    {
        int64_t ng = (int64_t)B * tlen * D;
        ProfScope ps(NCMB_K_VQ);
        LAUNCH(k_gather_codes, ew(ng), 256, 0, v->E[level], codes_dev, stride, rowmod, tlen, D, v->vocabs[level], ng, q);
    }
    if (v->resi) {
        up_to_full_dev(v, q, B, tlen, level, t3, t1, t2);
        int j = phi_index(v, level);
        conv1d(t3, nlc(D, L), v->phiW[j], v->phiB[j], up, nlc(D, L), B, D, D, L, 3, 1, 1, t3, v->resi_ratio);
    } else {
        up_to_full_dev(v, q, B, tlen, level, up, t1, t2);
    }
}

size_t vq_scratch_floats(const VQState *v, int B) { return 4 * (size_t)B * v->L * v->D + 64; }

// dst = src + sign * (level's increment), next (optional) = dst at the length of the next level. `up` (B*L*D floats) and
// scratch (4 x that) are used by the increments that are not a plain interpolation of the codes.
static void level_step(VQState *v, const int *codes, int stride, int rowmod, int level, int B, const float *src, float *dst, float sign,
                       int tnext, float *next, float *up, float *scratch) {
    const int D = v->D, L = v->L;
    const bool refined = v->has_all && level >= 1 && level <= v->n_levels - 2 && v->urefW[level];
    // whole float4s: the rows' width, and where the caller's buffers start
    const bool tiles = next && L % tnext == 0, vec = D % 4 == 0 && (((uintptr_t)src | (uintptr_t)dst | (uintptr_t)(tiles ? next : nullptr)) & 15) == 0;
    // k_level_step's table of interpolation weights; without one (a level of one step, a finished increment) it needs none
    const bool flat = v->levels[level] == 1 || L == 1;
    const size_t table = flat ? 0 : (size_t)L * 16;
    const bool plain = !(level == 0 && v->has_l1) && !v->resi && !refined && vec && table <= 48 * 1024;
    if (!plain) vq_increment_dev(v, codes, stride, rowmod, level, B, up, scratch);
    if (!vec) {                                               // one pass per operation
        const size_t n = (size_t)B * L * D;
        if (src != dst) {
            if (src) CUDA_CHECK(cudaMemcpyAsync(dst, src, n * 4, cudaMemcpyDeviceToDevice, stream()));
            else CUDA_CHECK(cudaMemsetAsync(dst, 0, n * 4, stream()));
        }
        ProfScope ps(NCMB_K_VQ);
        LAUNCH(k_axpy_inplace, ew((int64_t)n), 256, 0, dst, up, sign, (int64_t)n);
    } else {
        LevelStep a{};
        a.E = v->E[level]; a.codes = codes; a.stride = stride; a.rowmod = rowmod; a.tlen = v->levels[level]; a.V = v->vocabs[level];
        a.up_in = plain ? nullptr : up; a.src = src; a.dst = dst; a.next = tiles ? next : nullptr;
        a.sign = sign; a.L = L; a.D = D; a.tnext = tiles ? tnext : L; a.n4 = (int64_t)B * a.tnext * (D / 4);
        ProfScope ps(NCMB_K_VQ);
        LAUNCH(k_level_step, ew(a.n4), 256, plain ? table : 0, a);
        if (tiles) return;
    }
    if (next) interp_area(dst, nlc(D, L), next, nlc(D, tnext), B, D, L, tnext);
}

void vq_next_input_dev(VQState *v, const int *codes_dev, int stride, int rowmod, int level, float *z_hat, float *x_out, int B, float *scratch) {
    float *up = scratch + 4 * (size_t)B * v->L * v->D;        // caller provides 5n floats
    level_step(v, codes_dev, stride, rowmod, level, B, z_hat, z_hat, 1.0f, v->levels[level + 1], x_out, up, scratch);
}

void vq_encode_dev(VQState *v, const float *z, int B, int *idx_dev, float *scratch) {
    if (B <= 0) return;
    const int D = v->D, L = v->L, total = vq_total_codes(v);
    const size_t n = (size_t)B * L * D;
    float *z_rest = scratch + 5 * n, *down = scratch + 6 * n, *up = scratch + 4 * n;   // caller provides 7n floats
    const float *cur = z;
    int off = 0;
    for (int lv = 0; lv < v->n_levels; lv++) {
        const int tlen = v->levels[lv];
        const bool refined = v->has_all && lv >= 1 && lv <= v->n_levels - 2 && v->drefW[lv];
        const float *q = down;
        if (lv == 0) down_for_quant_dev(v, cur, B, L, lv, down, scratch, scratch + n);
        else if (refined) down_refine_dev(v, lv, B, down, scratch);
        else if (tlen == L) q = cur;                          // the mean over one position is the position
        nearest_codes(q, v->E[lv], (int64_t)B * tlen, v->vocabs[lv], D, idx_dev, tlen, total, off);
        if (lv + 1 < v->n_levels) {
            const int tn = v->levels[lv + 1];
            const bool next_refined = v->has_all && lv + 1 <= v->n_levels - 2 && v->drefW[lv + 1];
            level_step(v, idx_dev + off, total, 0, lv, B, cur, z_rest, -1.0f, tn, tn == L && !next_refined ? nullptr : down, up, scratch);
            cur = z_rest;
        }
        off += tlen;
    }
}

void vq_zhat_final_dev(VQState *v, const int *idx_dev, int B, float *z_hat, float **snapshots, float *scratch) {
    int total = vq_total_codes(v);
    size_t n = (size_t)B * v->L * v->D;
    float *up = scratch + 4 * n;
    int base = 0;
    for (int lv = 0; lv < v->n_levels; lv++) {
        level_step(v, idx_dev + base, total, 0, lv, B, lv ? z_hat : nullptr, z_hat, 1.0f, v->L, nullptr, up, scratch);
        if (snapshots && snapshots[lv] && snapshots[lv] != z_hat)
            CUDA_CHECK(cudaMemcpyAsync(snapshots[lv], z_hat, n * 4, cudaMemcpyDeviceToDevice, stream()));
        base += v->levels[lv];
    }
}

int *vq_codes_to_dev(VQState *v, const int *host, size_t n) {
    v->codes_ws.reserve(n * sizeof(int) + 256);
    v->codes_ws.reset();
    int *d = v->codes_ws.get<int>(n);
    upload_queued(d, host, n * sizeof(int));
    return d;
}

} // namespace ncmb

using namespace ncmb;

extern "C" {

// binds codebooks, Phi convs, cascade stages and refine convs by name (reference src/vq.c:75-192)
VQState *vq_load(const NCMConfig *c, WeightStore *ws, const char *prefix) {
    ensure_device();
    VQState *v = new VQState();
    v->n_levels = c->n_qlevels;
    for (int i = 0; i < v->n_levels; i++) { v->levels[i] = c->levels[i]; v->vocabs[i] = c->vq_vocab[i]; }
    v->D = c->vq_embed_dim;
    v->L = c->levels[c->n_qlevels - 1];
    for (int i = 0; i < v->n_levels; i++) v->E[i] = wneed(ws, "%sembeddings.%d.weight", prefix, i)->data;
    v->resi = c->quant_resi_enabled && fabsf(c->quant_resi_ratio) > 1e-6f;
    v->resi_ratio = c->quant_resi_ratio;
    if (v->resi) {
        int sm = c->quant_resi_share_mode;
        v->n_phi = sm == 0 ? v->n_levels : (sm == 1 ? 1 : sm);
        for (int i = 0; i < v->n_phi; i++) {
            Tensor *w = wget(ws, "%squant_resi.%d.weight", prefix, i), *b = wget(ws, "%squant_resi.%d.bias", prefix, i);
            if (!w && v->n_phi == 1) w = wget(ws, "%squant_resi.weight", prefix);
            if (!b && v->n_phi == 1) b = wget(ws, "%squant_resi.bias", prefix);
            if (!w || !b) { fprintf(stderr, "missing weight %squant_resi.%d\n", prefix, i); exit(1); }
            v->phiW[i] = w->data; v->phiB[i] = b->data;
            v->ticks[i] = (v->n_phi == 4) ? (i + 1.0 / 3.0) / v->n_phi : (i + 0.5) / v->n_phi;
        }
    }
    if (c->learned_l1_sampling) {
        v->has_l1 = 1; v->l1_norm = c->learned_l1_norm; v->l1_norm_final = c->learned_l1_norm_final;
        for (int s = 0; s < 16; s++) {
            Tensor *t = wget(ws, "%slearned_down_l1.%d.weight", prefix, s);
            if (t) {
                v->downW[v->n_down] = t->data; v->downK[v->n_down] = (int)t->shape[2];
                v->downB[v->n_down] = wneed(ws, "%slearned_down_l1.%d.bias", prefix, s)->data;
                v->n_down++;
            }
            t = wget(ws, "%slearned_up_l1.%d.weight", prefix, s);
            if (t) {
                v->upW[v->n_up] = t->data; v->upK[v->n_up] = (int)t->shape[2];
                v->upB[v->n_up] = wneed(ws, "%slearned_up_l1.%d.bias", prefix, s)->data;
                v->n_up++;
            }
        }
        if (!v->n_down) { fprintf(stderr, "learned_l1 weights missing\n"); exit(1); }
    }
    if (c->learned_all_sampling) {
        v->has_all = 1;
        for (int i = 1; i <= v->n_levels - 2; i++) {
            Tensor *t = wget(ws, "%slearned_down_refine.%d.weight", prefix, i);
            if (t) { v->drefW[i] = t->data; v->drefB[i] = wneed(ws, "%slearned_down_refine.%d.bias", prefix, i)->data; }
            t = wget(ws, "%slearned_up_refine.%d.weight", prefix, i);
            if (t) { v->urefW[i] = t->data; v->urefB[i] = wneed(ws, "%slearned_up_refine.%d.bias", prefix, i)->data; }
        }
    }
    return v;
}

void vq_free(VQState *vq) {
    if (!vq) return;
    vq->work.release(); vq->codes_ws.release();
    delete vq;
}
int vq_total_codes(const VQState *vq) { int s = 0; for (int i = 0; i < vq->n_levels; i++) s += vq->levels[i]; return s; }
int vq_nlevels(const VQState *vq) { return vq->n_levels; }
int vq_level_len(const VQState *vq, int k) { return vq->levels[k]; }
int vq_level_V(const VQState *vq, int k) { return vq->vocabs[k]; }
int vq_Ltotal(const VQState *vq) { return vq->L; }
int vq_Ddim(const VQState *vq) { return vq->D; }

static float *vq_scratch(VQState *vq, int B, int mult) {
    size_t n = (size_t)B * vq->L * vq->D;
    vq->work.reserve((mult * n + 1024) * sizeof(float));
    vq->work.reset();
    return vq->work.get<float>(mult * n);
}

void vq_next_input(VQState *vq, const int *codes, int level_idx, float *z_hat, float *x_out, int B) {
    int *cd = vq_codes_to_dev(vq, codes, (size_t)B * vq->levels[level_idx]);
    vq_next_input_dev(vq, cd, vq->levels[level_idx], 0, level_idx, z_hat, x_out, B, vq_scratch(vq, B, 5));
}

void vq_idx_to_zhats(VQState *vq, const int *idx, int B, float **zhats) {
    int *cd = vq_codes_to_dev(vq, idx, (size_t)B * vq_total_codes(vq));
    float *scr = vq_scratch(vq, B, 6);
    float *zh = scr + 5 * (size_t)B * vq->L * vq->D;
    vq_zhat_final_dev(vq, cd, B, zh, zhats, scr);
}

void vq_z_to_idx(VQState *vq, const float *z, int B, int *idx) {
    int total = vq_total_codes(vq);
    vq->codes_ws.reserve((size_t)B * total * sizeof(int) + 256);
    vq->codes_ws.reset();
    int *idx_dev = vq->codes_ws.get<int>((size_t)B * total);
    vq_encode_dev(vq, z, B, idx_dev, vq_scratch(vq, B, 7));
    mem_d2h(idx, idx_dev, (size_t)B * total * sizeof(int));
}

// idx [B][total] -> teacher-forcing input [B][T][D] (reference src/vq.c:601-674)
void vq_idx_to_ncm_input(VQState *vq, const int *idx, int B, float *x_out) {
    int D = vq->D, L = vq->L, total = vq_total_codes(vq), T = total - vq->levels[0];
    size_t n = (size_t)B * L * D;
    int *cd = vq_codes_to_dev(vq, idx, (size_t)B * total);
    float *scr = vq_scratch(vq, B, 7);
    float *up = scr + 4 * n, *z_hat = scr + 5 * n, *chunk = scr + 6 * n;
    int base = 0, off = 0;
    for (int li = 0; li < vq->n_levels - 1; li++) {
        int nlen = vq->levels[li + 1];
        level_step(vq, cd + base, total, 0, li, B, li ? z_hat : nullptr, z_hat, 1.0f, nlen, chunk, up, scr);
        CUDA_CHECK(cudaMemcpy2DAsync(x_out + (size_t)off * D, (size_t)T * D * 4, chunk, (size_t)nlen * D * 4,
                                     (size_t)nlen * D * 4, B, cudaMemcpyDeviceToDevice, stream()));
        base += vq->levels[li]; off += nlen;
    }
}

void ncmb_vq_encode_dev(VQState *vq, const float *z_dev, int B, int *idx_dev) {
    vq_encode_dev(vq, z_dev, B, idx_dev, vq_scratch(vq, B, 7));
}
void ncmb_vq_nearest_dev(VQState *vq, int level, const float *x_dev, long long n, int *idx_dev) {
    ensure_device();
    nearest_codes(x_dev, vq->E[level], n, vq->vocabs[level], vq->D, idx_dev, 1, 1, 0);
}

} // extern "C"
