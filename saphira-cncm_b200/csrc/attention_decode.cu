// Few-query attention: ONE query per sequence row against that row's K/V cache (the decoder-LM token loop,
// reference src/gpt2.c:92 / src/qwen.c:121 run with a KV cache instead of recomputing), or up to four queries
// per row against the cached prefix plus the row's own new tokens (the first levels of the NCP generate,
// reference src/ncp.c:990: level sizes 1 and 4).
//
// With one query there is nothing to tile over queries, so the keys are split instead: one CTA per
// (32-key chunk, kv head, row) computes the chunk's scores for every query head that shares the kv
// head (K and V are read once per group), a local softmax and the partial context, and writes
// (max, sum, context[hd]) per head to scratch. The last CTA of a (row, kv head) to finish -- an
// atomic counter tells it -- merges the partials with the usual log-sum-exp rescaling and writes the
// context row. A batch-1, 12-head step with 300 cached keys thus runs on ~120 CTAs instead of 12. With many
// rows a CTA takes several consecutive chunks (running maximum and sum), and a CTA that sees all keys of its
// row writes the context directly.
//
// step_d: optional device counter. When set, row lengths are read from k1_len + (*step_d) * len_step,
// so one captured CUDA graph serves every decode step.
#include "common.cuh"
#include "split.cuh"
#include "gemm_few.cuh"

#include <algorithm>

namespace ncmb {

// programmatic dependent launch (see launch_pdl) of clusters of nc CTAs along x
template <typename... KArgs, typename... Args>
static void launch_pdl_cluster(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, int nc, Args... args) {
    static const bool off = getenv("NCM_B200_NO_PDL") != nullptr;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream();
    cudaLaunchAttribute at[2];
    int n = 0;
    if (nc > 1) { at[n].id = cudaLaunchAttributeClusterDimension; at[n].val.clusterDim.x = (unsigned)nc; at[n].val.clusterDim.y = 1; at[n].val.clusterDim.z = 1; n++; }
    if (!off) { at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[n].val.programmaticStreamSerializationAllowed = 1; n++; }
    cfg.attrs = at; cfg.numAttrs = n;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
    if (e != cudaSuccess) fatal("decode attention: launch failed: %s", cudaGetErrorString(e));
    ctx().launches++;
}

constexpr int AD_KEYS = 32, AD_THREADS = 128, AD_MAXSPLIT = 64;   // up to 2048 keys per row
constexpr int AD_MAXG = 16;        // (query, head) pairs of one kv group handled together: G * queries per row <= 16

struct AttnDecDev {
    const float *q; int64_t ldq;
    const float *k, *v; int64_t ldk;
    const float *k2, *v2; int64_t ldk2; const int *k2_start;      // optional second key segment (this pass's own tokens)
    float *out; float *out_lo; int out_fmt; int64_t ldo;
    const int *q_start, *k_start, *k_len;
    const int *step_d; int64_t len_step;
    int H, Hkv, rows, max_split, cps;
    float scale;
    float *part; unsigned *count;
};

// GM: compile-time bound on the (query, head) pairs of a kv group (1, 4, 8 or 16). Every loop over them is unrolled
// to GM, so a one-head-per-kv-head model (GPT-2) does not issue the 16-wide context step of a grouped one.
template <int HD, int GM>
__global__ void __launch_bounds__(AD_THREADS) k_attention_decode(AttnDecDev a) {
    constexpr int DP = HD / 4;                         // dims per thread in the score step (4 threads per key)
    constexpr int QP = DP + 4;                         // pitch of a quarter in qs: the four quarters land in distinct banks
    constexpr int GROUPS = AD_THREADS / HD > 0 ? AD_THREADS / HD : 1;   // key groups in the PV step
    constexpr int KPG = AD_KEYS / GROUPS;
    __shared__ __align__(16) float qs[GM][4 * QP];
    __shared__ __align__(16) float sc[AD_KEYS][GM];    // scores, then probabilities, of the chunk: [key][head]
    __shared__ float red[GROUPS][GM][HD];
    __shared__ float mg[GM], lg[GM], alpha[GM];
    __shared__ int s_last;
    const int row = blockIdx.z, kvh = blockIdx.y, sp = blockIdx.x;
    const int Gh = a.H / a.Hkv;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_launch_dependents();          // programmatic dependent launch: the successor may start launching now,
    pdl_wait();                       // and nothing the predecessor wrote is read before this point
    const int *lens = a.k_len ? a.k_len + (a.step_d ? (int64_t)(*a.step_d) * a.len_step : 0) : nullptr;
    const int k00 = a.k_start[row], n1s = lens ? lens[row] : a.k_start[row + 1] - k00;
    const int k20 = a.k2_start ? a.k2_start[row] : 0, n2s = a.k2_start ? a.k2_start[row + 1] - k20 : 0;
    const int n1 = n1s + n2s;                          // keys of both segments, segment 1 first
    const int nchunks = (n1 + AD_KEYS - 1) / AD_KEYS;
    const int nsplit = (nchunks + a.cps - 1) / a.cps;   // CTAs that share the row's keys, cps 32-key chunks each
    if (sp >= nsplit) return;
    const int k0 = sp * a.cps * AD_KEYS;
    const int nch = min(a.cps, nchunks - sp * a.cps);
    const int q0 = a.q_start[row], nq = a.q_start[row + 1] - q0;
    const int G = Gh * nq;                             // virtual heads: vh = g * nq + qi
    // row pointer of key j of the row (either segment)
    auto krow = [&](int j) -> const float * {
        return j < n1s ? a.k + (int64_t)(k00 + j) * a.ldk : a.k2 + (int64_t)(k20 + j - n1s) * a.ldk2;
    };
    auto vrow = [&](int j) -> const float * {
        return j < n1s ? a.v + (int64_t)(k00 + j) * a.ldk : a.v2 + (int64_t)(k20 + j - n1s) * a.ldk2;
    };

    for (int i = tid; i < G * HD; i += AD_THREADS) {
        int vh = i / HD, d = i % HD;
        qs[vh][(d / DP) * QP + d % DP] = a.q[(int64_t)(q0 + vh % nq) * a.ldq + (kvh * Gh + vh / nq) * HD + d];
    }
    if (tid < GM) { mg[tid] = -INFINITY; lg[tid] = 0.f; alpha[tid] = 0.f; }
    for (int i = tid; i < AD_KEYS * GM; i += AD_THREADS) (&sc[0][0])[i] = 0.f;     // heads past G stay 0 in the context step
    // The CTA walks its cps chunks with a running maximum / sum per head (the usual rescaling when the maximum
    // grows). Loads run ahead of the arithmetic: the V elements of a chunk are requested before its scores are
    // formed, the K rows of the next chunk before the softmax of this one.
    const int sj = tid >> 2, spart = tid & 3;             // score step: four threads per key, a quarter of the head dim each
    const int grp = tid / HD, d = tid % HD;               // context step: thread = (key group, dim)
    float kr[DP];
    auto load_k = [&](int kbase) {
        if (kbase + sj < n1) {
            const float4 *kp = (const float4 *)(krow(kbase + sj) + kvh * HD + spart * DP);
#pragma unroll
            for (int i = 0; i < DP / 4; i++) { float4 t = kp[i]; kr[4 * i] = t.x; kr[4 * i + 1] = t.y; kr[4 * i + 2] = t.z; kr[4 * i + 3] = t.w; }
        } else {
#pragma unroll
            for (int i = 0; i < DP; i++) kr[i] = 0.f;
        }
    };
    float acc[GM];
#pragma unroll
    for (int g = 0; g < GM; g++) acc[g] = 0.f;
    load_k(k0);
    __syncthreads();
    for (int c = 0; c < nch; c++) {
        const int kb = k0 + c * AD_KEYS;
        float vr[KPG];                                   // all V loads of this thread in flight together
        if (grp < GROUPS) {
            if (kb + AD_KEYS <= n1s) {                    // the whole chunk lies in the first segment: one base, fixed strides
                const float *vb = a.v + (int64_t)(k00 + kb + grp * KPG) * a.ldk + kvh * HD + d;
#pragma unroll
                for (int jj = 0; jj < KPG; jj++) vr[jj] = vb[(int64_t)jj * a.ldk];
            } else {
#pragma unroll
                for (int jj = 0; jj < KPG; jj++) {
                    const int j = grp * KPG + jj;
                    vr[jj] = (kb + j < n1) ? vrow(kb + j)[kvh * HD + d] : 0.f;
                }
            }
        }
        {   // scores of the chunk
            const bool valid = kb + sj < n1;
#pragma unroll
            for (int g = 0; g < GM; g++) {
                if (g < G) {                              // warp-uniform
                    const float4 *qp = (const float4 *)&qs[g][spart * QP];
                    float dot = 0.f;
#pragma unroll
                    for (int i = 0; i < DP / 4; i++) {
                        const float4 t = qp[i];
                        dot = fmaf(kr[4 * i], t.x, dot); dot = fmaf(kr[4 * i + 1], t.y, dot);
                        dot = fmaf(kr[4 * i + 2], t.z, dot); dot = fmaf(kr[4 * i + 3], t.w, dot);
                    }
                    dot += __shfl_xor_sync(0xffffffffu, dot, 1);
                    dot += __shfl_xor_sync(0xffffffffu, dot, 2);
                    if (spart == 0) sc[sj][g] = valid ? dot * a.scale : -INFINITY;
                }
            }
        }
        if (c + 1 < nch) load_k(kb + AD_KEYS);
        __syncthreads();
        for (int g = warp; g < G; g += AD_THREADS / 32) {   // chunk softmax against the running maximum, one warp per head
            float s = sc[lane][g];
            float m = s;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            const float mold = mg[g];
            m = fmaxf(m, mold);
            float p = (s == -INFINITY) ? 0.f : expf(s - m);
            float l = p;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
            sc[lane][g] = p;
            __syncwarp();
            if (lane == 0) {
                const float al = (mold == -INFINITY) ? 0.f : expf(mold - m);
                alpha[g] = al; mg[g] = m; lg[g] = fmaf(lg[g], al, l);
            }
        }
        __syncthreads();
        if (grp < GROUPS) {
#pragma unroll
            for (int g = 0; g < GM; g++) acc[g] *= alpha[g];
#pragma unroll
            for (int jj = 0; jj < KPG; jj++) {
                const int j = grp * KPG + jj;
                if constexpr (GM % 4 == 0) {
#pragma unroll
                    for (int g4 = 0; g4 < GM / 4; g4++) {
                        const float4 pr = *(const float4 *)&sc[j][4 * g4];     // the same address for the whole warp: a broadcast
                        acc[4 * g4] = fmaf(pr.x, vr[jj], acc[4 * g4]); acc[4 * g4 + 1] = fmaf(pr.y, vr[jj], acc[4 * g4 + 1]);
                        acc[4 * g4 + 2] = fmaf(pr.z, vr[jj], acc[4 * g4 + 2]); acc[4 * g4 + 3] = fmaf(pr.w, vr[jj], acc[4 * g4 + 3]);
                    }
                } else {
#pragma unroll
                    for (int g = 0; g < GM; g++) acc[g] = fmaf(sc[j][g], vr[jj], acc[g]);
                }
            }
        }
        __syncthreads();                                  // sc and alpha are rewritten by the next chunk
    }
    if (grp < GROUPS) {
#pragma unroll
        for (int g = 0; g < GM; g++) red[grp][g][d] = acc[g];
    }
    __syncthreads();
    if (nsplit == 1) {                                    // the CTA saw every key of the row: no partials, no merge
        for (int i = tid; i < G * HD; i += AD_THREADS) {
            int g = i / HD, dd = i % HD;
            float o = 0.f;
#pragma unroll
            for (int r = 0; r < GROUPS; r++) o += red[r][g][dd];
            const float L = lg[g];
            const float r = L > 0.f ? o / L : 0.f;
            const int64_t at = (int64_t)(q0 + g % nq) * a.ldo + (kvh * Gh + g / nq) * HD + dd;
            if (a.out_lo) store_split1(a.out, a.out_lo, at, r, a.out_fmt);
            else a.out[at] = r;
        }
        return;
    }
    float *mine = a.part + ((int64_t)(row * a.Hkv + kvh) * a.max_split + sp) * AD_MAXG * (HD + 2);
    for (int i = tid; i < G * HD; i += AD_THREADS) {
        int g = i / HD, d = i % HD;
        float o = 0.f;
#pragma unroll
        for (int r = 0; r < GROUPS; r++) o += red[r][g][d];
        mine[g * (HD + 2) + 2 + d] = o;
        if (d == 0) { mine[g * (HD + 2)] = mg[g]; mine[g * (HD + 2) + 1] = lg[g]; }
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        unsigned old = atomicAdd(a.count + row * a.Hkv + kvh, 1u);
        s_last = (old == (unsigned)(nsplit - 1));
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // merge: the chunk partials of this (row, kv head), read through L2. Maxima and sums first (one load per
    // thread, all in flight together), then the rescaling weights once per head, then the context columns
    // with independent loads -- a chain of dependent L2 round trips per split would dominate the kernel.
    __shared__ float wsm[AD_MAXSPLIT][GM], lsm[AD_MAXSPLIT][GM], Lg[GM];
    const float *base = a.part + (int64_t)(row * a.Hkv + kvh) * a.max_split * AD_MAXG * (HD + 2);
    for (int i = tid; i < nsplit * G; i += AD_THREADS) {
        int s = i / G, g = i % G;
        const float *ps = base + ((int64_t)s * AD_MAXG + g) * (HD + 2);
        wsm[s][g] = __ldcg(ps); lsm[s][g] = __ldcg(ps + 1);
    }
    __syncthreads();
    if (tid < G) {
        float M = -INFINITY, L = 0.f;
        for (int s = 0; s < nsplit; s++) M = fmaxf(M, wsm[s][tid]);
        for (int s = 0; s < nsplit; s++) { float w = expf(wsm[s][tid] - M); wsm[s][tid] = w; L = fmaf(lsm[s][tid], w, L); }
        Lg[tid] = L;
    }
    __syncthreads();
    for (int i = tid; i < G * HD; i += AD_THREADS) {
        int g = i / HD, d = i % HD;
        float O = 0.f;
        int s = 0;
        for (; s + 4 <= nsplit; s += 4) {
            float o0 = __ldcg(base + ((int64_t)(s + 0) * AD_MAXG + g) * (HD + 2) + 2 + d);
            float o1 = __ldcg(base + ((int64_t)(s + 1) * AD_MAXG + g) * (HD + 2) + 2 + d);
            float o2 = __ldcg(base + ((int64_t)(s + 2) * AD_MAXG + g) * (HD + 2) + 2 + d);
            float o3 = __ldcg(base + ((int64_t)(s + 3) * AD_MAXG + g) * (HD + 2) + 2 + d);
            O = fmaf(o0, wsm[s][g], O); O = fmaf(o1, wsm[s + 1][g], O); O = fmaf(o2, wsm[s + 2][g], O); O = fmaf(o3, wsm[s + 3][g], O);
        }
        for (; s < nsplit; s++) O = fmaf(__ldcg(base + ((int64_t)s * AD_MAXG + g) * (HD + 2) + 2 + d), wsm[s][g], O);
        const float L = Lg[g];
        const float r = L > 0.f ? O / L : 0.f;
        const int64_t at = (int64_t)(q0 + g % nq) * a.ldo + (kvh * Gh + g / nq) * HD + d;
        if (a.out_lo) store_split1(a.out, a.out_lo, at, r, a.out_fmt);
        else a.out[at] = r;
    }
    if (tid == 0) a.count[row * a.Hkv + kvh] = 0;          // ready for the next launch
}

// ---- head dim 64, up to eight (query, head) pairs per kv head: lanes share keys, loads straight to registers ----
// LPK lanes hold a key: with sixteen (more than four pairs) a lane keeps four dims, with eight it keeps eight, of the key, of
// the query (in registers for all GM pairs) and of the context (accumulated in registers); a warp's loads are full 128-byte
// lines. The partial dot products of a key meet by a reduce-scatter that leaves one pair's score in a lane (eight shuffles for
// eight pairs), the softmax runs on those, and the probabilities travel back by one shuffle per pair and key. Nothing goes
// between lanes through shared memory until a warp's keys are done. A warp takes runs of four loads (8 or 16 keys); each lane
// keeps the loads of its next runs in flight with cp.async into slots of its own (a longer register file, no
// barrier): holding a run ahead in registers left 48 KB in flight per SM and a third of the bandwidth. The CTAs of a cluster share the keys of a (row, kv head) pair,
// their warps interleaving runs, and merge over distributed shared memory.
//
// FUSED (decode steps): q, k and v of the new token arrive as the slices of the QKV product. Every CTA adds what its heads
// need, rotates it, keeps the new key and value in shared memory and the first CTA of the cluster appends them to the cache.
// The cached keys and values of a warp's first run are requested before the kernel waits for that product; the reduce_norm
// kernel in front of the product starts its successor only after its own wait, so the cache and the step counter are final.
//
// Bound: the K|V cache read once; for few rows the chain product -> sums -> scores -> merge.
constexpr int ADG_NI = 4;              // loads of a run per lane
constexpr int adg_depth(int GM) { return GM > 4 ? 3 : 2; }   // runs in flight per warp, the current one included (12 or 16 KB per warp)
constexpr int ADG_MAXW = 4;            // warps of a CTA at most
constexpr int ADG_MAXC = 8;            // CTAs of a cluster at most

struct AttnFused {                     // see FewQkv: slices of the QKV product of a decode step, one token per row
    const float *part; int S; const float *bias;
    const float *cos_t, *sin_t; const int *pos; int64_t pos_step;
    float *kv; int64_t seq_pitch, step;      // cache position of the new token: kv + row * seq_pitch + *step_d * step, k | v of all kv heads
};

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool on) {      // off: the slot is zeroed
    const int n = on ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
// a slot holds NI loads of keys and NI of values per lane, 16 bytes each (twice where a lane keeps eight dims)
constexpr size_t adg_smem(int GM, int nw) { return (size_t)nw * adg_depth(GM) * 2 * ADG_NI * (GM > 4 ? 1 : 2) * 512; }

__device__ __forceinline__ float ld_cluster(const float *p, unsigned rank) {
    uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(r) : "memory");
    return v;
}

template <int GM, bool FUSED>
__global__ void __launch_bounds__(ADG_MAXW * 32) k_attention_dec_gqa(AttnDecDev a, AttnFused f) {
    extern __shared__ __align__(16) float4 adg_ring[];
    constexpr int HD = 64, LPK = GM > 4 ? 16 : 8, DPL = HD / LPK, NF = DPL / 4, KPI = 32 / LPK, NI = ADG_NI, RUN = NI * KPI, DEPTH = adg_depth(GM);
    constexpr int LOG = GM == 8 ? 3 : GM == 4 ? 2 : GM == 2 ? 1 : 0, HSH = (LPK == 16 ? 4 : 3) - LOG;   // lane dp holds pair dp >> HSH
    __shared__ float pm[ADG_MAXW][GM], pl[ADG_MAXW][GM], wg[ADG_MAXW][GM];
    __shared__ __align__(16) float po[ADG_MAXW][GM][HD];
    __shared__ __align__(16) float co[GM][HD];               // the CTA's context, maximum and sum, read by the cluster
    __shared__ float cm[GM], cl[GM], cw[ADG_MAXC][GM];
    __shared__ __align__(16) float qn[FUSED ? GM + 2 : 1][HD];   // the new token's queries, key, value
    const int rank = blockIdx.x, nc = gridDim.x;             // one cluster per (row, kv head)
    const int row = blockIdx.z, kvh = blockIdx.y;
    const int Gh = a.H / a.Hkv;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
    const int kg = lane / LPK, dp = lane % LPK;
    pdl_launch_dependents();
    if (!FUSED) pdl_wait();
    const int64_t st = a.step_d ? (int64_t)*a.step_d : 0;
    const int *lens = a.k_len ? a.k_len + st * a.len_step : nullptr;
    const int k00 = a.k_start[row], n1s = lens ? lens[row] : a.k_start[row + 1] - k00;
    const int k20 = a.k2_start ? a.k2_start[row] : 0, n2s = a.k2_start ? a.k2_start[row + 1] - k20 : 0;
    const int n1 = n1s + n2s, cached = FUSED ? n1 - 1 : n1;
    const int q0 = a.q_start[row], nq = FUSED ? 1 : a.q_start[row + 1] - q0;
    const int G = Gh * nq;                                   // virtual heads: vh = g * nq + qi
    const int first = (warp * nc + rank) * RUN, step = nw * nc * RUN;
    float4 *ring = adg_ring + (size_t)warp * DEPTH * 2 * NI * NF * 32 + lane;        // [slot][keys | values][load][half][lane]
    // dims of a lane: 4 dp .. (and 32 + 4 dp .. where it holds eight)
    int jl = first;                                          // first key of the next run to request
    auto request = [&](int slot) {
        float4 *dst = ring + slot * 2 * NI * NF * 32;
        if (jl < n1) {                                       // (positions without a cached key are zeroed)
#pragma unroll
            for (int i = 0; i < NI; i++) {
                const int j = jl + KPI * i + kg;
                const bool on = j < cached, seg1 = j < n1s;
                const int64_t at = on ? (seg1 ? (int64_t)(k00 + j) * a.ldk : (int64_t)(k20 + j - n1s) * a.ldk2) + kvh * HD + 4 * dp : 0;
                const float *kp = seg1 || !on ? a.k : a.k2, *vp = seg1 || !on ? a.v : a.v2;
#pragma unroll
                for (int h = 0; h < NF; h++) {
                    cp_async16(smem_addr(dst + (i * NF + h) * 32), kp + at + 32 * h, on);
                    cp_async16(smem_addr(dst + ((NI + i) * NF + h) * 32), vp + at + 32 * h, on);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        jl += step;
    };
#pragma unroll
    for (int r = 0; r < DEPTH - 1; r++) request(r);
    if constexpr (FUSED) {
        const int Wq = (a.H + 2 * a.Hkv) * HD;
        const int64_t rot = f.cos_t ? (int64_t)f.pos[st * f.pos_step + row] * HD : 0;
        pdl_wait();
        for (int it = tid; it < (Gh + 2) * 8; it += blockDim.x) {            // four rotation pairs (d, d + 32) each
            const int hh = it >> 3, d = (it & 7) * 4;
            const int h = hh < Gh ? kvh * Gh + hh : (hh == Gh ? a.H + kvh : a.H + a.Hkv + kvh);
            const float *p = f.part + (int64_t)row * Wq + h * HD + d;
            const int64_t ps = (int64_t)a.rows * Wq;
            float4 v0 = make_float4(0.f, 0.f, 0.f, 0.f), v1 = v0;
            for (int s = 0; s < f.S; s += 8) {
                float4 t0[8], t1[8];
#pragma unroll
                for (int u = 0; u < 8; u++)
                    if (s + u < f.S) { t0[u] = __ldcg((const float4 *)(p + (s + u) * ps)); t1[u] = __ldcg((const float4 *)(p + (s + u) * ps + HD / 2)); }
#pragma unroll
                for (int u = 0; u < 8; u++)
                    if (s + u < f.S) {
                        v0.x += t0[u].x; v0.y += t0[u].y; v0.z += t0[u].z; v0.w += t0[u].w;
                        v1.x += t1[u].x; v1.y += t1[u].y; v1.z += t1[u].z; v1.w += t1[u].w;
                    }
            }
            if (f.bias) {
                const float4 b0 = __ldg((const float4 *)(f.bias + h * HD + d)), b1 = __ldg((const float4 *)(f.bias + h * HD + d + HD / 2));
                v0.x += b0.x; v0.y += b0.y; v0.z += b0.z; v0.w += b0.w;
                v1.x += b1.x; v1.y += b1.y; v1.z += b1.z; v1.w += b1.w;
            }
            if (f.cos_t && hh <= Gh) {
                const float4 c0 = *(const float4 *)(f.cos_t + rot + d), c1 = *(const float4 *)(f.cos_t + rot + d + HD / 2);
                const float4 s0 = *(const float4 *)(f.sin_t + rot + d), s1 = *(const float4 *)(f.sin_t + rot + d + HD / 2);
                auto turn = [](float &x, float &y, float ca, float sa, float cb, float sb) {
                    const float y0 = __fadd_rn(__fmul_rn(x, ca), __fmul_rn(-y, sa)), y1 = __fadd_rn(__fmul_rn(y, cb), __fmul_rn(x, sb));
                    x = y0; y = y1;
                };
                turn(v0.x, v1.x, c0.x, s0.x, c1.x, s1.x); turn(v0.y, v1.y, c0.y, s0.y, c1.y, s1.y);
                turn(v0.z, v1.z, c0.z, s0.z, c1.z, s1.z); turn(v0.w, v1.w, c0.w, s0.w, c1.w, s1.w);
            }
            const int slot = hh < Gh ? hh : GM + hh - Gh;
            *(float4 *)&qn[slot][d] = v0; *(float4 *)&qn[slot][d + HD / 2] = v1;
            if (hh >= Gh && rank == 0) {
                float *kv = f.kv + (int64_t)row * f.seq_pitch + st * f.step + (h - a.H) * HD + d;
                *(float4 *)kv = v0; *(float4 *)(kv + HD / 2) = v1;
            }
        }
        __syncthreads();
    }
    float q[GM][DPL];
#pragma unroll
    for (int g = 0; g < GM; g++)
#pragma unroll
        for (int h = 0; h < NF; h++) {
            float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
            if (g < G) {
                if (FUSED) t = *(const float4 *)&qn[FUSED ? g : 0][4 * dp + 32 * h];
                else t = *(const float4 *)(a.q + (int64_t)(q0 + g % nq) * a.ldq + (kvh * Gh + g / nq) * HD + 4 * dp + 32 * h);
            }
            q[g][4 * h] = t.x * a.scale; q[g][4 * h + 1] = t.y * a.scale; q[g][4 * h + 2] = t.z * a.scale; q[g][4 * h + 3] = t.w * a.scale;
        }
    float acc[GM][DPL], m = -INFINITY, l = 0.f;
#pragma unroll
    for (int g = 0; g < GM; g++)
#pragma unroll
        for (int d = 0; d < DPL; d++) acc[g][d] = 0.f;
    int slot = 0;
    for (int j0 = first; j0 < n1; j0 += step) {
        request((slot + DEPTH - 1) % DEPTH);
        asm volatile("cp.async.wait_group %0;" ::"n"(DEPTH - 1) : "memory");
        float4 kf[NI][NF], vf[NI][NF];
#pragma unroll
        for (int i = 0; i < NI; i++)
#pragma unroll
            for (int h = 0; h < NF; h++) kf[i][h] = ring[(slot * 2 * NI * NF + i * NF + h) * 32];
        if constexpr (FUSED) {                                // the new token's key and value
#pragma unroll
            for (int i = 0; i < NI; i++)
                if (j0 + KPI * i + kg == cached) {
#pragma unroll
                    for (int h = 0; h < NF; h++) kf[i][h] = *(const float4 *)&qn[GM][4 * dp + 32 * h];
                }
        }
        float s[NI];
#pragma unroll
        for (int i = 0; i < NI; i++) {
            float v[GM];
#pragma unroll
            for (int g = 0; g < GM; g++) {
                float t = 0.f;
#pragma unroll
                for (int h = 0; h < NF; h++) {
                    t = fmaf(q[g][4 * h], kf[i][h].x, t); t = fmaf(q[g][4 * h + 1], kf[i][h].y, t);
                    t = fmaf(q[g][4 * h + 2], kf[i][h].z, t); t = fmaf(q[g][4 * h + 3], kf[i][h].w, t);
                }
                v[g] = t;
            }
            int o = LPK / 2;
#pragma unroll
            for (int w = GM / 2; w > 0; w >>= 1, o >>= 1) {   // halve the pairs a lane keeps
                const bool up = (dp & o) != 0;
#pragma unroll
                for (int g = 0; g < w; g++) {
                    const float give = up ? v[g] : v[g + w], keep = up ? v[g + w] : v[g];
                    v[g] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
            }
#pragma unroll
            for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
            s[i] = (j0 + KPI * i + kg < n1) ? v[0] : -INFINITY;
        }
#pragma unroll
        for (int i = 0; i < NI; i++)
#pragma unroll
            for (int h = 0; h < NF; h++) {
                vf[i][h] = ring[(slot * 2 * NI * NF + (NI + i) * NF + h) * 32];
                if (FUSED && j0 + KPI * i + kg == cached) vf[i][h] = *(const float4 *)&qn[FUSED ? GM + 1 : 0][4 * dp + 32 * h];
            }
        float mx = m;
#pragma unroll
        for (int i = 0; i < NI; i++) mx = fmaxf(mx, s[i]);
#pragma unroll
        for (int o = LPK; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));   // a run has at least one key: finite
        const float al = m == -INFINITY ? 0.f : expf(m - mx);
        l *= al;
        m = mx;
#pragma unroll
        for (int i = 0; i < NI; i++) { s[i] = expf(s[i] - m); l += s[i]; }
        if (__any_sync(0xffffffffu, al != 1.0f)) {
#pragma unroll
            for (int g = 0; g < GM; g++) {
                const float r = __shfl_sync(0xffffffffu, al, g << HSH);
#pragma unroll
                for (int d = 0; d < DPL; d++) acc[g][d] *= r;
            }
        }
#pragma unroll
        for (int i = 0; i < NI; i++) {
#pragma unroll
            for (int g = 0; g < GM; g++) {
                const float p = __shfl_sync(0xffffffffu, s[i], (lane & ~(LPK - 1)) | (g << HSH));
#pragma unroll
                for (int h = 0; h < NF; h++) {
                    acc[g][4 * h] = fmaf(p, vf[i][h].x, acc[g][4 * h]); acc[g][4 * h + 1] = fmaf(p, vf[i][h].y, acc[g][4 * h + 1]);
                    acc[g][4 * h + 2] = fmaf(p, vf[i][h].z, acc[g][4 * h + 2]); acc[g][4 * h + 3] = fmaf(p, vf[i][h].w, acc[g][4 * h + 3]);
                }
            }
        }
        slot = (slot + 1) % DEPTH;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    // the key groups of the warp, then the warps, then the CTAs of the cluster
#pragma unroll
    for (int o = LPK; o < 32; o <<= 1) {
        l += __shfl_xor_sync(0xffffffffu, l, o);
#pragma unroll
        for (int g = 0; g < GM; g++)
#pragma unroll
            for (int d = 0; d < DPL; d++) acc[g][d] += __shfl_xor_sync(0xffffffffu, acc[g][d], o);
    }
    if (kg == 0) {
        if ((dp & ((1 << HSH) - 1)) == 0) { pm[warp][dp >> HSH] = m; pl[warp][dp >> HSH] = l; }
#pragma unroll
        for (int g = 0; g < GM; g++)
#pragma unroll
            for (int h = 0; h < NF; h++)
                *(float4 *)&po[warp][g][4 * dp + 32 * h] = make_float4(acc[g][4 * h], acc[g][4 * h + 1], acc[g][4 * h + 2], acc[g][4 * h + 3]);
    }
    __syncthreads();
    if (tid < G) {
        float M = -INFINITY, L = 0.f;
        for (int w = 0; w < nw; w++) M = fmaxf(M, pm[w][tid]);
        for (int w = 0; w < nw; w++) {
            const float e = (pm[w][tid] == -INFINITY) ? 0.f : expf(pm[w][tid] - M);
            wg[w][tid] = e; L = fmaf(pl[w][tid], e, L);
        }
        cm[tid] = M; cl[tid] = L;
    }
    __syncthreads();
    auto store = [&](int g, int d, float r) {
        const int64_t at = (int64_t)(q0 + g % nq) * a.ldo + (kvh * Gh + g / nq) * HD + d;
        if (a.out_lo) store_split1(a.out, a.out_lo, at, r, a.out_fmt);
        else a.out[at] = r;
    };
    for (int i = tid; i < G * HD; i += blockDim.x) {
        const int g = i / HD, d = i % HD;
        float O = 0.f;
        for (int w = 0; w < nw; w++) O = fmaf(po[w][g][d], wg[w][g], O);
        if (nc == 1) store(g, d, cl[g] > 0.f ? O / cl[g] : 0.f);
        else co[g][d] = O;
    }
    if (nc == 1) return;
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (tid < G) {
        float mc[ADG_MAXC], M = -INFINITY, L = 0.f;
#pragma unroll
        for (int c = 0; c < ADG_MAXC; c++) { mc[c] = c < nc ? ld_cluster(&cm[tid], c) : -INFINITY; M = fmaxf(M, mc[c]); }
#pragma unroll
        for (int c = 0; c < ADG_MAXC; c++) {
            const float e = mc[c] == -INFINITY ? 0.f : expf(mc[c] - M);
            cw[c][tid] = e;
            if (c < nc) L = fmaf(ld_cluster(&cl[tid], c), e, L);
        }
        wg[0][tid] = L > 0.f ? 1.0f / L : 0.f;
    }
    __syncthreads();
    // every CTA closes its share of the pair's outputs
    for (int i = rank * blockDim.x + tid; i < G * HD; i += nc * blockDim.x) {
        const int g = i / HD, d = i % HD;
        float O = 0.f;
#pragma unroll
        for (int c = 0; c < ADG_MAXC; c++)
            if (c < nc) O = fmaf(ld_cluster(&co[g][d], c), cw[c][g], O);
        store(g, d, O * wg[0][g]);
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");   // co is read by the others
}

// ---- head dim 64, many (query, head) pairs per kv group: one WARP per run of 32-key chunks, products on mma.sync ----
// With 7 to 16 (query, head) pairs per kv group (grouped-query decode steps of many sequences, the 4-token NCP
// level) the kernels above spend their time re-reading q and the probabilities from shared memory, one load per four
// multiply-adds. Here the pairs are the 16 rows of an m16n8k8 tensor-core tile: S[16 x 32] = Q[16 x 64] K^T and
// O[16 x 64] += P[16 x 32] V per 32-key chunk, each product as three TF32 MMAs over hi/lo splits (fp32-grade, as
// the three-pass GEMM engine). Every K and V element of a chunk is loaded from global memory exactly once, straight
// into the lane that needs it as a B fragment, sixteen bytes at a time: which head dimension sits at which k position
// of a score MMA, and which at which column of an output tile, is free as long as both operands agree, so the
// positions are chosen to make a lane's elements contiguous (k-step 2 m + h holds dims 16 m + 4 tig + 2 h and + 1 at
// positions tig and tig + 4; column gid of output tile j is dim 8 gid + j). The hi / lo halves of Q sit in shared
// memory (a lane's A fragments of two k-steps are four 16-byte reads); the
// probabilities cross from the accumulator layout to the A-fragment layout through 2 KB of shared memory per warp.
// Loads run a phase ahead of the arithmetic (the next chunk's keys are requested when the score MMAs are done with
// their registers, the chunk's values before its score MMAs).
// A warp walks `cps` chunks with a running maximum and sum per row; the four warps of a CTA take every fourth chunk
// of the CTA's stretch of the (row, kv head)'s keys and their partials meet in shared memory; one partial per CTA goes to
// global memory, and only when the row needs more than one CTA (last CTA merges, as above). The tcgen05 path needs
// 64 rows at least: for 16 it would idle three quarters of the tile.
constexpr int ADM_WARPS = 4;
#ifndef ADM_MINB
#define ADM_MINB 2
#endif
__device__ __forceinline__ void adm_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void adm_split(float v, uint32_t &hi, uint32_t &lo) {
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(v));
    const float r = v - __uint_as_float(hi);
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(r));
}
__device__ __forceinline__ float adm_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__global__ void __launch_bounds__(ADM_WARPS * 32, ADM_MINB) k_attention_dec_mma(AttnDecDev a) {
    constexpr int HD = 64, GA = AD_MAXG;
    __shared__ __align__(8) float ps[ADM_WARPS][GA][36];      // a warp's probabilities of a chunk, [row][key] (padded rows)
    __shared__ __align__(16) uint32_t qsh[GA][68], qsl[GA][68];   // TF32 hi / lo halves of the query tile (padded rows)
    __shared__ float pm[ADM_WARPS][GA], pl[ADM_WARPS][GA], wg[ADM_WARPS][GA];
    __shared__ __align__(8) float po[ADM_WARPS][GA][HD];
    __shared__ float Mg[GA], Lg[GA];
    __shared__ int s_last;
    const int row = blockIdx.z, kvh = blockIdx.y, sp = blockIdx.x;
    const int Gh = a.H / a.Hkv;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int gid = lane >> 2, tig = lane & 3;                // fragment coordinates of the lane
    pdl_launch_dependents();
    pdl_wait();
    const int *lens = a.k_len ? a.k_len + (a.step_d ? (int64_t)(*a.step_d) * a.len_step : 0) : nullptr;
    const int k00 = a.k_start[row], n1s = lens ? lens[row] : a.k_start[row + 1] - k00;
    const int k20 = a.k2_start ? a.k2_start[row] : 0, n2s = a.k2_start ? a.k2_start[row + 1] - k20 : 0;
    const int n1 = n1s + n2s;
    const int per_warp = a.cps * 32, per_cta = ADM_WARPS * per_warp;
    const int nsplit = (n1 + per_cta - 1) / per_cta;
    if (sp >= nsplit) return;
    // the CTA's chunks are dealt to its warps in turn (warp w takes chunks w, w + 4, ...): rows shorter than the
    // longest the launch was sized for -- early steps of a graph-replayed decode loop -- still occupy all four warps
    const int kbeg = sp * per_cta + warp * 32;                // first key of this warp's first chunk
    constexpr int KSTEP = ADM_WARPS * 32;                     // keys from one of its chunks to the next
    const int q0 = a.q_start[row], nq = a.q_start[row + 1] - q0;
    const int G = Gh * nq;                                    // virtual heads (tile rows): vh = g * nq + qi
    auto krow = [&](int j) -> const float * {
        return j < n1s ? a.k + (int64_t)(k00 + j) * a.ldk : a.k2 + (int64_t)(k20 + j - n1s) * a.ldk2;
    };
    auto vrow = [&](int j) -> const float * {
        return j < n1s ? a.v + (int64_t)(k00 + j) * a.ldk : a.v2 + (int64_t)(k20 + j - n1s) * a.ldk2;
    };
    // Q as A fragments (16 x 8 per k-step: a0 (row gid, k tig), a1 (gid + 8, tig), a2 (gid, tig + 4), a3 (gid + 8, tig + 4)),
    // k positions mapped to head dims as described above. The hi / lo halves of the 16 x 64 tile are formed once per CTA
    // and kept in shared memory; a lane fetches its fragments of two k-steps with four 16-byte reads.
    {
        const int r = tid >> 3, d0 = (tid & 7) * 8;                  // 128 threads: row, eight dims
        const float *p = r < G ? a.q + (int64_t)(q0 + r % nq) * a.ldq + (kvh * Gh + r / nq) * HD + d0 : nullptr;
        const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 f0 = p ? *(const float4 *)p : z4, f1 = p ? *(const float4 *)(p + 4) : z4;
        uint4 h0, l0, h1, l1;
        adm_split(f0.x, h0.x, l0.x); adm_split(f0.y, h0.y, l0.y); adm_split(f0.z, h0.z, l0.z); adm_split(f0.w, h0.w, l0.w);
        adm_split(f1.x, h1.x, l1.x); adm_split(f1.y, h1.y, l1.y); adm_split(f1.z, h1.z, l1.z); adm_split(f1.w, h1.w, l1.w);
        *(uint4 *)&qsh[r][d0] = h0; *(uint4 *)&qsh[r][d0 + 4] = h1;
        *(uint4 *)&qsl[r][d0] = l0; *(uint4 *)&qsl[r][d0 + 4] = l1;
    }
    __syncthreads();
    const float sl2 = a.scale * 1.4426950408889634f;          // scores in the log2 domain
    float oacc[8][4];                                         // O[16 x 64]: tile j column n is dim 8 n + j, rows gid / gid + 8
#pragma unroll
    for (int j = 0; j < 8; j++) { oacc[j][0] = oacc[j][1] = oacc[j][2] = oacc[j][3] = 0.f; }
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f; // running maximum (log2 domain) and sum of rows gid, gid + 8
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    // Loads run a phase ahead of the arithmetic: the keys of chunk c + 1 are requested when the score MMAs of chunk c
    // are done with their registers (they arrive under the softmax and the P V MMAs), the values of chunk c before its
    // score MMAs.
    float4 kf[4][4];                                          // n-tile j = keys kc + 8 j + gid; the lane's sixteen dims, 16 m + 4 tig ..
    auto load_k = [&](int kc) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int key = kc + 8 * j + gid;
            const float *kp = key < n1 ? krow(key) + kvh * HD + 4 * tig : nullptr;
#pragma unroll
            for (int m = 0; m < 4; m++) kf[j][m] = kp ? *(const float4 *)(kp + 16 * m) : z4;
        }
    };
    if (kbeg < n1) load_k(kbeg);
    for (int c = 0; c < a.cps; c++) {
        const int kc = kbeg + c * KSTEP;
        if (kc >= n1) break;                                  // warp-uniform
        // the chunk's values: k-step s takes keys kc + 8 s + tig (b0) and + 4 (b1); column gid of output tile j is dim
        // 8 gid + j, so the lane's eight dims of a value row are two 16-byte loads
        float4 vf[4][4];
#pragma unroll
        for (int s = 0; s < 4; s++) {
            const int ka = kc + 8 * s + tig, kb = ka + 4;
            const float *va = ka < n1 ? vrow(ka) + kvh * HD + 8 * gid : nullptr, *vb = kb < n1 ? vrow(kb) + kvh * HD + 8 * gid : nullptr;
            vf[s][0] = va ? *(const float4 *)va : z4; vf[s][1] = va ? *(const float4 *)(va + 4) : z4;
            vf[s][2] = vb ? *(const float4 *)vb : z4; vf[s][3] = vb ? *(const float4 *)(vb + 4) : z4;
        }
        // ---- S = Q K^T ----
        float sacc[4][4];
#pragma unroll
        for (int j = 0; j < 4; j++) { sacc[j][0] = sacc[j][1] = sacc[j][2] = sacc[j][3] = 0.f; }
#pragma unroll
        for (int m = 0; m < 4; m++) {
            const uint4 h0 = *(const uint4 *)&qsh[gid][16 * m + 4 * tig], h1 = *(const uint4 *)&qsh[gid + 8][16 * m + 4 * tig];
            const uint4 q0l = *(const uint4 *)&qsl[gid][16 * m + 4 * tig], q1l = *(const uint4 *)&qsl[gid + 8][16 * m + 4 * tig];
            const uint32_t ah0[4] = {h0.x, h1.x, h0.y, h1.y}, al0[4] = {q0l.x, q1l.x, q0l.y, q1l.y};      // k-step 2 m
            const uint32_t ah1[4] = {h0.z, h1.z, h0.w, h1.w}, al1[4] = {q0l.z, q1l.z, q0l.w, q1l.w};      // k-step 2 m + 1
#pragma unroll
            for (int j = 0; j < 4; j++) {
                uint32_t bh0, bl0, bh1, bl1;
                adm_split(kf[j][m].x, bh0, bl0); adm_split(kf[j][m].y, bh1, bl1);
                adm_mma(sacc[j], al0, bh0, bh1);
                adm_mma(sacc[j], ah0, bl0, bl1);
                adm_mma(sacc[j], ah0, bh0, bh1);
                adm_split(kf[j][m].z, bh0, bl0); adm_split(kf[j][m].w, bh1, bl1);
                adm_mma(sacc[j], al1, bh0, bh1);
                adm_mma(sacc[j], ah1, bl0, bl1);
                adm_mma(sacc[j], ah1, bh0, bh1);
            }
        }
        if (c + 1 < a.cps && kc + KSTEP < n1) load_k(kc + KSTEP);   // the next chunk's keys, under the rest of this chunk
        // ---- softmax of the chunk, rows gid (c0, c1) and gid + 8 (c2, c3); columns 8 j + 2 tig, + 1 ----
        float cm0 = -INFINITY, cm1 = -INFINITY;
#pragma unroll
        for (int j = 0; j < 4; j++) {
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const bool ok = kc + 8 * j + 2 * tig + e < n1;
                sacc[j][e] = ok ? sacc[j][e] * sl2 : -INFINITY;
                sacc[j][2 + e] = ok ? sacc[j][2 + e] * sl2 : -INFINITY;
                cm0 = fmaxf(cm0, sacc[j][e]); cm1 = fmaxf(cm1, sacc[j][2 + e]);
            }
        }
        cm0 = fmaxf(cm0, __shfl_xor_sync(0xffffffffu, cm0, 1)); cm0 = fmaxf(cm0, __shfl_xor_sync(0xffffffffu, cm0, 2));
        cm1 = fmaxf(cm1, __shfl_xor_sync(0xffffffffu, cm1, 1)); cm1 = fmaxf(cm1, __shfl_xor_sync(0xffffffffu, cm1, 2));
        const float nm0 = fmaxf(m0, cm0), nm1 = fmaxf(m1, cm1);   // finite: the chunk has at least one key
        const float al0 = m0 == -INFINITY ? 0.f : adm_ex2(m0 - nm0), al1 = m1 == -INFINITY ? 0.f : adm_ex2(m1 - nm1);
        m0 = nm0; m1 = nm1;
        float cs0 = 0.f, cs1 = 0.f;
        __syncwarp();                                         // the previous chunk's reads of ps are done
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float p00 = adm_ex2(sacc[j][0] - nm0), p01 = adm_ex2(sacc[j][1] - nm0);
            const float p10 = adm_ex2(sacc[j][2] - nm1), p11 = adm_ex2(sacc[j][3] - nm1);
            cs0 += p00 + p01; cs1 += p10 + p11;
            *(float2 *)&ps[warp][gid][8 * j + 2 * tig] = make_float2(p00, p01);
            *(float2 *)&ps[warp][gid + 8][8 * j + 2 * tig] = make_float2(p10, p11);
        }
        cs0 += __shfl_xor_sync(0xffffffffu, cs0, 1); cs0 += __shfl_xor_sync(0xffffffffu, cs0, 2);
        cs1 += __shfl_xor_sync(0xffffffffu, cs1, 1); cs1 += __shfl_xor_sync(0xffffffffu, cs1, 2);
        l0 = fmaf(l0, al0, cs0); l1 = fmaf(l1, al1, cs1);
#pragma unroll
        for (int j = 0; j < 8; j++) { oacc[j][0] *= al0; oacc[j][1] *= al0; oacc[j][2] *= al1; oacc[j][3] *= al1; }
        __syncwarp();
        // ---- O += P V: A fragment of k-step s (keys kc + 8 s + tig, + 4) from ps ----
#pragma unroll
        for (int s = 0; s < 4; s++) {
            uint32_t ph[4], pl_[4];
            adm_split(ps[warp][gid][8 * s + tig], ph[0], pl_[0]);
            adm_split(ps[warp][gid + 8][8 * s + tig], ph[1], pl_[1]);
            adm_split(ps[warp][gid][8 * s + tig + 4], ph[2], pl_[2]);
            adm_split(ps[warp][gid + 8][8 * s + tig + 4], ph[3], pl_[3]);
            const float vb0[8] = {vf[s][0].x, vf[s][0].y, vf[s][0].z, vf[s][0].w, vf[s][1].x, vf[s][1].y, vf[s][1].z, vf[s][1].w};
            const float vb1[8] = {vf[s][2].x, vf[s][2].y, vf[s][2].z, vf[s][2].w, vf[s][3].x, vf[s][3].y, vf[s][3].z, vf[s][3].w};
#pragma unroll
            for (int j = 0; j < 8; j++) {
                uint32_t bh0, bl0, bh1, bl1;
                adm_split(vb0[j], bh0, bl0); adm_split(vb1[j], bh1, bl1);
                adm_mma(oacc[j], pl_, bh0, bh1);
                adm_mma(oacc[j], ph, bl0, bl1);
                adm_mma(oacc[j], ph, bh0, bh1);
            }
        }
    }
    // ---- the warps' partials meet in shared memory ----
    if (tig == 0) { pm[warp][gid] = m0; pm[warp][gid + 8] = m1; pl[warp][gid] = l0; pl[warp][gid + 8] = l1; }
#pragma unroll
    for (int j = 0; j < 8; j++) {                             // columns 2 tig, 2 tig + 1 of tile j are dims 16 tig + j, + 8
        po[warp][gid][16 * tig + j] = oacc[j][0]; po[warp][gid][16 * tig + 8 + j] = oacc[j][1];
        po[warp][gid + 8][16 * tig + j] = oacc[j][2]; po[warp][gid + 8][16 * tig + 8 + j] = oacc[j][3];
    }
    __syncthreads();
    if (tid < G) {
        float M = -INFINITY, L = 0.f;
        for (int w = 0; w < ADM_WARPS; w++) M = fmaxf(M, pm[w][tid]);
        for (int w = 0; w < ADM_WARPS; w++) {
            const float e = (pm[w][tid] == -INFINITY) ? 0.f : adm_ex2(pm[w][tid] - M);
            wg[w][tid] = e; L = fmaf(pl[w][tid], e, L);
        }
        Mg[tid] = M; Lg[tid] = L;
    }
    __syncthreads();
    float *mine = a.part + ((int64_t)(row * a.Hkv + kvh) * a.max_split + sp) * AD_MAXG * (HD + 2);
    for (int i = tid; i < G * HD; i += blockDim.x) {
        const int g = i / HD, d = i % HD;
        float O = 0.f;
        for (int w = 0; w < ADM_WARPS; w++) O = fmaf(po[w][g][d], wg[w][g], O);
        if (nsplit == 1) {
            const float L = Lg[g];
            const float r = L > 0.f ? O / L : 0.f;
            const int64_t at = (int64_t)(q0 + g % nq) * a.ldo + (kvh * Gh + g / nq) * HD + d;
            if (a.out_lo) store_split1(a.out, a.out_lo, at, r, a.out_fmt);
            else a.out[at] = r;
        } else {
            mine[g * (HD + 2) + 2 + d] = O;
            if (d == 0) { mine[g * (HD + 2)] = Mg[g]; mine[g * (HD + 2) + 1] = Lg[g]; }
        }
    }
    if (nsplit == 1) return;
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        unsigned old = atomicAdd(a.count + row * a.Hkv + kvh, 1u);
        s_last = (old == (unsigned)(nsplit - 1));
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // the last CTA of the (row, kv head) merges the CTAs' partials (maxima in the log2 domain here)
    const float *base = a.part + (int64_t)(row * a.Hkv + kvh) * a.max_split * AD_MAXG * (HD + 2);
    if (tid < G) {
        float M = -INFINITY, L = 0.f;
        for (int x = 0; x < nsplit; x++) M = fmaxf(M, __ldcg(base + ((int64_t)x * AD_MAXG + tid) * (HD + 2)));
        for (int x = 0; x < nsplit; x++) {
            const float *pp = base + ((int64_t)x * AD_MAXG + tid) * (HD + 2);
            const float mx = __ldcg(pp);
            L = fmaf(__ldcg(pp + 1), mx == -INFINITY ? 0.f : adm_ex2(mx - M), L);
        }
        Mg[tid] = M; Lg[tid] = L;
    }
    __syncthreads();
    for (int i = tid; i < G * HD; i += blockDim.x) {
        const int g = i / HD, d = i % HD;
        const float M = Mg[g];
        float O = 0.f;
        for (int x = 0; x < nsplit; x++) {
            const float *pp = base + ((int64_t)x * AD_MAXG + g) * (HD + 2);
            const float mx = __ldcg(pp);
            O = fmaf(__ldcg(pp + 2 + d), mx == -INFINITY ? 0.f : adm_ex2(mx - M), O);
        }
        const float L = Lg[g];
        const float r = L > 0.f ? O / L : 0.f;
        const int64_t at = (int64_t)(q0 + g % nq) * a.ldo + (kvh * Gh + g / nq) * HD + d;
        if (a.out_lo) store_split1(a.out, a.out_lo, at, r, a.out_fmt);
        else a.out[at] = r;
    }
    if (tid == 0) a.count[row * a.Hkv + kvh] = 0;
}

bool attention_decode_supported(const AttnArgs &a) {
    if (a.max_q < 1 || a.max_q > 4 || a.causal || a.window > 0) return false;      // a few queries per row, no mask
    if (a.hd != 16 && a.hd != 32 && a.hd != 64 && a.hd != 128) return false;
    if (a.Hkv <= 0 || a.H % a.Hkv || (a.H / a.Hkv) * a.max_q > AD_MAXG) return false;
    if (a.max_k1 <= 0 || a.max_k1 + a.max_k2 > AD_KEYS * AD_MAXSPLIT) return false;
    if ((a.ldk1 & 3) || ((uintptr_t)a.k1 & 15)) return false;
    if (a.k2 && ((a.ldk2 & 3) || ((uintptr_t)a.k2 & 15) || a.step_d)) return false;
    return true;
}

// The device arguments of a call whose rows are cut over max_split CTAs of cps chunks (or runs per warp), with the partial
// buffer and the completion counters it needs.
static AttnDecDev decode_args(const AttnArgs &a, int max_split, int cps) {
    static float *part = nullptr; static size_t part_cap = 0;
    static unsigned *count = nullptr; static size_t count_cap = 0;
    const size_t need = (size_t)a.rows * a.Hkv * max_split * AD_MAXG * (a.hd + 2), nc = (size_t)a.rows * a.Hkv;
    if (need > part_cap) {
        if (part) { CUDA_CHECK(cudaStreamSynchronize(stream())); dev_free(part); }
        part = (float *)dev_alloc(need * 4); part_cap = need;
    }
    if (nc > count_cap) {
        if (count) { CUDA_CHECK(cudaStreamSynchronize(stream())); dev_free(count); }
        count = (unsigned *)dev_alloc(nc * 4); count_cap = nc;
        CUDA_CHECK(cudaMemsetAsync(count, 0, nc * 4, stream()));
    }
    AttnDecDev d{};
    d.q = a.q; d.ldq = a.ldq; d.k = a.k1; d.v = a.v1; d.ldk = a.ldk1;
    d.k2 = a.k2; d.v2 = a.v2; d.ldk2 = a.ldk2; d.k2_start = a.k2 ? a.k2_start : nullptr; d.out = a.out; d.out_lo = a.out_lo; d.out_fmt = a.out_fmt; d.ldo = a.ldo;
    d.q_start = a.q_start; d.k_start = a.k1_start; d.k_len = a.k1_len;
    d.step_d = a.step_d; d.len_step = a.k1_len_step;
    d.H = a.H; d.Hkv = a.Hkv; d.max_split = max_split; d.cps = cps;
    d.scale = 1.0f / sqrtf((float)a.hd);
    d.part = part; d.count = count;
    return d;
}

static bool al16(const void *q) { return ((uintptr_t)q & 15) == 0; }
static bool gqa_shape(const AttnArgs &a) {
    return a.hd == 64 && (a.H / a.Hkv) * a.max_q <= 8 && (a.ldk1 & 3) == 0 && (!a.k2 || (a.ldk2 & 3) == 0) && al16(a.k1) && al16(a.v1) && (!a.k2 || (al16(a.k2) && al16(a.v2)));
}

// Warps and CTAs of a (row, kv head) pair. An SM holds about twelve of these warps; all pairs should be resident at once (a
// second wave of a few CTAs costs as much as the first), so many pairs get CTAs of two or three warps; few pairs get a cluster
// of up to eight CTAs, two per SM, each warp with at least a run of keys.
static void attention_gqa(const AttnArgs &a, const AttnFused &f, bool fused) {
    const int64_t pairs = (int64_t)a.rows * a.Hkv;
    const int gq = (a.H / a.Hkv) * a.max_q, gm = gq <= 1 ? 1 : gq <= 2 ? 2 : gq <= 4 ? 4 : 8, sms = ctx().sm_count;
    const int runs = (int)cdiv(a.max_k1 + a.max_k2, ADG_NI * (gm == 8 ? 2 : 4));
    int nw = std::min(ADG_MAXW, runs), nc = 1;
    while (nw > 2 && pairs > sms * (int64_t)(12 / nw)) nw--;
    while (nc < ADG_MAXC && pairs * nc * 2 <= 2 * (int64_t)sms && nw * nc < runs) nc *= 2;
    AttnDecDev d{};
    d.q = a.q; d.ldq = a.ldq; d.k = a.k1; d.v = a.v1; d.ldk = a.ldk1;
    d.k2 = a.k2; d.v2 = a.v2; d.ldk2 = a.ldk2; d.k2_start = a.k2 ? a.k2_start : nullptr; d.out = a.out; d.out_lo = a.out_lo; d.out_fmt = a.out_fmt; d.ldo = a.ldo;
    d.q_start = a.q_start; d.k_start = a.k1_start; d.k_len = a.k1_len;
    d.step_d = a.step_d; d.len_step = a.k1_len_step;
    d.H = a.H; d.Hkv = a.Hkv; d.rows = a.rows; d.scale = 1.0f / sqrtf((float)a.hd);
    const dim3 grid((unsigned)nc, (unsigned)a.Hkv, (unsigned)a.rows);
    ProfScope ps(NCMB_K_ATTN, 4.0 * (double)a.total_q * a.avg_keys * a.H * a.hd, 0);
#define GQA_LAUNCH(GM_) do { \
        static bool set = false; \
        if (!set) { \
            CUDA_CHECK(cudaFuncSetAttribute((k_attention_dec_gqa<GM_, true>), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)adg_smem(GM_, ADG_MAXW))); \
            CUDA_CHECK(cudaFuncSetAttribute((k_attention_dec_gqa<GM_, false>), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)adg_smem(GM_, ADG_MAXW))); \
            set = true; } \
        if (fused) launch_pdl_cluster(k_attention_dec_gqa<GM_, true>, grid, dim3(nw * 32), adg_smem(GM_, nw), nc, d, f); \
                             else launch_pdl_cluster(k_attention_dec_gqa<GM_, false>, grid, dim3(nw * 32), adg_smem(GM_, nw), nc, d, f); } while (0)
    if (gm == 1) GQA_LAUNCH(1);
    else if (gm == 2) GQA_LAUNCH(2);
    else if (gm == 4) GQA_LAUNCH(4);
    else GQA_LAUNCH(8);
#undef GQA_LAUNCH
}

bool attention_fused_supported(const AttnArgs &a) { return gqa_shape(a) && a.max_q == 1 && !a.k2 && a.k1_len && !a.causal && !a.window && a.max_k1 > 0; }
void attention_fused(const AttnArgs &a, const FewQkv &q) {
    AttnFused f{q.part, q.S, q.bias, q.cos_t, q.sin_t, q.pos, q.pos_step, q.kv, q.seq_pitch, q.step};
    attention_gqa(a, f, true);
}

void attention_decode(const AttnArgs &a) {
    // Keys of a row are shared out in 32-key chunks. With few (row, kv head) pairs every chunk gets a CTA of its own
    // (a batch-1 decode step has nothing else to fill the GPU with); with many pairs a CTA walks several chunks,
    // so that the fixed cost per CTA (query load, partials through L2, the merge) is paid about 8 x SMs times
    // and not once per chunk.
    const int max_chunks = (int)cdiv(a.max_k1 + a.max_k2, AD_KEYS);
    const int64_t pairs = (int64_t)a.rows * a.Hkv;
    const int gq_w = (a.H / a.Hkv) * a.max_q;
    // many (query, head) pairs per kv group and enough (row, kv head) pairs to fill the GPU with warps: the
    // tensor-core kernel (read per call: the tests run every kernel on the same inputs)
    const char *mma_s = getenv("NCM_B200_ATTN_DEC_MMA");
    const int mma_env = mma_s ? atoi(mma_s) : -1;
    const bool mma_takes = a.hd == 64 && gq_w <= AD_MAXG && ((a.ldk1 & 3) == 0) && (!a.k2 || (a.ldk2 & 3) == 0) && ((a.ldq & 3) == 0) &&
                           al16(a.q) && al16(a.k1) && al16(a.v1) && (!a.k2 || (al16(a.k2) && al16(a.v2)));
    const bool gqa_takes = gqa_shape(a) && ((a.ldq & 3) == 0) && al16(a.q) && mma_env != 1;
    // (measured: the 4-token level of config 2 -- 16 pairs per group, 9 chunks -- 2.99 -> 2.44 ms over its 12 layers. Up to eight
    // pairs per group go to k_attention_dec_gqa whatever their number; what is left for the second condition, groups of 9 to 11
    // pairs, follows the line measured for seven: gain from about 300 (row, kv head) pairs on, below the CTA-per-chunk kernels
    // spread a row over more SMs)
    static const int mma_min_g = getenv("NCM_B200_ATTN_DEC_MMA_MIN_G") ? atoi(getenv("NCM_B200_ATTN_DEC_MMA_MIN_G")) : 12;
    static const int mma_max_ch = getenv("NCM_B200_ATTN_DEC_MMA_MAX_CHUNKS") ? atoi(getenv("NCM_B200_ATTN_DEC_MMA_MAX_CHUNKS")) : 16;
    const bool mma_pays = (gq_w >= mma_min_g && max_chunks <= mma_max_ch && pairs * 4 >= (int64_t)ctx().sm_count) ||
                          (gq_w >= 6 && pairs >= 2 * (int64_t)ctx().sm_count);
    if (mma_takes && (mma_env == 1 || (mma_env != 0 && !gqa_takes && mma_pays))) {
        // chunks per warp: as few CTAs per (row, kv head) as still give every SM about eight warps
        const int64_t want_ctas = std::max<int64_t>(1, cdiv((int64_t)ctx().sm_count * 2, pairs));
        int cpw = (int)cdiv(max_chunks, ADM_WARPS * want_ctas);
        if (cpw < 1) cpw = 1;
        if (cpw > 16) cpw = 16;
        const int max_split = (int)cdiv(max_chunks, ADM_WARPS * cpw);
        if (max_split <= AD_MAXSPLIT) {
            AttnDecDev d = decode_args(a, max_split, cpw);
            dim3 grid((unsigned)max_split, (unsigned)a.Hkv, (unsigned)a.rows);
            ProfScope ps(NCMB_K_ATTN, 4.0 * (double)a.total_q * a.avg_keys * a.H * a.hd, 0);
            LAUNCH_PDL(k_attention_dec_mma, grid, ADM_WARPS * 32, 0, d);
            return;
        }
    }
    if (gqa_takes) { attention_gqa(a, AttnFused{}, false); return; }
    static const int per_sm = getenv("NCM_B200_ATTN_DEC_PER_SM") ? atoi(getenv("NCM_B200_ATTN_DEC_PER_SM")) : 8;
    int want_split = (int)std::min<int64_t>(max_chunks, cdiv((int64_t)ctx().sm_count * per_sm, pairs));
    if (want_split < 1) want_split = 1;
    static const int cps_env = getenv("NCM_B200_ATTN_DEC_CPS") ? atoi(getenv("NCM_B200_ATTN_DEC_CPS")) : 0;
    const int cps = cps_env > 0 ? std::min(cps_env, max_chunks) : (int)cdiv(max_chunks, want_split);
    const int max_split = (int)cdiv(max_chunks, cps);
    AttnDecDev d = decode_args(a, max_split, cps);
    dim3 grid((unsigned)max_split, (unsigned)a.Hkv, (unsigned)a.rows);
    ProfScope ps(NCMB_K_ATTN, 4.0 * (double)a.total_q * a.avg_keys * a.H * a.hd, 0);
    const int gq = (a.H / a.Hkv) * a.max_q;
#define AD_LAUNCH(HD_)                                                                              \
    do {                                                                                            \
        if (gq <= 1) LAUNCH_PDL((k_attention_decode<HD_, 1>), grid, AD_THREADS, 0, d);              \
        else if (gq <= 4) LAUNCH_PDL((k_attention_decode<HD_, 4>), grid, AD_THREADS, 0, d);         \
        else if (gq <= 8) LAUNCH_PDL((k_attention_decode<HD_, 8>), grid, AD_THREADS, 0, d);         \
        else LAUNCH_PDL((k_attention_decode<HD_, 16>), grid, AD_THREADS, 0, d);                     \
    } while (0)
    switch (a.hd) {
        case 16: AD_LAUNCH(16); break;
        case 32: AD_LAUNCH(32); break;
        case 64: AD_LAUNCH(64); break;
        default: AD_LAUNCH(128); break;
    }
#undef AD_LAUNCH
}

} // namespace ncmb
