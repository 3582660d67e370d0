// Device-side sampling of one level's positions for every row.
//
// One CTA per sequence row; positions are visited in order because the
// frequency / deficit / adjacency penalties of position t depend on the picks at
// positions < t (reference sample_level_rows, src/ncp.c:654-705). Per position:
//   CFG blend (1+w) cond - w uncond in fp64 (src/ncp.c:1112-1116), penalties in fp64,
//   then either first-index argmax (temp <= 0) or temperature / top-k / nucleus
//   sampling (src/kernels.c:794-825): the top `keep` logits are found with a
//   block-wide 4 x 8-bit radix select, sorted with a bitonic network, turned into
//   fp64 probabilities and walked sequentially in rank order exactly as the
//   reference does, using one pre-drawn uniform.
// The uniforms come either from the reference's xorshift64* stream (drawn on the
// host in the reference's (level, row, position) order) or from a counter-based
// generator keyed by (seed, global row, level, position).
#include "common.cuh"
#include "exp_tab.cuh"

#include <cub/device/device_radix_sort.cuh>
#include <vector>

namespace ncmb {

constexpr int SM_THREADS = 256;
constexpr int SM_MAXKEEP = 2048;           // exact sorted path handles keep <= this
constexpr int SM_SMEM_V = 16384;           // logits rows up to this many floats live in shared memory

struct SampleDev {
    SampleArgs a;
    int vals_in_smem;
};

__device__ __forceinline__ unsigned okey(float f) {      // order-preserving float -> uint
    unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float okey_inv(unsigned k) {
    unsigned u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    return __uint_as_float(u);
}

// splitmix64-style counter hash -> uniform double in [0, 1)
__device__ __forceinline__ double counter_uniform(unsigned long long seed, long long row, int level, int t) {
    unsigned long long z = seed ^ (0x9E3779B97F4A7C15ULL * (unsigned long long)(row + 1));
    z += 0xBF58476D1CE4E5B9ULL * (unsigned long long)(level + 1) + 0x94D049BB133111EBULL * (unsigned long long)(t + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    z = z ^ (z >> 31);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = z ^ (z >> 29);
    return (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

// the draw of model row b at position t: keyed by the sequence's global index, never by the row's place in the call
__device__ __forceinline__ double counter_uniform_row(const SampleArgs &a, int b, int t) {
    const bool twin = a.rng_wrap > 0 && b >= a.rng_wrap;
    return counter_uniform(a.rng_seed, a.rng_row0 + (twin ? b - a.rng_wrap : b), a.rng_level + (twin ? 64 : 0), t);
}

__global__ void __launch_bounds__(SM_THREADS) k_sample(SampleDev sd) {
    const SampleArgs &a = sd.a;
    extern __shared__ __align__(16) unsigned char smraw[];
    // layout: cand u64[SM_MAXKEEP] | probs f64[SM_MAXKEEP] | vals f32[V] (optional)
    unsigned long long *cand = (unsigned long long *)smraw;
    double *probs = (double *)(smraw + sizeof(unsigned long long) * SM_MAXKEEP);
    float *vals = sd.vals_in_smem ? (float *)(smraw + 16 * SM_MAXKEEP) : a.scratch + (size_t)blockIdx.x * a.V;
    __shared__ int hist[256];
    __shared__ unsigned long long red[SM_THREADS];
    __shared__ unsigned s_prefix, s_mask;
    __shared__ double s_den;
    __shared__ int s_remaining, s_ncand, s_pick, s_eqbase[SM_THREADS + 1];

    const int b = blockIdx.x, tid = threadIdx.x, V = a.V, Lc = a.Lc;
    double *cnt = a.cnt ? a.cnt + (size_t)b * a.cnt_stride : nullptr;
    int *hst = a.hist ? a.hist + (size_t)b * a.hist_stride : nullptr;
    int hl = a.hist_len ? a.hist_len[b] : 0;
    const bool penal = (a.freq > 0.f) || (a.adj_a != 0.f);

    for (int t = 0; t < Lc; t++) {
        const float *lc = a.logits + ((size_t)b * Lc + t) * V;
        const float *lu = a.uncond_off ? a.logits + (((size_t)b + a.uncond_off) * Lc + t) * V : nullptr;
        float *bo = a.blend_out ? a.blend_out + ((size_t)b * Lc + t) * V : nullptr;
        for (int v = tid; v < V; v += SM_THREADS) {
            float x = lc[v];
            if (lu) x = (float)((1.0 + a.cfg_w) * (double)x - a.cfg_w * (double)lu[v]);
            if (bo) bo[v] = x;
            if (penal) {
                double lg = x;
                if (a.freq > 0.f) {
                    double al = a.allow_dev ? a.allow_dev[v] * Lc : 0.0;
                    double c = cnt[v];
                    double excess = c - al;
                    if (excess < 0) excess = 0;
                    lg -= (double)a.freq * excess;
                    if (a.mu > 0.f && a.allow_dev) {
                        double def = al - c;
                        if (def < 0) def = 0;
                        lg += (double)a.mu * ((Lc - t) / (double)Lc) * def;
                    }
                }
                x = (float)lg;
            }
            vals[v] = x;
        }
        __syncthreads();
        if (a.adj_a != 0.f && tid == 0) {            // sequential: the same id may repeat in the window
            int w = a.adj_w > 0 ? a.adj_w : 1;
            int start = hl - w;
            if (start < 0) start = 0;
            for (int h = start; h < hl; h++) {
                double pen = (double)a.adj_a * pow((double)a.adj_d, (double)(hl - 1 - h));
                vals[hst[h]] -= (float)pen;
            }
        }
        __syncthreads();

        if (!(a.temp > 0.f)) {
            // first-index argmax: max over (ordered key, inverted index)
            unsigned long long best = 0;
            for (int v = tid; v < V; v += SM_THREADS) {
                unsigned long long c = ((unsigned long long)okey(vals[v]) << 32) | (unsigned)(0xffffffffu - (unsigned)v);
                if (c > best) best = c;
            }
            red[tid] = best;
            __syncthreads();
            for (int s = SM_THREADS / 2; s > 0; s >>= 1) {
                if (tid < s && red[tid + s] > red[tid]) red[tid] = red[tid + s];
                __syncthreads();
            }
            if (tid == 0) s_pick = (int)(0xffffffffu - (unsigned)(red[0] & 0xffffffffu));
            __syncthreads();
        } else {
            for (int v = tid; v < V; v += SM_THREADS) vals[v] = vals[v] / a.temp;
            int keep = (a.top_k > 0) ? (a.top_k < V ? a.top_k : V) : V;
            // ---- radix select: key of the keep-th largest value ----
            if (tid == 0) { s_prefix = 0; s_mask = 0; s_remaining = keep; }
            __syncthreads();
            for (int pass = 3; pass >= 0; pass--) {
                hist[tid] = 0;
                __syncthreads();
                unsigned prefix = s_prefix, mask = s_mask;
                for (int v = tid; v < V; v += SM_THREADS) {
                    unsigned k = okey(vals[v]);
                    if ((k & mask) == prefix) atomicAdd(&hist[(k >> (8 * pass)) & 0xff], 1);
                }
                __syncthreads();
                if (tid < 32) {
                    // the bin, scanning from 255 down, where the running count first reaches `rem`: lane l owns bins
                    // 255-8l .. 248-8l; lane totals are scanned with shuffles instead of one thread walking 256 bins
                    const int rem = s_remaining, top = 255 - 8 * tid;
                    int h8[8], tot = 0;
#pragma unroll
                    for (int i = 0; i < 8; i++) { h8[i] = hist[top - i]; tot += h8[i]; }
                    int incl = tot;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) { int t2 = __shfl_up_sync(0xffffffffu, incl, o); if (tid >= o) incl += t2; }
                    int cum = incl - tot;                               // count in all bins above this lane's
                    const bool here = cum < rem && incl >= rem;          // the crossing lies in this lane's bins
                    const unsigned who = __ballot_sync(0xffffffffu, here);
                    if (who == 0) {                                      // fewer than rem values in total: bin 0, as the serial walk ends
                        if (tid == 31) {
                            s_remaining = rem - (incl - h8[7]);
                            s_prefix = prefix; s_mask = mask | (0xffu << (8 * pass));
                        }
                    } else if (tid == __ffs(who) - 1) {
                        int bin = top;
                        for (int i = 0; i < 8; i++) {
                            bin = top - i;
                            if (bin == 0 || cum + h8[i] >= rem) break;
                            cum += h8[i];
                        }
                        s_remaining = rem - cum;
                        s_prefix = prefix | ((unsigned)bin << (8 * pass));
                        s_mask = mask | (0xffu << (8 * pass));
                    }
                }
                __syncthreads();
            }
            const unsigned thr = s_prefix;
            const int need_eq = s_remaining;          // how many values equal to the threshold are kept
            if (tid == 0) s_ncand = 0;
            __syncthreads();
            for (int v = tid; v < V; v += SM_THREADS) {
                unsigned k = okey(vals[v]);
                if (k > thr) {
                    int p = atomicAdd(&s_ncand, 1);
                    cand[p] = ((unsigned long long)k << 32) | (unsigned)(0xffffffffu - (unsigned)v);
                }
            }
            // threshold ties: lowest indices first (contiguous chunk per thread + exclusive scan)
            const int chunk = (V + SM_THREADS - 1) / SM_THREADS;
            const int v0 = tid * chunk, v1 = (v0 + chunk < V) ? v0 + chunk : V;
            int eq = 0;
            for (int v = v0; v < v1; v++) if (okey(vals[v]) == thr) eq++;
            s_eqbase[tid + 1] = eq;
            __syncthreads();
            {   // inclusive scan of the per-thread tie counts: warp shuffles, then the eight warp totals
                const int lane = tid & 31, wp = tid >> 5;
                int v = eq;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) { int t2 = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += t2; }
                if (lane == 31) hist[wp] = v;
                __syncthreads();
                int base = 0;
                for (int i = 0; i < wp; i++) base += hist[i];
                s_eqbase[tid + 1] = base + v;
                if (tid == 0) s_eqbase[0] = 0;
            }
            __syncthreads();
            {
                int rank = s_eqbase[tid], gt = s_ncand;
                for (int v = v0; v < v1 && rank < need_eq; v++)
                    if (okey(vals[v]) == thr) {
                        cand[gt + rank] = ((unsigned long long)thr << 32) | (unsigned)(0xffffffffu - (unsigned)v);
                        rank++;
                    }
            }
            __syncthreads();
            // ---- bitonic sort, descending: value desc, index asc ----
            int n2 = 1;
            while (n2 < keep) n2 <<= 1;
            for (int i = keep + tid; i < n2; i += SM_THREADS) cand[i] = 0;
            __syncthreads();
            for (int k = 2; k <= n2; k <<= 1)
                for (int j = k >> 1; j > 0; j >>= 1) {
                    for (int i = tid; i < n2; i += SM_THREADS) {
                        int ixj = i ^ j;
                        if (ixj > i) {
                            unsigned long long x = cand[i], y = cand[ixj];
                            bool desc = ((i & k) == 0);
                            if (desc ? (x < y) : (x > y)) { cand[i] = y; cand[ixj] = x; }
                        }
                    }
                    __syncthreads();
                }
            // ---- probabilities in rank order (fp64), nucleus cut, renormalise, walk ----
            const double mx = (double)okey_inv((unsigned)(cand[0] >> 32));
            for (int r = tid; r < keep; r += SM_THREADS)
                probs[r] = exp((double)okey_inv((unsigned)(cand[r] >> 32)) - mx);
            __syncthreads();
            // the sums run in rank order on one thread, as the reference's do; the divisions are independent
            if (tid == 0) {
                double den = 0;
                for (int r = 0; r < keep; r++) den += probs[r];
                s_den = den;
            }
            __syncthreads();
            {
                const double den = s_den;
                for (int r = tid; r < keep; r += SM_THREADS) probs[r] /= den;
            }
            __syncthreads();
            if (tid == 0) {
                double den;
                double cum = 0;
                int nkeep = keep;
                for (int r = 0; r < keep; r++) {
                    if (cum - probs[r] > (double)a.top_p) { nkeep = r; break; }
                    cum += probs[r];
                }
                den = 0;
                for (int r = 0; r < nkeep; r++) den += probs[r];
                double u01 = a.uniforms ? a.uniforms[(size_t)b * Lc + t]
                                        : counter_uniform_row(a, b, t);
                double u = u01 * den, acc = 0;
                int pr = nkeep - 1;
                for (int r = 0; r < nkeep; r++) { acc += probs[r]; if (u <= acc) { pr = r; break; } }
                s_pick = (int)(0xffffffffu - (unsigned)(cand[pr] & 0xffffffffu));
            }
            __syncthreads();
        }
        if (tid == 0) {
            int pick = s_pick;
            a.out[(size_t)b * a.out_stride + a.out_off + t] = pick;
            if (cnt) cnt[pick] += 1.0;
            if (hst) hst[hl] = pick;
        }
        hl++;
        __syncthreads();
    }
    if (tid == 0 && a.hist_len) a.hist_len[b] = hl;
}

// ---------------------------------------------------------------------------------------------
// Two-phase sampling. The sequential kernel above spends most of a position on work that does not
// depend on earlier picks: the blend and the 4096-wide selection. Penalties that only LOWER logits
// (frequency excess, adjacency with a >= 0; no deficit bonus) touch at most P tokens, the ones
// picked so far in the row, so the `keep` best penalised logits of a position lie among its
// keep + P best raw ones: a token of the penalised top-keep is preceded in raw order by at most
// keep - 1 unpenalised tokens (which precede it in penalised order too) and P penalised ones.
//   k_sample_topc  one CTA per (row, position), all positions at once: blend, the Kc >= keep + P
//                  best raw logits (same radix select, ties to the lowest index) -> candidates
//   k_sample_seq   one CTA per row, positions in order, Kc entries each: the same penalty, temperature,
//                  ordering (value descending, index ascending), fp64 probabilities and walk as above
// Picks equal the one-kernel path's bit for bit: every number a pick depends on is computed by the
// same operations in the same order.
constexpr int SC_MAXC = 256;

struct SampleCand {
    SampleArgs a;
    int Kc;
    unsigned long long *cand;       // [Bn][Lc][Kc]: ordered key << 32 | ~index of the raw (blended) logit
};

// The Kc best of the entries a CTA's threads hold, best first, to out[0, Kc). get(i) is a thread's i-th entry (0: none), Kc <= TC_T
// (entries are distinct: a key and an index).
//
// The Kc-th best of the threads' own maxima bounds the Kc-th best entry from below, so only entries from there on -- some Kc to
// 2 Kc of them, by the spread of entries over threads -- have to be ranked, by counting, in shared memory. Nothing is sorted and no
// entry touches a histogram; the bound comes out of 32 barriers that count. Where ties or an odd order of the entries put more
// than TC_LIST above the bound (a constant row), the cut is searched bit by bit over all entries instead.
constexpr int TC_T = 512, TC_LIST = 1024, TC_MAXPARTS = 32;
template <int N, class F>
__device__ __forceinline__ void topc_select(F get, int Kc, unsigned long long *out) {
    __shared__ unsigned long long list[TC_LIST];
    __shared__ int s_n;
    const int tid = threadIdx.x;
    unsigned top = 0;
#pragma unroll
    for (int i = 0; i < N; i++) top = max(top, (unsigned)(get(i) >> 32));
    unsigned cut = 0;
#pragma unroll 1
    for (unsigned bit = 0x80000000u; bit; bit >>= 1)
        if (__syncthreads_count(top >= (cut | bit)) >= Kc) cut |= bit;
    if (tid == 0) s_n = 0;
    __syncthreads();
    unsigned long long least = (unsigned long long)cut << 32;
    auto collect = [&]() {
#pragma unroll
        for (int i = 0; i < N; i++) {
            const unsigned long long k = get(i);
            if (k != 0 && k >= least) { const int at = atomicAdd(&s_n, 1); if (at < TC_LIST) list[at] = k; }
        }
        __syncthreads();
    };
    collect();
    if (s_n > TC_LIST) {
        unsigned long long c64 = 0;
#pragma unroll 1
        for (int bit = 63; bit >= 0; bit--) {
            const unsigned long long t = c64 | 1ull << bit;
            __syncthreads();
            if (tid == 0) s_n = 0;
            __syncthreads();
            int n = 0;
#pragma unroll
            for (int i = 0; i < N; i++) n += get(i) >= t;
            n = __reduce_add_sync(0xffffffffu, n);
            if ((tid & 31) == 0) atomicAdd(&s_n, n);
            __syncthreads();
            if (s_n >= Kc) c64 = t;
        }
        __syncthreads();
        if (tid == 0) s_n = 0;
        __syncthreads();
        least = c64;
        collect();
    }
    const int n = s_n;
    for (int e = tid; e < n; e += TC_T) {
        const unsigned long long k = list[e];
        int r = 0;
        for (int f = 0; f < n; f++) r += list[f] > k;
        if (r < Kc) out[r] = k;
    }
}

// CTA (part, row x position): the Kc best of one of gridDim.x equal parts (a part may hold fewer entries than Kc: zeros follow).
// Entries stay in registers, N per thread. Bound by latency: one trip to the logits, 32 barriers, one short list.
template <int N>
__global__ void __launch_bounds__(TC_T) k_sample_topc(SampleCand sc, unsigned long long *parts) {
    const SampleArgs &a = sc.a;
    const int tid = threadIdx.x, V = a.V, Lc = a.Lc, G = gridDim.x;
    const int b = blockIdx.y / Lc, t = blockIdx.y % Lc;
    const int v0 = (int)((long long)V * blockIdx.x / G), n = (int)((long long)V * (blockIdx.x + 1) / G) - v0;
    const float *lc = a.logits + ((size_t)b * Lc + t) * V + v0;
    const float *lu = a.uncond_off ? a.logits + (((size_t)b + a.uncond_off) * Lc + t) * V + v0 : nullptr;
    float *bo = a.blend_out ? a.blend_out + ((size_t)b * Lc + t) * V + v0 : nullptr;
    unsigned long long *out = (G > 1 ? parts : sc.cand) + ((size_t)blockIdx.y * G + blockIdx.x) * sc.Kc;
    float x[N];
#pragma unroll
    for (int i = 0; i < N; i++) { const int v = i * TC_T + tid; x[i] = v < n ? lc[v] : 0.f; }
    if (lu) {
#pragma unroll
        for (int i = 0; i < N; i++) { const int v = i * TC_T + tid; if (v < n) x[i] = (float)((1.0 + a.cfg_w) * (double)x[i] - a.cfg_w * (double)lu[v]); }
    }
    if (bo) {
#pragma unroll
        for (int i = 0; i < N; i++) { const int v = i * TC_T + tid; if (v < n) bo[v] = x[i]; }
    }
    auto get = [&](int i) -> unsigned long long {
        const int v = i * TC_T + tid;
        return v < n ? ((unsigned long long)okey(x[i]) << 32) | (unsigned)(0xffffffffu - (unsigned)(v0 + v)) : 0ull;
    };
    if (n < sc.Kc) for (int e = n + tid; e < sc.Kc; e += TC_T) out[e] = 0;
    topc_select<N>(get, sc.Kc < n ? sc.Kc : n, out);
}
template <int N>
__global__ void __launch_bounds__(TC_T) k_sample_merge(SampleCand sc, const unsigned long long *parts, int G) {
    const int tid = threadIdx.x, n = G * sc.Kc;
    unsigned long long k[N];
#pragma unroll
    for (int i = 0; i < N; i++) k[i] = i * TC_T + tid < n ? parts[(size_t)blockIdx.x * n + i * TC_T + tid] : 0;
    topc_select<N>([&](int i) { return k[i]; }, sc.Kc, sc.cand + (size_t)blockIdx.x * sc.Kc);
}

__global__ void __launch_bounds__(SC_MAXC) k_sample_seq(SampleCand sc) {
    const SampleArgs &a = sc.a;
    __shared__ unsigned long long cand[SC_MAXC];
    __shared__ double probs[SC_MAXC];
    __shared__ double s_den;
    __shared__ int s_pick;
    const int b = blockIdx.x, tid = threadIdx.x, Lc = a.Lc, Kc = sc.Kc;
    double *cnt = a.cnt ? a.cnt + (size_t)b * a.cnt_stride : nullptr;
    int *hst = a.hist ? a.hist + (size_t)b * a.hist_stride : nullptr;
    int hl = a.hist_len ? a.hist_len[b] : 0;
    const bool penal = (a.freq > 0.f) || (a.adj_a != 0.f);
    const int keep = (a.top_k > 0) ? (a.top_k < a.V ? a.top_k : a.V) : a.V;
    unsigned long long c_next = tid < Kc ? sc.cand[(size_t)b * Lc * Kc + tid] : 0;
    for (int t = 0; t < Lc; t++) {
        unsigned long long key = 0;
        const unsigned long long c = c_next;
        if (t + 1 < Lc && tid < Kc) c_next = sc.cand[((size_t)b * Lc + t + 1) * Kc + tid];   // in flight under this position's work
        if (tid < Kc) {
            const int v = (int)(0xffffffffu - (unsigned)(c & 0xffffffffu));
            float x = okey_inv((unsigned)(c >> 32));
            if (penal) {
                double lg = x;
                if (a.freq > 0.f) {
                    double al = a.allow_dev ? a.allow_dev[v] * Lc : 0.0;
                    double cc = cnt[v];
                    double excess = cc - al;
                    if (excess < 0) excess = 0;
                    lg -= (double)a.freq * excess;
                }
                x = (float)lg;
                if (a.adj_a != 0.f) {                    // window entries in order: the same id may repeat
                    int w = a.adj_w > 0 ? a.adj_w : 1;
                    int start = hl - w;
                    if (start < 0) start = 0;
                    for (int h = start; h < hl; h++)
                        if (hst[h] == v) {
                            double pen = (double)a.adj_a * pow((double)a.adj_d, (double)(hl - 1 - h));
                            x -= (float)pen;
                        }
                }
            }
            x = x / a.temp;
            key = ((unsigned long long)okey(x) << 32) | (unsigned)(0xffffffffu - (unsigned)v);
        }
        // bitonic sort, descending, one entry per thread: exchanges within a warp by shuffle, the few across
        // warps (partner distance >= 32) through shared memory
        for (int k = 2; k <= Kc; k <<= 1)
            for (int j = k >> 1; j > 0; j >>= 1) {
                unsigned long long other;
                if (j >= 32) {
                    cand[tid] = key;
                    __syncthreads();
                    other = cand[tid ^ j];
                    __syncthreads();
                } else {
                    other = __shfl_xor_sync(0xffffffffu, key, j);
                }
                const bool keep_max = (((tid & k) == 0) == ((tid & j) == 0));   // descending run: the lower index keeps the larger
                key = keep_max ? (key > other ? key : other) : (key < other ? key : other);
            }
        cand[tid] = key;
        __syncthreads();
        const double mx = (double)okey_inv((unsigned)(cand[0] >> 32));
        if (tid < keep) probs[tid] = exp((double)okey_inv((unsigned)(cand[tid] >> 32)) - mx);
        __syncthreads();
        if (tid == 0) {
            double den = 0;
            for (int r = 0; r < keep; r++) den += probs[r];
            s_den = den;
        }
        __syncthreads();
        if (tid < keep) probs[tid] /= s_den;
        __syncthreads();
        if (tid == 0) {
            // nucleus cut. The running sum of the kept ranks is at once the reference's renormaliser (its second sum
            // adds the same numbers in the same order) and, rank by rank, the accumulator of its final walk.
            double cum = 0;
            int nkeep = keep;
            for (int r = 0; r < keep; r++) {
                if (cum - probs[r] > (double)a.top_p) { nkeep = r; break; }
                cum += probs[r];
                probs[r] = cum;                          // from here on: inclusive running sums
            }
            const double u01 = a.uniforms ? a.uniforms[(size_t)b * Lc + t]
                                          : counter_uniform_row(a, b, t);
            s_den = u01 * cum;
            s_pick = nkeep;                              // handed to the search below
        }
        __syncthreads();
        {   // first rank whose running sum reaches u; the last kept rank if none does
            const int nkeep = s_pick;
            const double u = s_den;
            const bool hit = tid < nkeep && u <= probs[tid];
            __shared__ int s_first;
            if (tid == 0) s_first = nkeep - 1;
            __syncthreads();
            if (hit) atomicMin(&s_first, tid);
            __syncthreads();
            if (tid == 0) {
                const int pick = (int)(0xffffffffu - (unsigned)(cand[s_first] & 0xffffffffu));
                a.out[(size_t)b * a.out_stride + a.out_off + t] = pick;
                if (cnt) cnt[pick] += 1.0;
                if (hst) hst[hl] = pick;
            }
        }
        hl++;
        __syncthreads();                 // cnt / hist of this position are visible to the next one
    }
    if (tid == 0 && a.hist_len) a.hist_len[b] = hl;
}

// Kc for the two-phase path, or 0 when it does not apply
static int two_phase_width(const SampleArgs &a) {
    if (!(a.temp > 0.f) || a.top_k <= 0 || a.V > TC_MAXPARTS * TC_T * 32) return 0;
    const char *e = getenv("NCM_B200_SAMPLE_PHASES");          // 1 = one kernel always, 2 = two phases whenever valid
    const int mode = e ? atoi(e) : 0;
    if (mode == 1) return 0;
    const bool penal = (a.freq > 0.f) || (a.adj_a != 0.f);
    if (a.adj_a < 0.f || (a.adj_a != 0.f && a.adj_d < 0.f)) return 0;   // a negative adjacency weight (or decay) raises logits
    if (penal && a.freq > 0.f && a.mu > 0.f && a.allow_dev) return 0;   // so does the deficit bonus
    if (penal && a.picks_bound <= 0) return 0;
    const int keep = a.top_k < a.V ? a.top_k : a.V;
    int need = keep + (penal ? a.picks_bound : 0), Kc = 32;
    while (Kc < need) Kc <<= 1;
    if (Kc > SC_MAXC || Kc > a.V) return 0;
    if (mode != 2 && a.V < 8 * Kc) return 0;                    // nothing to gain on short rows
    return Kc;
}

size_t sample_scratch_floats(int Bn, int V) { return V > SM_SMEM_V ? (size_t)Bn * V : 0; }

// ---- large candidate sets (top_k = 0 or > 2048 over a big vocabulary, one position per row) ----
// The rows are sorted once (value descending, index ascending on ties: a stable device-wide
// radix sort) and one CTA per row then walks it with block-wide fp64 prefix sums: the
// nucleus cut "cum_before - p > top_p" and the draw "u <= cum" are monotone in the sorted
// rank, so each is the minimum rank that satisfies a predicate. Sums are formed in a
// different order than the reference's sequential loop (relative differences ~1e-16).
constexpr int SL_THREADS = 1024;

__global__ void k_sort_prep(const float *__restrict__ logits, float temp, int64_t n, int V, float *__restrict__ keys, int *__restrict__ idx) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        keys[i] = logits[i] / temp;
        idx[i] = (int)(i % V);
    }
}

// all rows in ONE device-wide sort: key = row << 32 | (0xffffffff - ordered value bits), ascending, so rows stay in
// order and every row comes out largest value first (the sort is stable: equal values keep ascending indices)
__global__ void k_sort_prep64(const float *__restrict__ logits, float temp, int64_t n, int V, unsigned long long *__restrict__ keys,
                              int *__restrict__ idx) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        keys[i] = ((unsigned long long)(i / V) << 32) | (unsigned long long)(0xffffffffu - okey(logits[i] / temp));
        idx[i] = (int)(i % V);
    }
}

__device__ __forceinline__ double block_excl_scan(double v, double *sm, double *total) {
    // exclusive scan of one value per thread over SL_THREADS threads
    int tid = threadIdx.x;
    sm[tid] = v;
    __syncthreads();
    for (int off = 1; off < SL_THREADS; off <<= 1) {
        double t = tid >= off ? sm[tid - off] : 0.0;
        __syncthreads();
        sm[tid] += t;
        __syncthreads();
    }
    double incl = sm[tid];
    *total = sm[SL_THREADS - 1];
    __syncthreads();
    return incl - v;
}

// K64: keys are the composite 64-bit keys of k_sort_prep64 (the value is recovered from the low word)
template <bool K64>
__global__ void __launch_bounds__(SL_THREADS) k_pick_sorted(const void *__restrict__ keys, const int *__restrict__ idx, double *__restrict__ pcache, int V, int keep,
                                                           float top_p, const double *__restrict__ uniforms,
                                                           unsigned long long seed, long long row0, int level,
                                                           int *__restrict__ out, int out_stride, int out_off) {
    __shared__ double sm[SL_THREADS];
    __shared__ int s_min;
    const int b = blockIdx.x, tid = threadIdx.x;
    const float *kf = (const float *)keys + (size_t)b * V;
    const unsigned long long *k8 = (const unsigned long long *)keys + (size_t)b * V;
    auto val = [&](int r) -> double {
        if (K64) return (double)okey_inv(0xffffffffu - (unsigned)(k8[r] & 0xffffffffull));
        return (double)kf[r];
    };
    const int *ir = idx + (size_t)b * V;
    const double mx = val(0);
    const int chunk = (keep + SL_THREADS - 1) / SL_THREADS;
    const int r0 = tid * chunk, r1 = min(r0 + chunk, keep);
    double local = 0;
    // the exponentials are taken once and kept: the passes below read them back. A thread's i-th entry sits at
    // [i][thread], so that a warp's accesses fall into one line although every thread walks its own run of ranks
    double *pc = pcache + (size_t)b * ((size_t)chunk * SL_THREADS) + tid;
    for (int r = r0; r < r1; r++) { const double p = exp(val(r) - mx); pc[(size_t)(r - r0) * SL_THREADS] = p; local += p; }
    double den;
    const double base = block_excl_scan(local, sm, &den);
    // nucleus cut: first rank with (cum_before - p) / den > top_p
    if (tid == 0) s_min = keep;
    __syncthreads();
    {
        double cum = base;
        for (int r = r0; r < r1; r++) {
            double p = pc[(size_t)(r - r0) * SL_THREADS];
            if ((cum - p) / den > (double)top_p) { atomicMin(&s_min, r); break; }
            cum += p;
        }
    }
    __syncthreads();
    const int nkeep = s_min;
    __syncthreads();
    // mass of the kept prefix
    double lk = 0;
    for (int r = r0; r < r1 && r < nkeep; r++) lk += pc[(size_t)(r - r0) * SL_THREADS];
    double den2;
    const double base2 = block_excl_scan(lk, sm, &den2);
    const double u01 = uniforms ? uniforms[b] : counter_uniform(seed, row0 + b, level, 0);
    const double u = u01 * den2;
    if (tid == 0) s_min = nkeep - 1;
    __syncthreads();
    {
        double acc = base2;
        for (int r = r0; r < r1 && r < nkeep; r++) {
            acc += pc[(size_t)(r - r0) * SL_THREADS];
            if (u <= acc) { atomicMin(&s_min, r); break; }
        }
    }
    __syncthreads();
    if (tid == 0) out[(size_t)b * out_stride + out_off] = ir[s_min < 0 ? 0 : s_min];
}

// ---- the same draw without sorting the row (top_k = 0: the nucleus is cut from the whole vocabulary) ----
// With seeded or near-uniform logits the nucleus holds most of a 150 K vocabulary, so the sort above is the
// sampler. Both the cut ("cum_before - p > top_p") and the draw ("u <= cum") are the first rank at which a
// monotone predicate over cumulative probability turns true. One sweep of the row sums its probability mass by distance
// below the maximum (bins of 1/64), one lists the elements of the bins the cut and the draw can fall into, and one CTA
// per row settles both on the lists. Lists that are too long (ties) are settled the way a radix select finds a rank: three
// passes over the row's ordered 32-bit keys (11 + 11 + 10 bits), descending into the bin where the predicate flips.
// Probabilities are accumulated as 64-bit fixed point (2^-44 steps, exact and order-independent integer
// sums, so runs are reproducible whatever order the atomics land in); the absolute error of a cumulative sum is
// below 1e-11 of the row's mass, which moves a draw only when it falls that close to a boundary. Ties of equal
// logits are ranked by ascending index, like the stable sort.
constexpr int NS_THREADS = 1024, ND_THREADS = 512;
constexpr int NS_BINS = 2048;
constexpr double NS_FIX = 17592186044416.0;                       // 2^44

struct NsHist {
    unsigned long long sum[NS_BINS];
    unsigned cnt[NS_BINS];
    unsigned kmin_inv[NS_BINS];       // ~(smallest key of the bin)
    __device__ __forceinline__ bool any(int i) const { return cnt[i] != 0; }
};
// Mass by distance below the row's largest value: bin NS_BINS - 1 holds [0, 1/64) and so on down to 32, where exp() is below half a
// unit of mass. Distances spread logits over most of the bins (top key bits put a whole octave of values into four).
struct NsDist {
    unsigned long long sum[NS_BINS];
    unsigned kmin_inv[NS_BINS];       // ~(smallest key of the bin); 0: empty
    __device__ __forceinline__ bool any(int i) const { return kmin_inv[i] != 0; }
};
// Per-row state; zeroed before the first kernel.
struct NsRow {
    unsigned maxkey;
    int n_nuc, n_pick;                 // entries on the row's two lists
    int nuc;                           // bin the nucleus cut lies in; -1: everything is kept
    unsigned long long total, nuc_above, pick_above;     // mass of the row; above the cut's bin; above the draw's first bin
};
constexpr int NS_LIST = 2048;          // (key, index) entries a list holds

__device__ __forceinline__ int ns_bin(float mx, float x) {        // monotone in x; -1: no mass
    const float d = mx - x;
    return d < 32.f ? NS_BINS - 1 - (int)(d * 64.f) : -1;
}
__device__ __forceinline__ unsigned long long ns_q_of_key(unsigned key, double mx, const double *tab) {
    // (adding 2^52 rounds to an integer, in the low bits of the sum)
    return (unsigned long long)__double_as_longlong(fma(exp_tab((double)okey_inv(key) - mx, tab), NS_FIX, 4503599627370496.0)) & 0xfffffffffffffull;
}

// exclusive block scan of one u64 per thread (NS_THREADS threads); every thread gets its prefix
__device__ __forceinline__ unsigned long long ns_block_excl_scan(unsigned long long v, unsigned long long *wsum) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    __syncthreads();                                               // wsum may still be read from an earlier call
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    unsigned long long base = 0;
    for (int w = 0; w < warp; w++) base += wsum[w];
    return base + x - v;
}

// One level of a descent over a histogram of `nbins` bins, highest bin first. NUCLEUS: the first bin whose LAST
// element satisfies cum_before - p > T (the cut then lies inside that bin or exactly in front of it; the descent
// into the bin settles which). Otherwise: the first bin with cum_incl >= T. Results through shared memory:
// *sel = bin (-1: no bin satisfies), *sel_above = mass above that bin.
template <bool NUCLEUS, class H>
__device__ void ns_decide(const H *h, int nbins, unsigned long long above, double T, double mx, const double *tab, unsigned long long *wsum, int *sel,
                          unsigned long long *sel_above) {
    const int tid = threadIdx.x;
    unsigned long long s[2]; int bin[2];
#pragma unroll
    for (int e = 0; e < 2; e++) {
        const int d = 2 * tid + e;
        bin[e] = nbins - 1 - d;
        s[e] = (d < nbins) ? h->sum[bin[e]] : 0ull;
    }
    if (tid == 0) *sel = 0x7fffffff;
    const unsigned long long ex = ns_block_excl_scan(s[0] + s[1], wsum);    // contains a __syncthreads after the init above
    unsigned long long ab = above + ex;
#pragma unroll
    for (int e = 0; e < 2; e++) {
        const int d = 2 * tid + e;
        if (d < nbins && h->any(bin[e])) {
            bool hit;
            if (NUCLEUS) {
                const unsigned kmin = ~h->kmin_inv[bin[e]];
                const long long g = (long long)(ab + s[e]) - 2ll * (long long)ns_q_of_key(kmin, mx, tab);
                hit = (double)g > T;
            } else {
                hit = (double)(ab + s[e]) >= T;
            }
            if (hit) atomicMin(sel, d);
        }
        ab += s[e];
    }
    __syncthreads();
    const int dsel = *sel;
    __syncthreads();
    if (dsel == 0x7fffffff) { if (tid == 0) *sel = -1; __syncthreads(); return; }
    if (dsel >> 1 == tid) {
        const int e = dsel & 1;
        const unsigned long long a0 = above + ex + (e ? s[0] : 0ull);
        *sel = bin[e];
        *sel_above = a0;
    }
    __syncthreads();
}

// (the largest quotient is the quotient of the largest: one division a thread, not one an element)
__global__ void __launch_bounds__(NS_THREADS) k_ns_max(const float *__restrict__ logits, float temp, int V, NsRow *rows) {
    const int b = blockIdx.y, stride = gridDim.x * NS_THREADS;
    const float *lg = logits + (size_t)b * V;
    float m = -INFINITY;
    for (int i0 = blockIdx.x * NS_THREADS + threadIdx.x; i0 < V; i0 += 8 * stride) {
        float x[8];
#pragma unroll
        for (int u = 0; u < 8; u++) x[u] = i0 + u * stride < V ? lg[i0 + u * stride] : -INFINITY;
#pragma unroll
        for (int u = 0; u < 8; u++) m = fmaxf(m, x[u]);
    }
    unsigned k = okey(m / temp);
    for (int o = 16; o; o >>= 1) k = max(k, __shfl_xor_sync(0xffffffffu, k, o));
    if ((threadIdx.x & 31) == 0) atomicMax(&rows[b].maxkey, k);
}

// mass by distance: one sweep over the logits, the masses as 16-bit limbs (mass below 2^32 or 2^16 -- most of a row -- takes fewer
// atomics); at most 2^16 elements per CTA
__global__ void __launch_bounds__(ND_THREADS) k_ns_dist(const float *__restrict__ logits, float temp, int V, const NsRow *rows, NsDist *dist) {
    __shared__ unsigned s0[NS_BINS], s1[NS_BINS], s2[NS_BINS], km[NS_BINS];
    __shared__ double tab[EXP_TAB];
    exp_tab_fill(tab);
    const int b = blockIdx.y, tid = threadIdx.x;
    const float *lg = logits + (size_t)b * V;
    const unsigned mk = rows[b].maxkey;
    const float mxf = okey_inv(mk);
    const double mx = (double)mxf;
    for (int i = tid; i < NS_BINS; i += ND_THREADS) { s0[i] = 0; s1[i] = 0; s2[i] = 0; km[i] = 0; }
    __syncthreads();
    const int v0 = (int)((long long)V * blockIdx.x / gridDim.x), v1 = (int)((long long)V * (blockIdx.x + 1) / gridDim.x);
    for (int i0 = v0 + tid; i0 < v1; i0 += 4 * ND_THREADS) {
        float x[4];
#pragma unroll
        for (int u = 0; u < 4; u++) x[u] = i0 + u * ND_THREADS < v1 ? lg[i0 + u * ND_THREADS] / temp : -INFINITY;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int bin = ns_bin(mxf, x[u]);
            if (bin < 0) continue;
            const unsigned k = okey(x[u]);
            const unsigned long long q = ns_q_of_key(k, mx, tab);
            const unsigned mid = (unsigned)(q >> 16) & 0xffffu, hi = (unsigned)(q >> 32);
            atomicAdd(&s0[bin], (unsigned)q & 0xffffu);
            if (mid) atomicAdd(&s1[bin], mid);
            if (hi) atomicAdd(&s2[bin], hi);
            if (~k > *(volatile unsigned *)&km[bin]) atomicMax(&km[bin], ~k);      // (rarely: a bin's minimum settles early)
        }
    }
    __syncthreads();
    NsDist *D = dist + b;
    for (int i = tid; i < NS_BINS; i += ND_THREADS)
        if (km[i]) {
            atomicAdd(&D->sum[i], (unsigned long long)s0[i] + ((unsigned long long)s1[i] << 16) + ((unsigned long long)s2[i] << 32));
            atomicMax(&D->kmin_inv[i], km[i]);
        }
}

// The bin of the nucleus cut and the bins the draw can fall into (the kept mass lies between the masses above and through the
// cut's bin); their elements go on the row's lists. Every CTA of a row repeats the decision.
__global__ void __launch_bounds__(NS_THREADS) k_ns_collect(const float *__restrict__ logits, float temp, int V, float top_p, const double *__restrict__ uniforms,
                                                           unsigned long long seed, long long row0, int level, NsRow *rows, const NsDist *dist,
                                                           unsigned long long *lists) {
    __shared__ unsigned long long wsum[32], s_above, s_total;
    __shared__ double tab[EXP_TAB];
    __shared__ int s_sel;
    exp_tab_fill(tab);
    const int b = blockIdx.y, tid = threadIdx.x;
    NsRow *row = rows + b;
    const NsDist *D = dist + b;
    const float mxf = okey_inv(row->maxkey);
    const double mx = (double)mxf;
    const unsigned long long two = D->sum[2 * tid] + D->sum[2 * tid + 1], ex = ns_block_excl_scan(two, wsum);
    if (tid == NS_THREADS - 1) s_total = ex + two;
    __syncthreads();
    const unsigned long long total = s_total;
    int nuc = -1;
    unsigned long long lo = total, hi = total, na = 0, pa = 0;       // bounds of the kept mass
    if (top_p < 1.0f) {
        ns_decide<true>(D, NS_BINS, 0ull, (double)top_p * (double)total, mx, tab, wsum, &s_sel, &s_above);
        nuc = s_sel;
        if (nuc >= 0) { na = s_above; lo = na; hi = na + D->sum[nuc]; }
        __syncthreads();
    }
    const double u01 = uniforms ? uniforms[b] : counter_uniform(seed, row0 + b, level, 0);
    ns_decide<false>(D, NS_BINS, 0ull, u01 * (double)lo, mx, tab, wsum, &s_sel, &s_above);
    const int p0 = s_sel < 0 ? NS_BINS - 1 : s_sel;
    if (s_sel >= 0) pa = s_above;
    __syncthreads();
    ns_decide<false>(D, NS_BINS, 0ull, u01 * (double)hi, mx, tab, wsum, &s_sel, &s_above);
    const int p1 = s_sel < 0 ? 0 : s_sel;                            // p1 <= p0: bins count downwards
    if (blockIdx.x == 0 && tid == 0) { row->nuc = nuc; row->total = total; row->nuc_above = na; row->pick_above = pa; }
    const float *lg = logits + (size_t)b * V;
    unsigned long long *Ln = lists + (size_t)b * 2 * NS_LIST, *Lp = Ln + NS_LIST;
    const int v0 = (int)((long long)V * blockIdx.x / gridDim.x), v1 = (int)((long long)V * (blockIdx.x + 1) / gridDim.x);
    // almost every element lies below all of these bins: told by one comparison, with room for the rounding of both sides
    const float far = (float)(NS_BINS - (nuc >= 0 ? min(nuc, p1) : p1)) / 64.f, least = (mxf - far) * temp - 1e-5f * (fabsf(mxf) + far + 1.f) * temp;
    for (int i0 = v0 + tid; i0 < v1; i0 += 8 * NS_THREADS) {
        float x[8];
#pragma unroll
        for (int u = 0; u < 8; u++) x[u] = i0 + u * NS_THREADS < v1 ? lg[i0 + u * NS_THREADS] : -INFINITY;
#pragma unroll
        for (int u = 0; u < 8; u++) {
            if (x[u] < least) continue;
            const float y = x[u] / temp;
            const int bin = ns_bin(mxf, y);
            if (bin < 0 || (bin != nuc && (bin > p0 || bin < p1))) continue;
            const unsigned long long e = ((unsigned long long)okey(y) << 32) | (unsigned)(0xffffffffu - (unsigned)(i0 + u * NS_THREADS));
            if (bin == nuc) { const int at = atomicAdd(&row->n_nuc, 1); if (at < NS_LIST) Ln[at] = e; }
            if (bin <= p0 && bin >= p1) { const int at = atomicAdd(&row->n_pick, 1); if (at < NS_LIST) Lp[at] = e; }
        }
    }
}

// Shared memory of the last kernel: a histogram over key bits with the limbs it is summed from, or a list and its masses.
struct NsWork { NsHist h; unsigned s0[NS_BINS], s1[NS_BINS], s2[NS_BINS]; };
struct NsListWork { unsigned long long e[NS_LIST], q[NS_LIST]; };
static_assert(sizeof(NsListWork) <= sizeof(NsWork), "the list fits the histogram's place");

// A list too long for NS_LIST (ties, or logits all but equal): one CTA finds the element by descending over the key's bits, 11, 11
// and 10 at a time, each level a sweep over the row. The 45-bit masses are summed as 15-bit limbs, 2^17 elements at a time.
// Returns the key; *above = mass above it, *cnt = elements that hold it; false: no element satisfies.
template <bool NUCLEUS>
__device__ bool ns_descend(const float *lg, float temp, int V, double mx, const double *tab, double T, NsWork *w, unsigned long long *wsum, int *s_sel,
                           unsigned long long *s_above, unsigned *key, unsigned long long *above, long long *cnt) {
    const int tid = threadIdx.x;
    unsigned prefix = 0;
    unsigned long long ab = 0;
    for (int level = 0; level < 3; level++) {
        const int nbins = level < 2 ? NS_BINS : 1024, shift = level == 0 ? 21 : level == 1 ? 10 : 0, fshift = level == 0 ? 32 : level == 1 ? 21 : 10;
        for (int i = tid; i < NS_BINS; i += NS_THREADS) { w->h.sum[i] = 0; w->h.cnt[i] = 0; w->h.kmin_inv[i] = 0; }
        for (int c0 = 0; c0 < V; c0 += 1 << 17) {
            for (int i = tid; i < NS_BINS; i += NS_THREADS) { w->s0[i] = 0; w->s1[i] = 0; w->s2[i] = 0; }
            __syncthreads();
            for (int i = c0 + tid; i < min(V, c0 + (1 << 17)); i += NS_THREADS) {
                const unsigned k = okey(lg[i] / temp);
                if (level > 0 && (k >> fshift) != prefix) continue;
                const int bin = (int)((k >> shift) & (unsigned)(nbins - 1));
                const unsigned long long q = ns_q_of_key(k, mx, tab);
                atomicAdd(&w->s0[bin], (unsigned)(q & 0x7fffull));
                atomicAdd(&w->s1[bin], (unsigned)((q >> 15) & 0x7fffull));
                atomicAdd(&w->s2[bin], (unsigned)(q >> 30));
                atomicAdd(&w->h.cnt[bin], 1u);
                atomicMax(&w->h.kmin_inv[bin], ~k);
            }
            __syncthreads();
            for (int i = tid; i < NS_BINS; i += NS_THREADS)
                w->h.sum[i] += (unsigned long long)w->s0[i] + ((unsigned long long)w->s1[i] << 15) + ((unsigned long long)w->s2[i] << 30);
            __syncthreads();
        }
        ns_decide<NUCLEUS>(&w->h, nbins, ab, T, mx, tab, wsum, s_sel, s_above);
        if (*s_sel < 0) {
            if (NUCLEUS) return false;
            __syncthreads();                                        // rounding put the draw past the last mass: the lowest occupied bin
            if (tid == 0) {
                int bin = 0;
                unsigned long long acc = ab, before = ab;
                for (int i = nbins - 1; i >= 0; i--) if (w->h.cnt[i]) { bin = i; before = acc; acc += w->h.sum[i]; }
                *s_sel = bin; *s_above = before;
            }
            __syncthreads();
        }
        prefix = level == 0 ? (unsigned)*s_sel : (prefix << (level == 1 ? 11 : 10)) | (unsigned)*s_sel;
        ab = *s_above;
        *cnt = (long long)w->h.cnt[*s_sel];
        __syncthreads();
    }
    *key = prefix; *above = ab;
    return true;
}

// The cut and the draw, one CTA per row. On a list, an element's cumulative mass is the mass above the list's bins plus that of the
// list's entries before and with it (key descending, index ascending), summed by every entry for itself.
__global__ void __launch_bounds__(NS_THREADS) k_ns_pick(const float *__restrict__ logits, float temp, int V, float top_p, const double *__restrict__ uniforms,
                                                        unsigned long long seed, long long row0, int level, const NsRow *rows,
                                                        const unsigned long long *lists, int *__restrict__ out, int out_stride, int out_off) {
    extern __shared__ __align__(16) unsigned char nsraw[];
    NsWork *W = (NsWork *)nsraw;
    NsListWork *L = (NsListWork *)nsraw;
    __shared__ unsigned long long wsum[32], s_above, s_hit;
    __shared__ double tab[EXP_TAB];
    __shared__ int s_sel;
    exp_tab_fill(tab);
    __syncthreads();
    const int b = blockIdx.x, tid = threadIdx.x;
    const NsRow *row = rows + b;
    const float *lg = logits + (size_t)b * V;
    const double mx = (double)okey_inv(row->maxkey);
    const unsigned long long total = row->total;
    const double u01 = uniforms ? uniforms[b] : counter_uniform(seed, row0 + b, level, 0);
    // largest entry e of a list for which pred(cumulative mass with e, mass of e) holds -> s_hit (0: none); returns its cumulative mass
    auto first = [&](const unsigned long long *list, int n, unsigned long long above, auto pred) -> unsigned long long {
        if (tid == 0) s_hit = 0;
        for (int i = tid; i < n; i += NS_THREADS) { L->e[i] = list[i]; L->q[i] = ns_q_of_key((unsigned)(list[i] >> 32), mx, tab); }
        __syncthreads();
        unsigned long long best = 0, bc = 0;
        for (int i = tid; i < n; i += NS_THREADS) {
            const unsigned long long e = L->e[i];
            unsigned long long cum = above;
            for (int f = 0; f < n; f++) if (L->e[f] >= e) cum += L->q[f];
            if (e > best && pred(cum, L->q[i])) { best = e; bc = cum; }
        }
        if (best) atomicMax(&s_hit, best);
        __syncthreads();
        if (best && best == s_hit) s_above = bc - ns_q_of_key((unsigned)(best >> 32), mx, tab);   // mass before it
        __syncthreads();
        return s_above;
    };
    // ---- the mass that is kept ----
    unsigned long long den = total;
    if (row->nuc >= 0) {
        const double T = (double)top_p * (double)total;
        if (row->n_nuc <= NS_LIST) {
            const unsigned long long before = first(lists + (size_t)b * 2 * NS_LIST, row->n_nuc, row->nuc_above,
                                                    [&](unsigned long long cum, unsigned long long q) { return (double)((long long)cum - 2ll * (long long)q) > T; });
            if (s_hit) den = before;
        } else {
            unsigned key; unsigned long long above; long long cnt;
            if (ns_descend<true>(lg, temp, V, mx, tab, T, W, wsum, &s_sel, &s_above, &key, &above, &cnt)) {
                // the j-th of the key's cnt elements (mass qk each, ascending index) has cum_before - p = above + (j - 1) qk; the
                // cut is the first j for which that exceeds T
                const unsigned long long qk = ns_q_of_key(key, mx, tab);
                long long j = 0;
                if (qk > 0) {
                    j = (long long)floor((T - (double)above) / (double)qk) + 1;
                    if (j < 0) j = 0;
                    if (j > cnt) j = cnt;
                    while (j > 0 && (double)((long long)above + (j - 2) * (long long)qk) > T) j--;
                    while (j < cnt && !((double)((long long)above + (j - 1) * (long long)qk) > T)) j++;
                }
                den = above + (unsigned long long)j * qk;
            }
        }
        __syncthreads();
    }
    // ---- the draw ----
    const double U = u01 * (double)den;
    int *o = out + (size_t)b * out_stride + out_off;
    if (row->n_pick <= NS_LIST) {
        first(lists + (size_t)b * 2 * NS_LIST + NS_LIST, row->n_pick, row->pick_above, [&](unsigned long long cum, unsigned long long) { return (double)cum >= U; });
        unsigned long long hit = s_hit;
        if (!hit) {                                                 // rounding put the draw past the last mass: the last entry
            if (tid == 0) { hit = ~0ull; for (int i = 0; i < row->n_pick; i++) hit = min(hit, L->e[i]); }
        }
        if (tid == 0) *o = (int)(0xffffffffu - (unsigned)(hit & 0xffffffffull));
        return;
    }
    unsigned key; unsigned long long above; long long cnt;
    ns_descend<false>(lg, temp, V, mx, tab, U, W, wsum, &s_sel, &s_above, &key, &above, &cnt);
    // the j-th tied element has cum_incl = above + (j + 1) qk: the first j for which that reaches U
    const unsigned long long qk = ns_q_of_key(key, mx, tab);
    long long j = 0;
    if (qk > 0 && cnt > 1) {
        j = (long long)ceil((U - (double)above) / (double)qk) - 1;
        if (j < 0) j = 0;
        if (j > cnt - 1) j = cnt - 1;
        while (j > 0 && (double)(above + (unsigned long long)j * qk) >= U) j--;
        while (j < cnt - 1 && !((double)(above + (unsigned long long)(j + 1) * qk) >= U)) j++;
    }
    // its index: matches per thread slice, scanned
    const int per = (V + NS_THREADS - 1) / NS_THREADS, i0 = min(V, tid * per), i1 = min(V, i0 + per);
    unsigned long long c = 0;
    for (int i = i0; i < i1; i++) c += okey(lg[i] / temp) == key;
    const unsigned long long ex = ns_block_excl_scan(c, wsum);
    if ((unsigned long long)j >= ex && (unsigned long long)j < ex + c) {
        long long need = j - (long long)ex;
        for (int i = i0; i < i1; i++)
            if (okey(lg[i] / temp) == key && need-- == 0) { *o = i; break; }
    }
}

static bool sample_rows_select(const SampleArgs &a) {
    // NCM_B200_SORT_SAMPLER=1 keeps the sort-based path (read per call: tests compare the two on the same rows);
    // NCM_B200_SELECT_MIN_V lowers the vocabulary size from which the selection path is taken (default 4096)
    const char *e = getenv("NCM_B200_SORT_SAMPLER"), *mv = getenv("NCM_B200_SELECT_MIN_V");
    if ((e && atoi(e)) || a.V < (mv ? atoi(mv) : 4096)) return false;
    static Workspace ws;
    const size_t n = (size_t)a.Bn * a.V;
    const size_t head = (size_t)a.Bn * (sizeof(NsDist) + sizeof(NsRow));
    const size_t need = head + (size_t)a.Bn * 2 * NS_LIST * 8 + 8192;
    if (need > ws.cap) ws.reserve(need + need / 8);
    ws.reset();
    NsDist *dist = (NsDist *)ws.alloc(head);
    NsRow *rows = (NsRow *)(dist + a.Bn);
    unsigned long long *lists = ws.get<unsigned long long>((size_t)a.Bn * 2 * NS_LIST);
    ProfScope ps(NCMB_K_SAMPLE, 0, (double)n * 12);
    CUDA_CHECK(cudaMemsetAsync(dist, 0, head, stream()));
    // CTAs per row: one wave of what is resident at once, where that gives every row one and no limb of a sum can wrap (2^16
    // elements a CTA); else about four waves, so that the last one's idle part is small
    auto parts = [&](int threads, int per_sm, int least) {
        const int res = per_sm * ctx().sm_count, one = res / a.Bn, most = std::min(32, (int)cdiv(a.V, 4 * threads));
        return (unsigned)std::max(std::max(std::min(one >= least ? one : 4 * res / a.Bn, most), least), 1);
    };
    static bool set = false;
    if (!set) { CUDA_CHECK(cudaFuncSetAttribute(k_ns_pick, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(NsWork))); set = true; }
    LAUNCH(k_ns_max, dim3(parts(NS_THREADS, 2, 1), (unsigned)a.Bn), NS_THREADS, 0, a.logits, a.temp, a.V, rows);
    LAUNCH(k_ns_dist, dim3(parts(ND_THREADS, 4, (int)cdiv(a.V, 1 << 16)), (unsigned)a.Bn), ND_THREADS, 0, a.logits, a.temp, a.V, (const NsRow *)rows, dist);
    LAUNCH(k_ns_collect, dim3(parts(NS_THREADS, 2, 1), (unsigned)a.Bn), NS_THREADS, 0, a.logits, a.temp, a.V, a.top_p, a.uniforms, a.rng_seed, a.rng_row0, a.rng_level,
           rows, (const NsDist *)dist, lists);
    LAUNCH(k_ns_pick, (unsigned)a.Bn, NS_THREADS, sizeof(NsWork), a.logits, a.temp, a.V, a.top_p, a.uniforms, a.rng_seed, a.rng_row0, a.rng_level,
           (const NsRow *)rows, (const unsigned long long *)lists, a.out, a.out_stride, a.out_off);
    return true;
}

static void sample_rows_large(const SampleArgs &a, int keep) {
    if (a.Lc != 1 || a.uncond_off || a.freq > 0.f || a.adj_a != 0.f)
        fatal("sampling: more than %d candidates (top_k=%d, V=%d) is supported for single-position rows "
              "without CFG or penalties only; set top_k <= %d", SM_MAXKEEP, a.top_k, a.V, SM_MAXKEEP);
    if (keep == a.V && sample_rows_select(a)) return;
    static Workspace ws;
    const int64_t n = (int64_t)a.Bn * a.V;
    // One row: a device-wide 32-bit radix sort. More rows: ONE device-wide sort of all rows on composite keys
    // (row index above the value bits); a segmented sort gives each row a single CTA, about a millisecond for a
    // 150 K vocabulary whatever the number of rows.
    const bool per_row = a.Bn == 1;
    int row_bits = 1;
    while ((1 << row_bits) < a.Bn) row_bits++;
    size_t temp_bytes = 0;
    if (per_row)
        cub::DeviceRadixSort::SortPairsDescending(nullptr, temp_bytes, (const float *)nullptr, (float *)nullptr,
                                                  (const int *)nullptr, (int *)nullptr, a.V, 0, 32, stream());
    else
        cub::DeviceRadixSort::SortPairs(nullptr, temp_bytes, (const unsigned long long *)nullptr, (unsigned long long *)nullptr,
                                        (const int *)nullptr, (int *)nullptr, n, 0, 32 + row_bits, stream());
    const size_t pc_per_row = (size_t)cdiv(keep, SL_THREADS) * SL_THREADS;
    size_t need = (size_t)n * 24 + (size_t)a.Bn * pc_per_row * 8 + temp_bytes + 8192;
    if (need > ws.cap) ws.reserve(need);
    ws.reset();
    ProfScope ps(NCMB_K_SAMPLE, 0, (double)n * 40);
    int64_t g = cdiv(n, 256), cap = (int64_t)ctx().sm_count * 16;
    cudaError_t e = cudaSuccess;
    if (per_row) {
        float *k_in = ws.get<float>(n), *k_out = ws.get<float>(n);
        int *i_in = ws.get<int>(n), *i_out = ws.get<int>(n);
        void *temp = ws.alloc(temp_bytes);
        double *pcache = ws.get<double>((size_t)a.Bn * pc_per_row);
        LAUNCH(k_sort_prep, (unsigned)(g > cap ? cap : g), 256, 0, a.logits, a.temp, n, a.V, k_in, i_in);
        e = cub::DeviceRadixSort::SortPairsDescending(temp, temp_bytes, k_in, k_out, i_in, i_out, a.V, 0, 32, stream());
        ctx().launches += 7;
        if (e != cudaSuccess) fatal("radix sort failed: %s", cudaGetErrorString(e));
        LAUNCH(k_pick_sorted<false>, (unsigned)a.Bn, SL_THREADS, 0, (const void *)k_out, (const int *)i_out, pcache, a.V, keep, a.top_p, a.uniforms, a.rng_seed,
               a.rng_row0, a.rng_level, a.out, a.out_stride, a.out_off);
    } else {
        unsigned long long *k_in = ws.get<unsigned long long>(n), *k_out = ws.get<unsigned long long>(n);
        int *i_in = ws.get<int>(n), *i_out = ws.get<int>(n);
        void *temp = ws.alloc(temp_bytes);
        double *pcache = ws.get<double>((size_t)a.Bn * pc_per_row);
        LAUNCH(k_sort_prep64, (unsigned)(g > cap ? cap : g), 256, 0, a.logits, a.temp, n, a.V, k_in, i_in);
        e = cub::DeviceRadixSort::SortPairs(temp, temp_bytes, k_in, k_out, i_in, i_out, n, 0, 32 + row_bits, stream());
        ctx().launches += 2 * ((32 + row_bits + 7) / 8) + 1;
        if (e != cudaSuccess) fatal("radix sort failed: %s", cudaGetErrorString(e));
        LAUNCH(k_pick_sorted<true>, (unsigned)a.Bn, SL_THREADS, 0, (const void *)k_out, (const int *)i_out, pcache, a.V, keep, a.top_p, a.uniforms, a.rng_seed,
               a.rng_row0, a.rng_level, a.out, a.out_stride, a.out_off);
    }
}

void sample_rows(const SampleArgs &a) {
    if (a.Bn <= 0 || a.Lc <= 0) return;
    if (a.temp > 0.f) {
        int keep = (a.top_k > 0) ? (a.top_k < a.V ? a.top_k : a.V) : a.V;
        if (keep > SM_MAXKEEP) { sample_rows_large(a, keep); return; }
    }
    if (const int Kc = two_phase_width(a)) {
        // parts of a row: one where the entries of a row fit a CTA's registers; long rows so that few of them still occupy the GPU
        const int rows = a.Bn * a.Lc;
        int G = 1;
        if (a.V > TC_T * 32) {
            const int want = (2 * ctx().sm_count + rows - 1) / rows, cap = std::min(std::min(TC_MAXPARTS, (int)cdiv(a.V, TC_T * 8)), TC_T * 16 / Kc);
            G = std::max((int)cdiv(a.V, TC_T * 32), std::min(want, cap));
        }
        static unsigned long long *cand = nullptr; static size_t cand_cap = 0;
        const size_t need = (size_t)rows * Kc * (G > 1 ? G + 1 : 1);
        if (need > cand_cap) {
            if (cand) { CUDA_CHECK(cudaStreamSynchronize(stream())); dev_free(cand); }
            cand = (unsigned long long *)dev_alloc(need * 8); cand_cap = need;
        }
        SampleCand sc;
        sc.a = a; sc.Kc = Kc; sc.cand = cand;
        unsigned long long *parts = cand + (size_t)rows * Kc;
        ProfScope ps(NCMB_K_SAMPLE, 0, (double)rows * a.V * (a.uncond_off ? 8 : 4));
        for (int r0 = 0; r0 < a.Bn; r0 += 65535 / a.Lc) {
            // (grid.y holds 65535 rows x positions)
            const int nb = std::min(a.Bn - r0, 65535 / a.Lc);
            SampleCand c = sc;
            const size_t at = (size_t)r0 * a.Lc;
            c.a.logits += at * a.V; if (c.a.blend_out) c.a.blend_out += at * a.V;
            c.cand += at * Kc;
            const dim3 grid((unsigned)G, (unsigned)(nb * a.Lc));
            const int64_t n = cdiv(a.V, G);
            if (n <= TC_T * 4) LAUNCH(k_sample_topc<4>, grid, TC_T, 0, c, parts + at * G * Kc);
            else if (n <= TC_T * 8) LAUNCH(k_sample_topc<8>, grid, TC_T, 0, c, parts + at * G * Kc);
            else if (n <= TC_T * 16) LAUNCH(k_sample_topc<16>, grid, TC_T, 0, c, parts + at * G * Kc);
            else LAUNCH(k_sample_topc<32>, grid, TC_T, 0, c, parts + at * G * Kc);
        }
        if (G > 1) {
            if (G * Kc <= TC_T * 4) LAUNCH(k_sample_merge<4>, (unsigned)rows, TC_T, 0, sc, (const unsigned long long *)parts, G);
            else LAUNCH(k_sample_merge<16>, (unsigned)rows, TC_T, 0, sc, (const unsigned long long *)parts, G);
        }
        LAUNCH(k_sample_seq, (unsigned)a.Bn, Kc, 0, sc);           // one thread per candidate
        return;
    }
    SampleDev sd;
    sd.a = a;
    sd.vals_in_smem = a.V <= SM_SMEM_V;
    if (!sd.vals_in_smem && !a.scratch) fatal("sampling: V=%d needs a scratch buffer", a.V);
    size_t smem = 16 * (size_t)SM_MAXKEEP + (sd.vals_in_smem ? sizeof(float) * (size_t)a.V : 0);
    static size_t attr = 0;
    if (smem > attr) {
        CUDA_CHECK(cudaFuncSetAttribute(k_sample, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(16 * SM_MAXKEEP + 4 * SM_SMEM_V)));
        attr = 16 * SM_MAXKEEP + 4 * SM_SMEM_V;
    }
    ProfScope ps(NCMB_K_SAMPLE, 0, (double)a.Bn * a.Lc * a.V * (a.uncond_off ? 8 : 4));
    LAUNCH(k_sample, (unsigned)a.Bn, SM_THREADS, smem, sd);
}

} // namespace ncmb

// Diagnostic: the device sampler on caller-supplied DEVICE rows, one position per row, no CFG and no penalties --
// sample_topkp's rule (src/kernels.c:794-825) with the uniform of row b taken from uniforms[b] (device doubles in
// [0, 1)). picks: device int[B].
extern "C" void ncmb_sample_rows_dev(const float *logits, int B, int V, float temp, int top_k, float top_p,
                                     const double *uniforms, int *picks) {
    using namespace ncmb;
    ensure_device();
    SampleArgs s{};
    s.logits = logits; s.Bn = B; s.Lc = 1; s.V = V; s.temp = temp; s.top_k = top_k; s.top_p = top_p;
    s.uniforms = uniforms; s.out = picks; s.out_stride = 1; s.out_off = 0; s.picks_bound = 1;
    float *scr = nullptr;
    const size_t need = sample_scratch_floats(B, V);
    if (need) { scr = (float *)dev_alloc(need * 4); s.scratch = scr; }
    sample_rows(s);
    CUDA_CHECK(cudaStreamSynchronize(stream()));
    if (scr) dev_free(scr);
}

// Host-side sampling helper of the reference kernel API (src/ncm.h:197): logits is a
// host row; same algorithm and the same single uniform draw per call.
static const float *g_sort_vals;
static int cmp_desc_idx(const void *pa, const void *pb) {
    float va = g_sort_vals[*(const int *)pa], vb = g_sort_vals[*(const int *)pb];
    return (va < vb) - (va > vb);
}
extern "C" int sample_topkp(const float *logits, int V, float temp, int top_k, float top_p, unsigned long long *rng) {
    if (!(temp > 0)) return argmax_row(logits, V);
    float *work = (float *)malloc((size_t)V * sizeof(float));
    int *ord = (int *)malloc((size_t)V * sizeof(int));
    double *probs = (double *)malloc((size_t)V * sizeof(double));
    if (!work || !ord || !probs) ncmb::fatal("oom in sample_topkp");
    for (int i = 0; i < V; i++) { work[i] = logits[i] / temp; ord[i] = i; }
    g_sort_vals = work;
    qsort(ord, (size_t)V, sizeof(int), cmp_desc_idx);
    int keep = (top_k > 0) ? (top_k < V ? top_k : V) : V;
    double mx = work[ord[0]], den = 0;
    for (int r = 0; r < keep; r++) { probs[r] = exp((double)work[ord[r]] - mx); den += probs[r]; }
    for (int r = 0; r < keep; r++) probs[r] /= den;
    double cum = 0;
    int nkeep = keep;
    for (int r = 0; r < keep; r++) { if (cum - probs[r] > top_p) { nkeep = r; break; } cum += probs[r]; }
    den = 0;
    for (int r = 0; r < nkeep; r++) den += probs[r];
    double u = (double)(rng_next(rng) >> 11) * (1.0 / 9007199254740992.0) * den, acc = 0;
    int pick = ord[nkeep - 1];
    for (int r = 0; r < nkeep; r++) { acc += probs[r]; if (u <= acc) { pick = ord[r]; break; } }
    free(work); free(ord); free(probs);
    return pick;
}
