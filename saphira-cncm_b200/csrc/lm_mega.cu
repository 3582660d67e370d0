// One decode step of one sequence (head dim 64) as ONE persistent kernel: every layer and the vocabulary projection.
//
// A step streams all weights once (4.6 us of HBM time a layer for the Qwen2 shape in bf16) through five products that depend on
// one another; as separate kernels each boundary and each cold start of the weight stream costs several times that (28 us a
// layer). Here one CTA per SM stays for the whole step:
//
//   * Weights. A model's rows are dealt to the CTAs once, and each CTA's rows of all layers lie in one buffer in the order it
//     uses them. A producer warp copies that stream through a 128 KB ring in shared memory (bulk copies of 8 KB), as far ahead
//     as the ring allows, whatever the other warps wait for: the stream only pauses when the ring is full.
//   * Exchange. A product's results are needed by all CTAs (the hidden state) or many (attention). They travel as 8-byte words
//     {value, tag}, written with one store and polled by whoever needs them; the tag is the layer's number in the generate, so
//     a word says itself whether it has arrived. That is one trip through L2 per hop instead of fence, barrier and read.
//     A buffer is written again one layer later, which cannot happen before every CTA has read it: the new value depends, by
//     way of the MLP that all CTAs take part in (I >= the number of CTAs), on results each of them produced after its read. The
//     MLP's own results are read by the CTAs that own hidden rows only, and the next ones depend on those rows.
//   * Products. Sixteen warps: four quarters of K x four groups of rows. A lane keeps its eight elements of the input in
//     registers; eight rows at a time meet in a reduce-scatter.
//
// One row only: 670 us a sampled step for the Qwen2 shape (the kernel chain: 757) and 306 for GPT-2 in fp32 (308). What is left is the
// six exchanges of a layer, about 1 us each, and the reductions between them; from two rows on the few-row kernel chain is faster
// (greedy steps of two rows 620 us and of four 725, against 837 and 1187 here with the sampler).
//
// Hops of a layer: hidden -> q k v -> attention partials -> hidden -> MLP -> hidden. Every wait is bounded (2 s): a wait that
// runs out records a code, the other CTAs see it and stop waiting, and the kernel ends.
#include "lm_mega.cuh"
#include "tc_common.cuh"
#include "tc_epilogue.cuh"

#include <algorithm>

namespace ncmb {

constexpr int MS_WARPS = 16, MS_T = MS_WARPS * 32;       // consumer threads; one more warp feeds the ring
constexpr int MS_CH = 8192, MS_SLOTS = 16, MS_RING = MS_CH * MS_SLOTS;
constexpr int MS_MAXC = 1024, MS_MAXI = 8192, MS_MAXNL = 256, MS_MAXSPLIT = 4, MS_PW = 66;       // words of an attention partial: max, sum, context
constexpr int MS_UPROWS = 128, MS_HROWS = 64;            // rows a CTA may have of an up-projection; vocabulary rows per round

// Rows of `rowb` bytes that may be in use at once: wherever in a chunk the first of them starts, they and what shares their chunks fit
// the ring. What needs more rows than that gives the first ones back in between, or the stream would wait for itself.
__host__ __device__ constexpr int ms_hold(long long rowb) { return (int)((MS_RING - MS_CH) / rowb); }
constexpr int MS_RGRP = 32;                              // rows of a [..][C] product in use at once: four groups of warps x eight rows
static_assert(ms_hold((long long)MS_MAXI * 4) >= 1, "a down-projection row has to fit the ring");

// contiguous share of n items for CTA c of g
__host__ __device__ __forceinline__ int ms_begin(int n, int c, int g) { return (int)((long long)n * c / g); }

struct MsLL {                                            // offsets of the exchange buffers, in words
    size_t x, x1, q, p, h, total;
    __host__ __device__ explicit MsLL(const MegaShape &s) {
        x = 0; x1 = x + s.C; q = x1 + s.C; p = q + s.C + 128 * (size_t)s.nkv; h = p + (size_t)s.H * MS_MAXSPLIT * MS_PW; total = h + s.I;
    }
};
__host__ __device__ __forceinline__ int ms_splits(const MegaShape &s, int grid) {
    const int n = grid / s.H;
    return n < 1 ? 1 : (n > MS_MAXSPLIT ? MS_MAXSPLIT : n);
}

struct MsSm {                                            // fixed part of shared memory, behind the ring
    unsigned long long full[MS_SLOTS], empty[MS_SLOTS];
    int dead;
    float red[2][MS_WARPS];
    float att[MS_WARPS][MS_PW + 2];
    alignas(16) float qn[3][64];                         // this CTA's query head; the new key and value (read as float4)
    float xres[8];                                       // hidden state of the rows this CTA owns
};

__device__ __forceinline__ void ms_bar() { asm volatile("bar.sync 1, %0;" ::"n"(MS_T) : "memory"); }
__device__ __forceinline__ void ll_store(uint2 *p, float v, unsigned tag) {
    asm volatile("st.volatile.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(__float_as_uint(v)), "r"(tag) : "memory");
}
__device__ __forceinline__ uint4 ll_load2(const uint2 *p) {
    uint4 v;
    asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}

struct MsCtx {
    MsSm *sm; int *err;
    // one slow step of a spin: false when the wait is over (limit, or another CTA gave up)
    __device__ __forceinline__ bool still(unsigned &it, unsigned long long &t0) const {
        if ((++it & 255u) != 0) return true;
        if (*(volatile int *)&sm->dead) return false;
        const unsigned long long now = gtime_ns();
        if (t0 == 0) t0 = now;
        if (*(volatile int *)err != 0) { *(volatile int *)&sm->dead = 1; return false; }
        if (now - t0 > TC_WAIT_NS) { atomicExch(err, 61); *(volatile int *)&sm->dead = 1; return false; }
        return true;
    }
    // N pairs of words at p[i] (16-byte aligned); absent ones (null) are zero
    template <int N>
    __device__ __forceinline__ void poll(const uint2 *const (&p)[N], unsigned tag, float2 (&v)[N]) const {
        unsigned it = 0;
        unsigned long long t0 = 0;
        for (;;) {
            uint4 w[N];
            bool ok = true;
#pragma unroll
            for (int i = 0; i < N; i++) w[i] = p[i] ? ll_load2(p[i]) : make_uint4(0u, tag, 0u, tag);
#pragma unroll
            for (int i = 0; i < N; i++) { ok = ok && w[i].y == tag && w[i].w == tag; v[i] = make_float2(__uint_as_float(w[i].x), __uint_as_float(w[i].z)); }
            if (ok || !still(it, t0)) return;
        }
    }
    __device__ __forceinline__ void wait(uint32_t bar, uint32_t parity) const {
        unsigned it = 0;
        unsigned long long t0 = 0;
        for (;;) {
            uint32_t ok;
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                         : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
            if (ok || !still(it, t0)) return;
        }
    }
};

// A warp's view of the weight stream: chunks known to have arrived, chunks given back. Lanes wait for (and give back) different
// chunks at once: one chunk after the other, by all lanes and returned by all warps, these took more of a layer than its products.
struct MsStream {
    const unsigned char *ring; uint32_t full, empty;
    int have = 0, rel = 0;
    __device__ __forceinline__ void ensure(const MsCtx &c, long long end, int lane) {
        const int need = (int)((end + MS_CH - 1) / MS_CH);
        if (need > have) {
            const int k = max(have, rel) + lane;             // (what was given back had arrived)
            if (k < need) c.wait(full + 8 * (k % MS_SLOTS), (uint32_t)(k / MS_SLOTS) & 1u);
            __syncwarp();
            have = need;
        }
    }
    // every byte below `upto` has been read by every warp (a barrier lies between); warp 0 tells the producer
    __device__ __forceinline__ void release(long long upto, int warp, int lane) {
        const int r = (int)(upto / MS_CH);
        if (warp == 0 && rel + lane < r) mbar_arrive(empty + 8 * ((rel + lane) % MS_SLOTS));
        rel = r;
    }
};

// eight weights at byte offset `off` of the stream
template <bool W16>
__device__ __forceinline__ void ms_w8(const unsigned char *ring, uint32_t off, float *w) {
    if (W16) {
        const uint4 u = *(const uint4 *)(ring + (off & (MS_RING - 1)));
        w[0] = __uint_as_float(u.x << 16); w[1] = __uint_as_float(u.x & 0xffff0000u);
        w[2] = __uint_as_float(u.y << 16); w[3] = __uint_as_float(u.y & 0xffff0000u);
        w[4] = __uint_as_float(u.z << 16); w[5] = __uint_as_float(u.z & 0xffff0000u);
        w[6] = __uint_as_float(u.w << 16); w[7] = __uint_as_float(u.w & 0xffff0000u);
    } else {
        const float4 a = *(const float4 *)(ring + (off & (MS_RING - 1))), b = *(const float4 *)(ring + ((off + 16) & (MS_RING - 1)));
        w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
    }
}
// eight sums of 32 lanes: afterwards lane l holds sum number l >> 2 (all four lanes of a group the same)
__device__ __forceinline__ float ms_reduce8(float (&v)[8], int lane) {
#pragma unroll
    for (int w = 4, o = 16; w > 0; w >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < w; i++) {
            const float give = up ? v[i] : v[i + w], keep = up ? v[i + w] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    return v[0];
}

// Rows [r0, r0 + n) of a [..][C] product whose stream begins at `base` (row r0's first byte): a warp takes quarter `warp & 3` of K
// and every fourth row; part[row][quarter].
template <bool W16>
__device__ __forceinline__ void ms_rows(const MsCtx &c, MsStream &st, long long base, int n, int C, const float *xs, float *part, int warp, int lane) {
    const int seg = warp & 3, rg = warp >> 2, L = C >> 5, esz = W16 ? 2 : 4;      // lanes of a quarter
    const bool on = lane < L;
    const long long rowb = (long long)C * esz, lo = (long long)(seg * (C >> 2) + lane * 8) * esz;
    float xr[8];
#pragma unroll
    for (int e = 0; e < 8; e += 4) {
        const float4 v = on ? *(const float4 *)(xs + seg * (C >> 2) + lane * 8 + e) : make_float4(0.f, 0.f, 0.f, 0.f);
        xr[e] = v.x; xr[e + 1] = v.y; xr[e + 2] = v.z; xr[e + 3] = v.w;
    }
    const uint32_t rb = (uint32_t)rowb, at = (uint32_t)(base & (MS_RING - 1)) + (uint32_t)lo + rg * rb;
    for (int b0 = 0; b0 < n; b0 += MS_RGRP) {
        if (b0 > 0) { ms_bar(); st.release(base + (long long)b0 * rowb, warp, lane); }
        st.ensure(c, base + (long long)min(n, b0 + MS_RGRP) * rowb, lane);
        const int i0 = b0 + rg;
        float acc[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            float w[8];
            if (i0 + 4 * j < n && on) ms_w8<W16>(st.ring, at + (b0 + 4 * j) * rb, w);
            else {
#pragma unroll
                for (int e = 0; e < 8; e++) w[e] = 0.f;
            }
            acc[j] = w[0] * xr[0];
#pragma unroll
            for (int e = 1; e < 8; e++) acc[j] = fmaf(w[e], xr[e], acc[j]);
        }
        const float s = ms_reduce8(acc, lane);
        const int r = i0 + 4 * (lane >> 2);
        if ((lane & 3) == 0 && r < n) part[r * 4 + seg] = s;
    }
}

// Down-projection rows [r0, r0 + n), n <= 8: the warp takes 256-wide pieces `warp`, `warp + 16` of K, whose inputs its lanes poll
// straight into registers; part[row][warp]. Rows that do not fit the ring together (seven of the Qwen2-0.5B shape in fp32 are 136 KB) are
// given back in groups. A CTA without rows does not wait for the inputs: nothing that it writes would keep them from being overwritten.
template <bool W16, bool GROUPS>
__device__ __forceinline__ void ms_down(const MsCtx &c, MsStream &st, long long base, int n, int I, const uint2 *hw, unsigned tag, float *part, int warp, int lane) {
    if (n == 0) return;
    const int esz = W16 ? 2 : 4;
    const long long rowb = (long long)I * esz;
    const uint32_t at = (uint32_t)(base & (MS_RING - 1)), rb = (uint32_t)rowb;
    float acc[8], xr[2][8];
#pragma unroll
    for (int j = 0; j < 8; j++) acc[j] = 0.f;
    {
        const uint2 *p[8];
        float2 v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int k = (warp + MS_WARPS * (i >> 2)) * 256 + lane * 8;
            p[i] = k < I ? hw + k + 2 * (i & 3) : nullptr;
        }
        c.poll<8>(p, tag, v);
#pragma unroll
        for (int i = 0; i < 8; i++) { xr[i >> 2][2 * (i & 3)] = v[i].x; xr[i >> 2][2 * (i & 3) + 1] = v[i].y; }
    }
    auto row = [&](int r, float &sum) {
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int k = (warp + MS_WARPS * u) * 256 + lane * 8;
            if (k < I) {
                float w[8];
                ms_w8<W16>(st.ring, at + r * rb + (uint32_t)(k * esz), w);
#pragma unroll
                for (int e = 0; e < 8; e++) sum = fmaf(w[e], xr[u][e], sum);
            }
        }
    };
    if (!GROUPS) {
#pragma unroll
        for (int r = 0; r < 8; r++) {
            if (r >= n) break;
            if ((r & 3) == 0) st.ensure(c, base + min(r + 4, n) * rowb, lane);
            row(r, acc[r]);
        }
    } else {
        const int hold = ms_hold(rowb);
        int g1 = 0;                                          // end of the group in use
#pragma unroll
        for (int r = 0; r < 8; r++) {
            if (r >= n) break;
            if (r == g1) {
                if (r > 0) { ms_bar(); st.release(base + r * rowb, warp, lane); }
                g1 = min(n, r + hold);
                st.ensure(c, base + g1 * rowb, lane);
            }
            row(r, acc[r]);
        }
    }
    const float s = ms_reduce8(acc, lane);
    if ((lane & 3) == 0 && (lane >> 2) < n) part[(lane >> 2) * MS_WARPS + warp] = s;
}

// norm of the row of C values held as pairs by threads t < C / 2, into xs
__device__ __forceinline__ void ms_norm(MsSm *sm, float2 v, int C, int kind, float2 w, float2 b, float eps, float *xs, int tid) {
    const int lane = tid & 31, warp = tid >> 5;
    const bool on = tid < (C >> 1);
    float mean = 0.f;
    auto sum = [&](float s, int k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) sm->red[k][warp] = s;
        ms_bar();
        float t = 0.f;
#pragma unroll
        for (int q = 0; q < MS_WARPS; q++) t += sm->red[k][q];
        return t;
    };
    if (kind == 1) mean = sum(on ? v.x + v.y : 0.f, 0) / (float)C;
    const float d0 = v.x - mean, d1 = v.y - mean;
    const float inv = 1.0f / sqrtf(sum(on ? d0 * d0 + d1 * d1 : 0.f, 1) / (float)C + eps);
    if (on) *(float2 *)(xs + 2 * tid) = make_float2(__fadd_rn(__fmul_rn(__fmul_rn(d0, inv), w.x), b.x), __fadd_rn(__fmul_rn(__fmul_rn(d1, inv), w.y), b.y));
    ms_bar();
}

// attention of query head h of row b over keys [k0, k1): `cached` keys in kv, key `cached` (the new token's) in sm->qn; the
// first four groups of 32 keys were requested by the caller (kf, vf). Partial to p.
struct MsKV { float4 k[4], v[4]; };
__device__ __forceinline__ void ms_kv_load(MsKV &f, const float *kv, int64_t pitch, int kvd, int j0, int k1, int cached, int warp, int lane) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int j = j0 + 32 * i + warp * 2 + (lane >> 4);
        if (j < k1 && j < cached) {
            const float *p = kv + (int64_t)j * pitch + 4 * (lane & 15);
            f.k[i] = *(const float4 *)p; f.v[i] = *(const float4 *)(p + kvd);
        } else f.k[i] = f.v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}
__device__ __forceinline__ void ms_attend(MsSm *sm, MsKV &f, const float *kv, int64_t pitch, int kvd, int k0, int k1, int cached, uint2 *out, unsigned tag, int tid) {
    const int lane = tid & 31, warp = tid >> 5, dp = lane & 15, kg = lane >> 4;
    const float4 q = *(const float4 *)&sm->qn[0][4 * dp];
    float m = -INFINITY, l = 0.f;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int j0 = k0; j0 < k1; j0 += 128) {
        if (j0 > k0) ms_kv_load(f, kv, pitch, kvd, j0, k1, cached, warp, lane);
        float s[4], mx = m;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int j = j0 + 32 * i + warp * 2 + kg;
            if (j == cached) { f.k[i] = *(const float4 *)&sm->qn[1][4 * dp]; f.v[i] = *(const float4 *)&sm->qn[2][4 * dp]; }
            float t = q.x * f.k[i].x;
            t = fmaf(q.y, f.k[i].y, t); t = fmaf(q.z, f.k[i].z, t); t = fmaf(q.w, f.k[i].w, t);
#pragma unroll
            for (int x = 8; x > 0; x >>= 1) t += __shfl_xor_sync(0xffffffffu, t, x);
            s[i] = j < k1 ? t * 0.125f : -INFINITY;          // 1 / sqrt(64)
            mx = fmaxf(mx, s[i]);
        }
        if (mx > -INFINITY) {
            const float al = m == -INFINITY ? 0.f : expf(m - mx);
            l *= al; o.x *= al; o.y *= al; o.z *= al; o.w *= al;
            m = mx;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float p = expf(s[i] - m);
                l += p;
                o.x = fmaf(p, f.v[i].x, o.x); o.y = fmaf(p, f.v[i].y, o.y); o.z = fmaf(p, f.v[i].z, o.z); o.w = fmaf(p, f.v[i].w, o.w);
            }
        }
    }
    // the two halves of the warp, then the warps
    const float m2 = __shfl_xor_sync(0xffffffffu, m, 16), M = fmaxf(m, m2), e = m == -INFINITY ? 0.f : expf(m - M);
    l *= e; o.x *= e; o.y *= e; o.z *= e; o.w *= e;
    l += __shfl_xor_sync(0xffffffffu, l, 16);
    o.x += __shfl_xor_sync(0xffffffffu, o.x, 16); o.y += __shfl_xor_sync(0xffffffffu, o.y, 16);
    o.z += __shfl_xor_sync(0xffffffffu, o.z, 16); o.w += __shfl_xor_sync(0xffffffffu, o.w, 16);
    if (kg == 0) {
        float *a = sm->att[warp];
        if (dp == 0) { a[0] = M; a[1] = l; }
        a[2 + 4 * dp] = o.x; a[3 + 4 * dp] = o.y; a[4 + 4 * dp] = o.z; a[5 + 4 * dp] = o.w;
    }
    ms_bar();
    if (warp < (MS_PW + 31) / 32) {
        const float mw = lane < MS_WARPS ? sm->att[lane][0] : -INFINITY;
        float X = mw;
#pragma unroll
        for (int x = 16; x > 0; x >>= 1) X = fmaxf(X, __shfl_xor_sync(0xffffffffu, X, x));
        const float ew = mw == -INFINITY ? 0.f : expf(mw - X);
        const int d = min(max(tid, 1), MS_PW - 1);
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < MS_WARPS; w++) {
            const float e1 = __shfl_sync(0xffffffffu, ew, w);
            if (e1 != 0.f) t = fmaf(sm->att[w][d], e1, t);
        }
        if (tid < MS_PW) ll_store(out + tid, tid == 0 ? X : t, tag);
    }
}

// GROUPS: a CTA's down-projection rows do not fit the ring together (a variant of its own: the others keep their registers)
template <bool W16, bool GROUPS>
__global__ void __launch_bounds__(MS_T + 32) k_lm_step(const __grid_constant__ MegaArgs a, const unsigned char *stream_w, const long long *stream_off, const unsigned char *head_w) {
    extern __shared__ __align__(1024) unsigned char ms_raw[];
    const MegaShape &S = a.s;
    unsigned char *ring = ms_raw;
    MsSm *sm = (MsSm *)(ring + MS_RING);
    float *xs = (float *)(((uintptr_t)(sm + 1) + 15) & ~(uintptr_t)15);          // [C] input of a product
    MegaLayer *layers = (MegaLayer *)(xs + S.C);                                 // [NL]
    float *part = (float *)(((uintptr_t)(layers + S.NL) + 15) & ~(uintptr_t)15);            // sums by quarter of K (or by warp)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cta = blockIdx.x, g = gridDim.x;
    const int C = S.C, I = S.I, kvd = S.nkv * 64, Wq = C + 2 * kvd, esz = W16 ? 2 : 4;
    // this CTA's share of every product
    const int q0 = ms_begin(Wq >> 1, cta, g), nq = ms_begin(Wq >> 1, cta + 1, g) - q0;        // pairs (d, d + 32) of a head
    const int c0 = ms_begin(C, cta, g), ncr = ms_begin(C, cta + 1, g) - c0;                   // rows of the o- and down-projections
    const int u0 = ms_begin(I, cta, g), nu = ms_begin(I, cta + 1, g) - u0, ur = S.gated ? 2 * nu : nu;
    const int v0 = ms_begin(S.V, cta, g), nv = ms_begin(S.V, cta + 1, g) - v0;
    const long long b_qkv = 2LL * nq * C * esz, b_o = (long long)ncr * C * esz, b_up = (long long)ur * C * esz, b_dn = (long long)ncr * I * esz;
    const long long b_layer = b_qkv + b_o + b_up + b_dn, b_all = b_layer * S.NL, b_head = (long long)nv * C * esz;
    const long long head_at = ((b_all + MS_CH - 1) / MS_CH) * MS_CH;                          // the head starts on a chunk of its own
    const uint32_t full = smem_u32(sm->full), empty = smem_u32(sm->empty);
    if (tid == 0) {
        for (int s = 0; s < MS_SLOTS; s++) { mbar_init(full + 8 * s, 1); mbar_init(empty + 8 * s, 1); }
        sm->dead = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < S.NL * (int)(sizeof(MegaLayer) / 8); i += MS_T + 32) ((unsigned long long *)layers)[i] = ((const unsigned long long *)a.layers)[i];
    __syncthreads();
    MsCtx c{sm, a.err};

    if (warp == MS_WARPS) {                                  // ---- the weight stream ----
        if (lane == 0) {
            const unsigned char *src = stream_w + stream_off[cta], *hsrc = head_w + (long long)v0 * C * esz;
            const int n_body = (int)(head_at / MS_CH), n_all = n_body + (int)((b_head + MS_CH - 1) / MS_CH);
            int k = 0;
            for (; k < n_all; k++) {
                const int s = k % MS_SLOTS;
                if (k >= MS_SLOTS) c.wait(empty + 8 * s, (uint32_t)(k / MS_SLOTS - 1) & 1u);
                if (*(volatile int *)&sm->dead) break;
                const bool body = k < n_body;
                const long long off = (long long)(body ? k : k - n_body) * MS_CH, left = (body ? b_all : b_head) - off;
                const uint32_t bytes = left < MS_CH ? (uint32_t)left : MS_CH;
                mbar_expect_tx(full + 8 * s, bytes);
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             ::"r"(smem_u32(ring + s * MS_CH)), "l"((body ? src : hsrc) + off), "r"(bytes), "r"(full + 8 * s) : "memory");
            }
            for (int j = k - MS_SLOTS < 0 ? 0 : k - MS_SLOTS; j < k; j++)       // every copy has landed before the CTA may end
                mbar_wait(full + 8 * (j % MS_SLOTS), (uint32_t)(j / MS_SLOTS) & 1u, a.err, 62);
        }
        return;
    }

    // ---- consumers ----
    MsStream st{ring, full, empty};
    const MsLL ll(S);
    uint2 *Lx = a.ll + ll.x, *Lx1 = a.ll + ll.x1, *Lq = a.ll + ll.q, *Lp = a.ll + ll.p, *Lh = a.ll + ll.h;
    const int step = *a.step_d, nsp = ms_splits(S, g);
    const unsigned tag0 = (unsigned)step * (unsigned)S.NL + 1u;
    const int pos = a.posmat[step + a.pos_base];
    const bool on2 = tid < (C >> 1);                          // this thread holds elements 2 tid, 2 tid + 1 of a hidden row
    auto pair_of = [&](const float *p, float none) { return p && on2 ? __ldg((const float2 *)p + tid) : make_float2(none, none); };
    // attention share: query head ah, part asp of its keys
    const bool att = cta < S.H * nsp;
    const int ah = att ? cta / nsp : 0, asp = cta % nsp, akv = ah / (S.H / S.nkv);
    const int n_keys = pos + 1, per = (n_keys + nsp - 1) / nsp;
    const int k0 = min(n_keys, asp * per), k1 = min(n_keys, k0 + per);
    auto one = [&](const float *p, bool on, int i) { return p && on ? __ldg(p + i) : 0.f; };
    long long at = 0;                                         // stream offset
    float2 xv[1];
    for (int li = 0; li < S.NL; li++) {
        const MegaLayer &L = layers[li];
        const unsigned tag = tag0 + (unsigned)li;
        const float *kvb = L.kv + akv * 64;
        if (att)                                              // this layer's keys and values: on their way from HBM during the product
            for (int i = tid; i < (k1 - k0) * 4; i += MS_T)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(kvb + (int64_t)(k0 + (i >> 2)) * 2 * kvd + (i & 2 ? kvd : 0) + (i & 1) * 32));
        // ---- hidden state, norm, q k v ----
        {
            const float2 w = pair_of(L.ln1w, 1.f), b = pair_of(L.ln1b, 0.f);
            if (li == 0) {
                xv[0] = make_float2(0.f, 0.f);
                if (on2) {
                    xv[0] = *((const float2 *)(a.wte + (int64_t)a.ids[0] * C) + tid);
                    if (a.wpe) { const float2 p = *((const float2 *)(a.wpe + (int64_t)pos * C) + tid); xv[0].x = __fadd_rn(xv[0].x, p.x); xv[0].y = __fadd_rn(xv[0].y, p.y); }
                }
            } else {
                const uint2 *p[1] = {on2 ? Lx + 2 * tid : nullptr};
                c.poll<1>(p, tag - 1u, xv);
            }
            const int r = 2 * tid - c0;
            if (on2 && r >= 0 && r < ncr) sm->xres[r] = xv[0].x;
            if (on2 && r + 1 >= 0 && r + 1 < ncr) sm->xres[r + 1] = xv[0].y;
            ms_norm(sm, xv[0], C, a.norm, w, b, a.eps, xs, tid);
        }
        ms_rows<W16>(c, st, at, 2 * nq, C, xs, part, warp, lane);
        at += b_qkv;
        ms_bar();
        if (tid < nq) {
            const int h = (q0 + tid) >> 5, d = (q0 + tid) & 31;
            const float4 p0 = *(const float4 *)(part + 8 * tid), p1 = *(const float4 *)(part + 8 * tid + 4);
            float y0 = (p0.x + p0.y) + (p0.z + p0.w), y1 = (p1.x + p1.y) + (p1.z + p1.w);
            y0 += one(L.qkvb, true, h * 64 + d); y1 += one(L.qkvb, true, h * 64 + d + 32);
            if (a.cosb && h < S.H + S.nkv) {
                const float *co = a.cosb + (int64_t)pos * 64 + d, *si = a.sinb + (int64_t)pos * 64 + d;
                const float z0 = __fadd_rn(__fmul_rn(y0, co[0]), __fmul_rn(-y1, si[0])), z1 = __fadd_rn(__fmul_rn(y1, co[32]), __fmul_rn(y0, si[32]));
                y0 = z0; y1 = z1;
            }
            uint2 *o = Lq + h * 64 + d;
            ll_store(o, y0, tag); ll_store(o + 32, y1, tag);
            if (h >= S.H) {
                float *kv = L.kv + (int64_t)pos * 2 * kvd + (h - S.H) * 64 + d;
                kv[0] = y0; kv[32] = y1;
            }
        }
        st.release(at, warp, lane);
        // ---- attention partials ----
        if (att) {
            MsKV f;
            ms_kv_load(f, kvb, 2 * kvd, kvd, k0, k1, pos, warp, lane);
            if (warp < 3) {
                const int h = warp == 0 ? ah : (warp == 1 ? S.H + akv : S.H + S.nkv + akv);
                const uint2 *p[1] = {warp == 0 || k1 == n_keys ? Lq + h * 64 + 2 * lane : nullptr};
                float2 v[1];
                c.poll<1>(p, tag, v);
                *(float2 *)&sm->qn[warp][2 * lane] = v[0];
            }
            ms_bar();
            ms_attend(sm, f, kvb, 2 * kvd, kvd, k0, k1, pos, Lp + ((size_t)ah * MS_MAXSPLIT + asp) * MS_PW, tag, tid);
        }
        // ---- context, o-projection, residual ----
        {
            const uint2 *p[2 * MS_MAXSPLIT];
            float2 v[2 * MS_MAXSPLIT];
#pragma unroll
            for (int s = 0; s < MS_MAXSPLIT; s++) {
                const uint2 *b = on2 && s < nsp ? Lp + ((size_t)(tid >> 5) * MS_MAXSPLIT + s) * MS_PW : nullptr;
                p[2 * s] = b; p[2 * s + 1] = b ? b + 2 + 2 * (tid & 31) : nullptr;
            }
            c.poll<2 * MS_MAXSPLIT>(p, tag, v);
            float M = -INFINITY;
#pragma unroll
            for (int s = 0; s < MS_MAXSPLIT; s++) if (s < nsp) M = fmaxf(M, v[2 * s].x);
            float l = 0.f, o0 = 0.f, o1 = 0.f;
#pragma unroll
            for (int s = 0; s < MS_MAXSPLIT; s++)
                if (s < nsp && v[2 * s].x != -INFINITY) {
                    const float e = expf(v[2 * s].x - M);
                    l = fmaf(v[2 * s].y, e, l); o0 = fmaf(v[2 * s + 1].x, e, o0); o1 = fmaf(v[2 * s + 1].y, e, o1);
                }
            const float inv = l > 0.f ? 1.0f / l : 0.f;
            if (on2) *(float2 *)(xs + 2 * tid) = make_float2(o0 * inv, o1 * inv);
        }
        ms_bar();
        ms_rows<W16>(c, st, at, ncr, C, xs, part, warp, lane);
        at += b_o;
        ms_bar();
        if (tid < ncr) {
            const float4 p = *(const float4 *)(part + 4 * tid);
            const float y = (p.x + p.y) + (p.z + p.w) + one(L.ob, true, c0 + tid) + sm->xres[tid];
            sm->xres[tid] = y;
            ll_store(Lx1 + c0 + tid, y, tag);
        }
        st.release(at, warp, lane);
        // ---- second norm, up-projection, activation ----
        {
            const float2 w = pair_of(L.ln2w, 1.f), b = pair_of(L.ln2b, 0.f);
            const uint2 *p[1] = {on2 ? Lx1 + 2 * tid : nullptr};
            c.poll<1>(p, tag, xv);
            ms_norm(sm, xv[0], C, a.norm, w, b, a.eps, xs, tid);
        }
        ms_rows<W16>(c, st, at, ur, C, xs, part, warp, lane);
        at += b_up;
        ms_bar();
        if (tid < nu) {
            float y;
            if (S.gated) {
                const float4 p0 = *(const float4 *)(part + 8 * tid), p1 = *(const float4 *)(part + 8 * tid + 4);
                const float gt = (p0.x + p0.y) + (p0.z + p0.w) + one(L.fcb, true, u0 + tid), up = (p1.x + p1.y) + (p1.z + p1.w) + one(L.fcb, true, I + u0 + tid);
                y = __fmul_rn(tc_act(gt, a.act), up);
            } else {
                const float4 p = *(const float4 *)(part + 4 * tid);
                y = tc_act((p.x + p.y) + (p.z + p.w) + one(L.fcb, true, u0 + tid), a.act);
            }
            ll_store(Lh + u0 + tid, y, tag);
        }
        st.release(at, warp, lane);
        ms_bar();                                             // part is rewritten by the down-projection
        // ---- down-projection, residual ----
        ms_down<W16, GROUPS>(c, st, at, ncr, I, Lh, tag, part, warp, lane);
        at += b_dn;
        ms_bar();
        if (tid < ncr) {
            // the product first, then the residual: added one by one to the larger residual, sixteen partial sums lose its last bits
            float q4[4];
#pragma unroll
            for (int q = 0; q < 4; q++) { const float4 p = *(const float4 *)(part + tid * MS_WARPS + 4 * q); q4[q] = (p.x + p.y) + (p.z + p.w); }
            const float y = ((q4[0] + q4[1]) + (q4[2] + q4[3])) + one(L.pb, true, c0 + tid) + sm->xres[tid];
            ll_store(Lx + c0 + tid, y, tag);
        }
        st.release(at, warp, lane);
    }
    // ---- final norm, vocabulary projection ----
    {
        const float2 w = pair_of(a.lnfw, 1.f), b = pair_of(a.lnfb, 0.f);
        const uint2 *p[1] = {on2 ? Lx + 2 * tid : nullptr};
        c.poll<1>(p, tag0 + (unsigned)S.NL - 1u, xv);
        ms_norm(sm, xv[0], C, a.norm, w, b, a.eps_f, xs, tid);
    }
    st.release(head_at, warp, lane);
    at = head_at;
    int buf = 0;
    for (int r0 = 0; r0 < nv; r0 += MS_HROWS, buf ^= 1) {
        const int n = min(MS_HROWS, nv - r0);
        float *pb = part + buf * MS_HROWS * 4;
        ms_rows<W16>(c, st, at, n, C, xs, pb, warp, lane);
        at += (long long)n * C * esz;
        ms_bar();                                             // (the other half of `part` is free by the next barrier)
        st.release(at, warp, lane);
        if (tid < n) {
            const float4 p = *(const float4 *)(pb + 4 * tid);
            a.logits[v0 + r0 + tid] = (p.x + p.y) + (p.z + p.w);
        }
    }
}

// one layer's rows into the CTAs' streams: block (cta, matrix)
__global__ void __launch_bounds__(256) k_mega_pack(MegaShape S, int li, int esz, const unsigned char *qkv, const unsigned char *o, const unsigned char *up, const unsigned char *dn,
                                                   const long long *off, unsigned char *dst) {
    const int cta = blockIdx.x, g = gridDim.x, mat = blockIdx.y, C = S.C, I = S.I, Wq = C + 128 * S.nkv;
    const int q0 = ms_begin(Wq >> 1, cta, g), nq = ms_begin(Wq >> 1, cta + 1, g) - q0;
    const int c0 = ms_begin(C, cta, g), ncr = ms_begin(C, cta + 1, g) - c0;
    const int u0 = ms_begin(I, cta, g), nu = ms_begin(I, cta + 1, g) - u0, ur = S.gated ? 2 * nu : nu;
    const long long rc = (long long)C * esz, rI = (long long)I * esz;
    const long long layer = 2LL * nq * rc + ncr * rc + ur * rc + ncr * rI;
    unsigned char *d = dst + off[cta] + li * layer + (mat > 0 ? 2LL * nq * rc : 0) + (mat > 1 ? ncr * rc : 0) + (mat > 2 ? ur * rc : 0);
    const int n = mat == 0 ? 2 * nq : mat == 1 ? ncr : mat == 2 ? ur : ncr;
    const long long row = mat == 3 ? rI : rc;
    const unsigned char *src = mat == 0 ? qkv : mat == 1 ? o : mat == 2 ? up : dn;
    for (int i = 0; i < n; i++) {
        int r;
        if (mat == 0) { const int pr = q0 + (i >> 1); r = (pr >> 5) * 64 + (pr & 31) + (i & 1) * 32; }
        else if (mat == 2) r = S.gated ? u0 + (i >> 1) + (i & 1) * I : u0 + i;
        else r = c0 + i;
        for (long long b = threadIdx.x * 16; b < row; b += 256 * 16) *(uint4 *)(d + i * row + b) = *(const uint4 *)(src + r * row + b);
    }
}

static int g_lm_persistent = -1;
void lm_mega_enable(int on) { g_lm_persistent = on ? 1 : 0; }
bool lm_mega_enabled() {
    if (g_lm_persistent < 0) { const char *e = getenv("NCM_B200_LM_PERSISTENT"); g_lm_persistent = e ? atoi(e) != 0 : 1; }
    return g_lm_persistent == 1;
}
static bool shape_fits(const MegaShape &s, int hd, bool qk_norm, int g) {
    return s.B == 1 && hd == 64 && s.C == s.H * 64 && s.C % 32 == 0 && s.C <= MS_MAXC && s.I % 8 == 0 && s.I >= g && s.I <= MS_MAXI && !qk_norm &&
           s.H % s.nkv == 0 && s.H <= g && cdiv(s.C, g) <= 8 && 2 * cdiv(s.I, g) <= MS_UPROWS && cdiv(s.C + 128 * s.nkv, g) + 2 <= MS_UPROWS &&
           (int64_t)s.C * 4 * MS_RGRP + 2 * MS_CH <= MS_RING && s.NL <= MS_MAXNL;
}
bool lm_mega_supported(const MegaShape &s, int hd, bool qk_norm) { return shape_fits(s, hd, qk_norm, ctx().sm_count); }

// The most chunks between what a CTA of g has given back and what it waits for, over the products of a step in the kernel's order (layers
// repeat at other offsets within a chunk); with more than MS_SLOTS the stream waits for a release that comes later. 0: not a shape of
// the kernel.
int lm_mega_ring_need(const MegaShape &s, int esz, int g) {
    if (!shape_fits(s, 64, false, g)) return 0;
    long long need = 0;
    for (int c = 0; c < g; c++) {
        auto share = [&](int n) { return ms_begin(n, c + 1, g) - ms_begin(n, c, g); };
        long long at = 0, rel = 0;
        auto product = [&](int n, int K, int group) {
            const long long rowb = (long long)K * esz;
            for (int r = 0; r < n; r += group) {
                rel = (at + r * rowb) / MS_CH;
                need = std::max(need, (at + std::min(n, r + group) * rowb + MS_CH - 1) / MS_CH - rel);
            }
            at += n * rowb;
        };
        const int ncr = share(s.C);
        for (int li = 0; li < s.NL; li++) {
            product(2 * share((s.C + 128 * s.nkv) >> 1), s.C, MS_RGRP);
            product(ncr, s.C, MS_RGRP);
            product((s.gated ? 2 : 1) * share(s.I), s.C, MS_RGRP);
            product(ncr, s.I, ms_hold((long long)s.I * esz));
        }
        at = (at + MS_CH - 1) / MS_CH * MS_CH;
        product(share(s.V), s.C, MS_RGRP);
    }
    return (int)need;
}

void lm_mega_free(MegaModel &m) {
    if (m.stream_w) dev_free(m.stream_w);
    if (m.stream_off) dev_free(m.stream_off);
    m = MegaModel();
}

void lm_mega_pack(MegaModel &m, const MegaShape &s, const std::vector<BlockWeights> &blocks, const float *wte, const unsigned short *wte16) {
    if (m.ready) return;
    const int g = ctx().sm_count;
    m.grid = g;
    m.w16 = wte16 != nullptr;
    for (auto &b : blocks) m.w16 = m.w16 && b.qkvw16 && b.ow16 && b.fcw16 && b.pw16;
    const int esz = m.w16 ? 2 : 4, Wq = s.C + 128 * s.nkv;
    std::vector<long long> off(g + 1, 0);
    for (int c = 0; c < g; c++) {
        const long long nq = ms_begin(Wq / 2, c + 1, g) - ms_begin(Wq / 2, c, g), nc = ms_begin(s.C, c + 1, g) - ms_begin(s.C, c, g);
        const long long nu = ms_begin(s.I, c + 1, g) - ms_begin(s.I, c, g);
        off[c + 1] = off[c] + s.NL * esz * ((2 * nq + nc + (s.gated ? 2 : 1) * nu) * s.C + nc * s.I);
    }
    m.stream_w = dev_alloc((size_t)off[g]);
    m.stream_off = (long long *)dev_alloc(sizeof(long long) * (g + 1));
    upload(m.stream_off, off.data(), sizeof(long long) * (g + 1));
    for (int li = 0; li < s.NL; li++) {
        const BlockWeights &b = blocks[li];
        auto pick = [&](const float *w, const unsigned short *w16) { return m.w16 ? (const unsigned char *)w16 : (const unsigned char *)w; };
        LAUNCH(k_mega_pack, dim3((unsigned)g, 4), 256, 0, s, li, esz, pick(b.qkvw, b.qkvw16), pick(b.ow, b.ow16), pick(b.fcw, b.fcw16), pick(b.pw, b.pw16),
               (const long long *)m.stream_off, (unsigned char *)m.stream_w);
    }
    m.head_w = m.w16 ? (const void *)wte16 : (const void *)wte;
    m.ready = true;
}

size_t lm_mega_exchange_words(const MegaShape &s) { return MsLL(s).total; }

template <bool W16, bool GROUPS>
static void launch_step(const MegaModel &m, const MegaArgs &a) {
    const MegaShape &s = a.s;
    const size_t part = (size_t)std::max<int64_t>(2 * MS_HROWS, 2 * cdiv(s.I, m.grid) + 2) * 4;
    const size_t smem = MS_RING + sizeof(MsSm) + 32 + ((size_t)s.C + part) * 4 + s.NL * sizeof(MegaLayer);
    static size_t set = 0;
    if (smem > set) { CUDA_CHECK(cudaFuncSetAttribute((k_lm_step<W16, GROUPS>), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); set = smem; }
    MegaArgs arg = a;
    const unsigned char *w = (const unsigned char *)m.stream_w, *h = (const unsigned char *)m.head_w;
    const long long *off = m.stream_off;
    void *params[] = {&arg, &w, &off, &h};
    cudaError_t e = cudaLaunchCooperativeKernel((const void *)(k_lm_step<W16, GROUPS>), dim3((unsigned)m.grid), dim3(MS_T + 32), params, smem, stream());
    if (e != cudaSuccess) fatal("lm_mega: cooperative launch failed: %s", cudaGetErrorString(e));
    ctx().launches++;
}
void lm_mega_launch(const MegaModel &m, const MegaArgs &a) {
    ProfScope ps(NCMB_K_GEMM, 0, 0);
    const bool groups = cdiv(a.s.C, m.grid) > ms_hold((long long)a.s.I * (m.w16 ? 2 : 4));
    if (m.w16) { if (groups) launch_step<true, true>(m, a); else launch_step<true, false>(m, a); }
    else if (groups) launch_step<false, true>(m, a);
    else launch_step<false, false>(m, a);
}

} // namespace ncmb
