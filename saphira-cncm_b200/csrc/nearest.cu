// Nearest code of a codebook: argmin_j |x_r - e_j|^2 for every row r, the lowest index among equals
// (reference src/vq.c:420-450).
//
// |x|^2 does not change the argmin, so a row looks for the smallest d_j = |e_j|^2 - 2 x.e_j. Finding it exactly needs
// fp32-grade products only where two codes are close, and for nearly every row that is one group of 32 codes out of
// hundreds. So the search runs in two passes:
//
//   1. k_nearest_coarse: ONE fp16 tensor-core pass over all codes (tcgen05, fp32 accumulate). The epilogue takes the
//      minimum of every group of 32 codes and keeps, per row and for each of four interleaved quarters of the groups,
//      the two groups with the smallest minimum and the value of the third. Products are not stored and indices inside
//      a group are not tracked: one multiply-add and half an instruction for the minimum (three-input min) per code.
//   2. k_nearest_refine: a bound on the rounding error of pass 1 (from the row's and the codes' norms) says which
//      groups can hold the true minimum. Their codes are evaluated again in fp32. A row where the third group of a
//      quarter cannot be ruled out goes to a list.
//   3. Few listed rows: k_nearest_scan evaluates all codes for them in fp32. Many (codes that lie close to one another against their
//      length, or repeat): k_nearest_coarse<., true> takes the products of the listed rows from fp16 pairs (22 bits, three MMAs) and
//      keeps the smallest distance and its code, whatever lies next to it.
//
// The result is the fp32 argmin; of a row that many codes are too close for pass 1, in a call with many such rows, it is that of
// distances with an error of about 2^-21 |x| |e|. The time depends on how close codes lie: see the table at nearest_codes().
#include "common.cuh"
#include "tc_common.cuh"
#include "split.cuh"
#include "nearest.cuh"

#include <algorithm>
#include <unordered_map>

namespace ncmb {

constexpr int NC_ROWS = 256;                 // rows of a work item: two 128-row MMA tiles share every code tile
constexpr int NC_CODES = 128;                // codes of a tile
constexpr int NC_GROUP = 32;                 // codes of a group
constexpr int NC_EPI = 16;                   // epilogue warps: four TMEM quadrants x the four groups of a tile
constexpr int NC_THREADS = 64 + 32 * NC_EPI;
constexpr int NC_TILE = 128 * 64 * 2;        // 128 rows of 64 halfs, 128-byte swizzle
constexpr float NEAR_BIG = 3.0e38f;          // starts a minimum: finite, so that the tile number in its low bits makes no NaN of it
constexpr int NC_MAXSLICE = 8;               // slices of the codebook a row block may be shared out to (four candidate lists each)
// kb: 64-wide blocks of a row; pair: two halves of every row and code
constexpr int nc_blocks(int kb, bool pair) { return pair ? 2 * kb : kb; }
constexpr int nc_stages(int kb, bool pair) { return nc_blocks(kb, pair) == 1 ? 6 : (nc_blocks(kb, pair) == 2 ? 2 : 1); }
constexpr int nc_xbufs(int kb, bool pair) { return nc_blocks(kb, pair) <= 2 ? 2 : 1; }
constexpr size_t nc_smem(int kb, bool pair) {
    return 1024 + (size_t)(2 * nc_xbufs(kb, pair) + nc_stages(kb, pair)) * nc_blocks(kb, pair) * NC_TILE + NC_EPI * 2 * NC_GROUP * 4 + (2 * nc_stages(kb, pair) + 8) * 8 + 16;
}

__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ unsigned ordered_bits(float v) {          // order-preserving float -> uint
    const unsigned u = __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float from_ordered(unsigned u) { return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u); }

// codebook constants, written by the preparation kernels
struct NearMeta { unsigned absmax; float scale; unsigned maxnorm, maxcn; };   // maxnorm: of scaled codes; both as bits of floats >= 0

__global__ void k_near_absmax(const float *__restrict__ E, int64_t n, NearMeta *meta) {
    unsigned m = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        m = max(m, __float_as_uint(fabsf(E[i])));
    for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(&meta->absmax, m);
}
// power of two that brings a largest element of m to [2^(top-1), 2^top)
__device__ __forceinline__ float pow2_scale(float m, int top) {
    if (!(m > 0.f) || !isfinite(m)) return 1.0f;
    int e;
    frexpf(m, &e);
    e = top - e;
    e = e > 40 ? 40 : (e < -40 ? -40 : e);
    return ldexpf(1.0f, e);
}
// one warp per code (Vp of them, V rounded up to a tile): fp16 row -2 s e and what it leaves (eh, el), |e|^2, and the fp32 row (padded to a multiple of four) in
// group order et[code / 32][d / 4][code % 32][4], which lets a warp with one code per lane read 512 contiguous bytes
__global__ void __launch_bounds__(256) k_near_codes(const float *__restrict__ E, int V, int Vp, int D, NearMeta *meta,
                                                    unsigned short *__restrict__ eh, unsigned short *__restrict__ el, float *__restrict__ cn, float *__restrict__ et) {
    const int code = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (code >= Vp) return;
    const float s = pow2_scale(__uint_as_float(meta->absmax), 14);
    const int Dp = (D + 3) & ~3;
    float *dst = et + (int64_t)(code / NC_GROUP) * Dp * NC_GROUP + (code % NC_GROUP) * 4;
    float q = 0.f;
    for (int d = lane; d < Dp; d += 32) {
        const float e = (code < V && d < D) ? E[(int64_t)code * D + d] : 0.f;
        q = fmaf(e, e, q);
        dst[(d / 4) * (NC_GROUP * 4) + (d & 3)] = e;
        if (code < V && d < D) {
            const float v = -2.0f * s * e;
            const unsigned short hi = f16_sat(v);
            eh[(int64_t)code * D + d] = hi;
            el[(int64_t)code * D + d] = f16_sat(v - __half2float(__ushort_as_half(hi)));
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
    if (lane == 0) {
        cn[code] = code < V ? q : INFINITY;
        if (code == 0) meta->scale = s;
        if (code < V) { atomicMax(&meta->maxnorm, __float_as_uint(sqrtf(q) * s)); atomicMax(&meta->maxcn, __float_as_uint(q)); }
    }
}

// rows -> fp16 rows scaled by a power of two each (largest element in [2^13, 2^14)); rinfo = (row factor x codebook factor,
// norm of the scaled row)
__global__ void __launch_bounds__(256) k_near_rows(const float *__restrict__ x, int64_t rows, int D, const NearMeta *__restrict__ meta,
                                                   unsigned short *__restrict__ xh, float2 *__restrict__ rinfo) {
    constexpr int RW = 4;                                   // rows of a warp, loads in flight together
    const int64_t r0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * RW;
    const int lane = threadIdx.x & 31;
    if (r0 >= rows) return;
    const float es = meta->scale;
    float2 v[RW][2];
#pragma unroll
    for (int i = 0; i < RW; i++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int d = lane * 2 + h * 64;
            v[i][h] = (r0 + i < rows && d < D) ? *(const float2 *)(x + (r0 + i) * D + d) : make_float2(0.f, 0.f);
        }
#pragma unroll
    for (int i = 0; i < RW; i++) {
        // bits of |v| order like the values, and a NaN orders above infinity, so a bad row keeps its mark
        unsigned m = max(max(__float_as_uint(fabsf(v[i][0].x)), __float_as_uint(fabsf(v[i][0].y))),
                         max(__float_as_uint(fabsf(v[i][1].x)), __float_as_uint(fabsf(v[i][1].y))));
        m = __reduce_max_sync(0xffffffffu, m);
        float q = (v[i][0].x * v[i][0].x + v[i][0].y * v[i][0].y) + (v[i][1].x * v[i][1].x + v[i][1].y * v[i][1].y);
#pragma unroll
        for (int o = 16; o; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
        if (r0 + i >= rows) break;
        const float mx = __uint_as_float(m), s = pow2_scale(mx, 14);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int d = lane * 2 + h * 64;
            if (d < D) *(ushort2 *)(xh + (r0 + i) * D + d) = make_ushort2(f16_sat(v[i][h].x * s), f16_sat(v[i][h].y * s));
        }
        // a row out of the scalable range compares false everywhere in pass 1 and is evaluated in full
        if (lane == 0) rinfo[r0 + i] = make_float2((mx * s < 32768.f) ? s * es : __uint_as_float(0x7fc00000u), sqrtf(q) * s);
    }
}

// Rows that pass 1 left undecided: list[0 .. na - 1]; rows that it cannot scale: list[rows - 1], list[rows - 2], ... (nb of them).
struct NearCount { unsigned na, nb; };
// from this many undecided rows on they go through the pair products: a wave of them takes as long as the scan of about 500 rows
constexpr unsigned NEAR_PAIR_MIN = 512;
__device__ __forceinline__ bool near_pairs(const NearCount &c, int64_t rows, int64_t min_rows) { return rows >= min_rows && c.na > NEAR_PAIR_MIN; }

// the undecided rows as fp16 pairs, in list order; rinfo as above. Four rows of a warp in flight.
__device__ __forceinline__ void near_make_pairs(const float *__restrict__ x, int D, float es, const int *__restrict__ list, unsigned n, unsigned short *__restrict__ xh,
                                                unsigned short *__restrict__ xl, float2 *__restrict__ rinfo) {
    constexpr int RW = 4;
    const int lane = threadIdx.x & 31;
    for (unsigned i0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * RW; i0 < n; i0 += ((gridDim.x * blockDim.x) >> 5) * RW) {
        float2 v[RW][2];
#pragma unroll
        for (int i = 0; i < RW; i++) {
            const float *xr = i0 + i < n ? x + (int64_t)list[i0 + i] * D : nullptr;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int d = lane * 2 + h * 64;
                v[i][h] = xr && d < D ? *(const float2 *)(xr + d) : make_float2(0.f, 0.f);
            }
        }
#pragma unroll
        for (int i = 0; i < RW; i++) {
            unsigned m = max(max(__float_as_uint(fabsf(v[i][0].x)), __float_as_uint(fabsf(v[i][0].y))),
                             max(__float_as_uint(fabsf(v[i][1].x)), __float_as_uint(fabsf(v[i][1].y))));
            const float s = pow2_scale(__uint_as_float(__reduce_max_sync(0xffffffffu, m)), 14);
            if (i0 + i >= n) break;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int d = lane * 2 + h * 64;
                uint32_t hi, lo;
                h16_pair2_raw(v[i][h].x * s, v[i][h].y * s, hi, lo, 1.0f);
                if (d < D) { *(uint32_t *)(xh + (int64_t)(i0 + i) * D + d) = hi; *(uint32_t *)(xl + (int64_t)(i0 + i) * D + d) = lo; }
            }
            if (lane == 0) rinfo[i0 + i] = make_float2(s * es, 0.f);
        }
    }
}

// 16 columns of two accumulators
__device__ __forceinline__ void tmem_ld16x2(uint32_t ta, uint32_t tb, uint32_t *a, uint32_t *b) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]), "=r"(a[4]), "=r"(a[5]), "=r"(a[6]), "=r"(a[7]),
                   "=r"(a[8]), "=r"(a[9]), "=r"(a[10]), "=r"(a[11]), "=r"(a[12]), "=r"(a[13]), "=r"(a[14]), "=r"(a[15]),
                   "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]), "=r"(b[4]), "=r"(b[5]), "=r"(b[6]), "=r"(b[7]),
                   "=r"(b[8]), "=r"(b[9]), "=r"(b[10]), "=r"(b[11]), "=r"(b[12]), "=r"(b[13]), "=r"(b[14]), "=r"(b[15])
                 : "r"(ta), "r"(tb) : "memory");
}

// ---- pass 1 ----
// Persistent CTAs over (256-row block, codebook slice) items. Warp 0: TMA producer (row tiles double-buffered, code tiles
// in a ring), warp 1: one lane issues the MMAs, warps 2-17: epilogue. A thread takes one row of each row
// tile and one of the tile's four groups: a norm read from shared memory serves two rows, and the candidates of both stay in
// registers over the whole slice. TMEM: two buffers of two 128-column accumulators, all 512 columns.
// Bound: the MMAs (1.83 ms at 2^20 rows and 16384 codes with the epilogue left out: 128-column MMAs are paced by their
// operand fetch) and the epilogue's issue and min throughput (2.2 ms alone) side by side: 2.8 ms. A code tile is fetched
// once per 256 rows. The whole search of 2^20 rows takes 3.8 ms; three TF32 passes with the argmin in the epilogue took 9.6.
//
// PAIR: the listed rows against all codes, rows and codes as pairs x1 + x2, e1 + e2 of which x2 e1 + x1 e2 + x1 e1 are taken; the epilogue
// keeps the smallest distance and its code (the lowest among equals) and adds them to best[] by atomicMin. How many rows there are, only
// the device knows: the work is dealt out here.
template <int KB, bool PAIR>
__global__ void __launch_bounds__(NC_THREADS, 1) k_nearest_coarse(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmE,
                                                                 const __grid_constant__ CUtensorMap tmX2, const __grid_constant__ CUtensorMap tmE2,
                                                                 const float *__restrict__ cn, const float2 *__restrict__ rinfo, int64_t rows,
                                                                 int ntiles, int nslice, int tps, int items,
                                                                 unsigned id_mask, float4 *__restrict__ cand, const NearCount *__restrict__ count,
                                                                 unsigned long long *__restrict__ best, int *err) {
    constexpr int NB = nc_blocks(KB, PAIR), ST = nc_stages(KB, PAIR), XB = nc_xbufs(KB, PAIR);
    if (PAIR) {
        pdl_wait();
        if (count->na <= NEAR_PAIR_MIN) return;
        rows = count->na;
        const int blocks = (int)((rows + NC_ROWS - 1) / NC_ROWS);
        nslice = max(1, min(min(NC_MAXSLICE, ntiles), (int)gridDim.x / blocks));
        tps = (ntiles + nslice - 1) / nslice;
        nslice = (ntiles + tps - 1) / tps;
        items = blocks * nslice;
    }
    extern __shared__ unsigned char near_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)near_raw + 1023) & ~(uintptr_t)1023);
    unsigned char *sX = smem, *sE = smem + 2 * XB * NB * NC_TILE;       // X: [buffer][row tile][k block]; E: [stage][k block]
    float *scn = (float *)(sE + ST * NB * NC_TILE);                     // per epilogue warp: two slots of 32 norms
    uint64_t *bars = (uint64_t *)(scn + NC_EPI * 2 * NC_GROUP);
    uint32_t *tmem_slot = (uint32_t *)(bars + 2 * ST + 8);
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + ST);
    const uint32_t xfull0 = smem_u32(bars + 2 * ST), xempty0 = xfull0 + 16, afull0 = xfull0 + 32, aempty0 = xfull0 + 48;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; s++) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
        for (int b = 0; b < 2; b++) {
            mbar_init(xfull0 + 8 * b, 1); mbar_init(xempty0 + 8 * b, 1);
            mbar_init(afull0 + 8 * b, 1); mbar_init(aempty0 + 8 * b, NC_EPI);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmX) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tmE) : "memory");
        if (PAIR) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tmX2) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tmE2) : "memory");
        }
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            int g = 0, it = 0, armed = 0, xarmed = 0;                   // code tiles / items issued so far
            bool ok = true;
            for (int w = blockIdx.x; w < items && ok; w += gridDim.x, it++) {
                const int rb = w / nslice, sl = w - rb * nslice;
                const int b = it % XB;
                ok = mbar_wait(xempty0 + 8 * b, (uint32_t)((it / XB) & 1) ^ 1u, err, 41);
                if (!ok) break;
                mbar_expect_tx(xfull0 + 8 * b, 2 * NB * NC_TILE);
                for (int h = 0; h < 2; h++)
                    for (int k = 0; k < NB; k++)
                        tma_load_2d(smem_u32(sX + ((b * 2 + h) * NB + k) * NC_TILE), k < KB ? &tmX : &tmX2, k % KB * 64, rb * NC_ROWS + h * 128, xfull0 + 8 * b);
                xarmed = it + 1;
                const int t1 = min(ntiles, (sl + 1) * tps);
                for (int t = sl * tps; t < t1; t++, g++) {
                    const int s = g % ST;
                    ok = mbar_wait(empty0 + 8 * s, (uint32_t)((g / ST) & 1) ^ 1u, err, 42);
                    if (!ok) break;
                    mbar_expect_tx(full0 + 8 * s, NB * NC_TILE);
                    for (int k = 0; k < NB; k++)
                        tma_load_2d(smem_u32(sE + (s * NB + k) * NC_TILE), k < KB ? &tmE : &tmE2, k % KB * 64, t * NC_CODES, full0 + 8 * s);
                    armed = g + 1;
                }
            }
            if (!ok) {                                                  // bounded wait for the copies already in flight
                for (int k = armed - ST < 0 ? 0 : armed - ST; k < armed; k++) mbar_wait(full0 + 8 * (k % ST), (uint32_t)((k / ST) & 1), err, 44);
                for (int k = xarmed - XB < 0 ? 0 : xarmed - XB; k < xarmed; k++) mbar_wait(xfull0 + 8 * (k % XB), (uint32_t)((k / XB) & 1), err, 44);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = umma_idesc_f16(128, NC_CODES);
            int g = 0, it = 0;
            bool ok = true;
            for (int w = blockIdx.x; w < items && ok; w += gridDim.x, it++) {
                const int sl = w % nslice, b = it % XB;
                ok = mbar_wait(xfull0 + 8 * b, (uint32_t)((it / XB) & 1), err, 45);
                const int t1 = min(ntiles, (sl + 1) * tps);
                for (int t = sl * tps; t < t1 && ok; t++, g++) {
                    const int acc = g & 1, s = g % ST;
                    ok = mbar_wait(aempty0 + 8 * acc, (uint32_t)((g >> 1) & 1) ^ 1u, err, 46) &&
                         mbar_wait(full0 + 8 * s, (uint32_t)((g / ST) & 1), err, 47);
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll
                    for (int h = 0; h < 2; h++)
#pragma unroll
                        for (int k = 0; k < (PAIR ? 3 * KB : KB); k++) {       // PAIR: x2 e1, x1 e2, x1 e1: the small products while the sum is small
                            const int kx = !PAIR ? k : (k < KB ? KB + k : (k < 2 * KB ? k - KB : k - 2 * KB)), ke = k < 2 * KB ? k : k - 2 * KB;
                            const uint64_t xd = umma_desc_sw128(smem_u32(sX + ((b * 2 + h) * NB + kx) * NC_TILE));
                            const uint64_t ed = umma_desc_sw128(smem_u32(sE + (s * NB + ke) * NC_TILE));
#pragma unroll
                            for (int i = 0; i < 4; i++)
                                umma_f16(tmem_base + (uint32_t)(acc * 256 + h * 128), xd + (uint64_t)(i * 2), ed + (uint64_t)(i * 2), idesc, (k | i) ? 1u : 0u);
                        }
                    umma_commit(empty0 + 8 * s);
                    umma_commit(afull0 + 8 * acc);
                }
                umma_commit(xempty0 + 8 * b);
            }
        }
    } else {
        const int q = warp & 3, c = (warp - 2) >> 2;
        float *slot = scn + (warp - 2) * 2 * NC_GROUP;
        int g = 0;
        bool ok = true;
        for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
            const int rb = w / nslice, sl = w - rb * nslice;
            const int64_t r0 = (int64_t)rb * NC_ROWS + q * 32 + lane;
            float s2[2], b1[2], b2[2], b3[2];
            float pd[2][2]; int pj[2][2];                                // PAIR: smallest distance of even and odd codes, their numbers
#pragma unroll
            for (int h = 0; h < 2; h++) {
                s2[h] = r0 + h * 128 < rows ? rinfo[r0 + h * 128].x : 0.f;
                b1[h] = b2[h] = b3[h] = INFINITY;
                pd[h][0] = pd[h][1] = INFINITY; pj[h][0] = pj[h][1] = 0x7fffffff;
            }
            const int t1 = min(ntiles, (sl + 1) * tps);
            float cnext = cn[sl * tps * NC_CODES + c * NC_GROUP + lane];     // a tile ahead: its latency would be most of a tile's time
            for (int t = sl * tps; t < t1; t++, g++) {
                const int acc = g & 1;
                float *sc = slot + acc * NC_GROUP;
                sc[lane] = cnext;
                __syncwarp();
                if (t + 1 < t1) cnext = cn[(t + 1) * NC_CODES + c * NC_GROUP + lane];
                ok = mbar_wait(afull0 + 8 * acc, (uint32_t)((g >> 1) & 1), err, 48);
                tc_fence_after();
                if (!ok) break;
                const uint32_t trow = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * 256 + c * NC_GROUP);
                float m[2][2] = {{NEAR_BIG, NEAR_BIG}, {NEAR_BIG, NEAR_BIG}};
#pragma unroll
                for (int e0 = 0; e0 < NC_GROUP; e0 += 16) {
                    uint32_t v[2][16];
                    tmem_ld16x2(trow + e0, trow + 128 + e0, v[0], v[1]);
                    if (e0 + 16 == NC_GROUP) {                          // both accumulators read: the MMAs may overwrite them
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(aempty0 + 8 * acc);
                    }
#pragma unroll
                    for (int j = 0; j < 16; j += 4) {
                        const float4 n4 = *(const float4 *)(sc + e0 + j);
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const float d0 = fmaf(n4.x, s2[h], __uint_as_float(v[h][j])), d1 = fmaf(n4.y, s2[h], __uint_as_float(v[h][j + 1]));
                            const float d2 = fmaf(n4.z, s2[h], __uint_as_float(v[h][j + 2])), d3 = fmaf(n4.w, s2[h], __uint_as_float(v[h][j + 3]));
                            if constexpr (PAIR) {
                                const int code = t * NC_CODES + c * NC_GROUP + e0 + j;
                                if (d0 < pd[h][0]) { pd[h][0] = d0; pj[h][0] = code; }
                                if (d1 < pd[h][1]) { pd[h][1] = d1; pj[h][1] = code + 1; }
                                if (d2 < pd[h][0]) { pd[h][0] = d2; pj[h][0] = code + 2; }
                                if (d3 < pd[h][1]) { pd[h][1] = d3; pj[h][1] = code + 3; }
                            } else {
                                m[h][0] = min3(m[h][0], d0, d1);
                                m[h][1] = min3(m[h][1], d2, d3);
                            }
                        }
                    }
                }
                // the tile's number replaces the low bits of the group's minimum, so the three smallest are kept without branches
                if constexpr (!PAIR) {
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const float mm = __uint_as_float((__float_as_uint(fminf(m[h][0], m[h][1])) & ~id_mask) | (unsigned)(t - sl * tps));
                        const float t2 = fmaxf(b1[h], mm), t3 = fmaxf(b2[h], t2);
                        b1[h] = fminf(b1[h], mm); b2[h] = fminf(b2[h], t2); b3[h] = fminf(b3[h], t3);
                    }
                }
            }
#pragma unroll
            for (int h = 0; h < 2; h++)
                if (PAIR) {
                    const bool odd = pd[h][1] < pd[h][0] || (pd[h][1] == pd[h][0] && pj[h][1] < pj[h][0]);
                    const float d = odd ? pd[h][1] : pd[h][0]; const int j = odd ? pj[h][1] : pj[h][0];
                    if (r0 + h * 128 < rows && ok && j != 0x7fffffff) atomicMin(best + r0 + h * 128, ((unsigned long long)ordered_bits(d) << 32) | (unsigned)j);
                } else if (r0 + h * 128 < rows && ok) cand[(int64_t)(sl * 4 + c) * rows + r0 + h * 128] = make_float4(b1[h], b2[h], b3[h], 0.f);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }
}

// ---- fp32 evaluation ----
// A row up to twice as long as the longest code is compared by |x - e|^2: near a code the squares of small differences have no
// error to speak of, where |e|^2 - 2 x.e cancels. A longer row's own length would cost that sum the digits that tell codes
// apart; it is compared by |e|^2 - 2 x.e, whose error is that of |x| |e|.
__device__ __forceinline__ bool near_direct(float xx, float max_ee) { return xx <= 4.0f * max_ee; }      // (NaN, infinity: false)

// Smallest d_j of the 32 codes of group g, fp32: lane = (code mod 8, quarter of the
// dims), four codes each, so that a row's elements are read four times instead of once per code.
__device__ __forceinline__ void group_best(const float *__restrict__ xr, const float *__restrict__ et, const float *__restrict__ cn, bool direct, int V, int g, int D,
                                           int lane, float &bd, int &bj) {
    const int cl = lane & 7, qd = lane >> 3;
    const float4 *ep = (const float4 *)(et + (int64_t)g * D * NC_GROUP) + cl;
    float a[4] = {0.f, 0.f, 0.f, 0.f};
    if (direct) {
#pragma unroll 4
        for (int d4 = qd; d4 < D / 4; d4 += 4) {
            const float4 v = __ldg((const float4 *)xr + d4);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float4 e = __ldg(ep + d4 * NC_GROUP + 8 * i);
                const float t0 = v.x - e.x, t1 = v.y - e.y, t2 = v.z - e.z, t3 = v.w - e.w;
                a[i] = fmaf(t0, t0, a[i]); a[i] = fmaf(t1, t1, a[i]); a[i] = fmaf(t2, t2, a[i]); a[i] = fmaf(t3, t3, a[i]);
            }
        }
    } else {
#pragma unroll 4
        for (int d4 = qd; d4 < D / 4; d4 += 4) {
            const float4 v = __ldg((const float4 *)xr + d4);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float4 e = __ldg(ep + d4 * NC_GROUP + 8 * i);
                a[i] = fmaf(v.x, e.x, a[i]); a[i] = fmaf(v.y, e.y, a[i]); a[i] = fmaf(v.z, e.z, a[i]); a[i] = fmaf(v.w, e.w, a[i]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        a[i] += __shfl_xor_sync(0xffffffffu, a[i], 8);
        a[i] += __shfl_xor_sync(0xffffffffu, a[i], 16);
        const int j = g * NC_GROUP + 8 * i + cl;
        const float d = direct ? a[i] : fmaf(-2.0f, a[i], cn[j]);
        if (j < V && (d < bd || (d == bd && j < bj))) { bd = d; bj = j; }
    }
}

// One warp per row, about 0.8 ms for 2^20 rows: 8 KB of codes per row out of L2 at 12 TB/s. Lane s holds candidate list s.
//
// Bound. With X = |x| s_r, E = max_j |e_j| s_e (scaled norms), each fp16 rounding is at most 2^-11 of the element plus
// 2^-25 (subnormals), so a dot product is off by at most X E (2^-10 + 2^-22) + 8 * 2^-25 (X + E) by the Cauchy-Schwarz
// inequality (8 covers sqrt(D) up to 64, and is taken as 12 for D up to 128); the fp32 accumulation of up to 128 products
// with truncation adds X E 2^-16. A code counts as a candidate when it is within twice the error of a distance (which is
// twice the dot product's) of the smallest; the tile number in the low bits of a minimum and the rounding of the distance
// itself add a relative part.
__global__ void __launch_bounds__(256) k_nearest_refine(const float *__restrict__ x, const float *__restrict__ et, const float *__restrict__ cn, int V,
                                                        const NearMeta *__restrict__ meta, const float2 *__restrict__ rinfo, int64_t rows, int D,
                                                        int nlists, int tps, unsigned id_mask, const float4 *__restrict__ cand,
                                                        int *__restrict__ idx_out, int out_tlen, int out_stride, int out_off,
                                                        int *__restrict__ list, NearCount *__restrict__ count, unsigned long long *__restrict__ best) {
    const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (r >= rows) return;
    const float *xr = x + r * D;
    float4 v = make_float4(INFINITY, INFINITY, INFINITY, 0.f);
    if (lane < nlists) v = cand[(int64_t)lane * rows + r];
    const float2 ri = rinfo[r];
    const float lo = from_ordered(__reduce_min_sync(0xffffffffu, ordered_bits(v.x)));
    const float rs = ri.x, X = ri.y, Em = __uint_as_float(meta->maxnorm), cm = __uint_as_float(meta->maxcn) * rs;
    const float dot_err = X * Em * (0x1p-10f + 0x1p-15f) + 12.0f * 0x1p-25f * (X + Em);
    const float margin = 1.01f * (4.0f * dot_err + (0x1p-21f + 0x1p-22f * (float)(id_mask + 1u)) * (2.0f * X * Em + cm));
    const float thr = lo + margin;
    // (comparisons written so that a NaN anywhere sends the row to a list)
    const bool bad = !(thr < INFINITY);
    if (bad || __any_sync(0xffffffffu, lane < nlists && !(v.z > thr))) {
        if (lane == 0) {
            const int64_t at = bad ? rows - 1 - atomicAdd(&count->nb, 1u) : (int64_t)atomicAdd(&count->na, 1u);
            list[at] = (int)r; best[at] = ~0ull;
        }
        return;
    }
    const float xn = X / (rs / meta->scale);                 // (powers of two: exact)
    const bool direct = near_direct(xn * xn, __uint_as_float(meta->maxcn));
    float bd = INFINITY; int bj = 0x7fffffff;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const float vk = k == 0 ? v.x : v.y;
        const int ck = ((lane >> 2) * tps + (int)(__float_as_uint(vk) & id_mask)) * (NC_CODES / NC_GROUP) + (lane & 3);    // list -> slice, group of a tile
        unsigned mask = __ballot_sync(0xffffffffu, lane < nlists && vk <= thr);
        while (mask) {
            const int src = __ffs(mask) - 1;
            mask &= mask - 1;
            const int g = __shfl_sync(0xffffffffu, ck, src);
            group_best(xr, et, cn, direct, V, g, D, lane, bd, bj);
        }
    }
    const unsigned u = ordered_bits(bd), um = __reduce_min_sync(0xffffffffu, u);
    const int j = (int)__reduce_min_sync(0xffffffffu, u == um ? (unsigned)bj : 0x7fffffffu);
    if (lane == 0) {
        const unsigned b = (unsigned)r / (unsigned)out_tlen;
        idx_out[(int64_t)b * out_stride + out_off + ((unsigned)r - b * (unsigned)out_tlen)] = j;
    }
}

// All codes for the listed rows (list == null: for rows 0 .. n_rows - 1). Work item: 8 rows x 256 codes, one code per
// thread; the minimum of a warp goes to best[] by atomicMin on (ordered distance, index). Undecided rows that go through the pair
// products are only converted for them here.
constexpr int NS_ROWS = 8, NS_CODES = 256;
__global__ void __launch_bounds__(NS_CODES) k_nearest_scan(const float *__restrict__ x, const float *__restrict__ et, const float *__restrict__ cn,
                                                           const NearMeta *__restrict__ meta, int V, int D,
                                                           const int *__restrict__ list, const NearCount *__restrict__ count, int n_rows, int64_t pair_rows,
                                                           unsigned short *__restrict__ xh, unsigned short *__restrict__ xl, float2 *__restrict__ rinfo,
                                                           unsigned long long *__restrict__ best) {
    extern __shared__ __align__(16) float near_xs[];                    // [Dp / 4][NS_ROWS][4]
    __shared__ int direct_s[NS_ROWS];
    const int Dp = (D + 3) & ~3;
    pdl_wait();
    const bool pairs = list && near_pairs(*count, n_rows, pair_rows);
    if (pairs) near_make_pairs(x, D, meta->scale, list, count->na, xh, xl, rinfo);
    const int nb = list ? (int)count->nb : 0, n = !list ? n_rows : (pairs ? 0 : (int)count->na), nsl = (V + NS_CODES - 1) / NS_CODES;
    const int64_t itb = (int64_t)((nb + NS_ROWS - 1) / NS_ROWS) * nsl, items = itb + (int64_t)((n + NS_ROWS - 1) / NS_ROWS) * nsl;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int64_t w = blockIdx.x; w < items; w += gridDim.x) {
        const bool back = w < itb;                                      // rows from the list's end
        const int64_t wi = back ? w : w - itb;
        const int r0 = (int)(wi / nsl) * NS_ROWS, j = (int)(wi % nsl) * NS_CODES + tid, nr = back ? nb : n;
        auto place = [&](int k) { return back ? (int64_t)n_rows - 1 - (r0 + k) : (int64_t)(r0 + k); };     // of row k in list[] and best[]
        __syncthreads();
        {                                                               // a warp per row
            const float *xr = r0 + warp < nr ? x + (int64_t)(list ? list[place(warp)] : r0 + warp) * D : nullptr;
            float q = 0.f;
            for (int d = lane; d < Dp; d += 32) {
                const float v = xr && d < D ? xr[d] : 0.f;
                near_xs[((d / 4) * NS_ROWS + warp) * 4 + (d & 3)] = v;
                q = fmaf(v, v, q);
            }
#pragma unroll
            for (int o = 16; o; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
            if (lane == 0) direct_s[warp] = near_direct(q, __uint_as_float(meta->maxcn));
        }
        __syncthreads();
        unsigned direct = 0;
#pragma unroll
        for (int k = 0; k < NS_ROWS; k++) direct |= (unsigned)direct_s[k] << k;
        const bool on = j < V;
        const int jj = on ? j : V - 1;
        const float4 *ep = (const float4 *)(et + (int64_t)(jj / NC_GROUP) * Dp * NC_GROUP) + jj % NC_GROUP;
        float dist[NS_ROWS];
#pragma unroll
        for (int k = 0; k < NS_ROWS; k++) dist[k] = INFINITY;
        if (direct) {
            float acc[NS_ROWS];
#pragma unroll
            for (int k = 0; k < NS_ROWS; k++) acc[k] = 0.f;
#pragma unroll 4
            for (int d = 0; d < Dp; d += 4) {
                const float4 e = __ldg(ep + (d / 4) * NC_GROUP);
#pragma unroll
                for (int k = 0; k < NS_ROWS; k++) {
                    const float4 v = *(const float4 *)&near_xs[(d * 2 + k) * 4];
                    const float t0 = v.x - e.x, t1 = v.y - e.y, t2 = v.z - e.z, t3 = v.w - e.w;
                    acc[k] = fmaf(t0, t0, acc[k]); acc[k] = fmaf(t1, t1, acc[k]); acc[k] = fmaf(t2, t2, acc[k]); acc[k] = fmaf(t3, t3, acc[k]);
                }
            }
#pragma unroll
            for (int k = 0; k < NS_ROWS; k++) if (direct >> k & 1) dist[k] = acc[k];
        }
        if (direct != (1u << NS_ROWS) - 1) {
            float acc[NS_ROWS];
#pragma unroll
            for (int k = 0; k < NS_ROWS; k++) acc[k] = 0.f;
#pragma unroll 4
            for (int d = 0; d < Dp; d += 4) {
                const float4 e = __ldg(ep + (d / 4) * NC_GROUP);
#pragma unroll
                for (int k = 0; k < NS_ROWS; k++) {
                    const float4 v = *(const float4 *)&near_xs[(d * 2 + k) * 4];
                    acc[k] = fmaf(v.x, e.x, acc[k]); acc[k] = fmaf(v.y, e.y, acc[k]); acc[k] = fmaf(v.z, e.z, acc[k]); acc[k] = fmaf(v.w, e.w, acc[k]);
                }
            }
            const float cj = cn[jj];
#pragma unroll
            for (int k = 0; k < NS_ROWS; k++) if (!(direct >> k & 1)) dist[k] = fmaf(-2.0f, acc[k], cj);
        }
#pragma unroll
        for (int k = 0; k < NS_ROWS; k++) {
            unsigned long long p = (on && dist[k] < INFINITY) ? ((unsigned long long)ordered_bits(dist[k]) << 32) | (unsigned)j : ~0ull;
#pragma unroll
            for (int o = 16; o; o >>= 1) { const unsigned long long t = __shfl_xor_sync(0xffffffffu, p, o); p = t < p ? t : p; }
            if (lane == 0 && r0 + k < nr && p != ~0ull) atomicMin(best + place(k), p);
        }
    }
}
static_assert(NS_CODES / 32 == NS_ROWS, "a warp loads a row");
__global__ void k_near_store(const unsigned long long *__restrict__ best, const int *__restrict__ list, const NearCount *__restrict__ count, int n_rows,
                             int *__restrict__ idx_out, int out_tlen, int out_stride, int out_off) {
    pdl_wait();
    const int na = list ? (int)count->na : n_rows, n = na + (list ? (int)count->nb : 0);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int64_t at = i < na ? i : (int64_t)n_rows - 1 - (i - na), r = list ? list[at] : at;
        const unsigned long long p = best[at];
        idx_out[(r / out_tlen) * out_stride + out_off + r % out_tlen] = p == ~0ull ? 0 : (int)(p & 0xffffffffull);   // no finite distance: code 0
    }
}

// ---- host side ----
struct CodeBook { int64_t n; int V, D; char *base; unsigned short *eh, *el; float *cn, *et; NearMeta *meta; };
static std::unordered_map<const float *, CodeBook> &codebooks() { static std::unordered_map<const float *, CodeBook> c; return c; }

void nearest_forget_weights() {
    for (auto &kv : codebooks()) dev_free(kv.second.base);
    codebooks().clear();
}
void nearest_forget_range(const void *p, size_t bytes) {
    auto &cb = codebooks();
    const char *lo = (const char *)p, *hi = lo + bytes;
    for (auto it = cb.begin(); it != cb.end();) {
        const char *w0 = (const char *)it->first, *w1 = w0 + (size_t)it->second.n * 4;
        if (w0 < hi && lo < w1) { dev_free(it->second.base); it = cb.erase(it); }
        else ++it;
    }
}

static const CodeBook &codebook(const float *E, int V, int D) {
    auto &cb = codebooks();
    auto it = cb.find(E);
    if (it != cb.end() && it->second.V == V && it->second.D == D) return it->second;
    if (it != cb.end()) { dev_free(it->second.base); cb.erase(it); }
    const int Vp = (int)cdiv(V, NC_CODES) * NC_CODES;
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t beh = up((size_t)V * D * 2), bcn = up((size_t)Vp * 4), bet = up((size_t)Vp * ((D + 3) & ~3) * 4);
    CodeBook c;
    c.n = (int64_t)V * D; c.V = V; c.D = D;
    c.base = (char *)dev_alloc(2 * beh + bcn + bet + 256);
    c.eh = (unsigned short *)c.base; c.el = (unsigned short *)(c.base + beh); c.cn = (float *)(c.base + 2 * beh);
    c.et = (float *)(c.base + 2 * beh + bcn); c.meta = (NearMeta *)(c.base + 2 * beh + bcn + bet);
    CUDA_CHECK(cudaMemsetAsync(c.meta, 0, sizeof(NearMeta), stream()));
    LAUNCH(k_near_absmax, (unsigned)std::min<int64_t>(cdiv(c.n, 256), ctx().sm_count * 4), 256, 0, E, c.n, c.meta);
    LAUNCH(k_near_codes, (unsigned)cdiv((int64_t)Vp * 32, 256), 256, 0, E, V, Vp, D, c.meta, c.eh, c.el, c.cn, c.et);
    return cb.emplace(E, c).first->second;
}

// Up to this many rows every code is evaluated in fp32 at once: at 16384 codes of 64 dims the four launches and the
// 256-row tiles of the two-pass search cost more than the extra arithmetic.
constexpr int64_t NEAR_SCAN_ROWS = 256;
// Calls of fewer rows never take the pair products: all their rows scanned are 0.2 to 0.3 ms.
constexpr int64_t NEAR_PAIR_ROWS = 1024;

static unsigned scan_grid(int64_t items) { return (unsigned)std::max<int64_t>(1, std::min<int64_t>(items, (int64_t)ctx().sm_count * 6)); }

// 2^20 rows against 16384 x 64 codes, by how close codes lie (three TF32 passes over everything took 9.1 to 10.1 ms for each):
//   random, or a code plus noise           3.7 - 3.9 ms      a tenth undecided (codes about a mean three times their spread)   5.1
//   unused codes at zero                   3.8               all undecided (repeated codes, tight clusters, a mean of 30 times   9.1 - 10.2
//                                                            the spread, unused codes near zero)
// With the scan alone the undecided took up to 144 ms. Calls of under 1024 rows: 42 us for 900 rows, 190 when all are undecided.
void nearest_codes(const float *x, const float *E, int64_t rows, int V, int D, int *idx_out, int out_tlen, int out_stride, int out_off) {
    if (rows <= 0) return;
    static Workspace ws;
    const CodeBook &cb = codebook(E, V, D);
    const int ntiles = (int)cdiv(V, NC_CODES), Dp = (D + 3) & ~3;
    const size_t scan_smem = (size_t)NS_ROWS * Dp * 4;
    const bool coarse = rows > NEAR_SCAN_ROWS && ctx().gemm_mode >= 1 && D <= 128 && D % 8 == 0 && ((uintptr_t)x & 15) == 0;
    if (rows > 0x7fffffff / 2) fatal("nearest: too many rows");
    ProfScope ps(NCMB_K_VQ, 2.0 * (double)rows * V * D, 4.0 * (double)rows * (D + 1));
    if (!coarse) {
        const size_t need = (size_t)rows * 8 + 1024;
        if (need > ws.cap) ws.reserve(need + need / 4);
        ws.reset();
        unsigned long long *best = ws.get<unsigned long long>(rows);
        CUDA_CHECK(cudaMemsetAsync(best, 0xff, (size_t)rows * 8, stream()));
        const int64_t items = cdiv(rows, NS_ROWS) * cdiv(V, NS_CODES);
        LAUNCH(k_nearest_scan, scan_grid(items), NS_CODES, scan_smem, x, cb.et, cb.cn, cb.meta, V, D, (const int *)nullptr, (const NearCount *)nullptr, (int)rows, NEAR_PAIR_ROWS,
               (unsigned short *)nullptr, (unsigned short *)nullptr, (float2 *)nullptr, best);
        LAUNCH_PDL(k_near_store, (unsigned)std::min<int64_t>(cdiv(rows, 256), ctx().sm_count * 4), 256, 0, best, (const int *)nullptr, (const NearCount *)nullptr, (int)rows,
               idx_out, out_tlen, out_stride, out_off);
        return;
    }
    // Row blocks share the SMs; where there are few, each is cut into slices of the codebook so that every SM has work.
    const int64_t blocks = cdiv(rows, NC_ROWS);
    int nslice = 1;
    if (blocks < 4 * (int64_t)ctx().sm_count) {
        double best_t = 1e30;
        for (int s = 1; s <= std::min(NC_MAXSLICE, ntiles); s++) {      // tiles of the busiest SM, and about two tiles' time per item to begin and end it
            const int tps = (int)cdiv(ntiles, s);
            const double t = (double)cdiv(blocks * cdiv(ntiles, tps), ctx().sm_count) * (tps + 2);
            if (t < best_t) { best_t = t; nslice = s; }
        }
    }
    const int tps = (int)cdiv(ntiles, nslice);
    nslice = (int)cdiv(ntiles, tps);
    const int64_t items = blocks * nslice;
    if (items > 0x7fffffff) fatal("nearest: too many work items");
    // (the second halves of the undecided rows take the place of the candidates, the first halves that of the fp16 rows)
    const size_t cand_b = std::max((size_t)nslice * 64, (size_t)D * 2);
    const size_t need = (size_t)rows * (D * 2 + 8 + 8 + 4 + cand_b) + 8192;
    if (need > ws.cap) ws.reserve(need + need / 8);
    ws.reset();
    unsigned short *xh = ws.get<unsigned short>((size_t)rows * D);
    float2 *rinfo = ws.get<float2>(rows);
    float4 *cand = (float4 *)ws.get<unsigned char>((size_t)rows * cand_b);
    unsigned id_mask = 0;
    while ((int)id_mask < tps - 1) id_mask = id_mask * 2 + 1;
    if (id_mask >= 1u << 20) fatal("nearest: codebook of %d rows is too large", V);
    unsigned long long *best = ws.get<unsigned long long>(rows);
    int *list = ws.get<int>(rows);
    NearCount *count = ws.get<NearCount>(1);
    CUDA_CHECK(cudaMemsetAsync(count, 0, sizeof(NearCount), stream()));
    LAUNCH(k_near_rows, (unsigned)cdiv(cdiv(rows, 4) * 32, 256), 256, 0, x, rows, D, cb.meta, xh, rinfo);
    unsigned short *xl = (unsigned short *)cand;
    const CUtensorMap mx = tc_get_map_h16(xh, rows, D, D, 128), me = tc_get_map_h16(cb.eh, V, D, D, 128);
    const int kb = D > 64 ? 2 : 1;
    const unsigned grid = (unsigned)std::min<int64_t>(items, ctx().sm_count);
    static bool set[3] = {false, false, false};
#define NEAR_LAUNCH(KB_)                                                                                                        \
    do {                                                                                                                        \
        if (!set[KB_]) {                                                                                                        \
            CUDA_CHECK(cudaFuncSetAttribute(k_nearest_coarse<KB_, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)nc_smem(KB_, false))); \
            CUDA_CHECK(cudaFuncSetAttribute(k_nearest_coarse<KB_, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)nc_smem(KB_, true))); \
            set[KB_] = true;                                                                                                    \
        }                                                                                                                       \
        if (!pair)                                                                                                              \
            LAUNCH((k_nearest_coarse<KB_, false>), grid, NC_THREADS, nc_smem(KB_, false), mx, me, mx, me, cb.cn, rinfo, rows, ntiles, nslice, tps, (int)items, \
                   id_mask, cand, (const NearCount *)nullptr, (unsigned long long *)nullptr, tc_err_flag());                    \
        else                                                                                                                    \
            LAUNCH_PDL((k_nearest_coarse<KB_, true>), (unsigned)ctx().sm_count, NC_THREADS, nc_smem(KB_, true), mx, me, mx2, me2, cb.cn, rinfo, rows, ntiles, 1, \
                       ntiles, 0, 0u, (float4 *)nullptr, (const NearCount *)count, best, tc_err_flag());                        \
    } while (0)
    auto products = [&](bool pair, const CUtensorMap &mx2, const CUtensorMap &me2) {
        if (kb == 2) NEAR_LAUNCH(2);
        else NEAR_LAUNCH(1);
    };
#undef NEAR_LAUNCH
    products(false, mx, me);
    LAUNCH(k_nearest_refine, (unsigned)cdiv(rows * 32, 256), 256, 0, x, cb.et, cb.cn, V, cb.meta, rinfo, rows, D, nslice * 4, tps, id_mask, cand,
           idx_out, out_tlen, out_stride, out_off, list, count, best);
    const int64_t max_items = cdiv(rows, NS_ROWS) * cdiv(V, NS_CODES);
    LAUNCH_PDL(k_nearest_scan, scan_grid(max_items), NS_CODES, scan_smem, x, cb.et, cb.cn, (const NearMeta *)cb.meta, V, D, (const int *)list, (const NearCount *)count, (int)rows,
               NEAR_PAIR_ROWS, xh, xl, rinfo, best);
    if (rows >= NEAR_PAIR_ROWS)                              // (ends at once where few rows are listed)
        products(true, tc_get_map_h16(xl, rows, D, D, 128), tc_get_map_h16(cb.el, V, D, D, 128));
    LAUNCH_PDL(k_near_store, (unsigned)std::min<int64_t>(cdiv(rows, 256), ctx().sm_count * 4), 256, 0, (const unsigned long long *)best, (const int *)list, (const NearCount *)count, (int)rows,
               idx_out, out_tlen, out_stride, out_off);
}

} // namespace ncmb
