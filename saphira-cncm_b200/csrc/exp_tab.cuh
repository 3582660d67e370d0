// exp() in fp64 of a difference x <= 0 by a table in shared memory.
#pragma once

namespace ncmb {

// exp() in fp64 of a difference x <= 0, by table and polynomial (Tang, "Table-driven implementation of the exponential function",
// ACM TOMS 15, 1989): x = (64 k + j) ln2 / 64 + r with |r| <= ln2 / 128, e^x = 2^k 2^(j/64) (1 + r + r^2/2 + ... + r^5/120). The
// truncation is below 2^-54; eleven fp64 operations a term instead of the library call's thirty-odd, which
// were what the kernels that take one per logit spent their time on. Largest error in 2e7 arguments from -40 to 0: 1.3 units in
// the last place (2 where an entry of the table is rounded the other way), which the sums over a vocabulary do not show: likelihoods of
// the Qwen2 shape are 2.3e-16 from 80-bit sums over the same logits, as with the library call.
constexpr int EXP_TAB = 64;
__device__ __forceinline__ void exp_tab_fill(double *tab) {      // by the first EXP_TAB threads; a barrier has to follow
    if (threadIdx.x < EXP_TAB) tab[threadIdx.x] = exp2((double)threadIdx.x / EXP_TAB);
}
__device__ __forceinline__ double exp_tab(double x, const double *tab) {
    if (x < -700.0) return 0.0;                                    // below any sum this is added to
    const double magic = 6755399441055744.0;                       // 1.5 * 2^52: adding it rounds to an integer
    const double t = fma(x, 92.332482616893656877, magic);         // 64 / ln 2
    const int n = __double2loint(t);
    const double kd = t - magic;
    double r = fma(kd, -0x1.62e42fefa0000p-7, x);                  // ln2 / 64 in two parts, the first short enough for an exact product
    r = fma(kd, -0x1.cf79abc9e3b39p-46, r);
    double q = fma(r, 1.0 / 120.0, 1.0 / 24.0);
    q = fma(r, q, 1.0 / 6.0);
    q = fma(r, q, 0.5);
    q = fma(r * r, q, r);
    const double b = tab[n & 63], e = fma(b, q, b);
    return __hiloint2double(__double2hiint(e) + ((n >> 6) << 20), __double2loint(e));
}

} // namespace ncmb
