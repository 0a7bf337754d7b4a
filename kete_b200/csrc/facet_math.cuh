// facet_math.cuh -- the elementary functions of the thermal models' facets (kernels.cu):
// reciprocal, reciprocal square root, exponential and logarithm over the ranges that the facets
// need, in fewer instructions than the library's.
//
// Errors over those ranges, as tests/test_gpu_facet_math.py holds them: 2^-52 relative for the
// reciprocals, 2^-51 for the exponential, 9e-16 absolute for the logarithm.
#pragma once

namespace kb {

// 1 / x of a normal x, and 1 / sqrt(x) of a normal x > 0, from the hardware's seeds (good to
// about 20 bits) by one third-order step: with e = 1 - x y, 1 / x = y (1 + e + e^2 + O(e^3)),
// and with e = 1 - x y^2, 1 / sqrt(x) = y (1 + e / 2 + 3 e^2 / 8 + O(e^3)).
__device__ __forceinline__ double recip3(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ double rsqrt3(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x * y, y, 1.0);
    return fma(y * e, fma(e, 0.375, 0.5), y);
}

// Constants of the facet arithmetic, as constant-bank operands: written as literals the compiler
// loads them into registers in every batch, two instructions each.
struct FacetConst {
    double log2e32, magic, ln2_hi, ln2_lo;  // 32 / ln 2, 1.5 x 2^52, ln 2 / 32 in two parts
    double e[5];                            // 1/6! .. 1/2!
    double artanh[10];                      // 1/21, 1/19 .. 1/3
    double ln2;
    double w1[5], w2[5], w3[5], w4[5];      // WISE corrections, highest power last
};
static __constant__ FacetConst c_fc = {
    46.16624130844683, 6755399441055744.0, 0x1.62e42fee00000p-6, 0x1.a39ef35793c76p-38,
    {1.0 / 720.0, 1.0 / 120.0, 1.0 / 24.0, 1.0 / 6.0, 0.5},
    {1.0 / 21.0, 1.0 / 19.0, 1.0 / 17.0, 1.0 / 15.0, 1.0 / 13.0, 1.0 / 11.0, 1.0 / 9.0, 1.0 / 7.0,
     1.0 / 5.0, 1.0 / 3.0},
    0.6931471805599453,
    {-3.78226591e-01, 3.50431748e-03, 1.45866307e-05, -6.67674083e-08, 7.03651986e-11},
    {-8.60229377e-01, 1.54988562e-02, -5.10705456e-05, 7.68314436e-08, -4.32238900e-11},
    {-1.29814355, 2.43268763e-02, -9.05178737e-05, 1.50095351e-07, -9.35433316e-11},
    {2.17247804e+01, -1.46084733e+01, 3.85364000e+00, -4.51512551e-01, 1.98397252e-02}};

// exp(x) for 0 <= x < 700: x = (32 n + j) ln 2 / 32 + r with ln 2 in two parts (Cody and Waite;
// the first has 32 significant bits, so its multiples are exact), the exponential's series to
// r^6 (the next term lies below 4e-18 for |r| <= ln 2 / 64), 2^(j/32) from the block's table,
// scaled by 2^n.
constexpr int EXP_TABLE = 32;
__device__ __forceinline__ double exp_positive(double x, const double* __restrict__ table) {
    const double t = fma(x, c_fc.log2e32, c_fc.magic);  // the low word is rint(32 x / ln 2)
    const double n = t - c_fc.magic;
    const int k = __double2loint(t);
    double r = fma(-n, c_fc.ln2_hi, x);
    r = fma(-n, c_fc.ln2_lo, r);
    double p = c_fc.e[0];
#pragma unroll
    for (int i = 1; i < 5; ++i) p = fma(p, r, c_fc.e[i]);
    p = fma(p * r, r, r);  // exp(r) - 1
    const double w = table[k & (EXP_TABLE - 1)];
    const double y = fma(w, p, w);
    return __hiloint2double(__double2hiint(y) + ((k >> 5) << 20), __double2loint(y));
}

// log(t) for 100 <= t <= 400: t = 2^e m with m in [2^-1/2, 2^1/2), log m = 2 artanh(s) with
// s = (m - 1) / (m + 1), |s| <= 0.1716, its series to s^21 (the next term lies below 3e-18).
__device__ __forceinline__ double log_kelvin(double t) {
    const int hi = __double2hiint(t);
    const int e = (hi - 0x3fe6a09e) >> 20;  // t / 2^e in [sqrt(1/2), sqrt(2))
    const double m = __hiloint2double(hi - (e << 20), __double2loint(t));
    const double s = (m - 1.0) * recip3(m + 1.0), z = s * s;
    double p = c_fc.artanh[0];
#pragma unroll
    for (int k = 1; k < 10; ++k) p = fma(p, z, c_fc.artanh[k]);
    const double l = fma(2.0 * s * z, p, 2.0 * s);
    return fma((double)e, c_fc.ln2, l);
}

}  // namespace kb
