// Inverse distances with FP64 accuracy on the FP32 pipe.
//
// This GPU issues one FP64 operation for about 64 FP32 ones, and a 1 / r in
// IEEE FP64 costs about 16 of them.  Here a pair costs about 140 FP32 and
// integer operations and two FP64 ones (the product with the charge and the
// accumulation), which run beside them on their own pipe.
//
// Coordinates are scaled by a power of two to |x| <= 1 and split exactly
// into x = a + b + c, a a multiple of 2^-23, b of 2^-47 with |b| <= 2^-24
// and c the rest (a float, |c| <= 2^-48).  On these common grids the
// differences of two points' a and b parts are exact, so a coordinate
// difference d1 + d2 + d3 (three non-overlapping floats) takes nine
// operations.  r^2 = R1 + Mh + Ml follows from error-free products
// (a b = fl(a b) + the FMA residual) and from sums in a window: a term t
// added to H = 1.5 2^k, k well above t, rounds to a grid that all partial
// sums share, so H + t - H is exact and t minus it is the rest (a fast
// two-sum whose order is known).  y0 is the hardware estimate of R1^-1/2,
// lowered by 2^-21 so that e = 1 - y0^2 r^2 > 0, and
//   1 / r = y0 (1 + e / 2 + 3 e^2 / 8) = y0 (1 + ci 2^-52),
// ci an unsigned 32-bit integer: the low word of the double 1 + ci 2^-52.
// Every quantity is carried to about 2^-58 relative; the one rounding to
// 2^-52 units makes the error of an IEEE rounding.  Pairs closer than
// 2^-19 of the largest |coordinate| (where the parts no longer hold all bits)
// are left to the caller's IEEE form.
#pragma once

#ifdef __CUDACC__
#include <cuda_runtime.h>

#include "edfmm_internal.cuh"

namespace edfmm {
#define GRID_FN __device__ __forceinline__
GRID_FN float g_add(float a, float b) { return __fadd_rn(a, b); }
GRID_FN float g_sub(float a, float b) { return __fsub_rn(a, b); }
GRID_FN float g_mul(float a, float b) { return __fmul_rn(a, b); }
GRID_FN float g_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
GRID_FN float g_rsqrt(float x) { return rsqrt_normal(x); }
GRID_FN int g_bits(float x) { return __float_as_int(x); }
GRID_FN float g_float(int x) { return __int_as_float(x); }
GRID_FN unsigned g_to_uint(float x) { return __float2uint_rn(x); }
#else
namespace edfmm {
#endif

constexpr float kGridNear2 = 0x1p-38f;  // below this scaled r^2 the caller evaluates in IEEE FP64

struct GridCoord {
    float a, b, c;
};

// |x| <= 1
GRID_FN GridCoord grid_split(double x) {
    const double a = (x + 0x1.8p29) - 0x1.8p29;  // to a multiple of 2^-23
    const double r = x - a;
    const double b = (r + 48.0) - 48.0;  // to a multiple of 2^-47
    return GridCoord{(float)a, (float)b, (float)(r - b)};
}

struct GridDiff {
    float d1, d2, d3;
};
GRID_FN GridDiff grid_diff(const GridCoord &x, const GridCoord &y) {
    const float a = g_sub(x.a, y.a), b = g_sub(x.b, y.b), c = g_sub(x.c, y.c);
    const float d1 = g_add(a, b);
    const float t = g_sub(b, g_sub(d1, a));
    const float d2 = g_add(t, c);
    return GridDiff{d1, d2, g_sub(c, g_sub(d2, t))};
}

// h += t on the window's grid, l += the rest
GRID_FN void grid_window(float t, float &h, float &l) {
    const float n = g_add(h, t);
    l = g_add(l, g_sub(t, g_sub(n, h)));
    h = n;
}
// s + f = a + b exactly
GRID_FN void grid_two_sum(float a, float b, float &s, float &f) {
    s = g_add(a, b);
    const float bb = g_sub(s, a);
    f = g_add(g_sub(a, g_sub(s, bb)), g_sub(b, bb));
}

// r^2 = R1 + Mh + Ml of the difference (x, y, z)
struct GridR2 {
    float R1, Mh, Ml;
};
GRID_FN GridR2 grid_r2(const GridDiff &x, const GridDiff &y, const GridDiff &z) {
    const float px = g_mul(x.d1, x.d1), py = g_mul(y.d1, y.d1), pz = g_mul(z.d1, z.d1);
    const float ex = g_fma(x.d1, x.d1, -px), ey = g_fma(y.d1, y.d1, -py), ez = g_fma(z.d1, z.d1, -pz);
    const float ux = g_add(x.d2, x.d2), uy = g_add(y.d2, y.d2), uz = g_add(z.d2, z.d2);
    const float cx = g_mul(x.d1, ux), cy = g_mul(y.d1, uy), cz = g_mul(z.d1, uz);
    float low = g_fma(x.d1, ux, -cx);
    low = g_add(low, g_fma(y.d1, uy, -cy));
    low = g_add(low, g_fma(z.d1, uz, -cz));
    low = g_fma(x.d2, x.d2, low);
    low = g_fma(y.d2, y.d2, low);
    low = g_fma(z.d2, z.d2, low);
    low = g_fma(x.d1, g_add(x.d3, x.d3), low);
    low = g_fma(y.d1, g_add(y.d3, y.d3), low);
    low = g_fma(z.d1, g_add(z.d3, z.d3), low);
    float s, f1, f2;
    GridR2 r;
    grid_two_sum(px, py, s, f1);
    grid_two_sum(s, pz, r.R1, f2);
    // the middle terms are below 2^-21.7 R1 in sum: window 1.5 2^(exponent(R1) - 13)
    const float K = g_float(((g_bits(r.R1) & 0x7f800000) - (13 << 23)) | 0x00400000);
    float h = g_add(K, cx), l = g_sub(cx, g_sub(h, K));
    grid_window(cy, h, l);
    grid_window(cz, h, l);
    grid_window(ex, h, l);
    grid_window(ey, h, l);
    grid_window(ez, h, l);
    grid_window(f1, h, l);
    grid_window(f2, h, l);
    r.Mh = g_sub(h, K);
    r.Ml = g_add(l, low);
    return r;
}

// 1 / sqrt(R1 + Mh + Ml) = y0 (1 + ci 2^-52); R1 >= kGridNear2
GRID_FN void grid_rsqrt(const GridR2 &r, float &y0, unsigned &ci) {
    const float y = g_rsqrt(r.R1);
    y0 = g_fma(y, -0x1p-21f, y);
    const float th = g_mul(y0, y0), tl = g_fma(y0, y0, -th);
    const float p = g_mul(th, r.R1), pe = g_fma(th, r.R1, -p);
    const float a = g_mul(tl, r.R1), ae = g_fma(tl, r.R1, -a);
    const float b = g_mul(th, r.Mh), be = g_fma(th, r.Mh, -b);
    float low = g_fma(th, r.Ml, be);
    low = g_fma(tl, r.Mh, low);
    low = g_add(low, ae);
    const float K = 0x1.8p-13f;
    float h = g_add(K, pe), l = g_sub(pe, g_sub(h, K));
    grid_window(a, h, l);
    grid_window(b, h, l);
    const float eh = g_sub(g_sub(1.0f, p), g_sub(h, K));  // exact: a multiple of 2^-36 below 2^-19
    const float n = g_add(l, low);                        // e = eh - n
    const float v = g_fma(g_mul(eh, eh), 0x1.8p50f, g_mul(n, -0x1p51f));  // 2^52 (3 eh^2 / 8 - n / 2)
    ci = g_to_uint(g_mul(eh, 0x1p51f)) + (unsigned)(g_bits(g_add(v, 0x1.8p23f)) - 0x4B400000);
}

// The same to two-float accuracy (about 2^-46) in about 60 operations: the third
// part of the differences is dropped and the middle terms are summed in FP32.
// 1 / r = y0 + z.
struct GridDiff2 {
    float d1, d2;
};
GRID_FN GridDiff2 grid_diff2(const GridCoord &x, const GridCoord &y) {
    const float a = g_sub(x.a, y.a), b = g_sub(x.b, y.b);
    const float d1 = g_add(a, b);
    return GridDiff2{d1, g_add(g_sub(b, g_sub(d1, a)), g_sub(x.c, y.c))};
}
GRID_FN float grid_r2_tf(const GridDiff2 &x, const GridDiff2 &y, const GridDiff2 &z, float &M) {
    const float px = g_mul(x.d1, x.d1), py = g_mul(y.d1, y.d1), pz = g_mul(z.d1, z.d1);
    float s, f1, R1, f2;
    grid_two_sum(px, py, s, f1);
    grid_two_sum(s, pz, R1, f2);
    float m = g_add(g_add(g_fma(x.d1, x.d1, -px), g_fma(y.d1, y.d1, -py)), g_fma(z.d1, z.d1, -pz));
    m = g_add(m, g_add(f1, f2));
    M = g_fma(2.0f, g_fma(z.d1, z.d2, g_fma(y.d1, y.d2, g_mul(x.d1, x.d2))), m);
    return R1;
}
GRID_FN void grid_rsqrt_tf(float R1, float M, float &y0, float &z) {
    y0 = g_rsqrt(R1);
    const float th = g_mul(y0, y0), tl = g_fma(y0, y0, -th);
    const float p = g_mul(th, R1), pe = g_fma(th, R1, -p);
    const float e = g_fma(-th, M, g_fma(-tl, R1, g_sub(g_sub(1.0f, p), pe)));
    z = g_mul(y0, g_mul(e, g_fma(0.375f, e, 0.5f)));
}

#ifdef __CUDACC__
// the double with the value of a positive normal float
GRID_FN double grid_double(float x) {
    const unsigned u = __float_as_uint(x);
    return __hiloint2double((int)((u >> 3) + 0x38000000u), (int)(u << 29));
}
// 1 + ci 2^-52
GRID_FN double grid_one_plus(unsigned ci) { return __hiloint2double(0x3FF00000, (int)ci); }
// exponent k with |x| < 2^k for the largest |x| whose high word is `hi`, and
// whether the split applies (finite, not zero, scales in range)
GRID_FN bool grid_exponent(unsigned hi, int &k) {
    const int e = (int)(hi >> 20);
    k = e - 1022;
    return e > 1023 - 300 && e < 1023 + 300;
}
GRID_FN double grid_pow2(int k) { return __hiloint2double((1023 + k) << 20, 0); }
#endif

#undef GRID_FN
}  // namespace edfmm
