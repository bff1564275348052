// Inverse distances with FP64 accuracy on the FP32 pipe.
//
// This GPU issues one FP64 operation for about 64 FP32 ones, and a 1 / r in
// IEEE FP64 costs about 16 of them.  Here a pair costs about 136 FP32
// operations, 20 integer ones and one FP64 multiply-add, which run beside them
// on their own pipes.  The functions take a float or, for two pairs at a time,
// a float2 (packed FP32x2 operations: the same roundings at half the issue
// slots; packed operands cannot be negated for free, so the middle terms
// carry the sign that needs the fewest negations).
//
// Coordinates (the FMM's less a centre, where that difference is exact) are
// scaled by a power of two to |x| <= 1 and split exactly
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
// ci an unsigned 32-bit integer, which an integer product with y0's mantissa
// adds to the bits of the double y0.
// Every quantity is carried to about 2^-58 relative; the roundings to 2^-52
// units make the error of an IEEE rounding.  Pairs closer than
// 2^-19 of the scale (where the parts no longer hold all bits)
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
GRID_FN double g_double(unsigned long long x) { return __longlong_as_double((long long)x); }
GRID_FN float2 g_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
GRID_FN float2 g_mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
GRID_FN float2 g_fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
GRID_FN float2 g_sub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
GRID_FN float2 g_neg(float2 a) { return __fmul2_rn(a, make_float2(-1.0f, -1.0f)); }
GRID_FN float2 g_rsqrt(float2 x) { return make_float2(g_rsqrt(x.x), g_rsqrt(x.y)); }
GRID_FN float2 g_set(float c, float2) { return make_float2(c, c); }
#else
namespace edfmm {
#endif

constexpr float kGridNear2 = 0x1p-38f;  // below this scaled r^2 the caller evaluates in IEEE FP64

GRID_FN float g_neg(float a) { return -a; }
GRID_FN float g_set(float c, float) { return c; }  // c in the second argument's type

template <typename V> struct GridCoordT {
    V a, b, c;
};
using GridCoord = GridCoordT<float>;

// |x| <= 1
GRID_FN GridCoord grid_split(double x) {
    const double a = (x + 0x1.8p29) - 0x1.8p29;  // to a multiple of 2^-23
    const double r = x - a;
    const double b = (r + 48.0) - 48.0;  // to a multiple of 2^-47
    return GridCoord{(float)a, (float)b, (float)(r - b)};
}

template <typename V> struct GridDiff {
    V d1, d2, d3;
};
template <typename V> GRID_FN GridDiff<V> grid_diff(const GridCoordT<V> &x, const GridCoordT<V> &y) {
    const V a = g_sub(x.a, y.a), b = g_sub(x.b, y.b), c = g_sub(x.c, y.c);
    const V d1 = g_add(a, b);
    const V t = g_sub(b, g_sub(d1, a));
    const V d2 = g_add(t, c);
    return GridDiff<V>{d1, d2, g_sub(c, g_sub(d2, t))};
}

// h += t on the window's grid, l += the rest
template <typename V> GRID_FN void grid_window(V t, V &h, V &l) {
    const V n = g_add(h, t);
    l = g_add(l, g_sub(t, g_sub(n, h)));
    h = n;
}
// s - nf = a + b exactly
template <typename V> GRID_FN void grid_two_sum_neg(V a, V b, V &s, V &nf) {
    s = g_add(a, b);
    const V bb = g_sub(s, a);
    nf = g_add(g_sub(g_sub(s, bb), a), g_sub(bb, b));
}
// s + f = a + b exactly
template <typename V> GRID_FN void grid_two_sum(V a, V b, V &s, V &f) {
    s = g_add(a, b);
    const V bb = g_sub(s, a);
    f = g_add(g_sub(a, g_sub(s, bb)), g_sub(b, bb));
}
// the window of the middle terms: 1.5 2^(exponent(R1) - 13)
GRID_FN float grid_window_of(float R1) { return g_float(((g_bits(R1) & 0x7f800000) - (13 << 23)) | 0x00400000); }
#ifdef __CUDACC__
GRID_FN float2 grid_window_of(float2 R1) { return make_float2(grid_window_of(R1.x), grid_window_of(R1.y)); }
#endif

// r^2 = R1 - Nh - Nl of the difference (x, y, z)
template <typename V> struct GridR2 {
    V R1, Nh, Nl;
};
template <typename V> GRID_FN GridR2<V> grid_r2(const GridDiff<V> &x, const GridDiff<V> &y, const GridDiff<V> &z) {
    const V nx = g_neg(x.d1), ny = g_neg(y.d1), nz = g_neg(z.d1);
    const V px = g_mul(x.d1, x.d1), py = g_mul(y.d1, y.d1), pz = g_mul(z.d1, z.d1);
    const V ex = g_fma(nx, x.d1, px), ey = g_fma(ny, y.d1, py), ez = g_fma(nz, z.d1, pz);  // p - d1^2
    const V tx = g_add(x.d1, x.d1), ty = g_add(y.d1, y.d1), tz = g_add(z.d1, z.d1);
    const V cx = g_mul(g_add(nx, nx), x.d2), cy = g_mul(g_add(ny, ny), y.d2), cz = g_mul(g_add(nz, nz), z.d2);
    V low = g_fma(tx, x.d2, cx);
    low = g_add(low, g_fma(ty, y.d2, cy));
    low = g_add(low, g_fma(tz, z.d2, cz));
    low = g_fma(x.d2, x.d2, low);
    low = g_fma(y.d2, y.d2, low);
    low = g_fma(z.d2, z.d2, low);
    low = g_fma(tx, x.d3, low);
    low = g_fma(ty, y.d3, low);
    low = g_fma(tz, z.d3, low);
    V s, f1, f2;
    GridR2<V> r;
    grid_two_sum_neg(px, py, s, f1);
    grid_two_sum_neg(s, pz, r.R1, f2);
    // the middle terms (negated) are below 2^-21.7 R1 in sum
    const V K = grid_window_of(r.R1);
    V h = g_add(K, cx), l = g_sub(cx, g_sub(h, K));
    grid_window(cy, h, l);
    grid_window(cz, h, l);
    grid_window(ex, h, l);
    grid_window(ey, h, l);
    grid_window(ez, h, l);
    grid_window(f1, h, l);
    grid_window(f2, h, l);
    r.Nh = g_sub(h, K);
    r.Nl = g_sub(l, low);
    return r;
}

// 1 / sqrt(R1 - Nh - Nl) = y0 (1 + ci 2^-52), ci = grid_ci(eh, v); R1 >= kGridNear2
template <typename V> GRID_FN void grid_rsqrt(const GridR2<V> &r, V &y0, V &ehs, V &vs) {
    const V y = g_rsqrt(r.R1);
    y0 = g_fma(y, g_set(-0x1p-21f, V()), y);
    const V ny = g_neg(y0);
    const V th = g_mul(y0, y0), nth = g_mul(ny, y0), ntl = g_fma(ny, y0, th);  // y0^2 = th - ntl
    const V p = g_mul(th, r.R1), pe = g_fma(nth, r.R1, p);                     // th R1 = p - pe
    const V a = g_mul(ntl, r.R1), ae = g_fma(g_neg(ntl), r.R1, a);             // ntl R1 = a - ae
    const V b = g_mul(th, r.Nh), be = g_fma(nth, r.Nh, b);                     // th Nh = b - be
    // 1 - e = p - (pe + a + b) + (ae + be) - th Nl + ntl Nh
    V low = g_fma(nth, r.Nl, be);
    low = g_fma(ntl, r.Nh, low);
    low = g_add(low, ae);
    const V K = g_set(0x1.8p-13f, V());
    V h = g_add(K, pe), l = g_sub(pe, g_sub(h, K));
    grid_window(a, h, l);
    grid_window(b, h, l);
    const V eh = g_add(g_sub(g_set(1.0f, V()), p), g_sub(h, K));  // exact: a multiple of 2^-36 below 2^-19
    const V n = g_sub(low, l);                                  // e = eh - n
    const V v = g_fma(g_mul(eh, eh), g_set(0x1.8p50f, V()), g_mul(n, g_set(-0x1p51f, V())));  // 2^52 (3 eh^2 / 8 - n / 2)
    ehs = g_mul(eh, g_set(0x1p51f, V()));
    vs = g_add(v, g_set(0x1.8p23f, V()));
}
GRID_FN unsigned grid_ci(float ehs, float vs) { return g_to_uint(ehs) + (unsigned)(g_bits(vs) - 0x4B400000); }

// y0 (1 + ci 2^-52) rounded to a double: y0's 24-bit mantissa times ci, in
// units of the double's last place, added to its bits; across a power of two
// the unit doubles
GRID_FN double grid_inv(float y0, unsigned ci) {
    const unsigned u = (unsigned)g_bits(y0);
    const unsigned long long base = ((unsigned long long)((u >> 3) + 0x38000000u) << 32) | (u << 29);
    const unsigned long long d = ((unsigned long long)((u & 0x7fffffu) | 0x800000u) * ci + 0x400000u) >> 23;
    unsigned long long r = base + d;
    if (((unsigned)(r >> 32) ^ (unsigned)(base >> 32)) >> 20) {
        const unsigned long long m = r & 0xfffffffffffffULL;
        r += (m >> 1) - m;
    }
    return g_double(r);
}

// The same to two-float accuracy (about 2^-46) in about 55 operations: the third
// part of the differences is dropped and the middle terms are summed in FP32.
// r^2 = R1 - N, 1 / r = y0 + z.
template <typename V> struct GridDiff2 {
    V d1, d2;
};
template <typename V> GRID_FN GridDiff2<V> grid_diff2(const GridCoordT<V> &x, const GridCoordT<V> &y) {
    const V a = g_sub(x.a, y.a), b = g_sub(x.b, y.b);
    const V d1 = g_add(a, b);
    return GridDiff2<V>{d1, g_add(g_sub(b, g_sub(d1, a)), g_sub(x.c, y.c))};
}
template <typename V>
GRID_FN V grid_r2_tf(const GridDiff2<V> &x, const GridDiff2<V> &y, const GridDiff2<V> &z, V &N) {
    const V px = g_mul(x.d1, x.d1), py = g_mul(y.d1, y.d1), pz = g_mul(z.d1, z.d1);
    V s, f1, R1, f2;
    grid_two_sum_neg(px, py, s, f1);
    grid_two_sum_neg(s, pz, R1, f2);
    V m = g_add(g_add(g_fma(g_neg(x.d1), x.d1, px), g_fma(g_neg(y.d1), y.d1, py)), g_fma(g_neg(z.d1), z.d1, pz));
    m = g_add(m, g_add(f1, f2));
    N = g_fma(g_set(-2.0f, V()), g_fma(z.d1, z.d2, g_fma(y.d1, y.d2, g_mul(x.d1, x.d2))), m);
    return R1;
}
template <typename V> GRID_FN void grid_rsqrt_tf(V R1, V N, V &y0, V &z) {
    y0 = g_rsqrt(R1);
    const V ny = g_neg(y0), th = g_mul(y0, y0), nth = g_mul(ny, y0), ntl = g_fma(ny, y0, th);
    const V p = g_mul(th, R1), pe = g_fma(nth, R1, p);
    const V e = g_fma(th, N, g_fma(ntl, R1, g_add(g_sub(g_set(1.0f, V()), p), pe)));
    z = g_mul(y0, g_mul(e, g_fma(g_set(0.375f, V()), e, g_set(0.5f, V()))));
}

#ifdef __CUDACC__
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
