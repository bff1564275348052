// Rotation-based M2L ("point and shoot").
//
// With d = (c_L - c_M) / a_L at polar angle theta and azimuth phi, rotate the
// frame so that d lies on +z, translate along z, rotate back:
//   M' = conj T(Q) M,   L' = axial(M', |d|),   L = T(Q)^T L',
//   Q = R_y(-theta) R_z(-phi),
// where T(Q) maps the solid harmonics under the rotation,
// R_n^m(Q v) = sum_m' T^n_{m m'}(Q) R_n^m'(v).  A z rotation is diagonal
// (e^{i m a}), and a y rotation is R_y(b) = Q_m R_z(b) Q_p with the fixed
// quarter turns Q_p, Q_m about x.  Their exact matrices (rotation_tables.h,
// real block basis [Re X0, Re X1, Im X1, ...] per degree, about 25% non-zero)
// are compile-time constants, so the zero entries cost nothing.  Along z,
// I_j^mu(0, 0, rho) = delta_mu0 j! / rho^(j+1), so
//   L'_n^m = (-1)^(n+m) sum_{k >= m} M'_k^m (n+k)! / rho^(n+k+1).
// Per pair this is about 2,300 multiply-adds at p = 8, against 7,300 for the
// azimuth-factored contraction.  One lane per (target, source) pair, one
// warp per target row; each lane accumulates its translated locals in
// private shared-memory slots, reduced over the warp at the end (fixed order).
#pragma once

#include <type_traits>

#include "edfmm_internal.cuh"
#include "harmonics.cuh"
#include "rotation_tables.h"
#include "twofloat.cuh"

namespace edfmm {
namespace {

constexpr float kRotExtremeRatio = 256.0f;  // FP32: beyond this (a_M/a_L)^k may overflow
constexpr int kRotThreads = 128;             // 4 warps; FP32: 3 blocks per SM at <= 168 registers

template <int TAB> __host__ __device__ constexpr double rot_entry(int i) {
    return TAB == 0 ? kRotFwdP[i] : TAB == 1 ? kRotFwdM[i] : TAB == 2 ? kRotBwdP[i] : kRotBwdM[i];
}

// y[I] = sum_J G[I][J] x[J] over the non-zero entries of table TAB, degree block at OFF
template <typename T, int TAB, int N, int OFF, int I, int J>
__device__ __forceinline__ void rot_dot(const T (&x)[N], T &acc) {
    constexpr double g = rot_entry<TAB>(OFF + I * N + J);
    if constexpr (g != 0.0) {
        if constexpr (std::is_same<T, tf32x2>::value) {
            // the table entries are dyadic rationals: nearly all exact in FP32
            constexpr float ghi = (float)g;
            constexpr float glo = (float)(g - (double)ghi);
            acc = tf_fma_const<glo == 0.0f>(ghi, glo, x[J], acc);
        } else {
            acc = fma((T)g, x[J], acc);
        }
    }
    if constexpr (J + 1 < N) rot_dot<T, TAB, N, OFF, I, J + 1>(x, acc);
}
template <typename T, int TAB, int N, int OFF, int I>
__device__ __forceinline__ void rot_apply(const T (&x)[N], T (&y)[N]) {
    T acc = T(0);
    rot_dot<T, TAB, N, OFF, I, 0>(x, acc);
    y[I] = acc;
    if constexpr (I + 1 < N) rot_apply<T, TAB, N, OFF, I + 1>(x, y);
}

// X_m <- X_m e^{i m a} on a degree block: (c[m], s[m]) = (cos m a, sin m a)
template <typename T, int N, int P>
__device__ __forceinline__ void zrot(T (&b)[N], const T (&c)[P + 1], const T (&s)[P + 1], T sign) {
#pragma unroll
    for (int m = 1; 2 * m < N; ++m) {
        const T re = b[2 * m - 1], im = b[2 * m], cm = c[m];
        if constexpr (std::is_same<T, tf32x2>::value) {
            const T sm = sign.hi < 0.0f ? -s[m] : s[m];
            b[2 * m - 1] = tf_cmul(re, cm, im, -sm);
            b[2 * m] = tf_cmul(im, cm, re, sm);
        } else {
            const T sm = sign * s[m];
            b[2 * m - 1] = re * cm - im * sm;
            b[2 * m] = re * sm + im * cm;
        }
    }
}

template <typename T, int P> struct Frame {
    T cp[P + 1], sp[P + 1];  // cos / sin (m phi)
    T ct[P + 1], st[P + 1];  // cos / sin (m theta)
};

template <typename T, int P>
__device__ __forceinline__ void powers(T c, T s, T (&cm)[P + 1], T (&sm)[P + 1]) {
    cm[0] = T(1);
    sm[0] = T(0);
#pragma unroll
    for (int m = 1; m <= P; ++m) {
        cm[m] = cm[m - 1] * c - sm[m - 1] * s;
        sm[m] = cm[m - 1] * s + sm[m - 1] * c;
    }
}

// register store of the (P+1)^2 real coefficients, or private shared-memory slots
template <typename T, int NV> struct RegV {
    T v[NV];
    __device__ __forceinline__ T get(int i) const { return v[i]; }
    __device__ __forceinline__ void set(int i, T x) { v[i] = x; }
};
// Shared-memory loads the compiler may not hoist or merge, so the FP64 kernel
// re-reads each coefficient where it is used instead of keeping them all in
// registers (FP64 FMAs are the cost there; shared-memory traffic is free).
__device__ __forceinline__ float lds_keep(const float *p) {
    float v;
    asm volatile("ld.volatile.shared.f32 %0, [%1];" : "=f"(v) : "r"((unsigned)__cvta_generic_to_shared(p)));
    return v;
}
__device__ __forceinline__ double lds_keep(const double *p) {
    double v;
    asm volatile("ld.volatile.shared.f64 %0, [%1];" : "=d"(v) : "r"((unsigned)__cvta_generic_to_shared(p)));
    return v;
}
// The matching stores are volatile too: volatile accesses keep their program
// order, which a plain store next to an asm load would not be guaranteed.
__device__ __forceinline__ void sts_keep(float *p, float v) {
    asm volatile("st.volatile.shared.f32 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(p)), "f"(v));
}
__device__ __forceinline__ void sts_keep(double *p, double v) {
    asm volatile("st.volatile.shared.f64 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(p)), "d"(v));
}
__device__ __forceinline__ tf32x2 lds_keep(const tf32x2 *p) {
    tf32x2 v;
    asm volatile("ld.volatile.shared.v2.f32 {%0, %1}, [%2];"
                 : "=f"(v.hi), "=f"(v.lo)
                 : "r"((unsigned)__cvta_generic_to_shared(p)));
    return v;
}
__device__ __forceinline__ void sts_keep(tf32x2 *p, tf32x2 v) {
    asm volatile("st.volatile.shared.v2.f32 [%0], {%1, %2};" ::"r"((unsigned)__cvta_generic_to_shared(p)), "f"(v.hi),
                 "f"(v.lo));
}
template <typename T, int STRIDE> struct SmemV {
    T *base;  // this lane's slot 0; slot i at base[i * STRIDE]
    __device__ __forceinline__ T get(int i) const { return lds_keep(base + i * STRIDE); }
    __device__ __forceinline__ void set(int i, T x) { sts_keep(base + i * STRIDE, x); }
};

// Per-lane accumulator of the translated locals (FP32): complex slot tri(n, m)
// at base[tri(n, m) * STRIDE] (one 8-byte word per lane, so a warp's access is
// conflict-free and each coefficient pair is one load and one store).  Plain
// accesses: the compiler keeps the slots in shared memory at 167 registers
// (volatile stores measured 5% slower).
template <int STRIDE> struct AccC {
    float2 *base;
    __device__ __forceinline__ float2 get(int q) const { return base[q * STRIDE]; }
    __device__ __forceinline__ void set(int q, float2 x) { base[q * STRIDE] = x; }
};

// forward rotation of degree n: scale by fn, R_z(+phi), Q_p, R_z(+theta), Q_m.
// BINOM: fn = c^n n! / rho^n (cr = c / rho); else fn = c^n (cr = c).
template <typename T, int P, bool BINOM, int n, typename V>
__device__ __forceinline__ void forward(V &v, T cr, T fn, const Frame<T, P> &F) {
    constexpr int N = 2 * n + 1, OV = n * n, OFF = kRotOff[n];
    T b[N], o[N];
#pragma unroll
    for (int i = 0; i < N; ++i) b[i] = v.get(OV + i) * fn;
    zrot<T, N, P>(b, F.cp, F.sp, T(1));
    rot_apply<T, 0, N, OFF, 0>(b, o);
    zrot<T, N, P>(o, F.ct, F.st, T(1));
    rot_apply<T, 1, N, OFF, 0>(o, b);
#pragma unroll
    for (int i = 0; i < N; ++i) v.set(OV + i, b[i]);
    if constexpr (n < P) forward<T, P, BINOM, n + 1>(v, cr, BINOM ? fn * cr * T(n + 1) : fn * cr, F);
}

// backward rotation of degree n (transposes in reverse order), added to acc;
// BINOM: scaled by hn = n! / rho^(n+1) as it is added
template <int P, bool BINOM, int n, typename V, typename A>
__device__ __forceinline__ void backward(V &v, A &acc, const Frame<float, P> &F, float hn, float irho) {
    constexpr int N = 2 * n + 1, OV = n * n, OFF = kRotOff[n];
    float b[N], o[N];
#pragma unroll
    for (int i = 0; i < N; ++i) b[i] = v.get(OV + i);
    rot_apply<float, 3, N, OFF, 0>(b, o);
    zrot<float, N, P>(o, F.ct, F.st, -1.0f);
    rot_apply<float, 2, N, OFF, 0>(o, b);
    zrot<float, N, P>(b, F.cp, F.sp, -1.0f);
    {
        float2 a = acc.get(tri(n, 0));
        a.x = BINOM ? fma(b[0], hn, a.x) : a.x + b[0];
        acc.set(tri(n, 0), a);
    }
#pragma unroll
    for (int m = 1; m <= n; ++m) {
        const float2 x = make_float2(b[2 * m - 1], b[2 * m]), a = acc.get(tri(n, m));
        acc.set(tri(n, m), BINOM ? __ffma2_rn(x, make_float2(hn, hn), a) : __fadd2_rn(a, x));
    }
    if constexpr (n < P) backward<P, BINOM, n + 1>(v, acc, F, hn * float(n + 1) * irho, irho);
}

// The axial translation with the factor table f[j] = j! / rho^(j+1):
// L'_n^m = (-1)^(n+m) sum_{k=m..P} M'_k^m f[n+k], in place; the complex
// (m >= 1) terms as packed pairs, f2[j] = (f[j], f[j]).
template <int P, int m, typename V>
__device__ __forceinline__ void axial_table(V &v, const float (&f)[2 * P + 1], const float2 (&f2)[2 * P + 1]) {
    if constexpr (m > 0) {
        float2 u[P + 1];
#pragma unroll
        for (int k = m; k <= P; ++k) u[k] = make_float2(v.get(k * k + 2 * m - 1), v.get(k * k + 2 * m));
#pragma unroll
        for (int n = m; n <= P; ++n) {
            float2 sum = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int k = m; k <= P; ++k) sum = __ffma2_rn(u[k], f2[n + k], sum);
            const float sg = ((n + m) & 1) ? -1.0f : 1.0f;
            v.set(n * n + 2 * m - 1, sg * sum.x);
            v.set(n * n + 2 * m, sg * sum.y);
        }
    } else {
        float u[P + 1], w[P + 1];
#pragma unroll
        for (int k = 0; k <= P; ++k) u[k] = v.get(k * k);
#pragma unroll
        for (int n = 0; n <= P; ++n) {
            float sum = 0.0f;
#pragma unroll
            for (int k = 0; k <= P; ++k) sum = fma(u[k], f[n + k], sum);
            w[n] = (n & 1) ? -sum : sum;
        }
#pragma unroll
        for (int n = 0; n <= P; ++n) v.set(n * n, w[n]);
    }
    if constexpr (m < P) axial_table<P, m + 1>(v, f, f2);
}

// The axial translation in binomial form (the FP32 kernel at p <= 7 and the
// two-float kernel; the FP32 kernel at p = 8 keeps the factor table, whose
// packed m >= 1 sums issue fewer instructions).  Along z,
//   L'_n^m = (-1)^(n+m) sum_{k=m..P} M'_k^m (n+k)! / rho^(n+k+1)
//          = h_n (-1)^(n+m) sum_k C(n+k, k) u_k^m,
// with u_k = M'_k k! / rho^k and h_n = n! / rho^(n+1).  The forward pass folds
// k! / rho^k into its scaling by c^k and the backward pass folds h_n into its
// accumulation, so the sums here have exact integer coefficients (at most
// C(16, 8) = 12,870), compile-time constants: no per-pair factor table.
__host__ __device__ constexpr double binom(int n, int k) {
    double r = 1.0;
    for (int i = 1; i <= k; ++i) r = r * (n - k + i) / i;
    return r;
}

// s = sum_{k=K..P} C(N+k, k) u[k] (K = the first term: a product)
template <typename T, int P, int N, int K, bool FIRST>
__device__ __forceinline__ void binom_dot(const T (&u)[P + 1], T &s) {
    constexpr double cb = binom(N + K, K);
    if constexpr (std::is_same<T, tf32x2>::value) {
        if constexpr (FIRST) {  // u * cb, cb exact in FP32
            const tf32x2 pr = tf_two_prod(u[K].hi, (float)cb);
            s = tf_fast_two_sum(pr.hi, __fmaf_rn(u[K].lo, (float)cb, pr.lo));
        } else {
            s = tf_fma_const<true>((float)cb, 0.0f, u[K], s);
        }
    } else if constexpr (FIRST) {
        s = u[K] * (T)cb;
    } else {
        s = fma((T)cb, u[K], s);
    }
    if constexpr (K < P) binom_dot<T, P, N, K + 1, false>(u, s);
}

template <typename T, int P, int m, int N, bool SCALE_OUT>
__device__ __forceinline__ void binom_rows(const T (&ur)[P + 1], const T (&ui)[P + 1], T (&wr)[P + 1],
                                           T (&wi)[P + 1], const T (&h)[P + 1]) {
    T sr, si = T(0);
    binom_dot<T, P, N, m, true>(ur, sr);
    if constexpr (m > 0) binom_dot<T, P, N, m, true>(ui, si);
    if constexpr (SCALE_OUT) {
        sr = sr * h[N];
        if constexpr (m > 0) si = si * h[N];
    }
    wr[N] = ((N + m) & 1) ? -sr : sr;
    wi[N] = ((N + m) & 1) ? -si : si;
    if constexpr (N < P) binom_rows<T, P, m, N + 1, SCALE_OUT>(ur, ui, wr, wi, h);
}

// u -> (-1)^(n+m) sum_k C(n+k, k) u_k^m in place (times h_n when SCALE_OUT)
template <typename T, int P, int m, bool SCALE_OUT, typename V>
__device__ __forceinline__ void axial(V &v, const T (&h)[P + 1]) {
    T ur[P + 1], ui[P + 1], wr[P + 1], wi[P + 1];
#pragma unroll
    for (int k = m; k <= P; ++k) {
        ur[k] = v.get(k * k + (m == 0 ? 0 : 2 * m - 1));
        ui[k] = m == 0 ? T(0) : v.get(k * k + 2 * m);
    }
    binom_rows<T, P, m, m, SCALE_OUT>(ur, ui, wr, wi, h);
#pragma unroll
    for (int n = m; n <= P; ++n) {
        v.set(n * n + (m == 0 ? 0 : 2 * m - 1), wr[n]);
        if (m > 0) v.set(n * n + 2 * m, wi[n]);
    }
    if constexpr (m < P) axial<T, P, m + 1, SCALE_OUT>(v, h);
}

// Which axial form the FP32 / FP64 kernel of order P runs (measured on the
// GB300: binomial 2.05 against 2.14 ms per M2L at p = 6, table 3.59 against
// 3.82 ms at p = 8)
template <typename T, int P> __host__ __device__ constexpr bool rot_binomial() { return !(sizeof(T) == 4 && P >= 8); }

// One pair (FP32): translated locals of the source with column Mcol added to acc.
template <int P, typename V, typename A>
__device__ __forceinline__ void rot_pair(V &v, A &acc, const float4 *Mcol, float c, float dx, float dy,
                                         float dz) {
    float4 x4{};
#pragma unroll
    for (int n = 0; n <= P; ++n) {
#pragma unroll
        for (int m = 0; m <= n; ++m) {
            const int q = tri(n, m);
            if ((q & 1) == 0) x4 = Mcol[(q >> 1) * kColNodes];  // two coefficients
            const float2 x = (q & 1) == 0 ? make_float2(x4.x, x4.y) : make_float2(x4.z, x4.w);
            if (m == 0) {
                v.set(n * n, x.x);
            } else {
                v.set(n * n + 2 * m - 1, x.x);
                v.set(n * n + 2 * m, x.y);
            }
        }
    }
    const float s2 = dx * dx + dy * dy, r2 = s2 + dz * dz;
    const float s = sqrt(s2), rho = sqrt(r2), irho = 1.0f / rho;
    Frame<float, P> F;
    float cphi = 1.0f, sphi = 0.0f;
    if (s2 > 0.0f) {
        const float is = 1.0f / s;
        cphi = dx * is;
        sphi = dy * is;
    }
    powers<float, P>(cphi, sphi, F.cp, F.sp);
    powers<float, P>(dz * irho, s * irho, F.ct, F.st);
    constexpr bool BINOM = rot_binomial<float, P>();
    forward<float, P, BINOM, 0>(v, BINOM ? c * irho : c, 1.0f, F);
    if constexpr (BINOM) {
        const float none[P + 1] = {};
        axial<float, P, 0, false>(v, none);
    } else {
        float f[2 * P + 1];
        f[0] = irho;
#pragma unroll
        for (int j = 1; j <= 2 * P; ++j) f[j] = f[j - 1] * (float)j * irho;
        float2 f2[2 * P + 1];
#pragma unroll
        for (int j = 0; j <= 2 * P; ++j) f2[j] = make_float2(f[j], f[j]);
        axial_table<P, 0>(v, f, f2);
    }
    backward<P, BINOM, 0>(v, acc, F, irho, irho);
}

// ---------------------------------------------------------------------------
// Packed layouts of the quarter-turn matrices.  In the real block basis each
// matrix of degree n is the direct sum of four dense blocks: an output
// coefficient reads only inputs of one class (real or imaginary part, m even
// or odd), and the four classes map to one another in pairs.  Pairing Re X_j
// with Im X_{j+1} (j = 0..n-1; Re X_n stays alone) puts two rows of
// different blocks into one packed FP32x2 operation whose operand is one
// input pair, for every input pair: 145 instead of 247 multiply-adds per
// matrix at p = 8, no cross terms.  Two layouts of a degree block are used:
//   RI: pair j = (Re X_j, Im X_{j+1});
//   XN: the same pairs with the halves swapped where j + n is odd;
// a forward matrix maps XN to RI, a backward one RI to XN.  The two-float
// kernel runs its matrices in this form (below).  (For the FP32 kernel the
// packed form measured slower: 4.43 against 3.59 ms per M2L at p = 8.)
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int ix_re(int m) { return m == 0 ? 0 : 2 * m - 1; }

// block index of half h of pair j of a degree-n block in layout L (0: RI, 1: XN)
template <int n, int L>
__host__ __device__ constexpr int pk_ix(int j, int h) {
    return ((L == 1 && ((j + n) & 1)) ? 1 - h : h) == 0 ? ix_re(j) : 2 * (j + 1);
}

// matrix entry (a, c) of table TAB, degree n
template <int TAB, int n>
__host__ __device__ constexpr double pk_g(int a, int c) {
    return rot_entry<TAB>(kRotOff[n] + a * (2 * n + 1) + c);
}

// does input pair i < I hold a non-zero for row A (half x) or row B (half y)?
template <int TAB, int n, int LIN, int A, int B>
__host__ __device__ constexpr bool pk_started(int I) {
    for (int i = 0; i < I; ++i)
        if (pk_g<TAB, n>(A, pk_ix<n, LIN>(i, 0)) != 0.0 || pk_g<TAB, n>(B, pk_ix<n, LIN>(i, 1)) != 0.0) return true;
    return false;
}

// One warp per target row, one lane per (target, source) pair.  The warps of
// a block run the same number of rounds of pairs, with a barrier between
// rounds, so that the warps of an SM walk the long straight-line pair code
// close together and share its instruction fetches.  Three warps a scheduler
// (168 registers, 46 KB of accumulators a block) must cover every latency:
// sources are read by columns and a round's source ids one round ahead.  30.6 M
// pairs of order 8: 3,178 us with rows (L1 at 64% of its wavefronts, a line
// per lane and load), 2,769 with columns (their copy, 8 us, included), 2,637
// with the ids ahead (1,620 us at the FP32 pipe's full rate; issue slots 64%
// used).  Reading the sources' centres ahead too: 2,766; four blocks (128
// registers, spills): 3,130.
template <int P>
__global__ void __launch_bounds__(kRotThreads, rot_binomial<float, P>() ? 4 : 3)
    k_m2l_rot(int64_t n_nodes, const int32_t *__restrict__ off, const int32_t *__restrict__ src,
              const int32_t *__restrict__ rows, const float4 *__restrict__ tcenter, const float4 *__restrict__ thalf,
              const float4 *__restrict__ center, const float4 *__restrict__ half, const float4 *Mcols,
              float2 *__restrict__ Lexp, int nc_pad, const InstMask mask) {
    using T = float;
    using T2 = float2;
    constexpr int NV = (P + 1) * (P + 1), NQ = (P + 1) * (P + 2) / 2, NT = kRotThreads;
    extern __shared__ __align__(16) unsigned char rot_smem[];
    __shared__ int max_rounds;
    chain_next();
    T2 *sq = reinterpret_cast<T2 *>(rot_smem);
    AccC<NT> acc{sq + threadIdx.x};
    // warp w takes target row rows[w] (rows by decreasing pair count), or row w
    const int64_t w = ((int64_t)blockIdx.x * NT + threadIdx.x) >> 5;
    const int64_t t = rows && w < n_nodes ? (int64_t)rows[w] : w;
    const int lane = threadIdx.x & 31;
    const bool live = t < n_nodes && inst_active(mask, (int)t);
    float4 ct{};
    T iaL = T(1);
    int b = 0, e = 0;
    if (live) {
        ct = tcenter[t];
        iaL = T(1) / thalf[t].w;
        b = off[t];
        e = off[t + 1];
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) acc.set(q, T2{});
    if (threadIdx.x == 0) max_rounds = 0;
    __syncthreads();
    if (lane == 0) atomicMax(&max_rounds, (e - b + 31) >> 5);
    __syncthreads();
    const int rounds = max_rounds;
    chain_wait();
    int sn = b + lane < e ? __ldg(src + b + lane) : 0;  // the next round's source
    for (int r = 0; r < rounds; ++r) {
        __syncthreads();
        const int k = b + r * 32 + lane;
        if (k >= e) continue;
        const int s = sn;
        if (k + 32 < e) sn = __ldg(src + k + 32);
        const float4 cs = center[s];
        const T c = half[s].w * iaL;
        if (c > kRotExtremeRatio) continue;  // translated by k_m2l_generic
        RegV<T, NV> v;
        rot_pair<P>(v, acc, Mcols + col_of(s, nc_pad >> 1), c, (ct.x - cs.x) * iaL, (ct.y - cs.y) * iaL,
                    (ct.z - cs.z) * iaL);
    }
    if (!live) return;
    T2 *out = Lexp + t * nc_pad;
#pragma unroll
    for (int n = 0; n <= P; ++n) {
#pragma unroll
        for (int m = 0; m <= n; ++m) {
            const int q = tri(n, m);
            const T2 a = acc.get(q);
            T re = a.x, im = a.y;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                re += __shfl_xor_sync(0xffffffffu, re, o);
                im += __shfl_xor_sync(0xffffffffu, im, o);
            }
            if ((q & 31) == lane) {
                T2 r;
                r.x = re * iaL;
                r.y = im * iaL;
                out[q] = r;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Two-float M2L for FP64 plans.  The same rotation algorithm on the FP32 pipe
// in two-float arithmetic (about 48 significant bits; twofloat.cuh).  The
// source multipoles and the node geometry arrive already split into (hi, lo)
// FP32 pairs (split once per node, not once per pair: a pair-time split
// costs hundreds of FP64-pipe conversions), the pair geometry is formed in
// two-float, and the locals are written back as FP64.  Each lane's
// translated locals go back into its own coefficient slots (81 two-float
// values at p = 8), and after every round of 32 pairs the warp adds the
// slots of its lanes, lane i owning coefficients i, i + 32, i + 64 in
// registers; so a block needs 81 KB of shared memory and two blocks share an
// SM (the FP64 kernel's per-lane accumulators allow one).  Pairs whose source
// scale exceeds 256x the target's are left to the caller (FP32 exponent
// range), as in the FP32 kernel.
// ---------------------------------------------------------------------------
template <typename T, int P, int n, typename V>
__device__ __forceinline__ void backward_v(V &v, const Frame<T, P> &F) {
    constexpr int N = 2 * n + 1, OV = n * n, OFF = kRotOff[n];
    T b[N], o[N];
#pragma unroll
    for (int i = 0; i < N; ++i) b[i] = v.get(OV + i);
    rot_apply<T, 3, N, OFF, 0>(b, o);
    zrot<T, N, P>(o, F.ct, F.st, T(-1));
    rot_apply<T, 2, N, OFF, 0>(o, b);
    zrot<T, N, P>(b, F.cp, F.sp, T(-1));
#pragma unroll
    for (int i = 0; i < N; ++i) v.set(OV + i, b[i]);
    if constexpr (n < P) backward_v<T, P, n + 1>(v, F);
}

// --- the two-float matrices on packed FP32x2 instructions ---
// Two two-float values of the rows of one packed pair: (hi.x, lo.x) and
// (hi.y, lo.y).  Each operation is the scalar two-float one (twofloat.cuh)
// on both halves at once; negations are folded into the constants or taken
// as fma(b, -1, a) = a - b, which rounds exactly like the subtraction, so
// the results are bit-identical to the scalar two-float matrices.
struct tfp {
    float2 hi, lo;
};
__device__ __forceinline__ float2 f2_sub(float2 a, float2 b) {
    return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a);
}
// x * g + c, g = (ghi + glo) per half; ng = -ghi, nglo = -glo (EXACT: glo = 0)
template <bool EXACT>
__device__ __forceinline__ tfp tfp_fma_const(float2 g, float2 ng, float2 nglo, const tfp &x, const tfp &c) {
    const float2 p = __fmul2_rn(x.hi, g);
    float2 ne = __ffma2_rn(x.hi, ng, p);  // -(x.hi g - p), the product's rounding error negated
    ne = __ffma2_rn(x.lo, ng, ne);        // -(error + x.lo g)
    if constexpr (!EXACT) ne = __ffma2_rn(x.hi, nglo, ne);
    const float2 s = __fadd2_rn(p, c.hi);  // two-sum of p and c.hi
    const float2 bb = f2_sub(s, p);
    const float2 es = __fadd2_rn(f2_sub(p, f2_sub(s, bb)), f2_sub(c.hi, bb));
    const float2 t = __fadd2_rn(es, f2_sub(c.lo, ne));
    const float2 h = __fadd2_rn(s, t);  // fast two-sum
    return tfp{h, f2_sub(t, f2_sub(h, s))};
}
// x * g (the first term of a row: the fma above with c = 0)
template <bool EXACT>
__device__ __forceinline__ tfp tfp_mul_const(float2 g, float2 ng, float2 nglo, const tfp &x) {
    const float2 p = __fmul2_rn(x.hi, g);
    float2 ne = __ffma2_rn(x.hi, ng, p);
    ne = __ffma2_rn(x.lo, ng, ne);
    if constexpr (!EXACT) ne = __ffma2_rn(x.hi, nglo, ne);
    const float2 h = f2_sub(p, ne);
    return tfp{h, f2_sub(f2_sub(p, h), ne)};
}

// a c + b s on both halves (tf_cmul)
__device__ __forceinline__ tfp tfp_cmul(const tfp &a, const tfp &c, const tfp &b, const tfp &s) {
    const float2 m1 = make_float2(-1.0f, -1.0f);
    const float2 nah = __fmul2_rn(a.hi, m1), nbh = __fmul2_rn(b.hi, m1);
    const float2 p = __fmul2_rn(a.hi, c.hi), q = __fmul2_rn(b.hi, s.hi);
    const float2 np = __ffma2_rn(nah, c.hi, p), nq = __ffma2_rn(nbh, s.hi, q);  // rounding errors, negated
    float2 l = __fmul2_rn(a.hi, c.lo);
    l = __ffma2_rn(a.lo, c.hi, l);
    l = __ffma2_rn(b.hi, s.lo, l);
    l = __ffma2_rn(b.lo, s.hi, l);
    l = f2_sub(f2_sub(l, np), nq);
    const float2 t = __fadd2_rn(p, q), bb = f2_sub(t, p);  // two-sum
    const float2 e = __fadd2_rn(f2_sub(p, f2_sub(t, bb)), f2_sub(q, bb));
    l = __fadd2_rn(l, e);
    const float2 h = __fadd2_rn(t, l);
    return tfp{h, f2_sub(l, f2_sub(h, t))};
}
// a * g, g the same two-float value for both halves
__device__ __forceinline__ tfp tfp_mul_tf(const tfp &a, tf32x2 g) {
    const float2 gh = make_float2(g.hi, g.hi), ngh = make_float2(-g.hi, -g.hi), ngl = make_float2(-g.lo, -g.lo);
    const float2 p = __fmul2_rn(a.hi, gh);
    float2 ne = __ffma2_rn(a.hi, ngh, p);
    ne = __ffma2_rn(a.hi, ngl, ne);
    ne = __ffma2_rn(a.lo, ngh, ne);
    const float2 h = f2_sub(p, ne);
    return tfp{h, f2_sub(f2_sub(p, h), ne)};
}

template <int n> struct PkT {  // one degree block of two-float values in a packed layout
    tfp p[n > 0 ? n : 1];
    tf32x2 r;  // Re X_n
};
template <int n, int L, int J>
__device__ __forceinline__ tf32x2 pkt_get(const PkT<n> &v) {
    if constexpr (J == ix_re(n)) {
        return v.r;
    } else {
        constexpr bool re = J == 0 || (J & 1);
        constexpr int j = re ? (J + 1) >> 1 : J / 2 - 1;
        constexpr bool y = re == (L == 1 && ((j + n) & 1));
        if constexpr (y) return tf32x2(v.p[j].hi.y, v.p[j].lo.y);
        else return tf32x2(v.p[j].hi.x, v.p[j].lo.x);
    }
}
template <int n, int L, int J>
__device__ __forceinline__ void pkt_set(PkT<n> &v, tf32x2 a) {
    if constexpr (J == ix_re(n)) {
        v.r = a;
    } else {
        constexpr bool re = J == 0 || (J & 1);
        constexpr int j = re ? (J + 1) >> 1 : J / 2 - 1;
        constexpr bool y = re == (L == 1 && ((j + n) & 1));
        if constexpr (y) {
            v.p[j].hi.y = a.hi;
            v.p[j].lo.y = a.lo;
        } else {
            v.p[j].hi.x = a.hi;
            v.p[j].lo.x = a.lo;
        }
    }
}

__host__ __device__ constexpr float tf_hi(double g) { return (float)g; }
__host__ __device__ constexpr float tf_lo(double g) { return (float)(g - (double)(float)g); }

template <int TAB, int n, int LIN, int A, int B, int I>
__device__ __forceinline__ void pkt_rows(const PkT<n> &x, tfp &acc) {
    if constexpr (I < n) {
        constexpr int C = pk_ix<n, LIN>(I, 0), D = pk_ix<n, LIN>(I, 1);
        constexpr double ga = pk_g<TAB, n>(A, C), gb = pk_g<TAB, n>(B, D);
        static_assert(pk_g<TAB, n>(A, D) == 0.0 && pk_g<TAB, n>(B, C) == 0.0,
                      "packed rotation layouts must leave no cross terms");
        if constexpr (ga != 0.0 || gb != 0.0) {
            constexpr bool exact = tf_lo(ga) == 0.0f && tf_lo(gb) == 0.0f;
            const float2 g = make_float2(tf_hi(ga), tf_hi(gb)), ng = make_float2(-tf_hi(ga), -tf_hi(gb));
            const float2 nglo = make_float2(-tf_lo(ga), -tf_lo(gb));
            if constexpr (pk_started<TAB, n, LIN, A, B>(I)) acc = tfp_fma_const<exact>(g, ng, nglo, x.p[I], acc);
            else acc = tfp_mul_const<exact>(g, ng, nglo, x.p[I]);
        }
        pkt_rows<TAB, n, LIN, A, B, I + 1>(x, acc);
    }
}

template <int TAB, int n, int LIN, int I, bool STARTED>
__device__ __forceinline__ void pkt_left_row(const PkT<n> &x, tf32x2 &acc) {
    constexpr int L = ix_re(n);
    if constexpr (I < n) {
        constexpr double ga = pk_g<TAB, n>(L, pk_ix<n, LIN>(I, 0));
        constexpr double gb = pk_g<TAB, n>(L, pk_ix<n, LIN>(I, 1));
        static_assert(ga == 0.0 || gb == 0.0, "one input class per row");
        if constexpr (ga != 0.0) {
            const tf32x2 v(x.p[I].hi.x, x.p[I].lo.x);
            acc = tf_fma_const<tf_lo(ga) == 0.0f>(tf_hi(ga), tf_lo(ga), v, STARTED ? acc : tf32x2(0.0f, 0.0f));
        }
        if constexpr (gb != 0.0) {
            const tf32x2 v(x.p[I].hi.y, x.p[I].lo.y);
            acc = tf_fma_const<tf_lo(gb) == 0.0f>(tf_hi(gb), tf_lo(gb), v, STARTED ? acc : tf32x2(0.0f, 0.0f));
        }
        pkt_left_row<TAB, n, LIN, I + 1, STARTED || ga != 0.0 || gb != 0.0>(x, acc);
    } else {
        constexpr double g = pk_g<TAB, n>(L, L);
        if constexpr (g != 0.0)
            acc = tf_fma_const<tf_lo(g) == 0.0f>(tf_hi(g), tf_lo(g), x.r, STARTED ? acc : tf32x2(0.0f, 0.0f));
        else if constexpr (!STARTED)
            acc = tf32x2(0.0f, 0.0f);
    }
}

template <int TAB, int n, int LIN, int LOUT, int J>
__device__ __forceinline__ void pkt_out_pairs(const PkT<n> &x, PkT<n> &y) {
    if constexpr (J < n) {
        constexpr int A = pk_ix<n, LOUT>(J, 0), B = pk_ix<n, LOUT>(J, 1), L = ix_re(n);
        constexpr double la = pk_g<TAB, n>(A, L), lb = pk_g<TAB, n>(B, L);
        tfp acc{make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
        if constexpr (pk_started<TAB, n, LIN, A, B>(n)) pkt_rows<TAB, n, LIN, A, B, 0>(x, acc);
        if constexpr (la != 0.0) {
            const tf32x2 r = tf_fma_const<tf_lo(la) == 0.0f>(tf_hi(la), tf_lo(la), x.r, tf32x2(acc.hi.x, acc.lo.x));
            acc.hi.x = r.hi;
            acc.lo.x = r.lo;
        }
        if constexpr (lb != 0.0) {
            const tf32x2 r = tf_fma_const<tf_lo(lb) == 0.0f>(tf_hi(lb), tf_lo(lb), x.r, tf32x2(acc.hi.y, acc.lo.y));
            acc.hi.y = r.hi;
            acc.lo.y = r.lo;
        }
        y.p[J] = acc;
        pkt_out_pairs<TAB, n, LIN, LOUT, J + 1>(x, y);
    }
}

template <int TAB, int n, int LIN, int LOUT>
__device__ __forceinline__ void pkt_apply(const PkT<n> &x, PkT<n> &y) {
    pkt_out_pairs<TAB, n, LIN, LOUT, 0>(x, y);
    pkt_left_row<TAB, n, LIN, 0, false>(x, y.r);
}

// X_m <- X_m e^{+-i m a} in two-float, x in layout LA, y in layout LB: pair j
// (Re X_j, Im X_{j+1}) at once, from (Re X_j, Im X_{j+1}) and (Im X_j, Re X_{j+1})
__device__ __forceinline__ tfp tfp_pair(tf32x2 a, tf32x2 b) {
    return tfp{make_float2(a.hi, b.hi), make_float2(a.lo, b.lo)};
}
template <int n, int LA, int LB, int P, int j>
__device__ __forceinline__ void pkt_zrot(const PkT<n> &x, PkT<n> &y, const tf32x2 (&c)[P + 1],
                                         const tf32x2 (&s)[P + 1], bool neg) {
    if constexpr (n == 0) {
        y.r = x.r;
    } else if constexpr (j < n) {
        const tf32x2 re0 = pkt_get<n, LA, ix_re(j)>(x), im1 = pkt_get<n, LA, 2 * (j + 1)>(x),
                     re1 = pkt_get<n, LA, ix_re(j + 1)>(x);
        const tf32x2 s1 = neg ? -s[j + 1] : s[j + 1];
        if constexpr (j == 0) {  // X_0 does not turn
            pkt_set<n, LB, 0>(y, re0);
            pkt_set<n, LB, 2>(y, tf_cmul(im1, c[1], re1, s1));
        } else {
            const tf32x2 im0 = pkt_get<n, LA, 2 * j>(x), s0 = neg ? s[j] : -s[j];
            const tfp o = tfp_cmul(tfp_pair(re0, im1), tfp_pair(c[j], c[j + 1]), tfp_pair(im0, re1), tfp_pair(s0, s1));
            pkt_set<n, LB, ix_re(j)>(y, tf32x2(o.hi.x, o.lo.x));
            pkt_set<n, LB, 2 * (j + 1)>(y, tf32x2(o.hi.y, o.lo.y));
        }
        pkt_zrot<n, LA, LB, P, j + 1>(x, y, c, s, neg);
    } else {
        const tf32x2 re = pkt_get<n, LA, ix_re(n)>(x), im = pkt_get<n, LA, 2 * n>(x);
        pkt_set<n, LB, ix_re(n)>(y, tf_cmul(re, c[n], im, neg ? s[n] : -s[n]));
    }
}

// all 2n + 1 values of a packed block to / from the slots of v (block index order)
template <int n, int L, int J, typename V>
__device__ __forceinline__ void pkt_store(V &v, const PkT<n> &x) {
    v.set(n * n + J, pkt_get<n, L, J>(x));
    if constexpr (J < 2 * n) pkt_store<n, L, J + 1>(v, x);
}
template <int n, int L, int J, typename V>
__device__ __forceinline__ void pkt_load(const V &v, PkT<n> &x) {
    pkt_set<n, L, J>(x, v.get(n * n + J));
    if constexpr (J < 2 * n) pkt_load<n, L, J + 1>(v, x);
}

// forward of degree n on the slots of v: scale by fn = c^n n! / rho^n,
// R_z(+phi), Q_p, R_z(+theta), Q_m
template <int P, int n, typename V>
__device__ __forceinline__ void forward_tf_pk(V &v, tf32x2 cr, tf32x2 fn, const Frame<tf32x2, P> &F) {
    PkT<n> a, b;
    pkt_load<n, 0, 0>(v, b);
#pragma unroll
    for (int j = 0; j < n; ++j) b.p[j] = tfp_mul_tf(b.p[j], fn);
    b.r = b.r * fn;
    pkt_zrot<n, 0, 1, P, 0>(b, a, F.cp, F.sp, false);
    pkt_apply<0, n, 1, 0>(a, b);
    pkt_zrot<n, 0, 1, P, 0>(b, a, F.ct, F.st, false);
    pkt_apply<1, n, 1, 0>(a, b);
    pkt_store<n, 0, 0>(v, b);
    if constexpr (n < P) forward_tf_pk<P, n + 1>(v, cr, fn * cr * tf32x2(n + 1), F);
}

// backward of degree n on the slots of v (transposes in reverse order)
template <int P, int n, typename V>
__device__ __forceinline__ void backward_tf_pk(V &v, const Frame<tf32x2, P> &F) {
    PkT<n> a, b;
    pkt_load<n, 0, 0>(v, a);
    pkt_apply<3, n, 0, 1>(a, b);
    pkt_zrot<n, 1, 0, P, 0>(b, a, F.ct, F.st, true);
    pkt_apply<2, n, 0, 1>(a, b);
    pkt_zrot<n, 1, 0, P, 0>(b, a, F.cp, F.sp, true);
    pkt_store<n, 0, 0>(v, a);
    if constexpr (n < P) backward_tf_pk<P, n + 1>(v, F);
}

// axial<tf32x2, P, m, true> with the real and imaginary parts of order m >= 1
// in the halves of packed operations
template <int P, int N, int K, int m>
__device__ __forceinline__ void pkt_binom(const tfp (&u)[P + 1], tfp &s) {
    constexpr float cb = (float)binom(N + K, K);
    const float2 g = make_float2(cb, cb), ng = make_float2(-cb, -cb), zero = make_float2(0.0f, 0.0f);
    if constexpr (K == m) s = tfp_mul_const<true>(g, ng, zero, u[K]);
    else s = tfp_fma_const<true>(g, ng, zero, u[K], s);
    if constexpr (K < P) pkt_binom<P, N, K + 1, m>(u, s);
}
template <int P, int m, int N, typename V>
__device__ __forceinline__ void axial_tf_rows(V &v, const tfp (&u)[P + 1], const tf32x2 (&h)[P + 1]) {
    tfp s;
    pkt_binom<P, N, m, m>(u, s);
    s = tfp_mul_tf(s, h[N]);
    const tf32x2 re(s.hi.x, s.lo.x), im(s.hi.y, s.lo.y);
    v.set(N * N + 2 * m - 1, ((N + m) & 1) ? -re : re);
    v.set(N * N + 2 * m, ((N + m) & 1) ? -im : im);
    if constexpr (N < P) axial_tf_rows<P, m, N + 1>(v, u, h);
}
template <int P, int m, typename V> __device__ __forceinline__ void axial_tf_pk(V &v, const tf32x2 (&h)[P + 1]) {
    if constexpr (m == 0) {
        tf32x2 ur[P + 1], ui[P + 1], wr[P + 1], wi[P + 1];
#pragma unroll
        for (int k = 0; k <= P; ++k) {
            ur[k] = v.get(k * k);
            ui[k] = tf32x2(0);
        }
        binom_rows<tf32x2, P, 0, 0, true>(ur, ui, wr, wi, h);
#pragma unroll
        for (int k = 0; k <= P; ++k) v.set(k * k, wr[k]);
    } else {
        tfp u[P + 1];
#pragma unroll
        for (int k = m; k <= P; ++k) u[k] = tfp_pair(v.get(k * k + 2 * m - 1), v.get(k * k + 2 * m));
        axial_tf_rows<P, m, m>(v, u, h);
    }
    if constexpr (m < P) axial_tf_pk<P, m + 1>(v, h);
}

// two-float slots split into a hi and a lo array (slot i of this thread at
// [i * STRIDE]), so that single values load straight into packed pairs
template <int STRIDE> struct SmemSplit {
    float *hi, *lo;
    __device__ __forceinline__ tf32x2 get(int i) const {
        return tf32x2(lds_keep(hi + i * STRIDE), lds_keep(lo + i * STRIDE));
    }
    __device__ __forceinline__ void set(int i, tf32x2 x) {
        sts_keep(hi + i * STRIDE, x.hi);
        sts_keep(lo + i * STRIDE, x.lo);
    }
};

// One pair: v <- the translated locals (real block basis) of the source with
// column Mcol (split multipoles: (re hi, re lo, im hi, im lo) per coefficient).
template <int P, bool PK, typename V>
__device__ __forceinline__ void rot_pair_tf(V &v, const float4 *Mcol, tf32x2 c, tf32x2 dx, tf32x2 dy,
                                            tf32x2 dz) {
    using T = tf32x2;
#pragma unroll
    for (int n = 0; n <= P; ++n) {
#pragma unroll
        for (int m = 0; m <= n; ++m) {
            const float4 x = Mcol[tri(n, m) * kColNodes];
            if (m == 0) {
                v.set(n * n, T(x.x, x.y));
            } else {
                v.set(n * n + 2 * m - 1, T(x.x, x.y));
                v.set(n * n + 2 * m, T(x.z, x.w));
            }
        }
    }
    const T s2 = fma(dy, dy, dx * dx), r2 = fma(dz, dz, s2);
    const T s = sqrt(s2), rho = sqrt(r2), irho = tf_recip(rho);
    Frame<T, P> F;
    T cphi = T(1), sphi = T(0);
    if (s2.hi > 0.0f) {
        const T is = tf_recip(s);
        cphi = dx * is;
        sphi = dy * is;
    }
    powers<T, P>(cphi, sphi, F.cp, F.sp);
    powers<T, P>(dz * irho, s * irho, F.ct, F.st);
    const T cr = c * irho;
    if constexpr (PK) forward_tf_pk<P, 0>(v, cr, T(1), F);
    else forward<T, P, true, 0>(v, cr, T(1), F);
    T h[P + 1];
    h[0] = irho;
#pragma unroll
    for (int j = 1; j <= P; ++j) h[j] = h[j - 1] * T(j) * irho;
    if constexpr (PK) axial_tf_pk<P, 0>(v, h);
    else axial<T, P, 0, true>(v, h);
    if constexpr (PK) backward_tf_pk<P, 0>(v, F);
    else backward_v<T, P, 0>(v, F);
}

// tnodes / snodes: per node (cx hi, cx lo, cy hi, cy lo), (cz hi, cz lo, a hi, a lo).
// NT = 128 (two blocks per SM) or 256 (one block of 8 warps per SM: one
// instruction-fetch stream per SM for the long pair code).  PK: the four
// matrices on packed FP32x2 instructions, with the slots split into hi and
// lo arrays (the same shared memory).
template <int P, int NT, bool PK>
__global__ void __launch_bounds__(NT, 256 / NT)
    k_m2l_rot_tf(int64_t n_nodes, const int32_t *__restrict__ off, const int32_t *__restrict__ src,
                 const int32_t *__restrict__ rows,
                 const float4 *__restrict__ tnodes, const double4 *__restrict__ thalf,
                 const float4 *__restrict__ snodes, const double4 *__restrict__ half,
                 const float4 *Mcols, double2 *__restrict__ Lexp, int nc_pad, const InstMask mask) {
    using T = tf32x2;
    constexpr int NV = (P + 1) * (P + 1), NR = (NV + 31) / 32;
    extern __shared__ __align__(16) unsigned char rot_smem[];
    __shared__ int max_rounds;
    chain_next();
    T *slots = reinterpret_cast<T *>(rot_smem);  // slot i of thread u at slots[i * NT + u]
    float *slots_hi = reinterpret_cast<float *>(rot_smem), *slots_lo = slots_hi + NV * NT;  // PK
    using VS = typename std::conditional<PK, SmemSplit<NT>, SmemV<T, NT>>::type;
    VS v;
    if constexpr (PK) v = VS{slots_hi + threadIdx.x, slots_lo + threadIdx.x};
    else v = VS{slots + threadIdx.x};
    // warp w takes target row rows[w] (rows by decreasing pair count), or row w
    const int64_t w = ((int64_t)blockIdx.x * NT + threadIdx.x) >> 5;
    const int64_t t = rows && w < n_nodes ? (int64_t)rows[w] : w;
    const int lane = threadIdx.x & 31;
    const int wbase = threadIdx.x & ~31;
    const bool live = t < n_nodes && inst_active(mask, (int)t);
    T ctx = T(0), cty = T(0), ctz = T(0), iaT = T(1);
    double iaL = 1.0;  // FP64, for the extreme-pair test (the same test as the pair lists of the FP64 kernel)
    int b = 0, e = 0;
    if (live) {
        const float4 u = tnodes[2 * t], w = tnodes[2 * t + 1];
        ctx = T(u.x, u.y);
        cty = T(u.z, u.w);
        ctz = T(w.x, w.y);
        iaT = tf_recip(T(w.z, w.w));
        iaL = 1.0 / thalf[t].w;
        b = off[t];
        e = off[t + 1];
    }
    T acc[NR];
#pragma unroll
    for (int j = 0; j < NR; ++j) acc[j] = T(0);
    if (threadIdx.x == 0) max_rounds = 0;
    __syncthreads();
    if (lane == 0) atomicMax(&max_rounds, (e - b + 31) >> 5);
    __syncthreads();
    const int rounds = max_rounds;
    chain_wait();
    for (int r = 0; r < rounds; ++r) {
        // the block's warps walk the (long, straight-line) pair code together
        // and share its instruction fetches; every thread runs `rounds` rounds
        __syncthreads();
        const int k = b + r * 32 + lane;
        bool have = false;
        if (k < e) {
            const int s = __ldg(src + k);
            if (!(half[s].w * iaL > (double)kRotExtremeRatio)) {
                have = true;
                const float4 u = snodes[2 * s], w = snodes[2 * s + 1];
                rot_pair_tf<P, PK>(v, Mcols + col_of(s, nc_pad), T(w.z, w.w) * iaT, (ctx - T(u.x, u.y)) * iaT,
                                   (cty - T(u.z, u.w)) * iaT, (ctz - T(w.x, w.y)) * iaT);
            }
        }
        if (!have) {
#pragma unroll
            for (int i = 0; i < NV; ++i) v.set(i, T(0));
        }
        __syncwarp();
        // coefficient i = lane + 32 j summed over the warp's lanes, starting at
        // this lane (conflict-free shared-memory reads; a fixed order per i)
#pragma unroll
        for (int j = 0; j < NR; ++j) {
            const int i = lane + 32 * j;
            if (i < NV) {
                T sum = acc[j];
                if constexpr (PK) {
                    const float *rh = slots_hi + i * NT + wbase, *rl = slots_lo + i * NT + wbase;
#pragma unroll 8
                    for (int l = 0; l < 32; ++l) {
                        const int o = (l + lane) & 31;
                        sum = sum + T(lds_keep(rh + o), lds_keep(rl + o));
                    }
                } else {
                    const T *row = slots + i * NT + wbase;
#pragma unroll 8
                    for (int l = 0; l < 32; ++l) sum = sum + lds_keep(row + ((l + lane) & 31));
                }
                acc[j] = sum;
            }
        }
        __syncwarp();
    }
    if (!live) return;
    double *out = reinterpret_cast<double *>(Lexp + t * nc_pad);
#pragma unroll
    for (int j = 0; j < NR; ++j) {
        const int i = lane + 32 * j;
        if (i < NV) {
            int n = 0;
            while ((n + 1) * (n + 1) <= i) ++n;
            const int q = i - n * n;  // 0: Re X0; 2m - 1: Re Xm; 2m: Im Xm
            const double val = tf_to_double(acc[j] * iaT);
            if (q == 0) {
                out[2 * tri(n, 0)] = val;
                out[2 * tri(n, 0) + 1] = 0.0;
            } else {
                out[2 * tri(n, (q + 1) >> 1) + ((q & 1) ? 0 : 1)] = val;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// FP64 M2L.  The pair's coefficients stay in its lane's shared-memory slots,
// read with loads the compiler may not hoist (81 doubles and the phases do
// not fit in registers), and after each round of 32 pairs the warp adds the
// slots of its lanes, lane i owning coefficients i, i + 32, i + 64.  The FP64
// pipe (64 cycles per warp operation) is the bound, so what counts is that
// every scheduler always has a warp to serve, and to the end: two blocks fit
// an SM, and the four warps of a block take the rounds of one row in turn.
// With the translated locals accumulated per lane one block filled an SM and
// its pipe idled through every shared-memory latency; with a row per warp, long
// rows that shared a scheduler ended long after the others.  180k pairs on a
// sphere of 20,011 points: 1,174 (accumulators per lane), 1,345 (a row per
// warp, ten warps per SM), 987 us (four warps a row; 590 us at the pipe's full rate).
// ---------------------------------------------------------------------------
template <int P>
__global__ void __launch_bounds__(kRotThreads, 2)
    k_m2l_rot_f64(int64_t n_nodes, const int32_t *__restrict__ off, const int32_t *__restrict__ src,
                  const int32_t *__restrict__ rows, const double4 *__restrict__ tcenter,
                  const double4 *__restrict__ thalf, const double4 *__restrict__ center,
                  const double4 *__restrict__ half, const double2 *Mexp, double2 *__restrict__ Lexp,
                  int nc_pad, const InstMask mask) {
    constexpr int NV = (P + 1) * (P + 1), NR = (NV + 31) / 32, NT = kRotThreads, NW = NT / 32;
    extern __shared__ __align__(16) unsigned char rot_smem[];
    double *slots = reinterpret_cast<double *>(rot_smem);  // slot i of thread u at slots[i * NT + u]
    chain_next();
    chain_wait();
    const int64_t t = rows ? (int64_t)rows[blockIdx.x] : (int64_t)blockIdx.x;
    if (t >= n_nodes || !inst_active(mask, (int)t)) return;
    const int lane = threadIdx.x & 31, wbase = threadIdx.x & ~31;
    SmemV<double, NT> v{slots + threadIdx.x};
    const double4 ct = tcenter[t];
    const double iaL = 1.0 / thalf[t].w;
    const int b = off[t], e = off[t + 1];
    double acc[NR];
#pragma unroll
    for (int j = 0; j < NR; ++j) acc[j] = 0.0;
    for (int k0 = b + wbase; k0 < e; k0 += NT) {
        const int k = k0 + lane;
        if (k < e) {
            const int s = __ldg(src + k);
            const double4 cs = center[s];
            const double2 *Mrow = Mexp + (int64_t)s * nc_pad;
#pragma unroll
            for (int n = 0; n <= P; ++n) {
#pragma unroll
                for (int m = 0; m <= n; ++m) {
                    const double2 x = Mrow[tri(n, m)];
                    if (m == 0) {
                        v.set(n * n, x.x);
                    } else {
                        v.set(n * n + 2 * m - 1, x.x);
                        v.set(n * n + 2 * m, x.y);
                    }
                }
            }
            const double dx = (ct.x - cs.x) * iaL, dy = (ct.y - cs.y) * iaL, dz = (ct.z - cs.z) * iaL;
            const double s2 = dx * dx + dy * dy, r2 = s2 + dz * dz;
            const double irho = rsqrt(r2);
            Frame<double, P> F;
            double cphi = 1.0, sphi = 0.0, s1 = 0.0;
            if (s2 > 0.0) {
                const double is = rsqrt(s2);
                s1 = s2 * is;
                cphi = dx * is;
                sphi = dy * is;
            }
            powers<double, P>(cphi, sphi, F.cp, F.sp);
            powers<double, P>(dz * irho, s1 * irho, F.ct, F.st);
            forward<double, P, true, 0>(v, half[s].w * iaL * irho, 1.0, F);
            double h[P + 1];
            h[0] = irho;
#pragma unroll
            for (int j = 1; j <= P; ++j) h[j] = h[j - 1] * (double)j * irho;
            axial<double, P, 0, true>(v, h);
            backward_v<double, P, 0>(v, F);
        } else {
#pragma unroll
            for (int i = 0; i < NV; ++i) v.set(i, 0.0);
        }
        __syncwarp();
        // starting at this lane: conflict-free shared-memory reads, a fixed order per coefficient
#pragma unroll
        for (int j = 0; j < NR; ++j) {
            const int i = lane + 32 * j;
            if (i < NV) {
                const double *row = slots + i * NT + wbase;
                double sum = acc[j];
#pragma unroll 8
                for (int l = 0; l < 32; ++l) sum += lds_keep(row + ((l + lane) & 31));
                acc[j] = sum;
            }
        }
        __syncwarp();
    }
    // the warps' sums, in warp order
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NR; ++j)
        if (lane + 32 * j < NV) slots[(wbase >> 5) * NV + lane + 32 * j] = acc[j];
    __syncthreads();
    double *out = reinterpret_cast<double *>(Lexp + t * nc_pad);
    for (int i = threadIdx.x; i < NV; i += NT) {
        double val = slots[i];
#pragma unroll
        for (int q = 1; q < NW; ++q) val += slots[q * NV + i];
        val *= iaL;
        int n = 0;
        while ((n + 1) * (n + 1) <= i) ++n;
        const int q = i - n * n;  // 0: Re X0; 2m - 1: Re Xm; 2m: Im Xm
        if (q == 0) {
            out[2 * tri(n, 0)] = val;
            out[2 * tri(n, 0) + 1] = 0.0;
        } else {
            out[2 * tri(n, (q + 1) >> 1) + ((q & 1) ? 0 : 1)] = val;
        }
    }
}

inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

template <int P, int NT, bool PK>
int launch_rot_tf(int64_t M, const int32_t *off, const int32_t *src, const int32_t *rows, const void *tnodes,
                  const void *thal,
                  const void *snodes, const void *hal, const void *Mx, void *Lx, int nc_pad, const InstMask &mask,
                  cudaStream_t s) {
    constexpr int NV = (P + 1) * (P + 1);
    constexpr size_t smem = (size_t)NV * NT * sizeof(tf32x2);
    static DeviceOnce once;
    EDFMM_CUDA_TRY(allow_smem(once, k_m2l_rot_tf<P, NT, PK>, smem));
    EDFMM_CUDA_TRY(chain_launch(chain_tree(M, EDFMM_F64, s), k_m2l_rot_tf<P, NT, PK>, nblk(M * 32, NT), NT, smem, s, M, off, src,
                                rows, static_cast<const float4 *>(tnodes), static_cast<const double4 *>(thal),
                                static_cast<const float4 *>(snodes), static_cast<const double4 *>(hal),
                                static_cast<const float4 *>(Mx), static_cast<double2 *>(Lx), nc_pad, mask));
    EDFMM_LAUNCH_CHECK("k_m2l_rot_tf");
    return EDFMM_OK;
}

template <int P>
int launch_rot_f64(int64_t M, const int32_t *off, const int32_t *src, const int32_t *rows, const void *tcen,
                   const void *thal, const void *cen, const void *hal, const void *Mx, void *Lx, int nc_pad,
                   const InstMask &mask, cudaStream_t s) {
    constexpr size_t smem = (size_t)(P + 1) * (P + 1) * kRotThreads * sizeof(double);
    static DeviceOnce once;
    EDFMM_CUDA_TRY(allow_smem(once, k_m2l_rot_f64<P>, smem));
    EDFMM_CUDA_TRY(chain_launch(chain_tree(M, EDFMM_F64, s), k_m2l_rot_f64<P>, (unsigned)M, kRotThreads, smem, s, M, off, src, rows,
                                static_cast<const double4 *>(tcen), static_cast<const double4 *>(thal),
                                static_cast<const double4 *>(cen), static_cast<const double4 *>(hal),
                                static_cast<const double2 *>(Mx), static_cast<double2 *>(Lx), nc_pad, mask));
    EDFMM_LAUNCH_CHECK("k_m2l_rot_f64");
    return EDFMM_OK;
}

template <int P>
int launch_rot(int64_t M, const int32_t *off, const int32_t *src, const int32_t *rows, const void *tcen,
               const void *thal, const void *cen, const void *hal, const void *Mx, void *Lx, int nc_pad,
               const InstMask &mask, cudaStream_t s) {
    constexpr int NQ = (P + 1) * (P + 2) / 2, NT = kRotThreads;
    constexpr size_t smem = (size_t)NQ * NT * sizeof(float2);
    static DeviceOnce once;
    EDFMM_CUDA_TRY(allow_smem(once, k_m2l_rot<P>, smem));
    EDFMM_CUDA_TRY(chain_launch(chain_tree(M, EDFMM_F32, s), k_m2l_rot<P>, nblk(M * 32, NT), NT, smem, s, M, off, src, rows,
                                static_cast<const float4 *>(tcen), static_cast<const float4 *>(thal),
                                static_cast<const float4 *>(cen), static_cast<const float4 *>(hal),
                                static_cast<const float4 *>(Mx), static_cast<float2 *>(Lx), nc_pad, mask));
    EDFMM_LAUNCH_CHECK("k_m2l_rot");
    return EDFMM_OK;
}

}  // namespace

// Entry points of the translation units that instantiate the kernels (they
// compile in parallel): FP32 and FP64 orders 1..8 (m2l_rot_f32.cu,
// m2l_rot_f64.cu; a..d = target centres, target halves, source centres,
// source halves) and two-float orders 6, 7 and 8 with 128 or 256 threads
// (m2l_rot_tf*.cu; a..d = target nodes, target halves, source nodes, source
// halves).
int m2l_rot_f32(int p, int64_t M, const int32_t *off, const int32_t *src, const int32_t *rows, const void *a, const void *b,
                const void *c, const void *d, const void *Mx, void *Lx, int nc_pad, const InstMask &mask,
                cudaStream_t s);
int m2l_rot_f64(int p, int64_t M, const int32_t *off, const int32_t *src, const int32_t *rows, const void *a, const void *b,
                const void *c, const void *d, const void *Mx, void *Lx, int nc_pad, const InstMask &mask,
                cudaStream_t s);
int m2l_rot_tf6(bool packed, int64_t M, const int32_t *off, const int32_t *src, const int32_t *rows, const void *a, const void *b,
                const void *c, const void *d, const void *Mx, void *Lx, int nc_pad, const InstMask &mask,
                cudaStream_t s);
int m2l_rot_tf7(bool packed, int64_t M, const int32_t *off, const int32_t *src, const int32_t *rows, const void *a, const void *b,
                const void *c, const void *d, const void *Mx, void *Lx, int nc_pad, const InstMask &mask,
                cudaStream_t s);
int m2l_rot_tf8(bool packed, int64_t M, const int32_t *off, const int32_t *src, const int32_t *rows, const void *a, const void *b,
                const void *c, const void *d, const void *Mx, void *Lx, int nc_pad, const InstMask &mask,
                cudaStream_t s);
int m2l_rot_tf8w(bool packed, int64_t M, const int32_t *off, const int32_t *src, const int32_t *rows, const void *a, const void *b,
                const void *c, const void *d, const void *Mx, void *Lx, int nc_pad, const InstMask &mask,
                cudaStream_t s);

}  // namespace edfmm
