// Far-field stages of the FMM: P2M, M2M, M2L, L2L.
//
// Coefficients are stored per node as (p+1)(p+2)/2 complex numbers (m >= 0),
// scaled by the node's expansion radius a (the tight-box radius, but at least
// 1/8 of the parent's a and 2^-40 of the root radius):
//   Mhat_n^m = M_n^m / a^n,  Lhat_n^m = L_n^m a^n.
// This keeps every coefficient O(1) in FP32 at any tree depth.
//
// M2L (the dominant stage) runs in the rotation form of m2l_rot.cuh for orders up
// to 8, in FP32, FP64 or two-float arithmetic; FP32 and two-float read the
// multipoles by columns (k_mult_columns).  With this scaling
//   Lhat_n^m = (-1)^(n+m) / a_L  sum_pairs sum_{k,l} Mhat_k^l (a_M/a_L)^k I_{n+k}^{l-m}(v),
// v = (c_L - c_M) / a_L, which is exact algebra; pairs whose source scale exceeds
// 256x the target's (only in strongly adaptive trees) would overflow (a_M/a_L)^k
// in FP32 and are instead translated by a shared-memory kernel using
//   Lhat_n^m = (-1)^(n+m) / a_L  (a_L/a_M)^(n+1) sum_{k,l} Mhat_k^l I_{n+k}^{l-m}((c_L - c_M)/a_M).
// FP64 has the range for any ratio; orders above 8 use the shared-memory kernel.
#include <algorithm>

#include "edfmm_internal.cuh"
#include "harmonics.cuh"
#include "twofloat.cuh"

namespace edfmm {

namespace {

constexpr float kExtremeRatio = 256.0f;
constexpr int kRotPMaxUsed = 8;  // rotation-based M2L (m2l_rot.cuh) for p <= 8

inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

__device__ __forceinline__ void coef_nm(int c, int &n, int &m) {
    n = 0;
    while ((n + 1) * (n + 2) / 2 <= c) ++n;
    m = c - n * (n + 1) / 2;
}

// ---------------------------------------------------------------------------
// charges
// ---------------------------------------------------------------------------
// grid: the split points of an FP64 tree (three float4 per point, the charge in
// the last two words, as a double or (tf) as two floats), or NULL; a == NULL
// keeps the charges that are set
template <typename T>
__global__ void k_set_charges(typename Vec4<T>::type *pts, float4 *grid, int tf, const int32_t *__restrict__ idx,
                              int64_t n, const T *__restrict__ a, const T *__restrict__ b) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    T q;
    if (a) {
        const int o = idx[i];
        q = b ? a[o] * b[o] : a[o];
        pts[i].w = q;
    } else {
        q = pts[i].w;
    }
    if constexpr (sizeof(T) == 8) {
        if (grid) {
            float2 w = make_float2(__int_as_float(__double2loint(q)), __int_as_float(__double2hiint(q)));
            if (tf) {
                const tf32x2 t = tf_from_double(q);
                w = make_float2(t.hi, t.lo);
            }
            *reinterpret_cast<float2 *>(&grid[3 * i + 2].z) = w;
        }
    }
}

// two-float mode: node geometry (cx, cy, cz, a) and FP64 complex
// coefficients split into (hi, lo) FP32 pairs
__global__ void k_split_nodes(const double4 *__restrict__ center, const double4 *__restrict__ half, int64_t n,
                              float4 *__restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double4 c = center[i];
    const tf32x2 x = tf_from_double(c.x), y = tf_from_double(c.y), z = tf_from_double(c.z),
                 a = tf_from_double(half[i].w);
    out[2 * i] = make_float4(x.hi, x.lo, y.hi, y.lo);
    out[2 * i + 1] = make_float4(z.hi, z.lo, a.hi, a.lo);
}
// Multipoles into the column layout that the M2L kernels read (m2l_rot.cuh):
// 16-byte words of 32 nodes' rows through shared memory, coalesced on both
// sides.  FP32: a word is two coefficients; SPLIT: an FP64 coefficient becomes
// (re hi, re lo, im hi, im lo).
template <bool SPLIT>
__global__ void __launch_bounds__(256) k_mult_columns(const float4 *in, int64_t n_nodes, int words, float4 *out) {
    extern __shared__ float4 col_tile[];  // [32][words + 1]
    chain_next();
    chain_wait();
    const int64_t n0 = (int64_t)blockIdx.x * kColNodes;
    const int nodes = (int)min((int64_t)kColNodes, n_nodes - n0);
    for (int k = threadIdx.x; k < nodes * words; k += blockDim.x) {
        float4 x = in[n0 * words + k];
        if constexpr (SPLIT) {
            const double2 c = *reinterpret_cast<const double2 *>(&x);
            const tf32x2 re = tf_from_double(c.x), im = tf_from_double(c.y);
            x = make_float4(re.hi, re.lo, im.hi, im.lo);
        }
        col_tile[(k / words) * (words + 1) + k % words] = x;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < words * kColNodes; k += blockDim.x) {
        const int s = k % kColNodes, w = k / kColNodes;
        if (s < nodes) out[n0 * words + k] = col_tile[s * (words + 1) + w];
    }
}
template <bool SPLIT>
int mult_columns(const FmmBuffers &buf, int64_t n_nodes, const DevBuf &out, bool chained, cudaStream_t s) {
    const int words = SPLIT ? buf.nc_pad : buf.nc_pad / 2;
    const size_t smem = sizeof(float4) * kColNodes * (size_t)(words + 1);
    EDFMM_CUDA_TRY(chain_launch(chained, k_mult_columns<SPLIT>, nblk(n_nodes, kColNodes), 256, smem, s,
                                dptr<float4>(buf.multipoles), n_nodes, words, dptr<float4>(out)));
    EDFMM_LAUNCH_CHECK("k_mult_columns");
    return EDFMM_OK;
}

// ---------------------------------------------------------------------------
// P2M: warp per leaf, lanes over points.  A lane's terms q R_n^m go straight to
// shared memory (row v = 2 tri(n, m) + part, one column per lane), and one
// lane per row adds the columns that hold points: at p = 8 and 20 points 90
// stores and 60 adds per lane, where a shuffle tree over register arrays
// takes 450 shuffles and 450 adds (and FP64 arrays of 180 values spill; an
// FP64 add takes 64 issue cycles).  Beside the near field, FP64, 2,468 leaves
// of 20 points: 282 -> 209 us; FP32, 9,856 leaves of 20 points (order 6): 39 ->
// 22 us.
// ---------------------------------------------------------------------------
template <typename T> constexpr int p2m_warps() { return sizeof(T) == 4 ? 4 : 2; }

// The columns m.. of q conj(R_n^m), row v = 2 tri(n, m) + part at sm[v * 33].
// R_n^m = R_m^m rho_n with a real rho (rho_m = 1): three operations a term and
// two products, q in the seed of R_m^m, where the complex recursion and the
// product with q took ten.  FP64, 2,468 leaves 109 -> 85 us, 1,254 leaves 71 -> 56.
template <typename T, int P, int M>
__device__ __forceinline__ void p2m_columns(T x, T y, T r2, const T (&zc)[P + 1], T dr, T di, T *sm) {
    sm[(2 * tri(M, M)) * 33] = dr;
    sm[(2 * tri(M, M) + 1) * 33] = -di;
    T rho = (T)1, last = (T)0;
#pragma unroll
    for (int n = M + 1; n <= P; ++n) {
        const T d = (T)(1.0 / ((n + M) * (n - M)));
        const T next = (n == M + 1 ? zc[n] : zc[n] * rho - r2 * last) * d;
        last = rho;
        rho = next;
        sm[(2 * tri(n, M)) * 33] = dr * rho;
        sm[(2 * tri(n, M) + 1) * 33] = M == 0 ? (T)0 : -(di * rho);  // m = 0 is real
    }
    if constexpr (M < P) {
        constexpr double c = -1.0 / (2.0 * (M + 1));
        const T sx = (T)c * x, sy = (T)c * y;
        p2m_columns<T, P, M + 1>(x, y, r2, zc, M == 0 ? sx * dr : sx * dr - sy * di, M == 0 ? sy * dr : sx * di + sy * dr,
                                 sm);
    }
}

template <typename T, int P>
__global__ void __launch_bounds__(32 * p2m_warps<T>())
    k_p2m(const int32_t *__restrict__ leaves, int64_t n_leaves, const typename Vec4<T>::type *__restrict__ pts,
          const typename Vec4<T>::type *__restrict__ center, const typename Vec4<T>::type *__restrict__ half,
          const int2 *__restrict__ range, Cplx<T> *__restrict__ Mexp, int nc_pad) {
    constexpr int NV = 2 * ncoef(P), NR = (NV + 31) / 32;
    extern __shared__ __align__(16) unsigned char p2m_smem[];
    chain_next();
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= n_leaves) return;
    T *sm = reinterpret_cast<T *>(p2m_smem) + (threadIdx.x >> 5) * (NV * 33);
    const int leaf = leaves[w];
    const typename Vec4<T>::type c = center[leaf];
    const T ia = (T)1 / half[leaf].w;
    const int2 rg = range[leaf];
    T acc[NR];
#pragma unroll
    for (int j = 0; j < NR; ++j) acc[j] = (T)0;
    for (int b = rg.x; b < rg.y; b += 32) {
        const int na = min(32, rg.y - b);
        __syncwarp();
        if (lane < na) {
            const typename Vec4<T>::type p = pts[b + lane];
            const T x = (p.x - c.x) * ia, y = (p.y - c.y) * ia, z = (p.z - c.z) * ia, q = p.w;
            const T r2 = x * x + y * y + z * z;
            T zc[P + 1];
#pragma unroll
            for (int n = 1; n <= P; ++n) zc[n] = (T)(2 * n - 1) * z;
            p2m_columns<T, P, 0>(x, y, r2, zc, q, (T)0, sm + lane);
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < NR; ++j) {
            const int v = lane + 32 * j;
            if (v < NV) {
                T t = acc[j];
                for (int l = 0; l < na; ++l) t += sm[v * 33 + l];
                acc[j] = t;
            }
        }
    }
    T *out = reinterpret_cast<T *>(Mexp + (int64_t)leaf * nc_pad);
#pragma unroll
    for (int j = 0; j < NR; ++j)
        if (lane + 32 * j < NV) out[lane + 32 * j] = acc[j];
}

// ---------------------------------------------------------------------------
// M2M: warp per internal node of one level, lanes over output coefficients
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(128) k_m2m(const int32_t *__restrict__ nodes, int n_nodes,
                                             const uint8_t *__restrict__ is_leaf, const int32_t *__restrict__ children,
                                             const typename Vec4<T>::type *__restrict__ center,
                                             const typename Vec4<T>::type *__restrict__ half, Cplx<T> *Mexp, int p,
                                             int nc_pad) {
    __shared__ Cplx<T> sR[4][ncoef(kPMax)], sM[4][ncoef(kPMax)];
    const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int w = blockIdx.x * 4 + wl;
    if (w >= n_nodes) return;
    const int node = nodes[w];
    if (is_leaf[node]) return;
    const int nc = ncoef(p);
    const typename Vec4<T>::type cp = center[node];
    const T aP = half[node].w, iaP = (T)1 / aP;
    Cplx<T> acc[3] = {{0, 0}, {0, 0}, {0, 0}};
    for (int o = 0; o < 8; ++o) {
        const int ch = children[8 * node + o];
        if (ch < 0) continue;
        const typename Vec4<T>::type cc = center[ch];
        const T ratio = half[ch].w * iaP;
        if (lane == 0) regular_harmonics_rt<T>((cc.x - cp.x) * iaP, (cc.y - cp.y) * iaP, (cc.z - cp.z) * iaP, p, sR[wl]);
        for (int k = lane; k < nc; k += 32) {
            int n, m;
            coef_nm(k, n, m);
            T sc = (T)1;
            for (int e = 0; e < n; ++e) sc *= ratio;
            Cplx<T> v = Mexp[(int64_t)ch * nc_pad + k];
            sM[wl][k] = Cplx<T>{v.re * sc, v.im * sc};
        }
        __syncwarp();
        for (int q = 0; q < 3; ++q) {
            const int k = lane + 32 * q;
            if (k >= nc) break;
            int n, m;
            coef_nm(k, n, m);
            Cplx<T> a = acc[q];
            for (int kk = 0; kk <= n; ++kk) {
                const int j = n - kk;
                for (int l = -kk; l <= kk; ++l) {
                    const int u = m - l;
                    if (u < -j || u > j) continue;
                    Cplx<T> r = harm_at(sR[wl], kk, l);
                    Cplx<T> mm = harm_at(sM[wl], j, u);
                    // conj(r) * mm
                    a.re += r.re * mm.re + r.im * mm.im;
                    a.im += r.re * mm.im - r.im * mm.re;
                }
            }
            acc[q] = a;
        }
        __syncwarp();
    }
    for (int q = 0; q < 3; ++q) {
        const int k = lane + 32 * q;
        if (k < nc) Mexp[(int64_t)node * nc_pad + k] = acc[q];
    }
}

// ---------------------------------------------------------------------------
// pair helpers: (sr, si) += (xr, xi) * (c0, c1) on coefficients held in
// separate re / im arrays, as one packed FMA (FFMA2)
// ---------------------------------------------------------------------------
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
template <typename T> struct Pair {};
template <> struct Pair<float> { using type = float2; };
template <> struct Pair<double> { using type = double2; };
__device__ __forceinline__ float2 mk2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ double2 mk2(double a, double b) { return make_double2(a, b); }
__device__ __forceinline__ void fma2_into(float &sr, float &si, float xr, float xi, float2 c) {
    const float2 r = __ffma2_rn(f2(xr, xi), c, f2(sr, si));
    sr = r.x;
    si = r.y;
}
// ---------------------------------------------------------------------------
// M2M / L2L fast paths (compile-time order), one launch per level.  Two forms:
// one thread per node (FP32, levels of many nodes: registers, packed FMAs),
// and one block per node (FP64, and small FP32 levels; below).  Both
// translations factor the azimuth out like the M2L.  With
// d = (c_C - c_P) / a_P = (s cos phi, s sin phi, z) and the real regular
// harmonics rho_k^l := R_k^l(s, 0, z) (R_k^l(d) = e^{i l phi} rho_k^l,
// rho_k^{-l} = (-1)^l rho_k^l):
//   M2M  Mhat_P,n^m = sum_C e^{-i m phi} sum_{k,l} rho_k^l Mt_{n-k}^{m-l},
//        Mt_j^u = e^{i u phi} (a_C/a_P)^j Mhat_C,j^u
//   L2L  Lhat_C,j^u += (a_C/a_P)^j e^{-i u phi} sum_{k,l} rho_k^l Lt_{j+k}^{u+l},
//        Lt_n^m = e^{i m phi} Lhat_P,n^m
// with negative orders through X^{-m} = (-1)^m conj(X^m).  The M2M runs from
// the deepest level up: a node first sums its children's translated
// multipoles (fixed order: deterministic), stores its own multipole, then
// writes its translation to the parent's centre for the next level up.
// ---------------------------------------------------------------------------
template <typename T, int MU, int K>
__device__ __forceinline__ T rho_coef(T z, T r2, T diag, T cm1, T cm2) {
    if constexpr (K == MU) {
        return diag;
    } else if constexpr (K == MU + 1) {
        return ((T)(2 * K - 1) / (T)((K + MU) * (K - MU))) * z * cm1;
    } else {
        return ((T)(2 * K - 1) * z * cm1 - r2 * cm2) * ((T)1 / (T)((K + MU) * (K - MU)));
    }
}

template <typename T, int P, int MU, int K, typename AR>
__device__ __forceinline__ void m2m_degree(AR &mr, AR &mi, T z, T r2, T diag, T cm1, T cm2, AR &Sr, AR &Si) {
    const T c = rho_coef<T, MU, K>(z, r2, diag, cm1, cm2);
    const auto cpp = mk2(c, c), cnn = mk2(-c, -c), cpn = mk2(c, -c), cnp = mk2(-c, c);
#pragma unroll
    for (int n = 0; n <= P; ++n) {
        if (n < K) continue;
        const int j = n - K;
#pragma unroll
        for (int m = 0; m <= P; ++m) {
            if (m > n) continue;
            {  // l = +mu, u = m - mu
                const int u = m - MU, au = u < 0 ? -u : u;
                if (au <= j) {
                    if (u >= 0)
                        fma2_into(Sr[tri(n, m)], Si[tri(n, m)], mr[tri(j, u)], mi[tri(j, u)], cpp);
                    else  // (-1)^|u| conj(Mt_j^|u|)
                        fma2_into(Sr[tri(n, m)], Si[tri(n, m)], mr[tri(j, au)], mi[tri(j, au)], (au & 1) ? cnp : cpn);
                }
            }
            if (MU > 0) {  // l = -mu: (-1)^mu rho, u = m + mu
                const int u = m + MU;
                if (u <= j) fma2_into(Sr[tri(n, m)], Si[tri(n, m)], mr[tri(j, u)], mi[tri(j, u)], (MU & 1) ? cnn : cpp);
            }
        }
    }
    if constexpr (K < P) m2m_degree<T, P, MU, K + 1>(mr, mi, z, r2, diag, c, cm1, Sr, Si);
}

template <typename T, int P, int MU, int K, typename AR>
__device__ __forceinline__ void l2l_degree(AR &lr, AR &li, T z, T r2, T diag, T cm1, T cm2, AR &Sr, AR &Si) {
    const T c = rho_coef<T, MU, K>(z, r2, diag, cm1, cm2);
    const auto cpp = mk2(c, c), cnn = mk2(-c, -c), cpn = mk2(c, -c), cnp = mk2(-c, c);
#pragma unroll
    for (int j = 0; j <= P; ++j) {
        if (j + K > P) continue;
        const int n = j + K;
#pragma unroll
        for (int u = 0; u <= P; ++u) {
            if (u > j) continue;
            {  // l = +mu, m' = u + mu
                const int mp = u + MU;
                if (mp <= n) fma2_into(Sr[tri(j, u)], Si[tri(j, u)], lr[tri(n, mp)], li[tri(n, mp)], cpp);
            }
            if (MU > 0) {  // l = -mu: (-1)^mu rho, m' = u - mu
                const int mp = u - MU;
                if (mp >= 0) {
                    fma2_into(Sr[tri(j, u)], Si[tri(j, u)], lr[tri(n, mp)], li[tri(n, mp)], (MU & 1) ? cnn : cpp);
                } else {  // (-1)^(mu + |m'|) conj(Lt_n^|m'|)
                    const int am = -mp;
                    if (am <= n)
                        fma2_into(Sr[tri(j, u)], Si[tri(j, u)], lr[tri(n, am)], li[tri(n, am)],
                                  ((MU + am) & 1) ? cnp : cpn);
                }
            }
        }
    }
    if constexpr (K < P) l2l_degree<T, P, MU, K + 1>(lr, li, z, r2, diag, c, cm1, Sr, Si);
}

// columns mu = 0..P of rho; diag carries rho_mu^mu = -s / (2 mu) rho_{mu-1}^{mu-1}
template <typename T, int P, bool L2L, int MU, typename AR>
__device__ __forceinline__ void shift_column(AR &xr, AR &xi, T s, T z, T r2, T &diag, AR &Sr, AR &Si) {
    if constexpr (MU > 0) diag *= -s * ((T)1 / (T)(2 * MU));
    if constexpr (L2L)
        l2l_degree<T, P, MU, MU>(xr, xi, z, r2, diag, (T)0, (T)0, Sr, Si);
    else
        m2m_degree<T, P, MU, MU>(xr, xi, z, r2, diag, (T)0, (T)0, Sr, Si);
    if constexpr (MU < P) shift_column<T, P, L2L, MU + 1>(xr, xi, s, z, r2, diag, Sr, Si);
}

// Load a coefficient row (16-byte aligned, nc_pad complex) into re / im arrays.
template <int P, typename AR>
__device__ __forceinline__ void load_row(const float2 *row, AR &xr, AR &xi) {
    constexpr int NC = ncoef(P);
    const float4 *r4 = reinterpret_cast<const float4 *>(row);
#pragma unroll
    for (int q = 0; q < (NC + 1) / 2; ++q) {
        const float4 v = r4[q];
        xr[2 * q] = v.x;
        xi[2 * q] = v.y;
        if (2 * q + 1 < NC) {
            xr[2 * q + 1] = v.z;
            xi[2 * q + 1] = v.w;
        }
    }
}
template <int P, typename AR>
__device__ __forceinline__ void store_row(float2 *row, AR &xr, AR &xi) {
    constexpr int NC = ncoef(P);
    float4 *o4 = reinterpret_cast<float4 *>(row);
#pragma unroll
    for (int q = 0; q < (NC + 1) / 2; ++q)
        o4[q] = make_float4(xr[2 * q], xi[2 * q], 2 * q + 1 < NC ? xr[2 * q + 1] : 0.0f,
                            2 * q + 1 < NC ? xi[2 * q + 1] : 0.0f);
}

// x_n^m <- e^{i m phi} f^n x_n^m  (f = 1 for the L2L)
template <int P, typename AR>
__device__ __forceinline__ void rotate_scale(AR &xr, AR &xi, float ec, float es, float f) {
    float wr = 1, wi = 0;
#pragma unroll
    for (int m = 0; m <= P; ++m) {
        if (m > 0) {
            const float nr = wr * ec - wi * es, ni = wr * es + wi * ec;
            wr = nr;
            wi = ni;
        }
        float fk = 1;
#pragma unroll
        for (int n = 0; n <= P; ++n) {
            if (n >= m) {
                const float fr = wr * fk, fi = wi * fk;
                const float2 x = f2(xr[tri(n, m)], xi[tri(n, m)]);
                const float2 y = __ffma2_rn(f2(x.y, x.x), f2(-fi, fi), __fmul2_rn(x, f2(fr, fr)));
                xr[tri(n, m)] = y.x;
                xi[tri(n, m)] = y.y;
            }
            fk *= f;
        }
    }
}

// frame of the translation child -> parent: d = (c_C - c_P) / a_P
template <typename T> struct Shift {
    T ratio, s, z, r2, ec, es;
};
template <typename T>
__device__ __forceinline__ Shift<T> shift_of(typename Vec4<T>::type cc, typename Vec4<T>::type cp, T a_child,
                                             T a_par) {
    Shift<T> f;
    const T iaP = (T)1 / a_par;
    f.ratio = a_child * iaP;
    const T dx = (cc.x - cp.x) * iaP, dy = (cc.y - cp.y) * iaP;
    f.z = (cc.z - cp.z) * iaP;
    const T s2 = dx * dx + dy * dy;
    f.s = sqrt(s2);
    f.r2 = s2 + f.z * f.z;
    f.ec = 1;
    f.es = 0;
    if (s2 > (T)0) {
        const T is = (T)1 / f.s;
        f.ec = dx * is;
        f.es = dy * is;
    }
    return f;
}

template <int P, typename AR>
__device__ __forceinline__ void m2m_node(int node, const uint8_t *__restrict__ is_leaf,
                                         const int32_t *__restrict__ children, const int32_t *__restrict__ parent,
                                         const float4 *__restrict__ center,
                                         const float4 *__restrict__ half,
                                         float2 *__restrict__ Mexp,
                                         float2 *__restrict__ moved, int nc_pad, AR &xr, AR &xi,
                                         AR &Sr, AR &Si) {
    constexpr int NC = ncoef(P);
    if (is_leaf[node]) {
        load_row<P>(Mexp + (int64_t)node * nc_pad, xr, xi);
    } else {
#pragma unroll
        for (int q = 0; q < NC; ++q) xr[q] = xi[q] = 0.0f;
        for (int o = 0; o < 8; ++o) {
            const int ch = children[8 * node + o];
            if (ch < 0) continue;
            load_row<P>(moved + (int64_t)ch * nc_pad, Sr, Si);
#pragma unroll
            for (int q = 0; q < NC; ++q) {
                xr[q] += Sr[q];
                xi[q] += Si[q];
            }
        }
        store_row<P>(Mexp + (int64_t)node * nc_pad, xr, xi);
    }
    const int par = parent[node];
    if (par < 0) return;
    const Shift<float> f = shift_of<float>(center[node], center[par], half[node].w, half[par].w);
    rotate_scale<P>(xr, xi, f.ec, f.es, f.ratio);
#pragma unroll
    for (int q = 0; q < NC; ++q) Sr[q] = Si[q] = 0.0f;
    float diag = 1;
    shift_column<float, P, false, 0>(xr, xi, f.s, f.z, f.r2, diag, Sr, Si);
    rotate_scale<P>(Sr, Si, f.ec, -f.es, 1.0f);  // e^{-i m phi}
    store_row<P>(moved + (int64_t)node * nc_pad, Sr, Si);
}

template <int P, typename AR>
__device__ __forceinline__ void l2l_node(int node, const int32_t *__restrict__ parent,
                                         const float4 *__restrict__ center,
                                         const float4 *__restrict__ half,
                                         float2 *__restrict__ Lexp, int nc_pad, AR &xr, AR &xi,
                                         AR &Sr, AR &Si) {
    constexpr int NC = ncoef(P);
    const int par = parent[node];
    if (par < 0) return;
    const Shift<float> f = shift_of<float>(center[node], center[par], half[node].w, half[par].w);
    load_row<P>(Lexp + (int64_t)par * nc_pad, xr, xi);
    rotate_scale<P>(xr, xi, f.ec, f.es, 1.0f);
#pragma unroll
    for (int q = 0; q < NC; ++q) Sr[q] = Si[q] = 0.0f;
    float diag = 1;
    shift_column<float, P, true, 0>(xr, xi, f.s, f.z, f.r2, diag, Sr, Si);
    rotate_scale<P>(Sr, Si, f.ec, -f.es, f.ratio);  // (a_C/a_P)^j e^{-i u phi}
    load_row<P>(Lexp + (int64_t)node * nc_pad, xr, xi);
#pragma unroll
    for (int q = 0; q < NC; ++q) {
        xr[q] += Sr[q];
        xi[q] += Si[q];
    }
    store_row<P>(Lexp + (int64_t)node * nc_pad, xr, xi);
}

constexpr int kFastThreads = 128;

template <int P>
__global__ void __launch_bounds__(kFastThreads) k_m2m_fast(
    const int32_t *__restrict__ nodes, int count, const uint8_t *__restrict__ is_leaf,
    const int32_t *__restrict__ children, const int32_t *__restrict__ parent, const float4 *__restrict__ center,
    const float4 *__restrict__ half, float2 *__restrict__ Mexp, float2 *__restrict__ moved, int nc_pad) {
    constexpr int NC = ncoef(P);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    float xr[NC], xi[NC], Sr[NC], Si[NC];
    m2m_node<P>(nodes[i], is_leaf, children, parent, center, half, Mexp, moved, nc_pad, xr, xi, Sr, Si);
}

template <int P>
__global__ void __launch_bounds__(kFastThreads) k_l2l_fast(const int32_t *__restrict__ nodes, int count,
                                                            const int32_t *__restrict__ parent,
                                                            const float4 *__restrict__ center,
                                                            const float4 *__restrict__ half, float2 *__restrict__ Lexp,
                                                            int nc_pad) {
    constexpr int NC = ncoef(P);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    float xr[NC], xi[NC], Sr[NC], Si[NC];
    l2l_node<P>(nodes[i], parent, center, half, Lexp, nc_pad, xr, xi, Sr, Si);
}

// ---------------------------------------------------------------------------
// The same translations with one block per node, its threads over the terms.
// A thread that owns a node walks about 2,600 dependent operations: 10 us
// however few nodes a level has in FP32, and 130 to 280 us in FP64, whose pipe
// issues a warp's operation in 64 cycles whether one lane is active or all (two
// FP64 lanes per SM and clock).  So what counts is the number of warp
// operations, along the chain and in all.  The terms (k, l) of all outputs are
// dealt to the threads in equal runs (12 at order 8 with 128 threads), each
// within one output, whose partial sums its first thread adds; the azimuth
// phases, harmonics and powers of the scale ratio of a node are laid out with
// the plan (ShiftFrame).  A warp per node that formed them itself and took whole
// outputs per lane (chains of 101 terms) needed 300 FP64 operations a node.
// FP64, 50k-panel torus, six levels: M2M 1,060 (a thread per node), 136 (a
// warp), 64 us; L2L 640, 138, 57.  FP32, 2,003 points, three and two levels:
// M2M 29 -> 24, L2L 24 -> 18 us, launches included.
// ---------------------------------------------------------------------------
// number of terms (k, l) of output (n, m): |l| <= k and |m - l| <= n - k (M2M),
// or k <= P - n, |l| <= k (L2L)
__host__ __device__ constexpr int shift_terms(int P, bool l2l, int n, int m) {
    int t = 0;
    for (int k = 0; k <= (l2l ? P - n : n); ++k)
        for (int l = -k; l <= k; ++l) {
            const int u = l2l ? m + l : m - l, j = l2l ? n + k : n - k;
            if (u >= -j && u <= j) ++t;
        }
    return t;
}
// threads of a block: about 12 terms each
template <int P> __host__ __device__ constexpr int shift_threads() { return P >= 7 ? 128 : (P >= 5 ? 64 : 32); }

// The terms of each thread: output (n, m), first term (k, l) and the number of
// terms; and for each output its first thread and the number of its threads.
template <int P, bool L2L> struct ShiftSplit {
    static constexpr int NT = shift_threads<P>();
    unsigned char n[NT], m[NT], k[NT], cnt[NT];
    signed char l[NT];
    unsigned char first[ncoef(P)], parts[ncoef(P)];
    __host__ __device__ constexpr ShiftSplit() : n(), m(), k(), cnt(), l(), first(), parts() {
        int cap = 1;  // the smallest run that fits the threads
        for (;; ++cap) {
            int used = 0;
            for (int n_ = 0; n_ <= P; ++n_)
                for (int m_ = 0; m_ <= n_; ++m_) used += (shift_terms(P, L2L, n_, m_) + cap - 1) / cap;
            if (used <= NT) break;
        }
        int t = 0, q = 0;
        for (int n_ = 0; n_ <= P; ++n_)
            for (int m_ = 0; m_ <= n_; ++m_, ++q) {
                const int terms = shift_terms(P, L2L, n_, m_), np = (terms + cap - 1) / cap;
                first[q] = (unsigned char)t;
                parts[q] = (unsigned char)np;
                int at = 0, part = 0;
                for (int kk = 0; kk <= (L2L ? P - n_ : n_); ++kk)
                    for (int ll = -kk; ll <= kk; ++ll) {
                        const int u = L2L ? m_ + ll : m_ - ll, j = L2L ? n_ + kk : n_ - kk;
                        if (u < -j || u > j) continue;
                        if (part < np && at == part * terms / np) {  // equal runs
                            n[t] = (unsigned char)n_;
                            m[t] = (unsigned char)m_;
                            k[t] = (unsigned char)kk;
                            l[t] = (signed char)ll;
                            cnt[t] = (unsigned char)((part + 1) * terms / np - at);
                            ++t;
                            ++part;
                        }
                        ++at;
                    }
            }
    }
};
template <int P, bool L2L> __device__ const ShiftSplit<P, L2L> d_shift_split{};

// What a node's translation from or to its parent needs, for any order up to
// 8: rho_k^l at k^2 + k + l, e^{i m phi}, (a_C / a_P)^n
constexpr int kFrameP = 8, kFramePh = (kFrameP + 1) * (kFrameP + 1), kFrameFr = kFramePh + 2 * (kFrameP + 1),
              kFrameSize = kFrameFr + kFrameP + 1;  // 108 values

template <typename T, int P> struct ShiftSmem {
    typename Pair<T>::type x[(P + 1) * (P + 1)];  // rotated input, all orders: (n, m) at n^2 + n + m
    typename Pair<T>::type part[shift_threads<P>()];
    T rho[(P + 1) * (P + 1)];
    T ph[2 * (P + 1)];
    T fr[P + 1];
};

template <typename T, int P> struct WarpShift {
    typename Pair<T>::type ph[P + 1];  // e^{i m phi}
    T rho[(P + 1) * (P + 1)];          // rho_k^l at k^2 + k + l
    T fr[P + 1];                       // (a_C / a_P)^n
};

// lanes 0..P: e^{i m phi}, ratio^m and column m of rho
template <typename T, int P>
__device__ __forceinline__ void warp_shift_frame(WarpShift<T, P> &S, const Shift<T> &f, int lane) {
    if (lane <= P) {
        const int m = lane;
        T wr = 1, wi = 0, fm = 1, diag = 1, ar = f.ec, ai = f.es, ra = f.ratio, sa = -f.s;
#pragma unroll
        for (int bit = 1; bit <= P; bit <<= 1) {  // powers by their binary digits
            if (m & bit) {
                const T nr = wr * ar - wi * ai, ni = wr * ai + wi * ar;
                wr = nr;
                wi = ni;
                fm *= ra;
                diag *= sa;
            }
            const T nr = ar * ar - ai * ai, ni = (T)2 * ar * ai;
            ar = nr;
            ai = ni;
            ra *= ra;
            sa *= sa;
        }
        S.ph[m] = mk2(wr, wi);
        S.fr[m] = fm;
        T inv = (T)1;
#pragma unroll
        for (int i = 1; i <= P; ++i)
            if (i <= m) inv *= (T)(1.0 / (2.0 * i));
        T cm1 = diag * inv, cm2 = 0;  // rho_m^m = (-s / 2)^m / m!
        const T sg = (m & 1) ? (T)-1 : (T)1;
        S.rho[m * m + 2 * m] = cm1;
        S.rho[m * m] = sg * cm1;
        for (int k = m + 1; k <= P; ++k) {
            const T d = (T)1 / (T)((k + m) * (k - m));
            const T c = ((T)(2 * k - 1) * f.z * cm1 - f.r2 * cm2) * d;
            cm2 = cm1;
            cm1 = c;
            S.rho[k * k + k + m] = c;
            S.rho[k * k + k - m] = sg * c;
        }
    }
}

// the frames of a level's nodes (a warp each)
template <typename T>
__global__ void __launch_bounds__(128) k_shift_frames(const int32_t *__restrict__ nodes, int count,
                                                      const int32_t *__restrict__ parent,
                                                      const typename Vec4<T>::type *__restrict__ center,
                                                      const typename Vec4<T>::type *__restrict__ half,
                                                      T *__restrict__ frames) {
    constexpr int P = kFrameP;
    __shared__ WarpShift<T, P> shifts[4];
    const int lane = threadIdx.x & 31, i = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (i >= count) return;
    WarpShift<T, P> &S = shifts[threadIdx.x >> 5];
    const int node = nodes[i], par = parent[node];
    if (par < 0) return;  // roots have no frame
    warp_shift_frame<T, P>(S, shift_of<T>(center[node], center[par], half[node].w, half[par].w), lane);
    __syncwarp();
    T *o = frames + (int64_t)i * kFrameSize;
    for (int q = lane; q < kFramePh; q += 32) o[q] = S.rho[q];
    if (lane <= P) {
        o[kFramePh + 2 * lane] = S.ph[lane].x;
        o[kFramePh + 2 * lane + 1] = S.ph[lane].y;
        o[kFrameFr + lane] = S.fr[lane];
    }
}

template <typename T, int P>
__device__ __forceinline__ void load_frame(ShiftSmem<T, P> &S, const T *__restrict__ fr) {
    constexpr int NT = shift_threads<P>(), NH = (P + 1) * (P + 1);
#pragma unroll
    for (int q = threadIdx.x; q < NH + 3 * (P + 1); q += NT) {
        if (q < NH) S.rho[q] = fr[q];
        else if (q < NH + 2 * (P + 1)) S.ph[q - NH] = fr[kFramePh + q - NH];
        else S.fr[q - NH - 2 * (P + 1)] = fr[kFrameFr + q - NH - 2 * (P + 1)];
    }
}

// x_n^m e^{i m phi} g, stored for orders m and -m (X^{-m} = (-1)^m conj X^m)
template <typename T, int P>
__device__ __forceinline__ void shift_put(ShiftSmem<T, P> &S, int n, int m, typename Pair<T>::type x, T g) {
    const T fr = S.ph[2 * m] * g, fi = S.ph[2 * m + 1] * g;
    const T yr = x.x * fr - x.y * fi, yi = x.x * fi + x.y * fr;
    const bool odd = m & 1;
    S.x[n * n + n - m] = mk2(odd ? -yr : yr, odd ? yi : -yi);
    S.x[n * n + n + m] = mk2(yr, yi);
}

// this thread's run of terms into its partial sum
template <typename T, int P, bool L2L>
__device__ __forceinline__ void shift_terms_sum(ShiftSmem<T, P> &S, int n, int m, int k, int l, int cnt) {
    typename Pair<T>::type s = mk2((T)0, (T)0);
    int j = L2L ? n + k : n - k;
    int ri = k * k + k + l, xi = j * j + j + (L2L ? m + l : m - l);
    int left = (L2L ? min(k, j - m) : min(k, m + j)) - l + 1;  // of degree k
    for (int t = 0; t < cnt; ++t) {
        const auto x = S.x[xi];
        const T r = S.rho[ri];
        s.x = fma(r, x.x, s.x);
        s.y = fma(r, x.y, s.y);
        ++ri;
        xi += L2L ? 1 : -1;
        if (--left == 0) {
            ++k;
            j = L2L ? n + k : n - k;
            // l from max(-k, m - j) (M2M) or max(-k, -j - m) (L2L) to min(k, m + j) or min(k, j - m)
            const int lo = max(-k, L2L ? -j - m : m - j), hi = min(k, L2L ? j - m : m + j);
            left = hi - lo + 1;
            ri = k * k + k + lo;
            xi = j * j + j + (L2L ? m + lo : m - lo);
        }
    }
    S.part[threadIdx.x] = s;
}
template <typename T, int P>
__device__ __forceinline__ typename Pair<T>::type shift_total(const ShiftSmem<T, P> &S, int first, int parts) {
    typename Pair<T>::type v = S.part[first];
    for (int p = 1; p < parts; ++p) {
        v.x += S.part[first + p].x;
        v.y += S.part[first + p].y;
    }
    return v;
}

template <typename T, int P>
__global__ void __launch_bounds__(shift_threads<P>()) k_m2m_node(
    const int32_t *__restrict__ nodes, const uint8_t *__restrict__ is_leaf, const int32_t *__restrict__ children,
    const T *__restrict__ frames, typename Pair<T>::type *__restrict__ Mexp, typename Pair<T>::type *__restrict__ moved,
    int nc_pad) {
    using T2 = typename Pair<T>::type;
    constexpr int NT = shift_threads<P>(), NC = ncoef(P);
    __shared__ ShiftSmem<T, P> S;
    const int tid = threadIdx.x, node = nodes[blockIdx.x];
    const ShiftSplit<P, false> &D = d_shift_split<P, false>;
    const int tn = D.n[tid], tm = D.m[tid], tk = D.k[tid], tl = D.l[tid], tc = D.cnt[tid];
    if (frames) load_frame<T, P>(S, frames + (int64_t)blockIdx.x * kFrameSize);
    const bool leaf = is_leaf[node];
    int child[8];
#pragma unroll
    for (int o = 0; o < 8; ++o) child[o] = leaf ? -1 : children[8 * node + o];
    chain_next();
    chain_wait();
    T2 x[(NC + NT - 1) / NT];
#pragma unroll
    for (int r = 0; r < (NC + NT - 1) / NT; ++r) {
        const int q = tid + r * NT;
        if (q >= NC) continue;
        if (leaf) {
            x[r] = Mexp[(int64_t)node * nc_pad + q];
        } else {
            T2 v[8];
#pragma unroll
            for (int o = 0; o < 8; ++o) {
                v[o] = child[o] >= 0 ? moved[(int64_t)child[o] * nc_pad + q] : mk2((T)0, (T)0);
            }
            x[r] = v[0];
#pragma unroll
            for (int o = 1; o < 8; ++o) {
                x[r].x += v[o].x;
                x[r].y += v[o].y;
            }
            Mexp[(int64_t)node * nc_pad + q] = x[r];
        }
    }
    if (!frames) return;  // the roots
    __syncthreads();
#pragma unroll
    for (int r = 0; r < (NC + NT - 1) / NT; ++r) {
        const int q = tid + r * NT;
        if (q >= NC) continue;
        int n = 0;
        while (tri(n + 1, 0) <= q) ++n;
        shift_put<T, P>(S, n, q - tri(n, 0), x[r], S.fr[n]);
    }
    __syncthreads();
    shift_terms_sum<T, P, false>(S, tn, tm, tk, tl, tc);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < (NC + NT - 1) / NT; ++r) {
        const int q = tid + r * NT;
        if (q >= NC) continue;
        int n = 0;
        while (tri(n + 1, 0) <= q) ++n;
        const int m = q - tri(n, 0);
        const T2 v = shift_total<T, P>(S, D.first[q], D.parts[q]);
        const T wx = S.ph[2 * m], wy = S.ph[2 * m + 1];
        moved[(int64_t)node * nc_pad + q] = mk2(v.x * wx + v.y * wy, v.y * wx - v.x * wy);  // e^{-i m phi}
    }
}

template <typename T, int P>
__global__ void __launch_bounds__(shift_threads<P>()) k_l2l_node(const int32_t *__restrict__ nodes,
                                                                 const int32_t *__restrict__ parent,
                                                                 const T *__restrict__ frames,
                                                                 typename Pair<T>::type *__restrict__ Lexp, int nc_pad) {
    using T2 = typename Pair<T>::type;
    constexpr int NT = shift_threads<P>(), NC = ncoef(P);
    __shared__ ShiftSmem<T, P> S;
    const int tid = threadIdx.x, node = nodes[blockIdx.x], par = parent[node];
    const ShiftSplit<P, true> &D = d_shift_split<P, true>;
    const int tn = D.n[tid], tm = D.m[tid], tk = D.k[tid], tl = D.l[tid], tc = D.cnt[tid];
    load_frame<T, P>(S, frames + (int64_t)blockIdx.x * kFrameSize);
    chain_next();
    chain_wait();
    T2 x[(NC + NT - 1) / NT], old[(NC + NT - 1) / NT];
#pragma unroll
    for (int r = 0; r < (NC + NT - 1) / NT; ++r) {
        const int q = tid + r * NT;
        if (q >= NC) continue;
        x[r] = Lexp[(int64_t)par * nc_pad + q];
        old[r] = Lexp[(int64_t)node * nc_pad + q];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < (NC + NT - 1) / NT; ++r) {
        const int q = tid + r * NT;
        if (q >= NC) continue;
        int n = 0;
        while (tri(n + 1, 0) <= q) ++n;
        shift_put<T, P>(S, n, q - tri(n, 0), x[r], (T)1);
    }
    __syncthreads();
    shift_terms_sum<T, P, true>(S, tn, tm, tk, tl, tc);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < (NC + NT - 1) / NT; ++r) {
        const int q = tid + r * NT;
        if (q >= NC) continue;
        int n = 0;
        while (tri(n + 1, 0) <= q) ++n;
        const int m = q - tri(n, 0);
        const T2 v = shift_total<T, P>(S, D.first[q], D.parts[q]);
        const T wx = S.ph[2 * m], wy = S.ph[2 * m + 1], g = S.fr[n];  // (a_C / a_P)^j e^{-i u phi}
        Lexp[(int64_t)node * nc_pad + q] =
            mk2(old[r].x + g * (v.x * wx + v.y * wy), old[r].y + g * (v.y * wx - v.x * wy));
    }
}

// ---------------------------------------------------------------------------
// M2L generic path: any precision / order; warp per target row, lanes over
// harmonics columns and output coefficients, operands in shared memory.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(128) k_m2l_generic(int64_t n_rows, const int32_t *__restrict__ row_ids,
                                                     const int32_t *__restrict__ off, const int32_t *__restrict__ src,
                                                     const typename Vec4<T>::type *__restrict__ tcenter,
                                                     const typename Vec4<T>::type *__restrict__ thalf,
                                                     const typename Vec4<T>::type *__restrict__ center,
                                                     const typename Vec4<T>::type *__restrict__ half,
                                                     const Cplx<T> *__restrict__ Mexp, Cplx<T> *Lexp, int p, int nc_pad,
                                                     int accumulate) {
    __shared__ Cplx<T> sI[4][ncoef(2 * kPMax)];
    __shared__ Cplx<T> sM[4][ncoef(kPMax)];
    const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t w = (int64_t)blockIdx.x * 4 + wl;
    if (w >= n_rows) return;
    const int t = row_ids ? row_ids[w] : (int)w;
    const int nc = ncoef(p);
    const typename Vec4<T>::type ct = tcenter[t];
    const T aL = thalf[t].w;
    Cplx<T> acc[3] = {{0, 0}, {0, 0}, {0, 0}};
    for (int k = off[t]; k < off[t + 1]; ++k) {
        const int s = src[k];
        const typename Vec4<T>::type cs = center[s];
        // Scale by the larger of the two radii so that every ratio is <= 1:
        //  source scale: A_n += (a_L/a_M)^(n+1) sum Mhat_k I_{n+k}(t / a_M)
        //  target scale: A_n += sum Mhat_k (a_M/a_L)^k I_{n+k}(t / a_L)
        const T aM = half[s].w;
        const bool by_src = aM >= aL;
        const T ia = (T)1 / (by_src ? aM : aL);
        const T f = by_src ? aL / aM : aM / aL;
        const T vx = (ct.x - cs.x) * ia, vy = (ct.y - cs.y) * ia, vz = (ct.z - cs.z) * ia;
        const T r2 = vx * vx + vy * vy + vz * vz, ir2 = (T)1 / r2;
        if (lane <= 2 * p) {
            const int mu = lane;
            T dr = (T)1 / sqrt(r2), di = (T)0;
            for (int i = 1; i <= mu; ++i) {
                const T sc = -(T)(2 * i - 1) * ir2;
                const T nr = sc * (vx * dr - vy * di), ni = sc * (vx * di + vy * dr);
                dr = nr;
                di = ni;
            }
            sI[wl][tri(mu, mu)] = Cplx<T>{dr, di};
            T pr = dr, pi = di, qr = 0, qi = 0;
            for (int j = mu + 1; j <= 2 * p; ++j) {
                const T a = (T)(2 * j - 1) * vz, b = (T)((j - 1 + mu) * (j - 1 - mu));
                const T nr = (a * pr - b * qr) * ir2, ni = (a * pi - b * qi) * ir2;
                sI[wl][tri(j, mu)] = Cplx<T>{nr, ni};
                qr = pr;
                qi = pi;
                pr = nr;
                pi = ni;
            }
        }
        for (int c = lane; c < nc; c += 32) {
            Cplx<T> mv = Mexp[(int64_t)s * nc_pad + c];
            if (!by_src) {
                int n, m;
                coef_nm(c, n, m);
                T fk = (T)1;
                for (int e = 0; e < n; ++e) fk *= f;
                mv.re *= fk;
                mv.im *= fk;
            }
            sM[wl][c] = mv;
        }
        __syncwarp();
        for (int q = 0; q < 3; ++q) {
            const int c = lane + 32 * q;
            if (c >= nc) break;
            int n, m;
            coef_nm(c, n, m);
            Cplx<T> sacc{0, 0};
            for (int kk = 0; kk <= p; ++kk)
                for (int l = -kk; l <= kk; ++l) {
                    Cplx<T> v = cmul(harm_at(sM[wl], kk, l), harm_at(sI[wl], n + kk, l - m));
                    sacc.re += v.re;
                    sacc.im += v.im;
                }
            T fn = (T)1;
            if (by_src) {
                fn = f;
                for (int e = 0; e < n; ++e) fn *= f;
            }
            acc[q].re += fn * sacc.re;
            acc[q].im += fn * sacc.im;
        }
        __syncwarp();
    }
    const T iaL = (T)1 / aL;
    for (int q = 0; q < 3; ++q) {
        const int c = lane + 32 * q;
        if (c >= nc) break;
        int n, m;
        coef_nm(c, n, m);
        const T sg = ((n + m) & 1) ? -iaL : iaL;
        Cplx<T> v{sg * acc[q].re, sg * acc[q].im};
        Cplx<T> *o = Lexp + (int64_t)t * nc_pad + c;
        if (accumulate) {
            v.re += o->re;
            v.im += o->im;
        }
        *o = v;
    }
}

// extreme pairs (source radius > 256x target radius) as a CSR by target
template <typename T4>
__global__ void k_extreme_flags(int64_t n_nodes, const int32_t *off, const int32_t *src, const T4 *thalf,
                                const T4 *half, int32_t *row_cnt) {
    using T = decltype(thalf->w);
    const int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (t >= n_nodes) return;
    const T iaL = (T)1 / thalf[t].w;
    int c = 0;
    for (int k = off[t] + lane; k < off[t + 1]; k += 32) c += (half[src[k]].w * iaL > (T)kExtremeRatio) ? 1 : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (lane == 0) row_cnt[t] = c;
}
template <typename T4>
__global__ void k_extreme_fill(int64_t n_nodes, const int32_t *off, const int32_t *src, const T4 *thalf,
                               const T4 *half, const int32_t *eoff, int32_t *esrc) {
    using T = decltype(thalf->w);
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_nodes) return;
    const T iaL = (T)1 / thalf[t].w;
    int j = eoff[t];
    for (int k = off[t]; k < off[t + 1]; ++k)
        if (half[src[k]].w * iaL > (T)kExtremeRatio) esrc[j++] = src[k];
}
__global__ void k_set_last(int32_t *off, int64_t rows, const int64_t *total) { off[rows] = (int32_t)*total; }
__global__ void k_nonempty_rows(int64_t n_nodes, const int32_t *cnt, const int32_t *pos, int32_t *rows) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n_nodes && cnt[t] > 0) rows[pos[t]] = (int32_t)t;
}
__global__ void k_flag_nonzero(int64_t n, const int32_t *cnt, int32_t *flag) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) flag[t] = cnt[t] > 0;
}

// ---------------------------------------------------------------------------
// L2L: warp per node of one level (level >= 1)
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(128) k_l2l(const int32_t *__restrict__ nodes, int n_nodes,
                                             const int32_t *__restrict__ parent,
                                             const typename Vec4<T>::type *__restrict__ center,
                                             const typename Vec4<T>::type *__restrict__ half, Cplx<T> *Lexp, int p,
                                             int nc_pad) {
    __shared__ Cplx<T> sR[4][ncoef(kPMax)], sL[4][ncoef(kPMax)];
    const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int w = blockIdx.x * 4 + wl;
    if (w >= n_nodes) return;
    const int node = nodes[w];
    const int par = parent[node];
    const int nc = ncoef(p);
    const typename Vec4<T>::type cc = center[node], cp = center[par];
    const T aP = half[par].w, iaP = (T)1 / aP, ratio = half[node].w * iaP;
    if (lane == 0) regular_harmonics_rt<T>((cc.x - cp.x) * iaP, (cc.y - cp.y) * iaP, (cc.z - cp.z) * iaP, p, sR[wl]);
    for (int k = lane; k < nc; k += 32) sL[wl][k] = Lexp[(int64_t)par * nc_pad + k];
    __syncwarp();
    for (int q = 0; q < 3; ++q) {
        const int c = lane + 32 * q;
        if (c >= nc) break;
        int j, u;
        coef_nm(c, j, u);
        Cplx<T> a{0, 0};
        for (int kk = 0; kk + j <= p; ++kk)
            for (int l = -kk; l <= kk; ++l) {
                const int nn = j + kk, mm = u + l;
                if (mm < -nn || mm > nn) continue;
                Cplx<T> v = cmul(harm_at(sL[wl], nn, mm), harm_at(sR[wl], kk, l));
                a.re += v.re;
                a.im += v.im;
            }
        T sc = (T)1;
        for (int e = 0; e < j; ++e) sc *= ratio;
        Cplx<T> *o = Lexp + (int64_t)node * nc_pad + c;
        o->re += sc * a.re;
        o->im += sc * a.im;
    }
}

template <typename T> int p2m_impl(const DevTree &tree, FmmBuffers &buf, cudaStream_t s) {
    using T4 = typename Vec4<T>::type;
    if (tree.n_leaves == 0) return EDFMM_OK;
    constexpr int NT = 32 * p2m_warps<T>();
    const unsigned grid = nblk(tree.n_leaves * 32, NT);
    const size_t smem = sizeof(T) * 33 * 2 * (size_t)ncoef(buf.p) * p2m_warps<T>();
#define EDFMM_P2M_CASE(PP)                                                                                          \
    case PP: {                                                                                                      \
        static DeviceOnce once;                                                                                     \
        EDFMM_CUDA_TRY(allow_smem(once, k_p2m<T, PP>, sizeof(T) * 33 * 2 * ncoef(PP) * p2m_warps<T>()));            \
        k_p2m<T, PP><<<grid, NT, smem, s>>>(dptr<int32_t>(tree.leaves), tree.n_leaves, dptr<T4>(tree.pts),           \
                                            dptr<T4>(tree.center), dptr<T4>(tree.half), dptr<int2>(tree.range),       \
                                            dptr<Cplx<T>>(buf.multipoles), buf.nc_pad);                              \
        break;                                                                                                      \
    }
    switch (buf.p) {
        EDFMM_P2M_CASE(1)
        EDFMM_P2M_CASE(2)
        EDFMM_P2M_CASE(3)
        EDFMM_P2M_CASE(4)
        EDFMM_P2M_CASE(5)
        EDFMM_P2M_CASE(6)
        EDFMM_P2M_CASE(7)
        EDFMM_P2M_CASE(8)
        EDFMM_P2M_CASE(9)
        EDFMM_P2M_CASE(10)
        default:
            return fail(EDFMM_ERR_UNSUPPORTED, "expansion order out of range");
    }
#undef EDFMM_P2M_CASE
    EDFMM_LAUNCH_CHECK("k_p2m");
    return EDFMM_OK;
}

// Far-field chains of trees up to these sizes overlap their launches
// (chain_launch).  FP32 matvecs of 2,003 points (73 nodes) take 60 us without and
// 43 with, 16,000 points (585 nodes) 125 and 102, the 200k-panel torus (11,705)
// 339 and 331, a million points (37,449) 4,600 and 4,624; FP64 2,000 points (65)
// 177 and 164, 20,011 points (1,500) 1,291 and 1,296, the 50k-panel torus in
// two-float (2,937) 1,602 and 1,655: blocks that wait for their predecessor hold
// places the near field would use.
constexpr int64_t kChainNodes32 = 16384, kChainNodes64 = 512;

// FP32 levels up to this many nodes take a block per node (FP64 all levels).
// M2M and L2L of the 200k-panel torus (levels of 2,344 and 6,968 nodes at order
// 6) take 62 and 43 us with the line at 2,048, 58 and 44 at 6,144, 58 and 49 at
// 12,288; of 1,048,576 points (4,096 and 32,768 nodes at order 8) 60 and 48, 56
// and 51, and 95 and 86 us with every level a block per node.
constexpr int kNodeLevel = 6144;

template <typename T, int P> int launch_m2m_fast(const DevTree &tree, FmmBuffers &buf, cudaStream_t s) {
    using T2 = typename Pair<T>::type;
    const bool chained = chain_tree(tree.n_nodes, tree.dtype, s);
    for (int lev = tree.max_level; lev >= 0; --lev) {
        const int lo = tree.level_offsets[lev], hi = tree.level_offsets[lev + 1];
        if (hi <= lo) continue;
        const int32_t *nodes = dptr<int32_t>(tree.level_nodes) + lo;
        const int64_t frames = tree.frame_off[lev];
        if (frames >= 0 || lev == 0) {
            EDFMM_CUDA_TRY(chain_launch(
                chained, k_m2m_node<T, P>, (unsigned)(hi - lo), shift_threads<P>(), 0, s, nodes,
                dptr<uint8_t>(tree.is_leaf), dptr<int32_t>(tree.children),
                lev == 0 ? (T *)nullptr : dptr<T>(tree.shift_frames) + frames * kFrameSize, dptr<T2>(buf.multipoles),
                dptr<T2>(buf.translated), buf.nc_pad));
        } else if constexpr (sizeof(T) == 4) {
            k_m2m_fast<P><<<nblk(hi - lo, kFastThreads), kFastThreads, 0, s>>>(
                nodes, hi - lo, dptr<uint8_t>(tree.is_leaf), dptr<int32_t>(tree.children), dptr<int32_t>(tree.parent),
                dptr<float4>(tree.center), dptr<float4>(tree.half), dptr<float2>(buf.multipoles),
                dptr<float2>(buf.translated), buf.nc_pad);
        }
        if (lev > 0) count_launch();
    }
    return EDFMM_OK;
}

template <typename T, int P> int launch_l2l_fast(const DevTree &tree, FmmBuffers &buf, cudaStream_t s) {
    using T2 = typename Pair<T>::type;
    const bool chained = chain_tree(tree.n_nodes, tree.dtype, s);
    for (int lev = 1; lev <= tree.max_level; ++lev) {
        const int lo = tree.level_offsets[lev], hi = tree.level_offsets[lev + 1];
        if (hi <= lo) continue;
        const int32_t *nodes = dptr<int32_t>(tree.level_nodes) + lo;
        const int64_t frames = tree.frame_off[lev];
        if (frames >= 0) {
            EDFMM_CUDA_TRY(chain_launch(chained, k_l2l_node<T, P>, (unsigned)(hi - lo), shift_threads<P>(), 0, s, nodes,
                                        dptr<int32_t>(tree.parent), dptr<T>(tree.shift_frames) + frames * kFrameSize,
                                        dptr<T2>(buf.locals), buf.nc_pad));
        } else if constexpr (sizeof(T) == 4) {
            k_l2l_fast<P><<<nblk(hi - lo, kFastThreads), kFastThreads, 0, s>>>(
                nodes, hi - lo, dptr<int32_t>(tree.parent), dptr<float4>(tree.center), dptr<float4>(tree.half),
                dptr<float2>(buf.locals), buf.nc_pad);
        }
        if (lev < tree.max_level) count_launch();
    }
    return EDFMM_OK;
}

template <typename T> int shift_prepare_impl(DevTree &tree, cudaStream_t s) {
    using T4 = typename Vec4<T>::type;
    const int levels = (int)tree.level_offsets.size() - 1;
    tree.frame_off.assign(std::max(levels, 0), -1);
    int64_t n = 0;
    for (int lev = 1; lev < levels; ++lev) {
        const int count = tree.level_offsets[lev + 1] - tree.level_offsets[lev];
        if (sizeof(T) == 4 && count > kNodeLevel) continue;
        tree.frame_off[lev] = n;
        n += count;
    }
    if (n == 0) return EDFMM_OK;
    if (int rc = tree.shift_frames.reserve(sizeof(T) * kFrameSize * (size_t)n)) return rc;
    for (int lev = 1; lev < levels;) {  // runs of levels that have frames lie one after another
        if (tree.frame_off[lev] < 0) {
            ++lev;
            continue;
        }
        int end = lev + 1;
        while (end < levels && tree.frame_off[end] >= 0) ++end;
        const int lo = tree.level_offsets[lev], hi = tree.level_offsets[end];
        if (hi > lo) {
            k_shift_frames<T><<<nblk(hi - lo, 4), 128, 0, s>>>(
                dptr<int32_t>(tree.level_nodes) + lo, hi - lo, dptr<int32_t>(tree.parent), dptr<T4>(tree.center),
                dptr<T4>(tree.half), dptr<T>(tree.shift_frames) + tree.frame_off[lev] * kFrameSize);
            EDFMM_LAUNCH_CHECK("k_shift_frames");
        }
        lev = end;
    }
    return EDFMM_OK;
}

template <typename T> int m2m_impl(const DevTree &tree, FmmBuffers &buf, cudaStream_t s) {
    using T4 = typename Vec4<T>::type;
    if (buf.p <= 8 && tree.n_nodes > 0) {
        int rc;
        switch (buf.p) {
            case 1: rc = launch_m2m_fast<T, 1>(tree, buf, s); break;
            case 2: rc = launch_m2m_fast<T, 2>(tree, buf, s); break;
            case 3: rc = launch_m2m_fast<T, 3>(tree, buf, s); break;
            case 4: rc = launch_m2m_fast<T, 4>(tree, buf, s); break;
            case 5: rc = launch_m2m_fast<T, 5>(tree, buf, s); break;
            case 6: rc = launch_m2m_fast<T, 6>(tree, buf, s); break;
            case 7: rc = launch_m2m_fast<T, 7>(tree, buf, s); break;
            default: rc = launch_m2m_fast<T, 8>(tree, buf, s); break;
        }
        if (rc) return rc;
        EDFMM_LAUNCH_CHECK("k_m2m_fast");
        return EDFMM_OK;
    }
    for (int lev = tree.max_level - 1; lev >= 0; --lev) {
        const int lo = tree.level_offsets[lev], hi = tree.level_offsets[lev + 1];
        if (hi <= lo) continue;
        k_m2m<T><<<nblk(hi - lo, 4), 128, 0, s>>>(dptr<int32_t>(tree.level_nodes) + lo, hi - lo, dptr<uint8_t>(tree.is_leaf),
                                                  dptr<int32_t>(tree.children), dptr<T4>(tree.center), dptr<T4>(tree.half),
                                                  dptr<Cplx<T>>(buf.multipoles), buf.p, buf.nc_pad);
        EDFMM_LAUNCH_CHECK("k_m2m");
    }
    return EDFMM_OK;
}

template <typename T> int l2l_impl(const DevTree &tree, FmmBuffers &buf, cudaStream_t s) {
    using T4 = typename Vec4<T>::type;
    if (buf.p <= 8) {
        if (tree.max_level < 1) return EDFMM_OK;
        int rc;
        switch (buf.p) {
            case 1: rc = launch_l2l_fast<T, 1>(tree, buf, s); break;
            case 2: rc = launch_l2l_fast<T, 2>(tree, buf, s); break;
            case 3: rc = launch_l2l_fast<T, 3>(tree, buf, s); break;
            case 4: rc = launch_l2l_fast<T, 4>(tree, buf, s); break;
            case 5: rc = launch_l2l_fast<T, 5>(tree, buf, s); break;
            case 6: rc = launch_l2l_fast<T, 6>(tree, buf, s); break;
            case 7: rc = launch_l2l_fast<T, 7>(tree, buf, s); break;
            default: rc = launch_l2l_fast<T, 8>(tree, buf, s); break;
        }
        if (rc) return rc;
        EDFMM_LAUNCH_CHECK("k_l2l_fast");
        return EDFMM_OK;
    }
    for (int lev = 1; lev <= tree.max_level; ++lev) {
        const int lo = tree.level_offsets[lev], hi = tree.level_offsets[lev + 1];
        if (hi <= lo) continue;
        k_l2l<T><<<nblk(hi - lo, 4), 128, 0, s>>>(dptr<int32_t>(tree.level_nodes) + lo, hi - lo, dptr<int32_t>(tree.parent),
                                                  dptr<T4>(tree.center), dptr<T4>(tree.half), dptr<Cplx<T>>(buf.locals),
                                                  buf.p, buf.nc_pad);
        EDFMM_LAUNCH_CHECK("k_l2l");
    }
    return EDFMM_OK;
}

// extreme-pair CSR for one orientation (float plans only)
template <typename T4>
int build_extreme(const DevTree &tree, const DevTree &stree, const int32_t *off, const int32_t *src, ExtremeRows &ext,
                  cudaStream_t s) {
    int rc;
    const int64_t M = tree.n_nodes;
    DevBuf cnt, tmp, total, flag, pos;
    if ((rc = cnt.reserve(sizeof(int32_t) * M)) || (rc = ext.off.reserve(sizeof(int32_t) * (M + 1))) ||
        (rc = tmp.reserve(scan_tmp_bytes(M))) || (rc = total.reserve(sizeof(int64_t))))
        return rc;
    k_extreme_flags<T4><<<nblk(M * 32, 128), 128, 0, s>>>(M, off, src, dptr<T4>(tree.half), dptr<T4>(stree.half),
                                                      dptr<int32_t>(cnt));
    EDFMM_LAUNCH_CHECK("k_extreme_flags");
    if ((rc = scan_exclusive(dptr<int32_t>(cnt), dptr<int32_t>(ext.off), M, dptr<int64_t>(total), tmp.p, s))) return rc;
    k_set_last<<<1, 1, 0, s>>>(dptr<int32_t>(ext.off), M, dptr<int64_t>(total));
    EDFMM_LAUNCH_CHECK("k_set_last");
    int64_t n_ext = 0;
    EDFMM_CUDA_TRY(cudaMemcpyAsync(&n_ext, total.p, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    EDFMM_CUDA_TRY(cudaStreamSynchronize(s));
    ext.n_pairs = n_ext;
    ext.n_rows = 0;
    ext.built = true;
    if (n_ext == 0) return EDFMM_OK;
    if ((rc = ext.src.reserve(sizeof(int32_t) * n_ext)) || (rc = flag.reserve(sizeof(int32_t) * M)) ||
        (rc = pos.reserve(sizeof(int32_t) * M)) || (rc = ext.rows.reserve(sizeof(int32_t) * M)))
        return rc;
    k_extreme_fill<T4><<<nblk(M, 128), 128, 0, s>>>(M, off, src, dptr<T4>(tree.half), dptr<T4>(stree.half),
                                                 dptr<int32_t>(ext.off), dptr<int32_t>(ext.src));
    EDFMM_LAUNCH_CHECK("k_extreme_fill");
    k_flag_nonzero<<<nblk(M, 256), 256, 0, s>>>(M, dptr<int32_t>(cnt), dptr<int32_t>(flag));
    EDFMM_LAUNCH_CHECK("k_flag_nonzero");
    if ((rc = scan_exclusive(dptr<int32_t>(flag), dptr<int32_t>(pos), M, dptr<int64_t>(total), tmp.p, s))) return rc;
    k_nonempty_rows<<<nblk(M, 256), 256, 0, s>>>(M, dptr<int32_t>(cnt), dptr<int32_t>(pos), dptr<int32_t>(ext.rows));
    EDFMM_LAUNCH_CHECK("k_nonempty_rows");
    int64_t nr = 0;
    EDFMM_CUDA_TRY(cudaMemcpyAsync(&nr, total.p, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    EDFMM_CUDA_TRY(cudaStreamSynchronize(s));
    ext.n_rows = nr;
    return EDFMM_OK;
}

// M2L from the source tree's multipoles (sbuf) into the target tree's locals
// (tbuf); for one tree, tree == stree and sbuf == tbuf.
template <typename T>
int m2l_impl(const DevTree &tree, const DevTree &stree, const DevLists &lists, const FmmBuffers &sbuf,
             FmmBuffers &buf, bool swapped, bool alone, cudaStream_t s) {
    using T4 = typename Vec4<T>::type;
    const int64_t M = tree.n_nodes;
    if (M == 0 || stree.n_nodes == 0) return EDFMM_OK;
    const int32_t *off = swapped ? dptr<int32_t>(lists.m2l_swapped_off) : dptr<int32_t>(lists.m2l_off);
    const int32_t *src = swapped ? dptr<int32_t>(lists.m2l_swapped_src) : dptr<int32_t>(lists.m2l_src);
    const int32_t *rows = swapped ? nullptr : dptr<int32_t>(lists.m2l_rows);
    // alone, the column copy begins the chain, with an ordinary launch
    const bool chained = !alone && chain_tree(stree.n_nodes, stree.dtype, s);
    if (buf.p > kRotPMaxUsed) {
        // orders above 8: the shared-memory kernel (scales by the larger radius)
        k_m2l_generic<T><<<nblk(M, 4), 128, 0, s>>>(M, nullptr, off, src, dptr<T4>(tree.center), dptr<T4>(tree.half),
                                                    dptr<T4>(stree.center), dptr<T4>(stree.half),
                                                    dptr<Cplx<T>>(sbuf.multipoles), dptr<Cplx<T>>(buf.locals), buf.p,
                                                    buf.nc_pad, 0);
        EDFMM_LAUNCH_CHECK("k_m2l_generic");
        return EDFMM_OK;
    }
    // FP64 plans in two-float mode: the rotation kernel on the FP32 pipe
    // (orders 6..8), which leaves extreme pairs like the FP32 kernel does
    bool two_float = false;
    if (sizeof(T) == 8 && buf.arith == EDFMM_ARITH_TWO_FLOAT && buf.p >= 6 && buf.p <= 8 && tree.nodes_tf.p &&
        stree.nodes_tf.p && sbuf.mult_tf.p) {
        // the source multipoles split once per node, then the pairs
        if (int rc = mult_columns<true>(sbuf, stree.n_nodes, sbuf.mult_tf, chained, s)) return rc;
        int rc = launch_m2l_rot_tf(buf.p, M, off, src, rows, tree.nodes_tf.p, tree.half.p, stree.nodes_tf.p, stree.half.p,
                                   sbuf.mult_tf.p, buf.locals.p, buf.nc_pad, buf.mask, buf.m2l_tf_block,
                                   buf.m2l_packed != 0, s);
        if (rc == EDFMM_OK) two_float = true;
        else if (rc != EDFMM_ERR_UNSUPPORTED) return rc;
    }
    if (!two_float) {
        // FP32 reads the multipoles by columns; `translated` is free once M2M has run
        if constexpr (sizeof(T) == 4) {
            if (int rc = mult_columns<false>(sbuf, stree.n_nodes, sbuf.translated, chained, s)) return rc;
        }
        if (int rc = launch_m2l_rot(sizeof(T) == 8 ? EDFMM_F64 : EDFMM_F32, buf.p, M, off, src, rows, tree.center.p,
                                    tree.half.p, stree.center.p, stree.half.p,
                                    sizeof(T) == 8 ? sbuf.multipoles.p : sbuf.translated.p, buf.locals.p,
                                    buf.nc_pad, buf.mask, s))
            return rc;
        if (sizeof(T) == 8) return EDFMM_OK;  // FP64 has the range for any scale ratio the tree produces
    }
    // FP32 and two-float: pairs whose source scale exceeds 256x the target's, skipped above
    const T4 *tc = dptr<T4>(tree.center), *th = dptr<T4>(tree.half);
    const T4 *cen = dptr<T4>(stree.center), *hal = dptr<T4>(stree.half);
    ExtremeRows &ext = swapped ? buf.extreme_swapped : buf.extreme;
    if (!ext.built) {
        int rc = build_extreme<T4>(tree, stree, off, src, ext, s);
        if (rc) return rc;
    }
    if (ext.n_pairs > 0) {
        k_m2l_generic<T><<<nblk(ext.n_rows, 4), 128, 0, s>>>(
            ext.n_rows, dptr<int32_t>(ext.rows), dptr<int32_t>(ext.off), dptr<int32_t>(ext.src), tc, th, cen, hal,
            dptr<Cplx<T>>(sbuf.multipoles), dptr<Cplx<T>>(buf.locals), buf.p, buf.nc_pad, 1);
        EDFMM_LAUNCH_CHECK("k_m2l_generic");
    }
    return EDFMM_OK;
}

}  // namespace

int set_charges(const DevTree &tree, const void *a, const void *b, cudaStream_t s) {
    if (tree.n_points == 0) return EDFMM_OK;
    const unsigned grid = nblk(tree.n_points, 256);
    if (tree.dtype == EDFMM_F64)
        k_set_charges<double><<<grid, 256, 0, s>>>(dptr<double4>(tree.pts), dptr<float4>(tree.pts_grid), tree.grid_tf,
                                                   dptr<int32_t>(tree.index_map), tree.n_points,
                                                   static_cast<const double *>(a), static_cast<const double *>(b));
    else
        k_set_charges<float><<<grid, 256, 0, s>>>(dptr<float4>(tree.pts), nullptr, 0, dptr<int32_t>(tree.index_map),
                                                  tree.n_points, static_cast<const float *>(a),
                                                  static_cast<const float *>(b));
    EDFMM_LAUNCH_CHECK("k_set_charges");
    return EDFMM_OK;
}

bool chain_tree(int64_t n_nodes, int dtype, cudaStream_t s) {
    return n_nodes <= (dtype == EDFMM_F64 ? kChainNodes64 : kChainNodes32) && chain_stream(s);
}
bool chain_stream(cudaStream_t s) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(s, &st) == cudaSuccess && st == cudaStreamCaptureStatusNone;
}

int shift_prepare(DevTree &tree, cudaStream_t s) {
    return tree.dtype == EDFMM_F64 ? shift_prepare_impl<double>(tree, s) : shift_prepare_impl<float>(tree, s);
}

int run_p2m(const DevTree &tree, FmmBuffers &buf, cudaStream_t s) {
    return tree.dtype == EDFMM_F64 ? p2m_impl<double>(tree, buf, s) : p2m_impl<float>(tree, buf, s);
}
int run_m2m(const DevTree &tree, FmmBuffers &buf, cudaStream_t s) {
    return tree.dtype == EDFMM_F64 ? m2m_impl<double>(tree, buf, s) : m2m_impl<float>(tree, buf, s);
}
int run_m2l(const DevTree &tree, const DevLists &lists, FmmBuffers &buf, bool swapped, bool alone, cudaStream_t s) {
    return tree.dtype == EDFMM_F64 ? m2l_impl<double>(tree, tree, lists, buf, buf, swapped, alone, s)
                                   : m2l_impl<float>(tree, tree, lists, buf, buf, swapped, alone, s);
}
int run_m2l_two(const DevTree &tgt_tree, const DevTree &src_tree, const DevLists &lists, const FmmBuffers &src_buf,
                FmmBuffers &tgt_buf, bool alone, cudaStream_t s) {
    return tgt_tree.dtype == EDFMM_F64
               ? m2l_impl<double>(tgt_tree, src_tree, lists, src_buf, tgt_buf, false, alone, s)
               : m2l_impl<float>(tgt_tree, src_tree, lists, src_buf, tgt_buf, false, alone, s);
}
int prepare_two_float(DevTree &tree, FmmBuffers &buf, cudaStream_t s) {
    if (tree.dtype != EDFMM_F64) return EDFMM_OK;
    const int64_t M = std::max<int64_t>(tree.n_nodes, 1);
    int rc;
    if ((rc = tree.nodes_tf.reserve(sizeof(float4) * 2 * (size_t)M))) return rc;
    if ((rc = buf.mult_tf.reserve(sizeof(float4) * (size_t)buf.nc_pad * (size_t)padded_nodes(tree.n_nodes)))) return rc;
    if (tree.n_nodes > 0) {
        k_split_nodes<<<nblk(tree.n_nodes, 256), 256, 0, s>>>(dptr<double4>(tree.center), dptr<double4>(tree.half),
                                                              tree.n_nodes, dptr<float4>(tree.nodes_tf));
        EDFMM_LAUNCH_CHECK("k_split_nodes");
    }
    return EDFMM_OK;
}

int prepare_extreme_rows(const DevTree &tree, const DevLists &lists, FmmBuffers &buf, cudaStream_t s) {
    if (buf.extreme.built || tree.n_nodes == 0) return EDFMM_OK;
    const int32_t *off = dptr<int32_t>(lists.m2l_off), *src = dptr<int32_t>(lists.m2l_src);
    return tree.dtype == EDFMM_F64 ? build_extreme<double4>(tree, tree, off, src, buf.extreme, s)
                                   : build_extreme<float4>(tree, tree, off, src, buf.extreme, s);
}
int run_l2l(const DevTree &tree, FmmBuffers &buf, cudaStream_t s) {
    return tree.dtype == EDFMM_F64 ? l2l_impl<double>(tree, buf, s) : l2l_impl<float>(tree, buf, s);
}

}  // namespace edfmm
