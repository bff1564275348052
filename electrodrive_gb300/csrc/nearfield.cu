// Near field (P2P) and the local-expansion evaluation with the matvec
// epilogue (L2P).
//
// P2P is the reference's kernels_cpu.py:83-153 contribution
//     q_s / max(|x_t - x_s|, eps)   (eps = machine epsilon of the dtype)
// evaluated as q_s * rsqrt(max(r^2, eps^2)), with the diagonal dropped only
// inside the self leaf pair.  L2P evaluates the leaf's local expansion at its
// points, adds the near sums and, for a full matvec, applies the epilogue of
// bem_fmm.py:718-749 (K_E, original order, self term, non-finite -> 0), so
// each output is written exactly once.
#include <cfloat>
#include <climits>
#include <type_traits>

#include "edfmm_internal.cuh"
#include "gridpoint.cuh"
#include "harmonics.cuh"
#include "twofloat.cuh"

namespace edfmm {

namespace {

__constant__ float2 c_rdiv_tf[kPMax + 1][kPMax + 1];  // (hi, lo) of 1 / ((n + m)(n - m)), 1 / n^2 at m = 0

// ---------------------------------------------------------------------------
// P2P.  One warp owns up to 64 (split forms: 32) targets of a leaf (a whole
// leaf at the usual leaf sizes); with few leaves the four warps of a block share one leaf, each
// walking a quarter of its row.
//
// Lanes: the nt targets are held R per lane by L = ceil(nt / R) lanes, and
// G = 32 / L such groups of lanes split the sources.  R is chosen per nt (table
// below) for the least time per interaction: a source read from shared memory
// serves R targets, and few lanes idle whatever nt is.  20 targets: R = 2, ten
// lanes, three groups; one lane per target would leave a third of the warp idle.
//
// Sources: the leaves of a row hold about 20 to 40 points each, so their
// points are packed back to back into chunks of 64 or 128 staged in shared
// memory: the ranges of 32 row entries are scanned over the warp, and a
// position's entry is found by counting the entries that start at or before
// it (one OR-reduction and population count per 32 positions).  Staging one
// leaf at a time, the fixed work per leaf was about half of the kernel on
// surface meshes.
// Alone: FP32, 200k-panel torus 295 -> 143 us, a million points in a cube 2,352
// -> 1,738 us (16 rsqrt per SM and clock: 58 and 935 us).  The split forms
// (gridpoint.cuh) take two sources in packed operations: FP64, 20,011 points on
// a sphere 2,486 -> 277 scalar -> 246 us packed (the FMA pipe's time is 65 us:
// leaves of about 16 points, three waves of blocks); two-float, 50k-panel torus
// 1,089 -> 327 -> 261 us (the FMA pipe's time: 110 us).
// ---------------------------------------------------------------------------
enum NearMode {
    kF32,   // packed pairs of sources on the FP32 pipe
    kTF,    // FP64 plan in two-float mode: the split coordinates to two-float accuracy
    kGrid,  // FP64 on the FP32 pipe from exactly split coordinates (gridpoint.cuh)
    kIeee   // FP64 between two trees (no common grid)
};

constexpr int kNearWarps = 4;

template <int MODE> struct NearCfg;
template <> struct NearCfg<kF32> {
    using T = float;
    // RS: the values of R compiled (bit R); A + B R: issue slots per source step.
    // R = 2, 3, 4: with 5 and 6 too a million points take 1,722 instead of 1,738 us,
    // but the warps of an SM then run six copies of the loop, and on surface
    // leaves (200k-panel torus 190 instead of 143 us, 24 dimers 427 instead of
    // 326) the instruction fetches cost more than the idle lanes.
    static constexpr int W = 64, CH = 128, REC = 1, RS = 0x1c, A = 5, B = 11;
};
// The split forms take one target a lane, 32 a window: the packed coordinates
// of a target are 18 registers, so that R = 2 and 3 spill at four blocks per SM
// (R = 1, 2, 3: 261 and 279 us on the two shapes above; R = 1, 2: 255 and 261;
// R = 1: 246 and 261; five blocks per SM 265 and 269).
template <> struct NearCfg<kTF> {
    using T = double;
    static constexpr int W = 32, CH = 64, REC = 3, RS = 0x2, A = 6, B = 75;
};
template <> struct NearCfg<kGrid> {
    using T = double;
    static constexpr int W = 32, CH = 64, REC = 3, RS = 0x2, A = 6, B = 150;
};
template <> struct NearCfg<kIeee> {
    using T = double;
    static constexpr int W = 64, CH = 64, REC = 2, RS = 0xe, A = 5, B = 128;
};

// targets per lane for nt targets: the least (A + B R) / G with G = 32 / ceil(nt / R)
template <int MODE> struct NearShape {
    unsigned char r[65];
    constexpr NearShape() : r() {
        using C = NearCfg<MODE>;
        for (int nt = 0; nt <= 64; ++nt) {
            r[nt] = 0;
            long best = 1L << 60;
            for (int R = 1; R < 8; ++R) {
                const int L = (nt + R - 1) / R;
                if (!(C::RS >> R & 1) || L < 1 || L > 32) continue;
                const long cost = (C::A + C::B * R) * 100000L / (32 / L);
                if (cost < best) {
                    best = cost;
                    r[nt] = (unsigned char)R;
                }
            }
        }
    }
};
template <int MODE> __device__ const NearShape<MODE> d_near_shape{};

template <typename T> struct NearParams {
    const int32_t *leaves;
    int64_t n_leaves;
    const int32_t *off;
    const int32_t *src;
    const typename Vec4<T>::type *pts;   // targets
    const int2 *range;                   // target leaves' point ranges
    const typename Vec4<T>::type *spts;  // sources (== pts for one tree)
    const float4 *spts_split;            // kTF, kGrid: three float4 per point
    const GridInfo *grid;                // kTF, kGrid: one per instance
    const int32_t *inst_off;             // batched plans: first node of each instance (NULL: one tree)
    int n_inst;
    const int2 *srange;
    int same;  // one tree: drop i == j in self pairs
    T eps2;
    InstMask mask;  // batched plans: leaves of inactive instances are skipped
    T *out;         // near sums, tree order
};

// the part of a leaf's row a warp walks, 32 entries at a time
struct RowBatch {
    int first, len, total;  // this lane's entry: position of its first point, number of points; points of the batch
    int seen;               // entries with points that start before the next window
};

template <typename T>
__device__ __forceinline__ void load_batch(const NearParams<T> &P, int k0, int kend, int skip, int lane, int *soff,
                                           RowBatch &b, bool &self) {
    const int k = k0 + lane;
    const int s = k < kend ? P.src[k] : -1;
    const int2 r = s >= 0 ? P.srange[s] : make_int2(0, 0);
    b.len = r.y - r.x;
    if (s >= 0 && s == skip) {
        self = true;
        b.len = 0;
    }
    int incl = b.len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    b.first = incl - b.len;
    b.total = __shfl_sync(0xffffffffu, incl, 31);
    b.seen = 0;
    const unsigned nz = __ballot_sync(0xffffffffu, b.len > 0);
    __syncwarp();
    if (b.len > 0) soff[__popc(nz & ((1u << lane) - 1u))] = r.x - b.first;
    __syncwarp();
}

// source indices of positions w + 2 lane and w + 2 lane + 1 of the batch (-1
// past its end), for consecutive windows w = 0, 64, 128, ...
__device__ __forceinline__ void window_sources(RowBatch &b, int w, int lane, const int *soff, int &i0, int &i1) {
    const int t = b.first - w;
    const bool in = b.len > 0 && t >= 0;
    const unsigned m0 = __reduce_or_sync(0xffffffffu, in && t < 32 ? 1u << (t & 31) : 0u);
    const unsigned m1 = __reduce_or_sync(0xffffffffu, in && t >= 32 && t < 64 ? 1u << (t & 31) : 0u);
    const unsigned m = lane < 16 ? m0 : m1;
    const int p = (2 * lane) & 31;
    const int e0 = b.seen + (lane < 16 ? 0 : __popc(m0)) + __popc(m & ((2u << p) - 1u)) - 1;
    const int e1 = e0 + (int)((m >> (p + 1)) & 1u);
    b.seen += __popc(m0) + __popc(m1);
    const int q = w + 2 * lane;
    i0 = q < b.total ? soff[e0] + q : -1;
    i1 = q + 1 < b.total ? soff[e1] + q + 1 : -1;
}

// a lane's targets
template <int MODE, int R> struct Targets;
template <int R> struct Targets<kF32, R> {
    float2 nx[R], ny[R], nz[R];  // -x of the target, in both halves
    float acc[R];
};
template <int R> struct Targets<kTF, R> {
    GridCoordT<float2> x[R], y[R], z[R];  // in both halves
    double acc[R];
};
template <int R> struct Targets<kGrid, R> {
    GridCoordT<float2> x[R], y[R], z[R];
    double acc[R];
};
__device__ __forceinline__ GridCoordT<float2> grid_both(const GridCoord &g) {
    return GridCoordT<float2>{make_float2(g.a, g.a), make_float2(g.b, g.b), make_float2(g.c, g.c)};
}
template <int R> struct Targets<kIeee, R> {
    double x[R], y[R], z[R], acc[R];
};

// staged sources to registers (the lane's two sources of a window) and on to shared memory
template <int MODE> struct Staged;
template <> struct Staged<kF32> {
    float4 a, b;
};
template <> struct Staged<kIeee> {
    double4 a, b;
};
template <> struct Staged<kTF> {
    float4 a[3], b[3];
};
template <> struct Staged<kGrid> {
    float4 a[3], b[3];
};
template <int MODE, typename T>
__device__ __forceinline__ void fetch(const NearParams<T> &P, int i0, int i1, Staged<MODE> &f) {
    if constexpr (MODE == kF32) {
        const float4 z = make_float4(0, 0, 0, 0);
        f.a = i0 >= 0 ? P.spts[i0] : z;
        f.b = i1 >= 0 ? P.spts[i1] : z;
    } else if constexpr (MODE == kIeee) {
        f.a = i0 >= 0 ? P.spts[i0] : double4{0, 0, 0, 0};
        f.b = i1 >= 0 ? P.spts[i1] : double4{0, 0, 0, 0};
    } else {
        constexpr int N = NearCfg<MODE>::REC;
#pragma unroll
        for (int c = 0; c < N; ++c) {
            f.a[c] = i0 >= 0 ? P.spts_split[(int64_t)N * i0 + c] : make_float4(0, 0, 0, 0);
            f.b[c] = i1 >= 0 ? P.spts_split[(int64_t)N * i1 + c] : make_float4(0, 0, 0, 0);
        }
        f.a[2].y = __int_as_float(i0);
        f.b[2].y = __int_as_float(i1);
    }
}
template <int MODE> __device__ __forceinline__ void stage(float4 *buf, int pair, const Staged<MODE> &f) {
    if constexpr (MODE == kF32) {  // (x, x', y, y'), (z, z', q, q')
        buf[2 * pair] = make_float4(f.a.x, f.b.x, f.a.y, f.b.y);
        buf[2 * pair + 1] = make_float4(f.a.z, f.b.z, f.a.w, f.b.w);
    } else if constexpr (MODE == kIeee) {
        double4 *d = reinterpret_cast<double4 *>(buf);
        d[2 * pair] = f.a;
        d[2 * pair + 1] = f.b;
    } else {
        // value by value like the FP32 records: the nine parts of both sources,
        // both indices and the charges (kGrid: two doubles; kTF: (hi, hi', lo, lo'))
        float4 *d = buf + 6 * pair;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            d[2 * c] = make_float4(f.a[c].x, f.b[c].x, f.a[c].y, f.b[c].y);
            d[2 * c + 1] = make_float4(f.a[c].z, f.b[c].z, f.a[c].w, f.b[c].w);
        }
        d[4] = make_float4(f.a[2].x, f.b[2].x, f.a[2].y, f.b[2].y);
        d[5] = MODE == kGrid ? make_float4(f.a[2].z, f.a[2].w, f.b[2].z, f.b[2].w)
                             : make_float4(f.a[2].z, f.b[2].z, f.a[2].w, f.b[2].w);
    }
}

template <int MODE, int R, typename T>
__device__ __forceinline__ void load_target(const NearParams<T> &P, int ti, int r, const GridInfo &g, Targets<MODE, R> &X) {
    const typename Vec4<T>::type x = P.pts[ti];
    if constexpr (MODE == kF32) {
        X.nx[r] = make_float2(-x.x, -x.x);
        X.ny[r] = make_float2(-x.y, -x.y);
        X.nz[r] = make_float2(-x.z, -x.z);
        X.acc[r] = 0.0f;
    } else if constexpr (MODE == kTF || MODE == kGrid) {
        X.x[r] = grid_both(grid_split((x.x - g.center[0]) * g.down));
        X.y[r] = grid_both(grid_split((x.y - g.center[1]) * g.down));
        X.z[r] = grid_both(grid_split((x.z - g.center[2]) * g.down));
        X.acc[r] = 0.0;
    } else {
        X.x[r] = x.x;
        X.y[r] = x.y;
        X.z[r] = x.z;
        X.acc[r] = 0.0;
    }
}

__device__ __forceinline__ double inv_dist(double r2, double eps2) { return rsqrt(fmax(r2, eps2)); }

// kGrid: a pair too close for the split, in IEEE FP64 (scaled by 2^k)
__device__ __noinline__ double grid_pair_ieee(const double4 *pts, int s, int t, double eps2, double up) {
    if (s < 0 || s == t) return 0.0;
    const double4 a = pts[t], b = pts[s];
    const double dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
    return b.w * inv_dist(dx * dx + dy * dy + dz * dz, eps2) * up;
}

// hi + lo -= (qh + ql) (y0 + z), both halves; nq = -qh
__device__ __forceinline__ void grid_sub_tf(float2 qh, float2 nq, float2 ql, float2 y0, float2 z, float2 &hi, float2 &lo) {
    const float2 p = g_mul(nq, y0);
    const float2 e = g_fma(ql, y0, g_fma(qh, z, g_fma(qh, y0, p)));
    float2 s, f;
    grid_two_sum(hi, p, s, f);
    hi = s;
    lo = g_add(lo, g_sub(f, e));
}
// a staged pair of split sources
struct GridPair {
    GridCoordT<float2> x, y, z;
    float4 idx, q;  // (-, -, index, index'), charges
};
__device__ __forceinline__ GridPair grid_pair(const float4 *d) {
    const float4 a = d[0], b = d[1], c = d[2], e = d[3];
    GridPair p;
    p.idx = d[4];
    p.q = d[5];
    p.x = GridCoordT<float2>{make_float2(a.x, a.y), make_float2(a.z, a.w), make_float2(b.x, b.y)};
    p.y = GridCoordT<float2>{make_float2(b.z, b.w), make_float2(c.x, c.y), make_float2(c.z, c.w)};
    p.z = GridCoordT<float2>{make_float2(e.x, e.y), make_float2(e.z, e.w), make_float2(p.idx.x, p.idx.y)};
    return p;
}

// sources part, part + G, ... of a staged chunk of cnt sources; SELF: the
// chunk holds points sbase .. of the targets' own leaf, and t0 + L r is the
// lane's target r (of targets up to last)
template <int MODE, int R, bool SELF, typename T>
__device__ __forceinline__ void accumulate(const NearParams<T> &P, const float4 *buf, int cnt, int part, int G, int sbase,
                                           int t0, int L, int last, const GridInfo &g,
                                           Targets<MODE, R> &X) {
    if constexpr (MODE == kF32) {
        const float eps2 = P.eps2;
        float2 ps[R];
#pragma unroll
        for (int r = 0; r < R; ++r) ps[r] = make_float2(0.0f, 0.0f);
        const int np = (cnt + 1) >> 1;
#pragma unroll 2
        for (int j = part; j < np; j += G) {
            const float4 u = buf[2 * j], v = buf[2 * j + 1];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float2 dx = __fadd2_rn(make_float2(u.x, u.y), X.nx[r]),
                             dy = __fadd2_rn(make_float2(u.z, u.w), X.ny[r]),
                             dz = __fadd2_rn(make_float2(v.x, v.y), X.nz[r]);
                const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
                float i0 = rsqrt_normal(fmaxf(r2.x, eps2)), i1 = rsqrt_normal(fmaxf(r2.y, eps2));
                if (SELF) {
                    if (sbase + 2 * j == t0 + L * r) i0 = 0.0f;
                    if (sbase + 2 * j + 1 == t0 + L * r) i1 = 0.0f;
                }
                ps[r] = __ffma2_rn(make_float2(v.z, v.w), make_float2(i0, i1), ps[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) X.acc[r] += ps[r].x + ps[r].y;  // per-chunk partial, then one add
    } else if constexpr (MODE == kTF) {
        float2 hi[R], lo[R];  // minus a chunk's sums, hi + lo, of at most 32 terms each; then FP64
        double ps[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            hi[r] = lo[r] = make_float2(0.0f, 0.0f);
            ps[r] = 0.0;
        }
        const int np = (cnt + 1) >> 1;
        for (int j = part; j < np; j += G) {
            const GridPair s = grid_pair(buf + 6 * j);
            const float2 qh = make_float2(s.q.x, s.q.y), ql = make_float2(s.q.z, s.q.w), nq = g_neg(qh);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                float2 N, y0, z;
                const float2 R1 = grid_r2_tf(grid_diff2(X.x[r], s.x), grid_diff2(X.y[r], s.y), grid_diff2(X.z[r], s.z), N);
                float2 h = qh, m = nq, l = ql;
                grid_rsqrt_tf(R1, N, y0, z);
                if (!(fminf(R1.x, R1.y) >= g.near2)) {  // the target itself, or a pair the split does not resolve
                    const int t = min(t0 + L * r, last);
                    if (!(R1.x >= g.near2)) {
                        ps[r] += grid_pair_ieee(P.pts, __float_as_int(s.idx.z), t, P.eps2, g.up);
                        h.x = m.x = l.x = y0.x = z.x = 0.0f;
                    }
                    if (!(R1.y >= g.near2)) {
                        ps[r] += grid_pair_ieee(P.pts, __float_as_int(s.idx.w), t, P.eps2, g.up);
                        h.y = m.y = l.y = y0.y = z.y = 0.0f;
                    }
                }
                grid_sub_tf(h, m, l, y0, z, hi[r], lo[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
            X.acc[r] += ps[r] - (((double)hi[r].x + (double)lo[r].x) + ((double)hi[r].y + (double)lo[r].y));
    } else if constexpr (MODE == kGrid) {
        double ps[R];
#pragma unroll
        for (int r = 0; r < R; ++r) ps[r] = 0.0;
        const int np = (cnt + 1) >> 1;
        for (int j = part; j < np; j += G) {
            const GridPair s = grid_pair(buf + 6 * j);
            const double wa = __hiloint2double(__float_as_int(s.q.y), __float_as_int(s.q.x)),
                         wb = __hiloint2double(__float_as_int(s.q.w), __float_as_int(s.q.z));
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const GridR2<float2> r2 =
                    grid_r2(grid_diff(X.x[r], s.x), grid_diff(X.y[r], s.y), grid_diff(X.z[r], s.z));
                float2 y0, eh, v;
                grid_rsqrt(r2, y0, eh, v);
                if (!(fminf(r2.R1.x, r2.R1.y) >= g.near2)) {  // the target itself, or a pair the split does not resolve
                    const int t = min(t0 + L * r, last);
                    if (!(r2.R1.x >= g.near2)) ps[r] += grid_pair_ieee(P.pts, __float_as_int(s.idx.z), t, P.eps2, g.up);
                    else ps[r] = fma(wa, grid_inv(y0.x, grid_ci(eh.x, v.x)), ps[r]);
                    if (!(r2.R1.y >= g.near2)) ps[r] += grid_pair_ieee(P.pts, __float_as_int(s.idx.w), t, P.eps2, g.up);
                    else ps[r] = fma(wb, grid_inv(y0.y, grid_ci(eh.y, v.y)), ps[r]);
                } else {
                    ps[r] = fma(wa, grid_inv(y0.x, grid_ci(eh.x, v.x)), ps[r]);
                    ps[r] = fma(wb, grid_inv(y0.y, grid_ci(eh.y, v.y)), ps[r]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) X.acc[r] += ps[r];
    } else {
        const double eps2 = P.eps2;
        const double4 *sp = reinterpret_cast<const double4 *>(buf);
        double ps[R];
#pragma unroll
        for (int r = 0; r < R; ++r) ps[r] = 0.0;
        for (int j = part; j < cnt; j += G) {
            const double4 q = sp[j];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const double dx = X.x[r] - q.x, dy = X.y[r] - q.y, dz = X.z[r] - q.z;
                double inv = inv_dist(dx * dx + dy * dy + dz * dz, eps2);
                if (SELF && sbase + j == t0 + L * r) inv = 0.0;
                ps[r] += q.w * inv;
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) X.acc[r] += ps[r];
    }
}

// targets tb .. tb + nt - 1 of leaf t; WPL warps share them (this is warp
// `wid` of the block)
template <int MODE, int R, int WPL, typename T>
__device__ __forceinline__ void near_targets(const NearParams<T> &P, int t, int tb, int nt, int2 rg, int wid,
                                             float4 *buf, int *soff, T *part, const GridInfo &g) {
    using C = NearCfg<MODE>;
    constexpr int NW = C::CH / 64;  // windows per chunk
    const int lane = threadIdx.x & 31;
    const int L = (nt + R - 1) / R, G = 32 / L;
    const int grp = lane / L, l = lane - grp * L;
    Targets<MODE, R> X;
#pragma unroll
    for (int r = 0; r < R; ++r) load_target<MODE, R>(P, tb + min(l + L * r, nt - 1), r, g, X);
    const int t0 = tb + l;
    const int first = grp < G ? grp : C::CH;  // lanes beyond the last group take no source
    int kbeg = P.off[t], kend = P.off[t + 1];
    if constexpr (WPL > 1) {
        const int per = (kend - kbeg + WPL - 1) / WPL;
        kbeg = min(kend, kbeg + wid * per);
        kend = min(kend, kbeg + per);
    }
    // the split forms drop the diagonal through their close-pair test
    const int skip = MODE != kGrid && MODE != kTF && P.same ? t : -2;
    bool self = false;
    for (int k0 = kbeg; k0 < kend; k0 += 32) {
        RowBatch b;
        load_batch(P, k0, kend, skip, lane, soff, b, self);
        Staged<MODE> f[NW];
#pragma unroll
        for (int i = 0; i < NW; ++i) {
            int i0, i1;
            window_sources(b, 64 * i, lane, soff, i0, i1);
            fetch<MODE>(P, i0, i1, f[i]);
        }
        for (int c = 0; c < b.total; c += C::CH) {
            __syncwarp();
#pragma unroll
            for (int i = 0; i < NW; ++i) stage<MODE>(buf, lane + 32 * i, f[i]);
            __syncwarp();
            if (c + C::CH < b.total) {  // the next chunk's points are loaded behind this one's arithmetic
#pragma unroll
                for (int i = 0; i < NW; ++i) {
                    int i0, i1;
                    window_sources(b, c + C::CH + 64 * i, lane, soff, i0, i1);
                    fetch<MODE>(P, i0, i1, f[i]);
                }
            }
            accumulate<MODE, R, false>(P, buf, min(C::CH, b.total - c), first, G, 0, t0, L, tb + nt - 1, g, X);
        }
    }
    if (__any_sync(0xffffffffu, self)) {
        for (int sb = rg.x; sb < rg.y; sb += C::CH) {
            __syncwarp();
#pragma unroll
            for (int i = 0; i < NW; ++i) {
                const int q = sb + 64 * i + 2 * lane;
                Staged<MODE> f;
                fetch<MODE>(P, q < rg.y ? q : -1, q + 1 < rg.y ? q + 1 : -1, f);
                stage<MODE>(buf, lane + 32 * i, f);
            }
            __syncwarp();
            accumulate<MODE, R, true>(P, buf, min(C::CH, rg.y - sb), first, G, sb, t0, L, tb + nt - 1, g, X);
        }
    }
    // the groups' sums per target, in group order (and in warp order)
    __syncwarp();
    T *red = reinterpret_cast<T *>(buf);  // G * nt <= 32 R values
    if (grp < G) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (l + L * r >= nt) continue;
            T v;
            if constexpr (MODE == kTF || MODE == kGrid) v = X.acc[r] * g.down;
            else v = X.acc[r];
            red[grp * nt + l + L * r] = v;
        }
    }
    __syncwarp();
    for (int i = lane; i < nt; i += 32) {
        T v = red[i];
        for (int q = 1; q < G; ++q) v += red[q * nt + i];
        if constexpr (WPL > 1) part[wid * 64 + i] = v;
        else P.out[tb + i] = v;
    }
    if constexpr (WPL > 1) {
        __syncthreads();
        for (int i = threadIdx.x; i < nt; i += 32 * WPL) {
            T v = part[i];
#pragma unroll
            for (int q = 1; q < WPL; ++q) v += part[q * 64 + i];
            P.out[tb + i] = v;
        }
        __syncthreads();
    } else {
        __syncwarp();
    }
}

template <int MODE> __host__ __device__ constexpr int near_blocks() { return MODE == kF32 ? 5 : 4; }

template <int MODE, int WPL>
__global__ void __launch_bounds__(32 * kNearWarps, near_blocks<MODE>())
    k_p2p(const NearParams<typename NearCfg<MODE>::T> P) {
    using C = NearCfg<MODE>;
    using T = typename C::T;
    __shared__ float4 buf[kNearWarps][C::CH * C::REC];
    __shared__ int soff[kNearWarps][32];
    __shared__ T part[WPL > 1 ? WPL * 64 : 1];
    const int wid = threadIdx.x >> 5;
    const int64_t w = WPL > 1 ? (int64_t)blockIdx.x : (int64_t)blockIdx.x * kNearWarps + wid;
    if (w >= P.n_leaves) return;
    const int t = P.leaves[w];
    if (!inst_active(P.mask, t)) return;  // uniform over the warps that share a leaf
    const int2 rg = P.range[t];
    GridInfo g{};
    if constexpr (MODE == kGrid || MODE == kTF) g = P.grid[instance_of_node(P.inst_off, P.n_inst, t)];
    for (int tb = rg.x; tb < rg.y; tb += C::W) {
        const int nt = min(C::W, rg.y - tb);
        const int R = d_near_shape<MODE>.r[nt];
#define EDFMM_NEAR_R(RR)                                                                                     \
    if constexpr ((C::RS >> RR) & 1) {                                                                           \
        if (R == RR) near_targets<MODE, RR, WPL>(P, t, tb, nt, rg, wid, buf[wid], soff[wid], part, g);       \
    }
        EDFMM_NEAR_R(1)
        EDFMM_NEAR_R(2)
        EDFMM_NEAR_R(3)
        EDFMM_NEAR_R(4)
#undef EDFMM_NEAR_R
    }
}

// ---------------------------------------------------------------------------
// L2P and epilogue: one warp per leaf, one lane per target
// ---------------------------------------------------------------------------
// Re sum_{n,m} L_n^m R_n^m(x, y, z) over m in [-n, n].  R_n^m = R_m^m rho_n with a
// real rho (rho_m = 1), so that a term takes five operations (three of the
// recursion, two sums) and a column one complex product at its end, where the
// complex recursion took nine a term.  FP64, 1,254 leaves 69 -> 47 us; two-float,
// 2,468 leaves 52 -> 41; FP32, 29,158 leaves at order 6 32 -> 26.
template <typename T, int P, int M>
__device__ __forceinline__ T l2p_columns(const Cplx<T> *L, T x, T y, T r2, const T (&zc)[P + 1], T dr, T di, T acc) {
    Cplx<T> lv = L[tri(M, M)];
    T re = lv.re, im = lv.im, rho = (T)1, last = (T)0;
#pragma unroll
    for (int n = M + 1; n <= P; ++n) {
        const T d = (T)(1.0 / ((n + M) * (n - M)));
        const T next = (n == M + 1 ? zc[n] : zc[n] * rho - r2 * last) * d;
        last = rho;
        rho = next;
        lv = L[tri(n, M)];
        re += lv.re * rho;
        if (M > 0) im += lv.im * rho;
    }
    acc += M == 0 ? re : (T)2 * (re * dr - im * di);
    if constexpr (M < P) {
        constexpr double c = -0.5 / (M + 1);
        const T sx = (T)c * x, sy = (T)c * y;
        return l2p_columns<T, P, M + 1>(L, x, y, r2, zc, M == 0 ? sx : sx * dr - sy * di,
                                        M == 0 ? sy : sx * di + sy * dr, acc);
    } else {
        return acc;
    }
}
template <typename T, int P>
__device__ __forceinline__ T l2p_point(const Cplx<T> *L, T x, T y, T z) {
    T zc[P + 1];
#pragma unroll
    for (int n = 1; n <= P; ++n) zc[n] = (T)(2 * n - 1) * z;
    return l2p_columns<T, P, 0>(L, x, y, x * x + y * y + z * z, zc, (T)1, (T)0, (T)0);
}

// l2p_point in two-float arithmetic, on two-float locals
__device__ __forceinline__ tf32x2 l2p_point_tf(const tf32x2c *L, int p, tf32x2 x, tf32x2 y, tf32x2 z) {
    using T = tf32x2;
    const T r2 = fma(z, z, fma(y, y, x * x)), n2 = -r2;
    T acc = T(0), dr = T(1), di = T(0);
    for (int m = 0; m <= p; ++m) {
        if (m > 0) {
            const float2 rd = c_rdiv_tf[m][0];
            const T sc = T(rd.x, rd.y) * T(-m) * T(0.5);  // -1 / (2m)
            const T nr = sc * (x * dr - y * di), ni = sc * (x * di + y * dr);
            dr = nr;
            di = ni;
        }
        tf32x2c lv = L[tri(m, m)];
        T re = lv.x, im = lv.y, rho = T(1), last = T(0);
        for (int n = m + 1; n <= p; ++n) {
            const float2 rd = c_rdiv_tf[n][m];
            const T next = fma(T(2 * n - 1) * z, rho, n2 * last) * T(rd.x, rd.y);
            last = rho;
            rho = next;
            lv = L[tri(n, m)];
            re = fma(lv.x, rho, re);
            im = fma(lv.y, rho, im);
        }
        const T col = re * dr - im * di;
        acc = m == 0 ? acc + col : acc + T(2) * col;
    }
    return acc;
}

template <typename T> struct L2pParams {
    const int32_t *leaves;
    int64_t n_leaves;
    const typename Vec4<T>::type *pts;
    const int2 *range;
    const typename Vec4<T>::type *center;
    const typename Vec4<T>::type *half;
    const Cplx<T> *Lexp;
    int nc_pad;
    int far;          // 0: the epilogue alone
    const T *add_in;  // near sums, tree order (nullable)
    InstMask mask;
    // epilogue
    int scatter;
    const int32_t *index_map;
    const T *sigma;
    const T *areas;
    const T *self_int;
    T k_e;
    T *out;
};

template <typename T, bool TF, int PP>
__global__ void __launch_bounds__(128) k_l2p(const L2pParams<T> P) {
    using T4 = typename Vec4<T>::type;
    constexpr int NC = ncoef(PP);
    __shared__ Cplx<T> sL[4][NC];
    const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t w = (int64_t)blockIdx.x * 4 + wl;
    if (w >= P.n_leaves) return;
    const int t = P.leaves[w];
    if (!inst_active(P.mask, t)) return;
    T4 c{};
    T ia = (T)1;
    if (P.far) {
        for (int k = lane; k < NC; k += 32) {
            const Cplx<T> v = P.Lexp[(int64_t)t * P.nc_pad + k];
            if constexpr (TF)  // staged as two-float (the same 16 bytes per coefficient)
                reinterpret_cast<tf32x2c *>(sL[wl])[k] = tf32x2c{tf_from_double(v.re), tf_from_double(v.im)};
            else
                sL[wl][k] = v;
        }
        c = P.center[t];
        ia = (T)1 / P.half[t].w;
        __syncwarp();
    }
    const int2 rg = P.range[t];
    for (int ti = rg.x + lane; ti < rg.y; ti += 32) {
        T v = P.add_in ? P.add_in[ti] : (T)0;
        if (P.far) {
            const T4 x = P.pts[ti];
            if constexpr (TF)
                v += tf_to_double(l2p_point_tf(reinterpret_cast<const tf32x2c *>(sL[wl]), PP,
                                               tf_from_double((x.x - c.x) * ia), tf_from_double((x.y - c.y) * ia),
                                               tf_from_double((x.z - c.z) * ia)));
            else
                v += l2p_point<T, PP>(sL[wl], (x.x - c.x) * ia, (x.y - c.y) * ia, (x.z - c.z) * ia);
        }
        if (P.scatter) {
            const int o = P.index_map[ti];
            v = v * P.k_e;
            if (P.self_int) v += P.self_int[o] * P.sigma[o] * P.areas[o];
            if (!isfinite(v)) v = (T)0;
            P.out[o] = v;
        } else {
            P.out[ti] = v;
        }
    }
}

// ---------------------------------------------------------------------------
// FP64 trees: the exact split of the points (gridpoint.cuh)
// ---------------------------------------------------------------------------
// A batched plan has one scale per instance, so that each instance's results are
// those of its own plan.  node_off NULL: one tree.
__device__ __forceinline__ int instance_of_point(const int32_t *node_off, int n_inst, const int2 *range, int64_t i) {
    if (!node_off) return 0;
    int lo = 0, hi = n_inst - 1;  // last instance whose root's points start at or before i
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (range[node_off[mid]].x <= i) lo = mid; else hi = mid - 1;
    }
    return lo;
}
// doubles to integers of the same order (NaN beyond the infinity of its sign)
__device__ __forceinline__ long long ord_of(double x) {
    const long long i = __double_as_longlong(x);
    return i >= 0 ? i : i ^ 0x7fffffffffffffffLL;
}
__device__ __forceinline__ double from_ord(long long i) {
    return __longlong_as_double(i >= 0 ? i : i ^ 0x7fffffffffffffffLL);
}
// memset's pattern for "no point yet": below every number of a usable scale
constexpr int kNoExtent = 0x80;

__global__ void k_grid_extent(const double4 *__restrict__ pts, int64_t n, const int32_t *node_off, int n_inst,
                              const int2 *__restrict__ range, GridInfo *info) {
    // a block takes a run of points, mostly of one instance; a thread adds its
    // points up as long as the instance stays the same
    const int64_t per = (n + gridDim.x - 1) / gridDim.x, b = blockIdx.x * per, e = min(n, b + per);
    long long m[6] = {LLONG_MIN, LLONG_MIN, LLONG_MIN, LLONG_MIN, LLONG_MIN, LLONG_MIN};
    int k = -1;  // none yet, or past the end
    auto flush = [&] {  // the warp's extents of its instance, or a lane's own
        const int k0 = __shfl_sync(0xffffffffu, k, 0);
        const bool one = __all_sync(0xffffffffu, k == k0 || k < 0);
#pragma unroll
        for (int a = 0; a < 6; ++a) {
            long long v = m[a];
            if (one) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v = max(v, (long long)__shfl_xor_sync(0xffffffffu, v, o));
            }
            if (k >= 0 && (!one || (threadIdx.x & 31) == 0)) atomicMax(&info[k].ext[a], v);
        }
    };
    for (int64_t i0 = b; i0 < e; i0 += blockDim.x) {
        const int64_t i = i0 + threadIdx.x;
        const int ki = i < e ? instance_of_point(node_off, n_inst, range, i) : k;
        if (__any_sync(0xffffffffu, ki != k)) {
            flush();
            k = ki;
#pragma unroll
            for (int a = 0; a < 6; ++a) m[a] = LLONG_MIN;
        }
        if (i < e) {
            const double4 p = pts[i];
            const double x[3] = {p.x, p.y, p.z};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                m[a] = max(m[a], ord_of(x[a]));
                m[3 + a] = max(m[3 + a], ord_of(-x[a]));
            }
        }
    }
    flush();
}
// Each frame from its points' extents.  An axis on which the points lie within a
// sixteenth of their distance from the origin has its centre at the nearest of
// them: a coordinate and the centre are then within a factor of two of one
// another, so that their difference is exact, and the scale is that of the
// extent.  Without it a geometry far from the origin has all its near pairs
// closer than the split resolves, each formed a second time in IEEE FP64 (20,011
// points on a sphere at x = 1e6, two-float: 1,590 us against 148 at the origin).
// The scale of an axis without a centre is at most 2^4 times its extent.
__global__ void k_grid_frames(int n_inst, GridInfo *info) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_inst) return;
    unsigned reach = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double hi = from_ord(info[i].ext[a]), lo = -from_ord(info[i].ext[3 + a]);
        const double c = lo > 0.0 && hi <= 1.0625 * lo ? lo : hi < 0.0 && lo >= 1.0625 * hi ? hi : 0.0;
        info[i].center[a] = c;
        reach = max(reach, (unsigned)__double2hiint(hi - c) & 0x7fffffffu);
        reach = max(reach, (unsigned)__double2hiint(lo - c) & 0x7fffffffu);
    }
    int k;
    const bool ok = grid_exponent(reach, k);
    if (!ok) k = 0;
    info[i].down = grid_pow2(-k);
    info[i].up = grid_pow2(k);
    // without a usable scale every pair is evaluated in IEEE FP64: no r^2 is >= NaN
    info[i].near2 =
        ok ? fmaxf(kGridNear2, (float)(1.0001 * DBL_EPSILON * DBL_EPSILON * info[i].down * info[i].down)) : NAN;
}
// three float4 per point: (xa, xb, xc, ya), (yb, yc, za, zb), (zc, -, charge);
// set_charges writes the charge
__global__ void k_grid_points(const double4 *__restrict__ pts, int64_t n, const int32_t *node_off, int n_inst,
                              const int2 *__restrict__ range, const GridInfo *__restrict__ info,
                              float4 *__restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const GridInfo g = info[instance_of_point(node_off, n_inst, range, i)];
    const double4 p = pts[i];
    GridCoord x{}, y{}, z{};
    if (g.near2 >= 0.0f) {  // not NaN
        x = grid_split((p.x - g.center[0]) * g.down);
        y = grid_split((p.y - g.center[1]) * g.down);
        z = grid_split((p.z - g.center[2]) * g.down);
    }
    out[3 * i] = make_float4(x.a, x.b, x.c, y.a);
    out[3 * i + 1] = make_float4(y.b, y.c, z.a, z.b);
    out[3 * i + 2] = make_float4(z.c, 0.0f, 0.0f, 0.0f);
}

}  // namespace

// The split points of an FP64 tree (48 bytes per point), without their charges
int grid_prepare(DevTree &tree, cudaStream_t s) {
    if (tree.dtype != EDFMM_F64 || tree.n_points == 0) return EDFMM_OK;
    int rc;
    const int K = std::max(tree.n_inst, 1);
    if ((rc = tree.pts_grid.reserve(sizeof(float4) * 3 * (size_t)tree.n_points)) ||
        (rc = tree.grid_info.reserve(sizeof(GridInfo) * (size_t)K)))
        return rc;
    GridInfo *info = dptr<GridInfo>(tree.grid_info);
    const int32_t *node_off = tree.n_inst > 0 ? dptr<int32_t>(tree.inst_node_off) : nullptr;
    const int2 *range = dptr<int2>(tree.range);
    EDFMM_CUDA_TRY(cudaMemsetAsync(info, kNoExtent, sizeof(GridInfo) * (size_t)K, s));
    const int64_t nb = (tree.n_points + 255) / 256;
    k_grid_extent<<<(unsigned)(nb < 608 ? nb : 608), 256, 0, s>>>(dptr<double4>(tree.pts), tree.n_points, node_off, K,
                                                                  range, info);
    EDFMM_LAUNCH_CHECK("k_grid_extent");
    k_grid_frames<<<(unsigned)((K + 127) / 128), 128, 0, s>>>(K, info);
    EDFMM_LAUNCH_CHECK("k_grid_frames");
    k_grid_points<<<(unsigned)nb, 256, 0, s>>>(dptr<double4>(tree.pts), tree.n_points, node_off, K, range, info,
                                               dptr<float4>(tree.pts_grid));
    EDFMM_LAUNCH_CHECK("k_grid_points");
    return EDFMM_OK;
}

// The two-float table; __constant__ data lives in each device context, so
// every plan creation uploads it on its device.
int upload_tables() {
    float2 ht[kPMax + 1][kPMax + 1];
    for (int n = 0; n <= kPMax; ++n)
        for (int m = 0; m <= kPMax; ++m) {
            int d = (n + m) * (n - m);
            if (m == 0 && n > 0) d = n * n;
            const double v = d != 0 ? 1.0 / d : 0.0;
            ht[n][m].x = (float)v;
            ht[n][m].y = (float)(v - (double)ht[n][m].x);
        }
    EDFMM_CUDA_TRY(cudaMemcpyToSymbol(c_rdiv_tf, ht, sizeof(ht)));
    return EDFMM_OK;
}

namespace {

// Below this many leaves the four warps of a block share a leaf.  With one warp
// per leaf 2,003 points (64 leaves) keep 64 warps busy: 84 us against 23.  The
// FP64 forms take ten times as long per interaction, so their last wave
// weighs more: 2,468 leaves in two-float (at 106 operations an interaction)
// 874 us with a warp per leaf, 406 shared; FP32 with 9,856 leaves 143 and 162 us.
template <int MODE> constexpr int64_t shared_leaves() { return MODE == kF32 ? 152 * 16 : 152 * 64; }

template <int MODE, typename T> int near_launch(const NearParams<T> &P, cudaStream_t s) {
    if (P.n_leaves < shared_leaves<MODE>())
        k_p2p<MODE, kNearWarps><<<(unsigned)P.n_leaves, 32 * kNearWarps, 0, s>>>(P);
    else
        k_p2p<MODE, 1><<<(unsigned)((P.n_leaves + kNearWarps - 1) / kNearWarps), 32 * kNearWarps, 0, s>>>(P);
    EDFMM_LAUNCH_CHECK("k_p2p");
    return EDFMM_OK;
}

template <typename T>
int near_impl(const DevTree &tree, const DevLists &lists, const FmmBuffers &buf, const DevTree *src_tree, void *out,
              cudaStream_t s) {
    using T4 = typename Vec4<T>::type;
    if (tree.n_leaves == 0) return EDFMM_OK;
    NearParams<T> P{};
    P.leaves = lists.p2p_leaves.p ? dptr<int32_t>(lists.p2p_leaves) : dptr<int32_t>(tree.leaves);
    P.n_leaves = tree.n_leaves;
    P.off = dptr<int32_t>(lists.p2p_off);
    P.src = dptr<int32_t>(lists.p2p_src);
    P.pts = dptr<T4>(tree.pts);
    P.range = dptr<int2>(tree.range);
    P.spts = src_tree ? dptr<T4>(src_tree->pts) : P.pts;
    P.srange = src_tree ? dptr<int2>(src_tree->range) : P.range;
    P.same = src_tree ? 0 : 1;
    const T eps = sizeof(T) == 8 ? (T)DBL_EPSILON : (T)FLT_EPSILON;
    P.eps2 = eps * eps;
    P.mask = src_tree ? InstMask{} : buf.mask;
    P.out = static_cast<T *>(out);
    if constexpr (sizeof(T) == 4) {
        return near_launch<kF32>(P, s);
    } else {
        if (src_tree) return near_launch<kIeee>(P, s);
        P.spts_split = dptr<float4>(tree.pts_grid);
        P.grid = dptr<GridInfo>(tree.grid_info);
        P.inst_off = tree.n_inst > 0 ? dptr<int32_t>(tree.inst_node_off) : nullptr;
        P.n_inst = tree.n_inst;
        return tree.grid_tf ? near_launch<kTF>(P, s) : near_launch<kGrid>(P, s);
    }
}

template <typename T>
int l2p_impl(const DevTree &tree, const FmmBuffers &buf, const L2pArgs &a, cudaStream_t s) {
    using T4 = typename Vec4<T>::type;
    if (tree.n_leaves == 0) return EDFMM_OK;
    L2pParams<T> P{};
    P.leaves = dptr<int32_t>(tree.leaves);
    P.n_leaves = tree.n_leaves;
    P.pts = dptr<T4>(tree.pts);
    P.range = dptr<int2>(tree.range);
    P.center = dptr<T4>(tree.center);
    P.half = dptr<T4>(tree.half);
    P.Lexp = dptr<Cplx<T>>(buf.locals);
    P.nc_pad = buf.nc_pad;
    P.far = a.far ? 1 : 0;
    P.add_in = static_cast<const T *>(a.add_in);
    P.mask = buf.mask;
    P.scatter = a.scatter ? 1 : 0;
    P.index_map = dptr<int32_t>(tree.index_map);
    P.sigma = static_cast<const T *>(a.sigma);
    P.areas = static_cast<const T *>(a.areas);
    P.self_int = static_cast<const T *>(a.self_int);
    P.k_e = (T)a.k_e;
    P.out = static_cast<T *>(a.out);
    const unsigned grid = (unsigned)((tree.n_leaves + 3) / 4);
    const bool tf = sizeof(T) == 8 && buf.arith == EDFMM_ARITH_TWO_FLOAT;
    switch (buf.p) {
#define EDFMM_L2P_CASE(PP)                                                  \
    case PP:                                                                \
        if (sizeof(T) == 8 && tf) k_l2p<T, (sizeof(T) == 8), PP><<<grid, 128, 0, s>>>(P); \
        else k_l2p<T, false, PP><<<grid, 128, 0, s>>>(P);                   \
        break;
        EDFMM_L2P_CASE(1)
        EDFMM_L2P_CASE(2)
        EDFMM_L2P_CASE(3)
        EDFMM_L2P_CASE(4)
        EDFMM_L2P_CASE(5)
        EDFMM_L2P_CASE(6)
        EDFMM_L2P_CASE(7)
        EDFMM_L2P_CASE(8)
        EDFMM_L2P_CASE(9)
        EDFMM_L2P_CASE(10)
#undef EDFMM_L2P_CASE
        default:
            return fail(EDFMM_ERR_UNSUPPORTED, "expansion order out of range");
    }
    EDFMM_LAUNCH_CHECK("k_l2p");
    return EDFMM_OK;
}

}  // namespace

int run_p2p(const DevTree &tree, const DevLists &lists, const FmmBuffers &buf, const DevTree *src_tree, void *out,
            cudaStream_t s) {
    return tree.dtype == EDFMM_F64 ? near_impl<double>(tree, lists, buf, src_tree, out, s)
                                   : near_impl<float>(tree, lists, buf, src_tree, out, s);
}

int run_l2p(const DevTree &tree, const FmmBuffers &buf, const L2pArgs &args, cudaStream_t s) {
    return tree.dtype == EDFMM_F64 ? l2p_impl<double>(tree, buf, args, s) : l2p_impl<float>(tree, buf, args, s);
}

namespace {

// Gradient of the local expansion sum_{n,m} w_m Re(L_n^m R_n^m(x, y, z))
// (w_0 = 1, w_m = 2) in the node's scaled frame, from
//   d/dz R_n^m = R_{n-1}^m,  (d/dx + i d/dy) R_n^m = R_{n-1}^{m+1},
//   (d/dx - i d/dy) R_n^m = -R_{n-1}^{m-1}
// (negative orders through R^{-m} = (-1)^m conj(R^m)).
template <typename T>
__device__ void l2p_gradient(const Cplx<T> *L, int p, T x, T y, T z, T &gx, T &gy, T &gz) {
    Cplx<T> R[ncoef(kPMax - 1)];
    gx = gy = gz = (T)0;
    if (p < 1) return;
    regular_harmonics_rt<T>(x, y, z, p - 1, R);
    for (int n = 1; n <= p; ++n) {
        for (int m = 0; m <= n; ++m) {
            const Cplx<T> l = L[tri(n, m)];
            const Cplx<T> zero{(T)0, (T)0};
            const Cplx<T> dp = m + 1 <= n - 1 ? R[tri(n - 1, m + 1)] : zero;
            Cplx<T> dm = zero;
            if (m - 1 >= -(n - 1) && m - 1 <= n - 1) {
                const Cplx<T> h = harm_at<T>(R, n - 1, m - 1);
                dm = Cplx<T>{-h.re, -h.im};
            }
            const Cplx<T> dz = m <= n - 1 ? R[tri(n - 1, m)] : zero;
            const T w = m == 0 ? (T)1 : (T)2;
            const Cplx<T> sp = cmul(l, Cplx<T>{dp.re + dm.re, dp.im + dm.im});
            const Cplx<T> sm = cmul(l, Cplx<T>{dp.re - dm.re, dp.im - dm.im});
            gx += w * (T)0.5 * sp.re;
            gy += w * (T)0.5 * sm.im;
            gz += w * cmul(l, dz).re;
        }
    }
}

// Field at the points of a target tree from a source plan: one warp per
// target leaf, one lane per target.  Near part: sum_j q_j (x - y_j) / r^3
// over the leaf's P2P row (the gradient of the potential kernel
// q / max(r, eps), zero where r <= eps); far part: minus the gradient of the
// leaf's local expansion.  out[3 * index_map[i] + c] = k_e * E_c.
template <typename T>
__global__ void __launch_bounds__(128) k_targets_field(
    const int32_t *__restrict__ leaves, int64_t n_leaves, const int32_t *__restrict__ off,
    const int32_t *__restrict__ src, const typename Vec4<T>::type *__restrict__ pts, const int2 *__restrict__ range,
    const typename Vec4<T>::type *__restrict__ spts, const int2 *__restrict__ srange,
    const typename Vec4<T>::type *__restrict__ center, const typename Vec4<T>::type *__restrict__ half,
    const Cplx<T> *__restrict__ Lexp, int p, int nc_pad, T eps2, int near, int far,
    const int32_t *__restrict__ index_map, T k_e, T *__restrict__ out) {
    using T4 = typename Vec4<T>::type;
    __shared__ T4 sp[4][32];
    const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t w = (int64_t)blockIdx.x * 4 + wl;
    if (w >= n_leaves) return;
    const int t = leaves[w];
    const int2 rg = range[t];
    T4 c{};
    T ia = (T)1;
    if (far) {
        c = center[t];
        ia = (T)1 / half[t].w;
    }
    for (int tb = rg.x; tb < rg.y; tb += 32) {
        const int ti = tb + lane;
        const bool valid = ti < rg.y;
        const T4 x = pts[valid ? ti : rg.x];
        T ex = 0, ey = 0, ez = 0;
        if (near) {
            for (int k = off[t]; k < off[t + 1]; ++k) {
                const int2 sr = srange[src[k]];
                for (int sb = sr.x; sb < sr.y; sb += 32) {
                    const int cnt = min(32, sr.y - sb);
                    __syncwarp();
                    if (lane < cnt) sp[wl][lane] = spts[sb + lane];
                    __syncwarp();
                    for (int j = 0; j < cnt; ++j) {
                        const T4 q = sp[wl][j];
                        const T dx = x.x - q.x, dy = x.y - q.y, dz = x.z - q.z;
                        const T r2 = dx * dx + dy * dy + dz * dz;
                        if (r2 > eps2) {
                            const T ir = (T)1 / sqrt(r2);
                            const T wq = q.w * ir * ir * ir;
                            ex += wq * dx;
                            ey += wq * dy;
                            ez += wq * dz;
                        }
                    }
                }
            }
        }
        if (far && valid) {
            T gx, gy, gz;
            l2p_gradient<T>(Lexp + (int64_t)t * nc_pad, p, (x.x - c.x) * ia, (x.y - c.y) * ia, (x.z - c.z) * ia, gx, gy,
                            gz);
            ex -= gx * ia;
            ey -= gy * ia;
            ez -= gz * ia;
        }
        if (valid) {
            const int o = index_map[ti];
            out[3 * o] = k_e * ex;
            out[3 * o + 1] = k_e * ey;
            out[3 * o + 2] = k_e * ez;
        }
    }
}

template <typename T>
int field_impl(const DevTree &tree, const DevLists &lists, const FmmBuffers &buf, const DevTree &stree, double k_e,
               bool near, bool far, void *out, cudaStream_t s) {
    using T4 = typename Vec4<T>::type;
    if (tree.n_leaves == 0) return EDFMM_OK;
    const T eps = sizeof(T) == 8 ? (T)DBL_EPSILON : (T)FLT_EPSILON;
    k_targets_field<T><<<(unsigned)((tree.n_leaves + 3) / 4), 128, 0, s>>>(
        dptr<int32_t>(tree.leaves), tree.n_leaves, dptr<int32_t>(lists.p2p_off), dptr<int32_t>(lists.p2p_src),
        dptr<T4>(tree.pts), dptr<int2>(tree.range), dptr<T4>(stree.pts), dptr<int2>(stree.range),
        dptr<T4>(tree.center), dptr<T4>(tree.half), dptr<Cplx<T>>(buf.locals), buf.p, buf.nc_pad, eps * eps,
        near ? 1 : 0, far ? 1 : 0, dptr<int32_t>(tree.index_map), (T)k_e, static_cast<T *>(out));
    EDFMM_LAUNCH_CHECK("k_targets_field");
    return EDFMM_OK;
}

}  // namespace

int run_targets_field(const DevTree &tree, const DevLists &lists, const FmmBuffers &buf, const DevTree &stree,
                      double k_e, bool near, bool far, void *out, cudaStream_t s) {
    return tree.dtype == EDFMM_F64 ? field_impl<double>(tree, lists, buf, stree, k_e, near, far, out, s)
                                   : field_impl<float>(tree, lists, buf, stree, k_e, near, far, out, s);
}

}  // namespace edfmm
