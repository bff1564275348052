// Dense single-layer operator (the reference's torch-tiled A(x),
// electrodrive/core/bem_kernel.py:157-230 and :341-381):
//   V_i = k_e sum_{j != i} sigma_j A_j / sqrt(max(|c_i - c_j|^2, 1e-24))
//         + self_integrals_i sigma_i A_i        (self term only if given);
//   non-finite V_i -> 0,
// and the induced potential and field at separate targets.
//
// One block owns a tile of targets; the sources are split over the blocks of
// a thread-block cluster and, inside a block, over its warps, so that small
// problems fill every SM.  The partial sums are added in a fixed order, over
// the block's warps and then over the cluster's blocks through distributed
// shared memory: no scratch in device memory, no second launch.
//
// FP32 (k_dense_f32): each lane keeps several targets, so that a source pair
// read from shared memory (two 16-byte broadcasts) serves all of them;
// distances run as packed pairs.  An interaction is 7 FMA-pipe operations,
// one maximum and one MUFU.RSQ (16 per SM and clock: the bound).  19,997
// panels, one matvec: 175 -> 123 us (5.03e12 rsqrt/s: 79 us).
//
// FP64 (k_dense_f64): the inverse distances run on the FP32 pipe at FP64
// accuracy (gridpoint.cuh), two pairs in packed operations; one FP64 operation
// per interaction remains, beside 16 in IEEE arithmetic, whose pipe bounded
// the kernel (15.8 operations at 2 per SM and clock).  5,120 panels, one
// matvec: 770 -> 160 us.  A tile of sources
// whose coordinates are not finite, or all zero, and pairs too close for the
// split run in IEEE FP64.
#include <algorithm>
#include <cmath>

#include "edfmm_internal.cuh"
#include "gridpoint.cuh"

namespace edfmm {

namespace {

// kBoth: field and potential in one pass; kTable: every 1 / r of the operator written out
enum DenseKind { kMatvec = 0, kPotential = 1, kField = 2, kBoth = 3, kTable = 4 };
template <int KIND> __host__ __device__ constexpr bool has_field() { return KIND == kField || KIND == kBoth; }
// sums per target: the field's three, the potential
template <int KIND> __host__ __device__ constexpr int dense_comp() { return KIND == kField ? 3 : KIND == kBoth ? 4 : 1; }

constexpr int kThreads = 128;     // 4 warps
constexpr int kTile32 = 256;      // sources staged per shared-memory tile, FP32
constexpr int kTile64 = 128;      // FP64
constexpr int kMaxCluster = 8;    // the portable cluster size

__device__ __forceinline__ float inv_r(float r2) { return rsqrt_normal(fmaxf(r2, 1e-24f)); }
__device__ __forceinline__ double inv_r(double r2) { return rsqrt(fmax(r2, 1e-24)); }

template <typename T> struct DenseArgs {
    const T *tgt;  // (m, 3) targets (the centroids themselves for kMatvec)
    int64_t m;
    const T *c, *sigma, *areas;  // (n, 3), (n), (n)
    int64_t n;
    int64_t chunk;  // sources per block of the cluster (even)
    int cs;         // cluster size
    T k_e;
    const T *self_int;  // kMatvec only
    T *out;
    T *out_v;  // kBoth: the potential
    int64_t ld;  // kTable: distance of out's rows
};

__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// element of the same shared-memory variable in block `rank` of the cluster
__device__ __forceinline__ float dsm_load(const float *p, int rank) {
    unsigned a;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ double dsm_load(const double *p, int rank) {
    unsigned a;
    double v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
    return v;
}

// Sum over the block's source groups and the cluster's blocks, and write the
// rows.  part[(g * ROWS + row) * COMP + comp]: group g's sums of this block.
template <typename T, int KIND, int ROWS, int GROUPS>
__device__ __forceinline__ void dense_finish(const DenseArgs<T> &A, T *part, int64_t row0, int rank) {
    constexpr int COMP = dense_comp<KIND>(), NV = ROWS * COMP;
    __syncthreads();
    for (int q = threadIdx.x; q < NV; q += kThreads) {
        T v = part[q];
#pragma unroll
        for (int g = 1; g < GROUPS; ++g) v += part[g * NV + q];
        part[q] = v;
    }
    if (A.cs > 1) cluster_sync_all();
    else __syncthreads();
    if (rank == 0) {
        for (int q = threadIdx.x; q < NV; q += kThreads) {
            const int64_t i = row0 + q / COMP;
            if (i >= A.m) continue;
            T v = part[q];
            for (int r = 1; r < A.cs; ++r) v += dsm_load(part + q, r);
            if (KIND == kMatvec) {
                v *= A.k_e;
                if (A.self_int) v += A.self_int[i] * A.sigma[i] * A.areas[i];
                A.out[i] = isfinite(v) ? v : (T)0;
            } else if (KIND == kPotential) {
                A.out[i] = v * A.k_e;
            } else if (KIND == kBoth && q % COMP == 3) {
                A.out_v[i] = v * A.k_e;
            } else {
                A.out[i * 3 + q % COMP] = isfinite(v) ? v : (T)0;
            }
        }
    }
    if (A.cs > 1) cluster_sync_all();  // the other blocks' shared memory stays until it has been read
}

// the block's target tile and its share of the sources (rank of the cluster)
template <typename T>
__device__ __forceinline__ void dense_ranges(const DenseArgs<T> &A, int rows, int64_t &row0, int &rank, int64_t &j0,
                                             int64_t &j1) {
    row0 = (int64_t)(blockIdx.x / (unsigned)A.cs) * rows;
    rank = (int)(blockIdx.x % (unsigned)A.cs);
    j0 = min(A.n, rank * A.chunk);
    j1 = min(A.n, j0 + A.chunk);
}

// ---------------------------------------------------------------------------
// FP32: 32 * TPT targets per block, the four warps take every fourth source
// pair of a tile.  The field weight is formed in the reference's order (k_e
// times 1/r^3, times sigma A), so a near-coincident pair overflows where the
// reference's does, and non-finite components become zero at the end
// (bem_kernel.py:990-997).
// ---------------------------------------------------------------------------
template <int KIND> __host__ __device__ constexpr int tpt32() { return has_field<KIND>() ? 2 : 4; }

template <int KIND, bool SELF, int TPT>
__device__ __forceinline__ void dense_tile_f32(const float4 *src, int npairs, int wid, float k_e, const float2 (&nx)[TPT],
                                               const float2 (&ny)[TPT], const float2 (&nz)[TPT], int self0,
                                               float2 (&ax)[TPT], float2 (&ay)[TPT], float2 (&az)[TPT],
                                               float2 (&av)[TPT]) {
#pragma unroll 2
    for (int k = wid; k < npairs; k += 4) {
        const float4 u = src[2 * k], v = src[2 * k + 1];  // (x, x', y, y'), (z, z', q, q')
        const float2 qw = make_float2(v.z, v.w);
#pragma unroll
        for (int t = 0; t < TPT; ++t) {
            const float2 dx = __fadd2_rn(make_float2(u.x, u.y), nx[t]), dy = __fadd2_rn(make_float2(u.z, u.w), ny[t]),
                         dz = __fadd2_rn(make_float2(v.x, v.y), nz[t]);
            const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
            const float2 ir = make_float2(inv_r(r2.x), inv_r(r2.y));
            if (has_field<KIND>()) {
                const float2 ke2 = make_float2(k_e, k_e);
                const float2 w = __fmul2_rn(__fmul2_rn(ke2, __fmul2_rn(__fmul2_rn(ir, ir), ir)), qw);
                ax[t] = __ffma2_rn(w, dx, ax[t]);  // source minus target: the sign is taken at the end
                ay[t] = __ffma2_rn(w, dy, ay[t]);
                az[t] = __ffma2_rn(w, dz, az[t]);
            }
            if (KIND != kField) {
                float2 v = __ffma2_rn(qw, ir, av[t]);
                if (SELF) {  // not the target itself, at self0 + 32 t of this tile (its charge may be infinite)
                    if (2 * k == self0 + 32 * t) v.x = av[t].x;
                    if (2 * k + 1 == self0 + 32 * t) v.y = av[t].y;
                }
                av[t] = v;
            }
        }
    }
}

template <int KIND>
__global__ void __launch_bounds__(kThreads) k_dense_f32(const DenseArgs<float> A) {
    constexpr int TPT = tpt32<KIND>(), ROWS = 32 * TPT, COMP = dense_comp<KIND>();
    __shared__ float4 src[kTile32];
    __shared__ float part[4 * ROWS * COMP];
    int64_t row0, j0, j1;
    int rank;
    dense_ranges(A, ROWS, row0, rank, j0, j1);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float2 nx[TPT], ny[TPT], nz[TPT];
    float ex[TPT], ey[TPT], ez[TPT], ev[TPT];
#pragma unroll
    for (int t = 0; t < TPT; ++t) {
        const int64_t i = min(row0 + lane + 32 * t, A.m - 1);
        nx[t].x = nx[t].y = -A.tgt[3 * i];
        ny[t].x = ny[t].y = -A.tgt[3 * i + 1];
        nz[t].x = nz[t].y = -A.tgt[3 * i + 2];
        ex[t] = ey[t] = ez[t] = ev[t] = 0.0f;
    }
    float *sf = reinterpret_cast<float *>(src);
    for (int64_t jb = j0; jb < j1; jb += kTile32) {
        const int cnt = (int)min((int64_t)kTile32, j1 - jb);
        __syncthreads();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int q = threadIdx.x + h * kThreads;
            // past its end a tile holds its last source, without charge: a point of
            // its own there could meet a target, whose weight k_e / r^3 then
            // overflows and is NaN times no charge
            const int64_t j = jb + min(q, cnt - 1);
            const float x = A.c[3 * j], y = A.c[3 * j + 1], z = A.c[3 * j + 2], w = A.sigma[j] * A.areas[j];
            float *o = sf + (q >> 1) * 8 + (q & 1);
            o[0] = x;
            o[2] = y;
            o[4] = z;
            o[6] = q < cnt ? w : 0.0f;
        }
        __syncthreads();
        // two-level sum (tile, then chunk) bounds FP32 rounding growth
        float2 ax[TPT], ay[TPT], az[TPT], av[TPT];
#pragma unroll
        for (int t = 0; t < TPT; ++t) ax[t] = ay[t] = az[t] = av[t] = make_float2(0.0f, 0.0f);
        const int np = (cnt + 1) >> 1;
        if (KIND == kMatvec && jb < row0 + ROWS && row0 < jb + cnt)
            dense_tile_f32<KIND, true>(src, np, wid, A.k_e, nx, ny, nz, (int)(row0 - jb) + lane, ax, ay, az, av);
        else
            dense_tile_f32<KIND, false>(src, np, wid, A.k_e, nx, ny, nz, 0, ax, ay, az, av);
#pragma unroll
        for (int t = 0; t < TPT; ++t) {
            if (has_field<KIND>()) {
                ex[t] += ax[t].x + ax[t].y;
                ey[t] += ay[t].x + ay[t].y;
                ez[t] += az[t].x + az[t].y;
            }
            if (KIND != kField) ev[t] += av[t].x + av[t].y;
        }
    }
#pragma unroll
    for (int t = 0; t < TPT; ++t) {
        float *p = part + (wid * ROWS + lane + 32 * t) * COMP;
        if (has_field<KIND>()) {
            p[0] = -ex[t];
            p[1] = -ey[t];
            p[2] = -ez[t];
        }
        if (KIND != kField) p[COMP - 1] = ev[t];
    }
    dense_finish<float, KIND, ROWS, 4>(A, part, row0, rank);
}

// ---------------------------------------------------------------------------
// FP64: 128 / GROUPS targets per block, one per thread; the groups of threads
// take every GROUPS-th pair of sources of a tile, two pairs at a time (packed
// operations issue in half the slots, and two independent chains cover their
// latency).  The FMA pipe is the bound, 141 cycles of a scheduler per 32
// interactions: 5,120 panels 165 us scalar, one source at a time, with two FP64
// operations an interaction; 154 packed (75% of the pipe's time; the rest is
// the exact split of each tile's sources, again for every 64 targets, and the
// uneven number of blocks per SM).
// ---------------------------------------------------------------------------
// Sources lie in the tile in pairs, value by value (24 words a pair: the nine
// parts of both, a gap, both charges), so that a load gives packed operands.
constexpr int kPairWords = 24, kPairCharge = 10;  // the charges as doubles 10 and 11 of a pair
struct Tgt64 {
    double x, y, z;
    GridCoordT<float2> gx, gy, gz;  // scaled, in both halves
};
__device__ __forceinline__ GridCoordT<float2> grid_both(const GridCoord &g) {
    return GridCoordT<float2>{make_float2(g.a, g.a), make_float2(g.b, g.b), make_float2(g.c, g.c)};
}

__device__ __forceinline__ unsigned high_abs(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }

// one source in IEEE FP64, from device memory (w: the charge)
template <int KIND>
__device__ __noinline__ void dense_pair_ieee(const double *c, int64_t j, int64_t self, double x, double y, double z,
                                             double w, double k_e, double &ex, double &ey, double &ez, double &ev) {
    ex = ey = ez = ev = 0.0;
    if ((KIND == kMatvec || KIND == kTable) && j == self) return;
    const double dx = x - c[3 * j], dy = y - c[3 * j + 1], dz = z - c[3 * j + 2];
    const double ir = inv_r(dx * dx + dy * dy + dz * dz);
    if (has_field<KIND>()) {
        const double f = (k_e * (ir * ir * ir)) * w;
        ex = f * dx;
        ey = f * dy;
        ez = f * dz;
    }
    ev = w * ir;
}

template <int KIND, int GROUPS>
__global__ void __launch_bounds__(kThreads) k_dense_f64(const DenseArgs<double> A) {
    constexpr int COMP = dense_comp<KIND>(), ROWS = kThreads / GROUPS;
    __shared__ __align__(16) float src[kTile64 / 2 * kPairWords];
    __shared__ double xyz[has_field<KIND>() ? 3 * kTile64 : 1];
    __shared__ double part[kThreads * COMP];
    __shared__ unsigned s_hi[4];
    int64_t row0, j0, j1;
    int rank;
    dense_ranges(A, ROWS, row0, rank, j0, j1);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, grp = threadIdx.x / ROWS;
    const int64_t i = row0 + threadIdx.x % ROWS;
    Tgt64 T;
    {
        const int64_t q = min(i, A.m - 1);
        T.x = A.tgt[3 * q];
        T.y = A.tgt[3 * q + 1];
        T.z = A.tgt[3 * q + 2];
    }
    const unsigned thi = max(high_abs(T.x), max(high_abs(T.y), high_abs(T.z)));
    int kprev = INT32_MIN;
    double ex = 0, ey = 0, ez = 0, ev = 0;
    auto charge = [&](int q) -> double & {
        return reinterpret_cast<double *>(src)[(q >> 1) * (kPairWords / 2) + kPairCharge + (q & 1)];
    };
    for (int64_t jb = j0; jb < j1; jb += kTile64) {
        const int cnt = (int)min((int64_t)kTile64, j1 - jb);
        double x = 0, y = 0, z = 0, w = 0;
        if ((int)threadIdx.x < cnt) {
            const int64_t j = jb + threadIdx.x;
            x = A.c[3 * j];
            y = A.c[3 * j + 1];
            z = A.c[3 * j + 2];
            w = KIND == kTable ? 1.0 : A.sigma[j] * A.areas[j];
        }
        // the tile's scale: a power of two above every |coordinate| of its sources and targets
        const unsigned hi = __reduce_max_sync(0xffffffffu, max(max(thi, high_abs(x)), max(high_abs(y), high_abs(z))));
        __syncthreads();  // the previous tile has been read
        if (lane == 0) s_hi[wid] = hi;
        __syncthreads();
        int k;
        const bool split = grid_exponent(max(max(s_hi[0], s_hi[1]), max(s_hi[2], s_hi[3])), k);
        if (!split) {
            if ((int)threadIdx.x < cnt) charge(threadIdx.x) = w;
            __syncthreads();
            for (int s = grp; s < cnt; s += GROUPS) {
                double px, py, pz, pv;
                dense_pair_ieee<KIND>(A.c, jb + s, i, T.x, T.y, T.z, charge(s), A.k_e, px, py, pz, pv);
                if (KIND == kTable && i < A.m) A.out[(jb + s) * A.ld + i] = pv;
                ex += px;
                ey += py;
                ez += pz;
                ev += pv;
            }
            continue;
        }
        const double down = grid_pow2(-k);
        if (k != kprev) {
            T.gx = grid_both(grid_split(T.x * down));
            T.gy = grid_both(grid_split(T.y * down));
            T.gz = grid_both(grid_split(T.z * down));
            kprev = k;
        }
        if ((int)threadIdx.x < ((cnt + 4 * GROUPS - 1) & ~(4 * GROUPS - 1))) {
            // padding: no charge, outside the scaled box
            const bool real = (int)threadIdx.x < cnt;
            const GridCoord out{3.0f, 0.0f, 0.0f};
            const GridCoord a = real ? grid_split(x * down) : out, b = real ? grid_split(y * down) : out,
                            c = real ? grid_split(z * down) : out;
            float *q = src + (threadIdx.x >> 1) * kPairWords + (threadIdx.x & 1);
            q[0] = a.a;
            q[2] = a.b;
            q[4] = a.c;
            q[6] = b.a;
            q[8] = b.b;
            q[10] = b.c;
            q[12] = c.a;
            q[14] = c.b;
            q[16] = c.c;
            charge(threadIdx.x) = w;
            if (has_field<KIND>()) {
                xyz[3 * threadIdx.x] = x;
                xyz[3 * threadIdx.x + 1] = y;
                xyz[3 * threadIdx.x + 2] = z;
            }
        }
        __syncthreads();
        // closer than the split resolves, or than the clamp: IEEE
        const float near2 = fmaxf(kGridNear2, (float)(1.0001e-24 * down * down));
        double tx = 0, ty = 0, tz = 0, tv = 0;  // two-level sum: tile, then chunk; the split pairs in scaled units
        double sx = 0, sy = 0, sz = 0, sv = 0;
        auto add = [&](int s, float y0, float eh, float v, double w) {
            const double ir = grid_inv(y0, grid_ci(eh, v));
            if (has_field<KIND>()) {  // every FP64 operation is 64 cycles: k_e at the end, w / r shared
                const double wr = w * ir, f = wr * (ir * ir);
                tx = fma(f, T.x - xyz[3 * s], tx);
                ty = fma(f, T.y - xyz[3 * s + 1], ty);
                tz = fma(f, T.z - xyz[3 * s + 2], tz);
                if (KIND == kBoth) tv += wr;
            } else if (KIND == kTable) {
                if (s < cnt && i < A.m) A.out[(jb + s) * A.ld + i] = ir * down;
            } else {
                tv = fma(w, ir, tv);
            }
        };
        auto ieee = [&](int s, double w) {
            if (s >= cnt) return;  // padding
            double px, py, pz, pv;
            dense_pair_ieee<KIND>(A.c, jb + s, i, T.x, T.y, T.z, w, A.k_e, px, py, pz, pv);
            sx += px;
            sy += py;
            sz += pz;
            sv += pv;
            if (KIND == kTable && i < A.m) A.out[(jb + s) * A.ld + i] = pv;
        };
        struct Pair2 {
            float2 R1, y0, eh, v;
            double2 w;
        };
        auto pair_of = [&](int s, Pair2 &p) {
            const float4 *q = reinterpret_cast<const float4 *>(src + (s >> 1) * kPairWords);
            const float4 q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3];
            const float2 q4 = *reinterpret_cast<const float2 *>(q + 4);
            p.w = *reinterpret_cast<const double2 *>(q + 5);
            const GridR2<float2> r2 = grid_r2(
                grid_diff(T.gx, GridCoordT<float2>{make_float2(q0.x, q0.y), make_float2(q0.z, q0.w), make_float2(q1.x, q1.y)}),
                grid_diff(T.gy, GridCoordT<float2>{make_float2(q1.z, q1.w), make_float2(q2.x, q2.y), make_float2(q2.z, q2.w)}),
                grid_diff(T.gz, GridCoordT<float2>{make_float2(q3.x, q3.y), make_float2(q3.z, q3.w), q4}));
            p.R1 = r2.R1;
            grid_rsqrt(r2, p.y0, p.eh, p.v);
        };
        auto add_pair = [&](int s, const Pair2 &p) {
            add(s, p.y0.x, p.eh.x, p.v.x, p.w.x);
            add(s + 1, p.y0.y, p.eh.y, p.v.y, p.w.y);
        };
        auto add_close = [&](int s, const Pair2 &p) {
            if (p.R1.x < near2) ieee(s, p.w.x);
            else add(s, p.y0.x, p.eh.x, p.v.x, p.w.x);
            if (p.R1.y < near2) ieee(s + 1, p.w.y);
            else add(s + 1, p.y0.y, p.eh.y, p.v.y, p.w.y);
        };
        for (int s = 2 * grp; s < cnt; s += 4 * GROUPS) {  // two pairs of sources in the padded tile
            Pair2 a, b;
            pair_of(s, a);
            pair_of(s + 2 * GROUPS, b);
            if (fminf(fminf(a.R1.x, a.R1.y), fminf(b.R1.x, b.R1.y)) < near2) {
                add_close(s, a);
                add_close(s + 2 * GROUPS, b);
            } else {
                add_pair(s, a);
                add_pair(s + 2 * GROUPS, b);
            }
        }
        if (has_field<KIND>()) {
            const double unscale = down * down * down;
            ex += A.k_e * (tx * unscale) + sx;
            ey += A.k_e * (ty * unscale) + sy;
            ez += A.k_e * (tz * unscale) + sz;
        }
        if (KIND != kField) ev += tv * down + sv;
    }
    if (KIND == kTable) return;
    double *p = part + threadIdx.x * COMP;
    if (has_field<KIND>()) {
        p[0] = ex;
        p[1] = ey;
        p[2] = ez;
    }
    if (KIND != kField) p[COMP - 1] = ev;
    dense_finish<double, KIND, ROWS, GROUPS>(A, part, row0, rank);
}

int sm_count() {
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 152;
    if (dev < 64 && cached[dev]) return cached[dev];
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (dev < 64) cached[dev] = sms;
    return sms;
}

// Cluster size: the number of blocks that share a target tile's sources.  A
// block costs its sources plus about 40 sources' worth of set-up and
// reduction, and the fullest SM decides.  FP64: up to four blocks per SM run at
// once, beyond that blocks follow one another and the last one costs half its
// time on average; and fewer than three blocks leave the pipes waiting, so an
// SM takes the time of three.  3,000 panels: 142 us with clusters of 3 (one
// block per SM), 92 with 8; 5,120: 207 with 6, 182 with 7, 189 with 8; 12,000:
// 892 with 4, 796 with 8.  FP32 lanes hold several targets:
// 1,000 targets, 5,120 sources take 34 us with clusters chosen for one block
// per SM and 36 for three.
int cluster_size(int64_t tiles, int64_t n, bool f64) {
    const int64_t sms = sm_count();
    if (tiles >= 8 * sms) return 1;
    int best = 1;
    double cost = 1e300;
    for (int cs = 1; cs <= kMaxCluster; ++cs) {
        const double per_sm = (double)(tiles * cs) / (double)sms, whole = std::ceil(per_sm);
        const double blocks = !f64 ? whole : per_sm <= 4.0 ? std::max(whole, 3.0) : per_sm + 0.5;
        const double t = blocks * (std::ceil((double)n / cs) + 40.0);
        if (t < cost) {
            cost = t;
            best = cs;
        }
    }
    return best;
}

template <typename T, int KIND>
int dense_launch(const T *tgt, int64_t m, const T *c, const T *sigma, const T *areas, int64_t n, T k_e,
                 const T *self_int, T *out, T *out_v, cudaStream_t s, int64_t ld = 0) {
    // FP64: 64 targets per block, or 32 when those would leave SMs without a block
    // even in clusters of eight; the smaller tile splits every source for half
    // the targets (1,000 targets, 5,120 sources: 89 and 290 us, potential and
    // field, with 64, 76 and 180 with 32)
    const bool narrow = sizeof(T) == 8 && KIND != kTable && (m + 63) / 64 * kMaxCluster < 2 * sm_count();
    const int ROWS = sizeof(T) == 4 ? 32 * tpt32<KIND>() : narrow ? 32 : 64;
    const int64_t tiles = (m + ROWS - 1) / ROWS;
    DenseArgs<T> A{tgt, m, c, sigma, areas, n, 0, cluster_size(tiles, n, sizeof(T) == 8), k_e, self_int, out, out_v, ld};
    A.chunk = ((n + A.cs - 1) / A.cs + 1) & ~(int64_t)1;
    if (tiles * A.cs > INT32_MAX) return fail(EDFMM_ERR_ARG, "too many targets for one launch");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * A.cs));
    cfg.blockDim = dim3(kThreads);
    cfg.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)A.cs;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = A.cs > 1 ? 1 : 0;
    cudaError_t e;
    if constexpr (sizeof(T) == 4) e = cudaLaunchKernelEx(&cfg, k_dense_f32<KIND>, A);
    else e = narrow ? cudaLaunchKernelEx(&cfg, k_dense_f64<KIND, 4>, A) : cudaLaunchKernelEx(&cfg, k_dense_f64<KIND, 2>, A);
    if (e != cudaSuccess) return fail(EDFMM_ERR_CUDA, std::string("launch of k_dense failed: ") + cudaGetErrorString(e));
    EDFMM_LAUNCH_CHECK("k_dense");
    return EDFMM_OK;
}

// ---------------------------------------------------------------------------
// The FP64 operator of repeated applications: its 1 / r as a table (symmetric,
// so row j serves source j's column), and their matrix-vector product.  A pair
// then costs 8 bytes and one FP64 multiply-add in place of 136 FP32 operations.
// A lane owns two targets, a warp 64; the eight warps of a block and the blocks
// of a cluster of eight take every 64th source, and their sums are added in
// a fixed order as in the kernels above.  5,120 panels: 162 us an application
// from the coordinates, 63 with the table (210 MB; the FP64 pipe's time is 45 us),
// 180 once to fill it; 20,000 panels (3.2 GB) 2,035 and 734 us.
// ---------------------------------------------------------------------------
constexpr size_t kTableCharges = 32768;  // bytes of a block's charges
constexpr int kTableThreads = 256, kTableRows = 64, kTableWarps = kTableThreads / 32;

__global__ void __launch_bounds__(kTableThreads) k_dense_table(const double *__restrict__ table, int64_t ld,
                                                               const DenseArgs<double> A) {
    __shared__ double part[kTableWarps * kTableRows];
    extern __shared__ double charge[];  // this block's sources: a product a warp would otherwise form again
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t row0 = (int64_t)(blockIdx.x / (unsigned)A.cs) * kTableRows;
    const int rank = (int)(blockIdx.x % (unsigned)A.cs);
    const int64_t j0 = min(A.n, rank * A.chunk);
    const int cnt = (int)(min(A.n, j0 + A.chunk) - j0);
    for (int q = threadIdx.x; q < cnt; q += kTableThreads) charge[q] = A.sigma[j0 + q] * A.areas[j0 + q];
    __syncthreads();
    const double *col = table + j0 * ld + row0 + 2 * lane;
    double ax = 0, ay = 0;
    int j = wid;
    constexpr int U = 8;  // loads in flight
    for (; j + (U - 1) * kTableWarps < cnt; j += U * kTableWarps) {
        double2 k[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            k[u] = __ldg(reinterpret_cast<const double2 *>(col + (int64_t)(j + u * kTableWarps) * ld));
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const double w = charge[j + u * kTableWarps];
            ax = fma(k[u].x, w, ax);
            ay = fma(k[u].y, w, ay);
        }
    }
    for (; j < cnt; j += kTableWarps) {
        const double2 k = __ldg(reinterpret_cast<const double2 *>(col + (int64_t)j * ld));
        ax = fma(k.x, charge[j], ax);
        ay = fma(k.y, charge[j], ay);
    }
    part[wid * kTableRows + 2 * lane] = ax;
    part[wid * kTableRows + 2 * lane + 1] = ay;
    __syncthreads();
    if (threadIdx.x < kTableRows) {
        double v = part[threadIdx.x];
#pragma unroll
        for (int g = 1; g < kTableWarps; ++g) v += part[g * kTableRows + threadIdx.x];
        part[threadIdx.x] = v;
    }
    if (A.cs > 1) cluster_sync_all();
    else __syncthreads();
    const int64_t i = row0 + threadIdx.x;
    if (rank == 0 && threadIdx.x < kTableRows && i < A.m) {
        double v = part[threadIdx.x];
        for (int r = 1; r < A.cs; ++r) v += dsm_load(part + threadIdx.x, r);
        if (!isfinite(v) && !isfinite(A.sigma[i] * A.areas[i])) {  // its own charge times the diagonal's 0: the sum without it
            v = 0.0;
            for (int64_t j = 0; j < A.n; ++j)
                if (j != i) v = fma(table[j * ld + i], A.sigma[j] * A.areas[j], v);
        }
        v *= A.k_e;
        if (A.self_int) v += A.self_int[i] * A.sigma[i] * A.areas[i];
        A.out[i] = isfinite(v) ? v : 0.0;
    }
    if (A.cs > 1) cluster_sync_all();  // the other blocks' shared memory stays until it has been read
}

inline int64_t table_ld(int64_t n) { return (n + kTableRows - 1) / kTableRows * kTableRows; }

template <int KIND>
int dense_any(const void *tgt, int64_t m, const void *c, const void *sigma, const void *areas, int64_t n, int dtype,
              double k_e, const void *self_int, void *out, void *out_v, cudaStream_t s) {
    if (dtype == EDFMM_F64)
        return dense_launch<double, KIND>((const double *)tgt, m, (const double *)c, (const double *)sigma,
                                          (const double *)areas, n, k_e, (const double *)self_int, (double *)out,
                                          (double *)out_v, s);
    return dense_launch<float, KIND>((const float *)tgt, m, (const float *)c, (const float *)sigma, (const float *)areas,
                                     n, (float)k_e, (const float *)self_int, (float *)out, (float *)out_v, s);
}

}  // namespace

}  // namespace edfmm

using namespace edfmm;

#define EDFMM_DENSE_NOALLOC_MAX_N 262144

extern "C" EDFMM_API int edfmm_dense_matvec(const void *centroids, const void *sigma, const void *areas,
                                            const void *self_integrals, int64_t n, int dtype, double k_e, void *out,
                                            void *stream) {
    if (n < 0) return fail(EDFMM_ERR_ARG, "n must be >= 0");
    if (dtype != EDFMM_F32 && dtype != EDFMM_F64) return fail(EDFMM_ERR_ARG, "dtype must be EDFMM_F32 or EDFMM_F64");
    if (n == 0) return EDFMM_OK;
    if (!centroids || !sigma || !areas || !out) return fail(EDFMM_ERR_ARG, "centroids, sigma, areas, out must be non-NULL");
    return dense_any<kMatvec>(centroids, n, centroids, sigma, areas, n, dtype, k_e, self_integrals, out,
                              nullptr, static_cast<cudaStream_t>(stream));
}

extern "C" EDFMM_API int edfmm_dense_matvec_noalloc(const void *centroids, const void *sigma, const void *areas,
                                                    const void *self_integrals, int64_t n, int dtype, double k_e,
                                                    void *out, void *stream) {
    if (n > EDFMM_DENSE_NOALLOC_MAX_N)
        return fail(EDFMM_ERR_ARG, "edfmm_dense_matvec_noalloc: n = " + std::to_string(n) + " exceeds its limit of " +
                                       std::to_string(EDFMM_DENSE_NOALLOC_MAX_N) + " panels; use edfmm_dense_matvec");
    return edfmm_dense_matvec(centroids, sigma, areas, self_integrals, n, dtype, k_e, out, stream);
}

extern "C" EDFMM_API size_t edfmm_dense_workspace_bytes(int64_t, int) { return 0; }

extern "C" EDFMM_API int edfmm_dense_matvec_ws(const void *centroids, const void *sigma, const void *areas,
                                               const void *self_integrals, int64_t n, int dtype, double k_e, void *out,
                                               void *, size_t, void *stream) {
    return edfmm_dense_matvec(centroids, sigma, areas, self_integrals, n, dtype, k_e, out, stream);
}

extern "C" EDFMM_API int edfmm_dense_field_targets(const void *targets, int64_t m, const void *centroids,
                                                   const void *sigma, const void *areas, int64_t n, int dtype,
                                                   double k_e, void *out, void *stream) {
    if (m < 0 || n < 0) return fail(EDFMM_ERR_ARG, "sizes must be >= 0");
    if (dtype != EDFMM_F32 && dtype != EDFMM_F64) return fail(EDFMM_ERR_ARG, "bad dtype");
    if (m == 0) return EDFMM_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (n == 0) {
        EDFMM_CUDA_TRY(cudaMemsetAsync(out, 0, (size_t)m * 3 * (dtype == EDFMM_F64 ? 8 : 4), s));
        return EDFMM_OK;
    }
    if (!targets || !centroids || !sigma || !areas || !out) return fail(EDFMM_ERR_ARG, "NULL argument");
    return dense_any<kField>(targets, m, centroids, sigma, areas, n, dtype, k_e, nullptr, out, nullptr, s);
}

extern "C" EDFMM_API int edfmm_dense_potential_targets(const void *targets, int64_t m, const void *centroids,
                                                       const void *sigma, const void *areas, int64_t n, int dtype,
                                                       double k_e, void *out, void *stream) {
    if (m < 0 || n < 0) return fail(EDFMM_ERR_ARG, "sizes must be >= 0");
    if (dtype != EDFMM_F32 && dtype != EDFMM_F64) return fail(EDFMM_ERR_ARG, "bad dtype");
    if (m == 0) return EDFMM_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (n == 0) {
        EDFMM_CUDA_TRY(cudaMemsetAsync(out, 0, (size_t)m * (dtype == EDFMM_F64 ? 8 : 4), s));
        return EDFMM_OK;
    }
    if (!targets || !centroids || !sigma || !areas || !out) return fail(EDFMM_ERR_ARG, "NULL argument");
    return dense_any<kPotential>(targets, m, centroids, sigma, areas, n, dtype, k_e, nullptr, out, nullptr, s);
}

extern "C" EDFMM_API int edfmm_dense_potential_field_targets(const void *targets, int64_t m, const void *centroids,
                                                             const void *sigma, const void *areas, int64_t n, int dtype,
                                                             double k_e, void *potential, void *field, void *stream) {
    if (m < 0 || n < 0) return fail(EDFMM_ERR_ARG, "sizes must be >= 0");
    if (dtype != EDFMM_F32 && dtype != EDFMM_F64) return fail(EDFMM_ERR_ARG, "bad dtype");
    if (m == 0) return EDFMM_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (!targets || !potential || !field) return fail(EDFMM_ERR_ARG, "NULL argument");
    if (n == 0) {
        const size_t row = (size_t)m * (dtype == EDFMM_F64 ? 8 : 4);
        EDFMM_CUDA_TRY(cudaMemsetAsync(potential, 0, row, s));
        EDFMM_CUDA_TRY(cudaMemsetAsync(field, 0, 3 * row, s));
        return EDFMM_OK;
    }
    if (!centroids || !sigma || !areas) return fail(EDFMM_ERR_ARG, "NULL argument");
    return dense_any<kBoth>(targets, m, centroids, sigma, areas, n, dtype, k_e, nullptr, field, potential, s);
}

extern "C" EDFMM_API size_t edfmm_dense_table_bytes(int64_t n) {
    return n > 0 && n <= (int64_t)(kTableCharges / sizeof(double)) * kMaxCluster ? (size_t)n * (size_t)table_ld(n) * sizeof(double) : 0;
}

extern "C" EDFMM_API int edfmm_dense_table_build(const void *centroids, int64_t n, void *table, void *stream) {
    if (n < 0) return fail(EDFMM_ERR_ARG, "n must be >= 0");
    if (n == 0) return EDFMM_OK;
    if (!centroids || !table) return fail(EDFMM_ERR_ARG, "NULL argument");
    if (edfmm_dense_table_bytes(n) == 0) return fail(EDFMM_ERR_ARG, "edfmm_dense_table_build: too many panels");
    const double *c = static_cast<const double *>(centroids);
    return dense_launch<double, kTable>(c, n, c, nullptr, nullptr, n, 1.0, nullptr, static_cast<double *>(table),
                                        nullptr, static_cast<cudaStream_t>(stream), table_ld(n));
}

extern "C" EDFMM_API int edfmm_dense_table_matvec(const void *table, const void *sigma, const void *areas,
                                                  const void *self_integrals, int64_t n, double k_e, void *out,
                                                  void *stream) {
    if (n < 0) return fail(EDFMM_ERR_ARG, "n must be >= 0");
    if (n == 0) return EDFMM_OK;
    if (!table || !sigma || !areas || !out) return fail(EDFMM_ERR_ARG, "table, sigma, areas, out must be non-NULL");
    const int64_t tiles = (n + kTableRows - 1) / kTableRows;
    const int64_t chunk = (n + kMaxCluster - 1) / kMaxCluster;
    if (chunk * sizeof(double) > kTableCharges)
        return fail(EDFMM_ERR_ARG, "edfmm_dense_table_matvec: at most " +
                                       std::to_string(kTableCharges / sizeof(double) * kMaxCluster) + " panels");
    DenseArgs<double> A{nullptr, n, nullptr, (const double *)sigma, (const double *)areas, n, chunk, kMaxCluster, k_e,
                        (const double *)self_integrals, (double *)out, nullptr, 0};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * A.cs));
    cfg.blockDim = dim3(kTableThreads);
    cfg.dynamicSmemBytes = (size_t)chunk * sizeof(double);
    cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)A.cs;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k_dense_table, static_cast<const double *>(table), table_ld(n), A);
    if (e != cudaSuccess) return fail(EDFMM_ERR_CUDA, std::string("launch of k_dense_table failed: ") + cudaGetErrorString(e));
    EDFMM_LAUNCH_CHECK("k_dense_table");
    return EDFMM_OK;
}
