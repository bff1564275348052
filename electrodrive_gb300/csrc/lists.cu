// GPU dual-tree traversal producing the P2P and M2L interaction lists.
//
// The reference walks (src, tgt) node pairs from (root, root) with a LIFO
// stack (electrodrive/fmm3d/interaction_lists.py:419-472).  Every reachable
// pair has a unique parent pair, so the traversal is a tree of pairs and the
// output is a set; here it is expanded breadth first, one frontier of pairs
// per launch.  The decisions reproduce the
// reference bit for bit:
//   * MAC (interaction_lists.py:273-297): dist = |c_s - c_t| rounded in the
//     tree dtype as sqrt(fma(dz, dz, fma(dy, dy, dx * dx))), d = 2 * radius in
//     the tree dtype, accept iff dist != 0 and max(d_s, d_t) / dist < theta
//     evaluated in double; never for the same node;
//   * leaf-leaf -> P2P (self pairs included);
//   * refinement side (interaction_lists.py:306-337): the non-leaf side,
//     else the side whose diameter exceeds the other's by 1.01x, else the side
//     with more (or equal: src) points.
// The output is stored as CSR rows by target with sources ascending, i.e.
// the reference's (tgt, src) sort order (interaction_lists.py:474-485).
#include <algorithm>
#include <climits>

#include "edfmm_internal.cuh"

namespace edfmm {

namespace {

__device__ __forceinline__ float rn_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double rn_sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float rn_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double rn_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float rn_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double rn_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float rn_sqrt(float a) { return __fsqrt_rn(a); }
__device__ __forceinline__ double rn_sqrt(double a) { return __dsqrt_rn(a); }

enum { kM2L = 0, kP2P = 1, kRefineSrc = 2, kRefineTgt = 3 };

// max(d_s, d_t) / dist < theta in double.  The quotient's FP64 division is half
// of a pair's cost, so an FP32 tree decides by FP32 products first: they are
// within 2^-22 of the exact ones for distances far from the ends of the range,
// and only pairs within 2^-20 of the bound go on to the division.
__device__ __forceinline__ bool mac_accepts(float mx, float dist, double theta) {
    const float th = (float)theta;
    if (dist > 1e-30f && dist < 1e30f && th > 1e-6f) {
        const float b = th * dist;
        if (mx < b * (1.0f - 9.5367431640625e-7f)) return true;
        if (mx > b * (1.0f + 9.5367431640625e-7f)) return false;
    }
    return __ddiv_rn((double)mx, (double)dist) < theta;
}
__device__ __forceinline__ bool mac_accepts(double mx, double dist, double theta) {
    return __ddiv_rn(mx, dist) < theta;
}

// s indexes the source tree (sc, sleaf, srange), t the target tree; `same`
// marks the single-tree case, where a node is never paired with itself by M2L.
template <typename T>
__device__ __forceinline__ int classify(int s, int t, const typename Vec4<T>::type *__restrict__ sc,
                                        const uint8_t *__restrict__ sleaf, const int2 *__restrict__ srange,
                                        const typename Vec4<T>::type *__restrict__ tc,
                                        const uint8_t *__restrict__ tleaf, const int2 *__restrict__ trange,
                                        int same, double theta) {
    typename Vec4<T>::type cs = sc[s], ct = tc[t];
    const T ds = rn_mul((T)2, cs.w), dt = rn_mul((T)2, ct.w);
    if (!(same && s == t)) {
        T dx = rn_sub(cs.x, ct.x), dy = rn_sub(cs.y, ct.y), dz = rn_sub(cs.z, ct.z);
        const T dist = rn_sqrt(rn_fma(dz, dz, rn_fma(dy, dy, rn_mul(dx, dx))));
        if (dist != (T)0 && mac_accepts(ds >= dt ? ds : dt, dist, theta)) return kM2L;
    }
    bool sl = sleaf[s], tl = tleaf[t];
    if (sl && tl) return kP2P;
    if (sl) return kRefineTgt;
    if (tl) return kRefineSrc;
    if ((double)ds > __dmul_rn((double)dt, 1.01)) return kRefineSrc;
    if ((double)dt > __dmul_rn((double)ds, 1.01)) return kRefineTgt;
    int ns = srange[s].y - srange[s].x, nt = trange[t].y - trange[t].x;
    return ns >= nt ? kRefineSrc : kRefineTgt;
}

// the arrays of one tree that the traversal reads
template <typename T> struct TravTree {
    const typename Vec4<T>::type *center;
    const uint8_t *is_leaf;
    const int2 *range;
    const int32_t *children;
};

// ---------------------------------------------------------------------------
// The traversal keeps its counters on the device: front d reads the number of
// its pairs from what front d - 1 counted, so all fronts are launched at once
// and the host reads the counters a single time.  A front whose output does
// not fit writes what fits, goes on counting, and marks itself; later fronts
// then do nothing, and the host grows what was short and starts again at the
// marked front, whose input is still whole.
// ---------------------------------------------------------------------------
constexpr int kMaxLevel = 64;                // max_depth's bound
constexpr int kMaxFronts = 2 * kMaxLevel + 1;  // a refinement adds one level on one side

constexpr int kNoFront = 0x7f7f7f7f;  // four equal bytes

enum { kCntM2L = 0, kCntP2P = 1, kCntNext = 2 };

struct TravState {
    unsigned long long n[kMaxFronts][3];  // M2L pairs, P2P pairs and refined pairs of each front
    unsigned long long interactions;      // sum over P2P pairs of n_source * n_target
    long long scan_total;                 // both lists' pairs
    int full_front;                       // first front whose output did not fit (kNoFront: none)
    int max_row[2];                       // longest P2P and M2L row
};

__global__ void k_trav_init(TravState *st) {
    unsigned long long *z = &st->n[0][0];
    for (int i = threadIdx.x; i < 3 * kMaxFronts; i += blockDim.x) z[i] = 0;
    if (threadIdx.x == 0) st->full_front = kNoFront;
}

constexpr int kFrontThreads = 256;
constexpr unsigned kSrcSide = 0x80000000u;  // a front's pair refines its source side

// One front: the children of every pair of the previous one's refined pairs
// (a thread each), classified and appended to the M2L list, the P2P list or
// the pairs to refine.  Front 0 classifies the roots: (root, root) for every
// root of a same-tree forest, else the pair of both trees' roots (DFS id 0).
// Only pairs that go on are stored: the last front of 100,000 points in a cube
// meets 3.05 M pairs of which none does.  A block counts its 256 pairs by
// ballots, takes its room in the three outputs with one atomic each, and
// writes; the order of the pairs is free, because the CSR rows are sorted and
// the next front is a set.  The nine fronts of 100,000 points take 81 us; with
// every pair stored, three prefix sums and a read by the host in each front
// (and FP64 divisions for all pairs) the fronts took about 1.1 ms.
template <typename T>
__global__ void __launch_bounds__(kFrontThreads) k_front(const int2 *__restrict__ front, int d,
                                                         const int32_t *__restrict__ roots, int64_t n_roots,
                                                         TravTree<T> S, TravTree<T> Tt, int same, double theta,
                                                         int2 *m2l, int64_t cap_m2l, int2 *p2p, int64_t cap_p2p,
                                                         int2 *next, int64_t cap_next, TravState *st) {
    constexpr int kWarps = kFrontThreads / 32;
    __shared__ int wtot[kWarps][3];
    __shared__ int64_t sbase[3];
    if (*(volatile int *)&st->full_front < d) return;
    const int64_t items = d == 0 ? n_roots : 8 * (int64_t)st->n[d - 1][kCntNext];
    if ((int64_t)blockIdx.x * kFrontThreads >= items) return;
    int64_t start = 0;  // where this front's pairs begin in list threadIdx.x
    if (threadIdx.x < kCntNext)
        for (int e = 0; e < d; ++e) start += (int64_t)st->n[e][threadIdx.x];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    for (int64_t t0 = (int64_t)blockIdx.x * kFrontThreads; t0 < items; t0 += (int64_t)gridDim.x * kFrontThreads) {
        const int64_t i = t0 + threadIdx.x;
        int2 pr = make_int2(0, 0);
        bool live = i < items;
        if (live && d == 0) {
            if (n_roots > 1) pr.x = pr.y = roots[i];
        } else if (live) {
            pr = front[i >> 3];
            const bool src = (unsigned)pr.x & kSrcSide;
            pr.x = (int)((unsigned)pr.x & ~kSrcSide);
            const int c = src ? S.children[8 * (int64_t)pr.x + (i & 7)] : Tt.children[8 * (int64_t)pr.y + (i & 7)];
            live = c >= 0;
            if (src) pr.x = c;
            else pr.y = c;
        }
        int code = -1;
        if (live)
            code = classify<T>(pr.x, pr.y, S.center, S.is_leaf, S.range, Tt.center, Tt.is_leaf, Tt.range, same, theta);
        const unsigned bm = __ballot_sync(0xffffffffu, code == kM2L);
        const unsigned bp = __ballot_sync(0xffffffffu, code == kP2P);
        const unsigned br = __ballot_sync(0xffffffffu, code >= kRefineSrc);
        if (lane == 0) {
            wtot[w][kCntM2L] = __popc(bm);
            wtot[w][kCntP2P] = __popc(bp);
            wtot[w][kCntNext] = __popc(br);
        }
        __syncthreads();
        if (threadIdx.x < 3) {
            const int k = threadIdx.x;
            int run = 0;
#pragma unroll
            for (int ww = 0; ww < kWarps; ++ww) {
                const int v = wtot[ww][k];
                wtot[ww][k] = run;
                run += v;
            }
            const int64_t base = start + (run > 0 ? (int64_t)atomicAdd(&st->n[d][k], (unsigned long long)run) : 0);
            sbase[k] = base;
            const int64_t cap = k == kCntM2L ? cap_m2l : (k == kCntP2P ? cap_p2p : cap_next);
            if (run > 0 && base + run > cap) atomicMin(&st->full_front, d);
        }
        __syncthreads();
        if (code == kM2L) {
            const int64_t q = sbase[kCntM2L] + wtot[w][kCntM2L] + __popc(bm & lt);
            if (q < cap_m2l) m2l[q] = pr;
        } else if (code == kP2P) {
            const int64_t q = sbase[kCntP2P] + wtot[w][kCntP2P] + __popc(bp & lt);
            if (q < cap_p2p) p2p[q] = pr;
        } else if (code >= kRefineSrc) {
            const int64_t q = sbase[kCntNext] + wtot[w][kCntNext] + __popc(br & lt);
            if (code == kRefineSrc) pr.x = (int)((unsigned)pr.x | kSrcSide);
            if (q < cap_next) next[q] = pr;
        }
        __syncthreads();  // wtot and sbase are written again
    }
}

// ---------------------------------------------------------------------------
// CSR rows of up to two pair lists at once (list = blockIdx.y): list 0 is
// P2P, list 1 M2L.  Row counts of both lists lie in one array, cnt[l * rows + r],
// so that one prefix sum serves both.
// ---------------------------------------------------------------------------
struct PairLists {
    const int2 *pairs[2];
    int64_t n[2];         // pairs of each list; -1: counted on the device
    const TravState *st;  // the traversal's counters (n == -1)
    int key_x;            // rows keyed by .x (the swapped pair order) instead of .y
};

__device__ __forceinline__ int64_t list_size(const PairLists &P, int l) {
    if (P.n[l] >= 0) return P.n[l];
    if (P.st->full_front != kNoFront) return 0;  // the traversal starts again
    int64_t n = 0;
    for (int e = 0; e < kMaxFronts; ++e) n += (int64_t)P.st->n[e][l == 0 ? kCntP2P : kCntM2L];
    return n;
}

// pairs of each row, and for list 0 the source points of each row (work)
__global__ void __launch_bounds__(256) k_row_counts(PairLists P, int64_t rows, int32_t *cnt, int32_t *work,
                                                    const int2 *__restrict__ srange) {
    const int l = blockIdx.y;
    __shared__ int64_t sn;
    if (threadIdx.x == 0) sn = list_size(P, l);
    __syncthreads();
    const int64_t n = sn;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int2 p = P.pairs[l][i];
        const int r = P.key_x ? p.y : p.x;  // the pair's value
        const int64_t row = P.key_x ? p.x : p.y;
        atomicAdd(&cnt[l * rows + row], 1);
        if (l == 0 && work) atomicAdd(&work[row], srange[r].y - srange[r].x);
    }
}

// row offsets from the prefix sum over both lists' counts (list l's rows start
// at sum[l * rows]; the difference is exact modulo 2^32), the longest rows and
// the number of near-field interactions
__global__ void __launch_bounds__(256) k_rows_finish(const int32_t *__restrict__ cnt, const int32_t *__restrict__ sum,
                                                     int64_t rows, int32_t *off0, int32_t *off1,
                                                     const int32_t *__restrict__ work,
                                                     const int2 *__restrict__ trange, TravState *st) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int c0 = 0, c1 = 0;
    unsigned long long v = 0;
    const int32_t base1 = off1 ? sum[rows] : 0;
    if (i < rows) {
        c0 = cnt[i];
        off0[i] = sum[i];
        if (i == rows - 1) off0[rows] = sum[i] + c0;
        if (off1) {
            c1 = cnt[rows + i];
            off1[i] = sum[rows + i] - base1;
            if (i == rows - 1) off1[rows] = sum[rows + i] - base1 + c1;
        }
        if (work) v = (unsigned long long)work[i] * (unsigned long long)(trange[i].y - trange[i].x);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        c0 = max(c0, __shfl_xor_sync(0xffffffffu, c0, o));
        c1 = max(c1, __shfl_xor_sync(0xffffffffu, c1, o));
        v += __shfl_xor_sync(0xffffffffu, v, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (c0 > 0) atomicMax(&st->max_row[0], c0);
        if (c1 > 0) atomicMax(&st->max_row[1], c1);
        if (v > 0) atomicAdd(&st->interactions, v);
    }
}

// each pair's value into its row, from the row's end (cnt counts down)
__global__ void __launch_bounds__(256) k_row_fill(PairLists P, int64_t rows, int32_t *cnt,
                                                  const int32_t *__restrict__ off0, const int32_t *__restrict__ off1,
                                                  int32_t *vals0, int32_t *vals1) {
    const int l = blockIdx.y;
    const int64_t n = P.n[l];
    const int32_t *off = l ? off1 : off0;
    int32_t *vals = l ? vals1 : vals0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int2 p = P.pairs[l][i];
        const int row = P.key_x ? p.x : p.y;
        vals[off[row] + atomicSub(&cnt[l * rows + row], 1) - 1] = P.key_x ? p.y : p.x;
    }
}

// ---------------------------------------------------------------------------
// Launch orders: the target tree's leaves by decreasing near-field work, in
// buckets of log2(work) in quarter steps, and its nodes by decreasing M2L pair
// count, in 256 buckets of equal width (single counts up to a longest row of
// 255).  A stable counting sort by chunks of 1024: histograms of both orders
// in one launch, one prefix sum over (bucket, chunk), stable ranks inside a
// chunk; within a bucket the tree order stays, so the orders are
// deterministic.
// ---------------------------------------------------------------------------
constexpr int kOrderChunk = 1024;
constexpr int kBuckets = 256;

struct OrderArgs {
    const int32_t *leaves;  // order 0: items are leaves[i]
    int64_t n[2];           // leaves, nodes
    int nb;                 // chunks of the longer order
    const int32_t *work;    // source points per target node
    const int2 *trange;
    const int32_t *m2l_off;
    const TravState *st;
};

__device__ __forceinline__ int order_bucket(const OrderArgs &A, int l, int64_t i) {
    int b;
    if (l == 0) {
        const int t = A.leaves[i];
        // one more than the interactions: a leaf without sources still writes its result
        const long long v = (long long)A.work[t] * (A.trange[t].y - A.trange[t].x) + 1;
        const int e = 63 - __clzll(v);  // v = 2^e * m, m in [1, 2)
        const float m = (float)((double)v / (double)(1ll << e));
        b = 4 * e + (m >= 1.68179283f ? 3 : (m >= 1.41421356f ? 2 : (m >= 1.18920712f ? 1 : 0)));
    } else {
        const int c = A.m2l_off[i + 1] - A.m2l_off[i], top = A.st->max_row[1];
        b = top < kBuckets ? c : (int)((int64_t)c * (kBuckets - 1) / top);
    }
    return kBuckets - 1 - min(b, kBuckets - 1);
}

__global__ void __launch_bounds__(kOrderChunk) k_order_hist(OrderArgs A, int32_t *hist) {
    const int l = blockIdx.y;
    __shared__ int h[kBuckets];
    if (threadIdx.x < kBuckets) h[threadIdx.x] = 0;
    __syncthreads();
    const int64_t i = (int64_t)blockIdx.x * kOrderChunk + threadIdx.x;
    if (i < A.n[l]) atomicAdd(&h[order_bucket(A, l, i)], 1);
    __syncthreads();
    if (threadIdx.x < kBuckets) hist[((int64_t)l * kBuckets + threadIdx.x) * A.nb + blockIdx.x] = h[threadIdx.x];
}

__global__ void __launch_bounds__(kOrderChunk) k_order_place(OrderArgs A, const int32_t *__restrict__ sum,
                                                             int32_t *out0, int32_t *out1) {
    constexpr int kWarps = kOrderChunk / 32;
    const int l = blockIdx.y;
    __shared__ unsigned short wc[kWarps][kBuckets];
    for (int k = threadIdx.x; k < kWarps * kBuckets; k += kOrderChunk) (&wc[0][0])[k] = 0;
    __syncthreads();
    const int64_t i = (int64_t)blockIdx.x * kOrderChunk + threadIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const bool live = i < A.n[l];
    const int b = live ? order_bucket(A, l, i) : kBuckets;
    const unsigned peers = __match_any_sync(0xffffffffu, b);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    if (live && rank == 0) wc[w][b] = (unsigned short)__popc(peers);
    __syncthreads();
    if (threadIdx.x < kBuckets) {
        int run = 0;
        for (int ww = 0; ww < kWarps; ++ww) {
            const int v = wc[ww][threadIdx.x];
            wc[ww][threadIdx.x] = (unsigned short)run;
            run += v;
        }
    }
    __syncthreads();
    if (!live) return;
    int64_t q = (int64_t)sum[((int64_t)l * kBuckets + b) * A.nb + blockIdx.x] + wc[w][b] + rank;
    if (l == 0) out0[q] = A.leaves[i];
    else out1[q - A.n[0]] = (int32_t)i;
}

// transposed CSR from a CSR: pairs (row -> val) become (val -> row)
__global__ void k_csr_to_pairs(const int32_t *off, const int32_t *vals, int64_t rows, int2 *pairs) {
    int64_t r = (int64_t)blockIdx.x * blockDim.y + threadIdx.y;
    if (r >= rows) return;
    for (int k = off[r] + threadIdx.x; k < off[r + 1]; k += blockDim.x) pairs[k] = make_int2(vals[k], (int)r);
}

inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }
// blocks of a grid-stride pass over n items (the passes are memory bound: 8
// blocks of 256 threads fill an SM)
inline unsigned stride_blocks(int64_t n) { return (unsigned)std::min<int64_t>(std::max<int64_t>(nblk(n, 256), 1), 152 * 8); }

// growable pair buffer
struct PairBuf {
    DevBuf buf;
    int64_t cap = 0;
    // room for `want` pairs, at least doubled; the first `keep` pairs stay
    int grow(int64_t want, int64_t keep, cudaStream_t s) {
        if (want <= cap) return EDFMM_OK;
        const int64_t nc = std::max<int64_t>(want, cap * 2);
        DevBuf nb;
        if (int rc = nb.reserve(sizeof(int2) * nc)) return rc;
        if (keep > 0) EDFMM_CUDA_TRY(cudaMemcpyAsync(nb.p, buf.p, sizeof(int2) * keep, cudaMemcpyDeviceToDevice, s));
        EDFMM_CUDA_TRY(cudaStreamSynchronize(s));  // the old block may be freed
        buf = std::move(nb);
        cap = nc;
        return EDFMM_OK;
    }
};

// L.p2p_leaves and L.m2l_rows
int order_rows(const DevTree &tree, const int32_t *work, const TravState *st, DevLists &L, cudaStream_t s) {
    const int64_t nl = std::max<int64_t>(tree.n_leaves, 0), M = tree.n_nodes;
    int rc;
    DevBuf hist, sum, tmp;
    OrderArgs A;
    A.leaves = dptr<int32_t>(tree.leaves);
    A.n[0] = nl;
    A.n[1] = M;
    A.nb = (int)((std::max(nl, M) + kOrderChunk - 1) / kOrderChunk);
    A.work = work;
    A.trange = dptr<int2>(tree.range);
    A.m2l_off = dptr<int32_t>(L.m2l_off);
    A.st = st;
    const int64_t nh = 2 * (int64_t)kBuckets * A.nb;
    if ((rc = L.p2p_leaves.reserve(sizeof(int32_t) * std::max<int64_t>(nl, 1))) ||
        (rc = L.m2l_rows.reserve(sizeof(int32_t) * M)) || (rc = hist.reserve(sizeof(int32_t) * nh)) ||
        (rc = sum.reserve(sizeof(int32_t) * nh)) || (rc = tmp.reserve(scan_tmp_bytes(nh))))
        return rc;
    const dim3 grid((unsigned)A.nb, 2);
    k_order_hist<<<grid, kOrderChunk, 0, s>>>(A, dptr<int32_t>(hist));
    EDFMM_LAUNCH_CHECK("k_order_hist");
    if ((rc = scan_exclusive(dptr<int32_t>(hist), dptr<int32_t>(sum), nh, nullptr, tmp.p, s))) return rc;
    k_order_place<<<grid, kOrderChunk, 0, s>>>(A, dptr<int32_t>(sum), dptr<int32_t>(L.p2p_leaves),
                                               dptr<int32_t>(L.m2l_rows));
    EDFMM_LAUNCH_CHECK("k_order_place");
    return EDFMM_OK;
}

template <typename T>
int lists_impl(const DevTree &stree, const DevTree &tree, double theta, DevLists &L, cudaStream_t s) {
    using T4 = typename Vec4<T>::type;
    int rc;
    const int64_t M = tree.n_nodes;  // rows: target-tree nodes
    const int same = &stree == &tree ? 1 : 0;
    const TravTree<T> S{dptr<T4>(stree.center), dptr<uint8_t>(stree.is_leaf), dptr<int2>(stree.range),
                        dptr<int32_t>(stree.children)};
    const TravTree<T> Tt{dptr<T4>(tree.center), dptr<uint8_t>(tree.is_leaf), dptr<int2>(tree.range),
                         dptr<int32_t>(tree.children)};
    L = DevLists();
    if (M == 0 || stree.n_nodes == 0) {  // rows of nothing
        const size_t rows = sizeof(int32_t) * (size_t)(M + 1);
        if ((rc = L.p2p_off.reserve(rows)) || (rc = L.m2l_off.reserve(rows)) || (rc = L.p2p_src.reserve(4)) ||
            (rc = L.m2l_src.reserve(4)))
            return rc;
        EDFMM_CUDA_TRY(cudaMemsetAsync(L.p2p_off.p, 0, rows, s));
        EDFMM_CUDA_TRY(cudaMemsetAsync(L.m2l_off.p, 0, rows, s));
        return EDFMM_OK;
    }
    // a same-tree forest (batched plan) starts from every (root, root) pair;
    // no pair ever joins two trees, so each tree gets its own lists
    const int n_roots = same && tree.level_offsets.size() > 1 ? tree.level_offsets[1] - tree.level_offsets[0] : 1;
    const int n_fronts = std::min(stree.max_level + tree.max_level + 1, kMaxFronts);
    // first capacities: 640 M2L, 160 P2P and 160 front pairs a node hold the
    // lists of 100,000 points in a cube (589, 103 and 89 at theta 0.5; a
    // surface's are a fifth of that); at most 32 MB each before any pair is known
    const int64_t nodes = std::max(M, stree.n_nodes), most = 4 << 20;
    const int64_t g_m2l = std::min(640 * nodes, most), g_p2p = std::min(160 * nodes, most);
    PairBuf m2l, p2p, front[2];
    DevBuf state, cnt, work, sum, tmp;
    if ((rc = state.reserve(sizeof(TravState))) || (rc = cnt.reserve(sizeof(int32_t) * 3 * M)) ||
        (rc = sum.reserve(sizeof(int32_t) * 2 * M)) || (rc = tmp.reserve(scan_tmp_bytes(2 * M))) ||
        (rc = L.p2p_off.reserve(sizeof(int32_t) * (M + 1))) || (rc = L.m2l_off.reserve(sizeof(int32_t) * (M + 1))) ||
        (rc = m2l.grow(g_m2l, 0, s)) || (rc = p2p.grow(g_p2p, 0, s)) ||
        (rc = front[0].grow(g_p2p, 0, s)) || (rc = front[1].grow(g_p2p, 0, s)))
        return rc;
    TravState *st = dptr<TravState>(state);
    int32_t *wk = dptr<int32_t>(cnt) + 2 * M;
    TravState h;
    k_trav_init<<<1, 256, 0, s>>>(st);
    EDFMM_LAUNCH_CHECK("k_trav_init");
    PairLists P;
    for (int d0 = 0;;) {
        for (int d = d0; d < n_fronts; ++d) {
            PairBuf &out = front[(d + 1) & 1];
            k_front<T><<<152 * 4, kFrontThreads, 0, s>>>(dptr<int2>(front[d & 1].buf), d, dptr<int32_t>(tree.level_nodes),
                                                         n_roots, S, Tt, same, theta,
                                                         dptr<int2>(m2l.buf), m2l.cap, dptr<int2>(p2p.buf), p2p.cap,
                                                         dptr<int2>(out.buf), out.cap, st);
            EDFMM_LAUNCH_CHECK("k_front");
        }
        // rows of both lists (of nothing, when a front did not fit)
        P = PairLists{{dptr<int2>(p2p.buf), dptr<int2>(m2l.buf)}, {-1, -1}, st, 0};
        EDFMM_CUDA_TRY(cudaMemsetAsync(cnt.p, 0, sizeof(int32_t) * 3 * M, s));
        EDFMM_CUDA_TRY(cudaMemsetAsync(st->max_row, 0, sizeof(st->max_row), s));
        EDFMM_CUDA_TRY(cudaMemsetAsync(&st->interactions, 0, sizeof(st->interactions), s));
        k_row_counts<<<dim3(152 * 4, 2), 256, 0, s>>>(P, M, dptr<int32_t>(cnt), wk, dptr<int2>(stree.range));
        EDFMM_LAUNCH_CHECK("k_row_counts");
        if ((rc = scan_exclusive(dptr<int32_t>(cnt), dptr<int32_t>(sum), 2 * M, nullptr, tmp.p, s))) return rc;
        k_rows_finish<<<nblk(M, 256), 256, 0, s>>>(dptr<int32_t>(cnt), dptr<int32_t>(sum), M, dptr<int32_t>(L.p2p_off),
                                                   dptr<int32_t>(L.m2l_off), wk, dptr<int2>(tree.range), st);
        EDFMM_LAUNCH_CHECK("k_rows_finish");
        EDFMM_CUDA_TRY(cudaMemcpyAsync(&h, st, sizeof(h), cudaMemcpyDeviceToHost, s));
        EDFMM_CUDA_TRY(cudaStreamSynchronize(s));
        const int last = std::min(h.full_front, n_fronts - 1);  // fronts after a full one counted nothing
        int64_t nm = 0, np = 0;
        for (int d = 0; d <= last; ++d) {
            nm += (int64_t)h.n[d][kCntM2L];
            np += (int64_t)h.n[d][kCntP2P];
            if (nm >= INT32_MAX || np >= INT32_MAX || (int64_t)h.n[d][kCntNext] >= INT32_MAX)
                return fail(EDFMM_ERR_ARG, "interaction lists exceed 2^31 pairs");
        }
        if (h.full_front == kNoFront) {
            L.n_m2l = nm;
            L.n_p2p = np;
            break;
        }
        // grow what front d0 did not fit into, forget its counts, run it again
        d0 = h.full_front;
        PairBuf &out = front[(d0 + 1) & 1];
        if ((rc = m2l.grow(nm, std::min(nm - (int64_t)h.n[d0][kCntM2L], m2l.cap), s)) ||
            (rc = p2p.grow(np, std::min(np - (int64_t)h.n[d0][kCntP2P], p2p.cap), s)) ||
            (rc = out.grow((int64_t)h.n[d0][kCntNext], 0, s)))
            return rc;
        EDFMM_CUDA_TRY(cudaMemsetAsync(st->n[d0], 0, sizeof(st->n[d0]), s));
        EDFMM_CUDA_TRY(cudaMemsetAsync(&st->full_front, 0x7f, sizeof(int), s));
    }
    L.p2p_interactions = (int64_t)h.interactions;
    L.max_p2p_row = h.max_row[0];
    L.max_m2l_row = h.max_row[1];
    if ((rc = L.p2p_src.reserve(sizeof(int32_t) * std::max<int64_t>(L.n_p2p, 1))) ||
        (rc = L.m2l_src.reserve(sizeof(int32_t) * std::max<int64_t>(L.n_m2l, 1))))
        return rc;
    P.n[0] = L.n_p2p;
    P.n[1] = L.n_m2l;
    k_row_fill<<<dim3(stride_blocks(std::max(L.n_p2p, L.n_m2l)), 2), 256, 0, s>>>(
        P, M, dptr<int32_t>(cnt), dptr<int32_t>(L.p2p_off), dptr<int32_t>(L.m2l_off), dptr<int32_t>(L.p2p_src),
        dptr<int32_t>(L.m2l_src));
    EDFMM_LAUNCH_CHECK("k_row_fill");
    if ((rc = sort_csr_rows(dptr<int32_t>(L.p2p_off), dptr<int32_t>(L.p2p_src), M, L.max_p2p_row, stree.n_nodes, s)) ||
        (rc = sort_csr_rows(dptr<int32_t>(L.m2l_off), dptr<int32_t>(L.m2l_src), M, L.max_m2l_row, stree.n_nodes, s)))
        return rc;
    return order_rows(tree, wk, st, L, s);
}

}  // namespace

int lists_build(const DevTree &tree, double theta, DevLists &lists, cudaStream_t s) {
    if (tree.dtype == EDFMM_F64) return lists_impl<double>(tree, tree, theta, lists, s);
    return lists_impl<float>(tree, tree, theta, lists, s);
}

int lists_build_two(const DevTree &src_tree, const DevTree &tgt_tree, double theta, DevLists &lists, cudaStream_t s) {
    if (src_tree.dtype != tgt_tree.dtype) return fail(EDFMM_ERR_ARG, "source and target trees differ in dtype");
    if (src_tree.dtype == EDFMM_F64) return lists_impl<double>(src_tree, tgt_tree, theta, lists, s);
    return lists_impl<float>(src_tree, tgt_tree, theta, lists, s);
}

int lists_build_swapped(const DevTree &tree, DevLists &L, cudaStream_t s) {
    if (L.have_m2l_swapped) return EDFMM_OK;
    int rc;
    const int64_t M = tree.n_nodes;
    DevBuf pairs;
    if ((rc = pairs.reserve(sizeof(int2) * std::max<int64_t>(L.n_m2l, 1)))) return rc;
    if (M > 0) {
        dim3 blk(32, 8);
        k_csr_to_pairs<<<nblk(M, 8), blk, 0, s>>>(dptr<int32_t>(L.m2l_off), dptr<int32_t>(L.m2l_src), M, dptr<int2>(pairs));
        EDFMM_LAUNCH_CHECK("k_csr_to_pairs");
    }
    // pairs are (src, tgt); the swapped rows are keyed on src
    const int64_t rows = std::max<int64_t>(M, 1), n = L.n_m2l;
    DevBuf state, cnt, sum, tmp;
    if ((rc = state.reserve(sizeof(TravState))) || (rc = cnt.reserve(sizeof(int32_t) * rows)) ||
        (rc = sum.reserve(sizeof(int32_t) * rows)) || (rc = tmp.reserve(scan_tmp_bytes(rows))) ||
        (rc = L.m2l_swapped_off.reserve(sizeof(int32_t) * (rows + 1))) ||
        (rc = L.m2l_swapped_src.reserve(sizeof(int32_t) * std::max<int64_t>(n, 1))))
        return rc;
    TravState *st = dptr<TravState>(state);
    const PairLists P{{dptr<int2>(pairs), nullptr}, {n, 0}, nullptr, 1};
    int mx = 0;
    EDFMM_CUDA_TRY(cudaMemsetAsync(cnt.p, 0, sizeof(int32_t) * rows, s));
    EDFMM_CUDA_TRY(cudaMemsetAsync(st->max_row, 0, sizeof(st->max_row), s));
    k_row_counts<<<stride_blocks(n), 256, 0, s>>>(P, rows, dptr<int32_t>(cnt), nullptr, nullptr);
    EDFMM_LAUNCH_CHECK("k_row_counts");
    if ((rc = scan_exclusive(dptr<int32_t>(cnt), dptr<int32_t>(sum), rows, nullptr, tmp.p, s))) return rc;
    k_rows_finish<<<nblk(rows, 256), 256, 0, s>>>(dptr<int32_t>(cnt), dptr<int32_t>(sum), rows,
                                                  dptr<int32_t>(L.m2l_swapped_off), nullptr, nullptr, nullptr, st);
    EDFMM_LAUNCH_CHECK("k_rows_finish");
    k_row_fill<<<stride_blocks(n), 256, 0, s>>>(P, rows, dptr<int32_t>(cnt), dptr<int32_t>(L.m2l_swapped_off), nullptr,
                                                dptr<int32_t>(L.m2l_swapped_src), nullptr);
    EDFMM_LAUNCH_CHECK("k_row_fill");
    EDFMM_CUDA_TRY(cudaMemcpyAsync(&mx, &st->max_row[0], sizeof(int), cudaMemcpyDeviceToHost, s));
    EDFMM_CUDA_TRY(cudaStreamSynchronize(s));
    if ((rc = sort_csr_rows(dptr<int32_t>(L.m2l_swapped_off), dptr<int32_t>(L.m2l_swapped_src), rows, mx, rows, s))) return rc;
    L.have_m2l_swapped = true;
    return EDFMM_OK;
}

}  // namespace edfmm
