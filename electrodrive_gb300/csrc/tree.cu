// GPU construction of the adaptive tight-bbox octree.
//
// The reference builds the tree with a depth-first Python recursion
// (electrodrive/fmm3d/tree.py:801-960).  Here the same tree is built one
// level at a time:
//   * every node of a level reduces the tight bounding box of its point range
//     (exact min/max via order-preserving integer atomics, so the result does
//     not depend on the reduction order);
//   * centre = 0.5 * (min + max), half = max(0.5 * (max - min), 0) and the
//     radius = sqrt(fma(hz, hz, fma(hy, hy, hx * hx))) * (1 + 1e-12) are
//     formed with the same roundings as the reference's torch ops;
//   * a node splits unless n <= leaf_size, level >= max_depth or
//     max(half) < 1e-7 (tree.py:895-897);
//   * points are partitioned stably by octant (x > cx) + 2 (y > cy) + 4 (z > cz)
//     with chunked counting (per-chunk octant counts, per-node prefix over its
//     chunks, ballot ranks inside a chunk), which reproduces the reference's
//     stable counting sort (tree.py:921-939);
//   * the final DFS pre-order numbering (tree.py:878-889) equals the rank of
//     each node by (range start, level): nodes sharing a start form a chain
//     of first children, so dfs = #nodes with smaller start + depth inside
//     the chain.
// Points move between two buffers level by level; a leaf's points go to their
// final place in the level that finds the leaf.  The set-up is bound by
// launches and by the host's one read a level (the number of children): a
// level whose nodes all hold at most 1024 points, which is every level but
// the first two or three, is a single kernel with a block per node.  A whole
// plan (tree, lists, buffers), created and destroyed: 100,003 points in a
// cube 4.9 -> 0.90 ms, 2,003 points 1.17 -> 0.58 ms, 1,048,576 points 14.4 ->
// 3.9 ms against two reads a level, 13 launches a level and a copy of the
// points back into place.
#include <algorithm>
#include <cfloat>

#include "edfmm_internal.cuh"

namespace edfmm {

namespace {

constexpr int kChunk = 1024;  // points per chunk, one thread per point

// order-preserving float <-> int maps for exact atomic min / max
__device__ __forceinline__ int ord_of(float f) {
    int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float from_ord(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }
__device__ __forceinline__ long long ord_of(double f) {
    long long i = __double_as_longlong(f);
    return i >= 0 ? i : i ^ 0x7fffffffffffffffLL;
}
__device__ __forceinline__ double from_ord(long long i) {
    return __longlong_as_double(i >= 0 ? i : i ^ 0x7fffffffffffffffLL);
}

template <typename T> struct OrdT {};
template <> struct OrdT<float> {
    using type = int;
    static constexpr int hi = 0x7fffffff;
    static constexpr int lo = (int)0x80000000;
};
template <> struct OrdT<double> {
    using type = long long;
    static constexpr long long hi = 0x7fffffffffffffffLL;
    static constexpr long long lo = (long long)0x8000000000000000ULL;
};

// exact-rounding helpers (no contraction across these)
__device__ __forceinline__ float rn_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double rn_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float rn_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double rn_sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float rn_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double rn_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float rn_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double rn_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float rn_sqrt(float a) { return __fsqrt_rn(a); }
__device__ __forceinline__ double rn_sqrt(double a) { return __dsqrt_rn(a); }

// radius = ||h|| * (1 + 1e-12) rounded in T (tree.py:331)
__device__ __forceinline__ float radius_of(float hx, float hy, float hz) {
    float r = rn_sqrt(rn_fma(hz, hz, rn_fma(hy, hy, rn_mul(hx, hx))));
    return rn_mul(r, (float)(1.0 + 1e-12));
}
__device__ __forceinline__ double radius_of(double hx, double hy, double hz) {
    double r = rn_sqrt(rn_fma(hz, hz, rn_fma(hy, hy, rn_mul(hx, hx))));
    return rn_mul(r, 1.0 + 1e-12);
}

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------

// what the host reads back after each level
struct BuildState {
    int64_t next;          // nodes of the next level
    int32_t leaves, warn;  // leaves so far, leaves above leaf_size at max_depth
    int32_t max_child[66]; // points of the largest node of each level
};

// points into tree layout, and the roots (one, or one per instance)
template <typename T>
__global__ void k_init_points(const T *__restrict__ pts, int64_t n, typename Vec4<T>::type *xyz, int32_t *perm,
                              const int64_t *inst_off, int K0, int2 *rng, int32_t *parent, int32_t *root) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < K0) {
        rng[i] = inst_off ? make_int2((int)inst_off[i], (int)inst_off[i + 1]) : make_int2(0, (int)n);
        parent[i] = -1;
        root[i] = (int32_t)i;
    }
    if (i >= n) return;
    typename Vec4<T>::type v;
    v.x = pts[3 * i];
    v.y = pts[3 * i + 1];
    v.z = pts[3 * i + 2];
    v.w = 0;
    xyz[i] = v;
    perm[i] = (int32_t)i;
}

// chunk counts per node of the level; empty bounding boxes
template <typename T>
__global__ void k_chunk_counts(const int2 *rng, int K, int32_t *cnt, typename OrdT<T>::type *bb) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= K) return;
    int n = rng[i].y - rng[i].x;
    cnt[i] = (n + kChunk - 1) / kChunk;
    for (int a = 0; a < 3; ++a) {
        bb[6 * i + a] = OrdT<T>::hi;      // min
        bb[6 * i + 3 + a] = OrdT<T>::lo;  // max
    }
}

__global__ void k_chunk_fill(const int2 *rng, int K, const int32_t *chunk_off, int32_t *chunk_node) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= K) return;
    int n = rng[i].y - rng[i].x;
    int c = (n + kChunk - 1) / kChunk;
    int b = chunk_off[i];
    for (int k = 0; k < c; ++k) chunk_node[b + k] = i;
}

template <typename T>
__global__ void __launch_bounds__(kChunk) k_bbox(const typename Vec4<T>::type *__restrict__ xyz, const int2 *rng,
                                                 const int32_t *chunk_node, const int32_t *chunk_off,
                                                 const int64_t *n_chunks, typename OrdT<T>::type *bb) {
    using O = typename OrdT<T>::type;
    int q = blockIdx.x;
    if (q >= *n_chunks) return;  // the grid is a bound on the level's chunks
    int node = chunk_node[q];
    int k = q - chunk_off[node];
    int s = rng[node].x + k * kChunk;
    int e = min(rng[node].y, s + kChunk);
    int i = s + threadIdx.x;
    O mn[3] = {OrdT<T>::hi, OrdT<T>::hi, OrdT<T>::hi}, mx[3] = {OrdT<T>::lo, OrdT<T>::lo, OrdT<T>::lo};
    if (i < e) {
        typename Vec4<T>::type v = xyz[i];
        mn[0] = mx[0] = ord_of(v.x);
        mn[1] = mx[1] = ord_of(v.y);
        mn[2] = mx[2] = ord_of(v.z);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            O y = __shfl_xor_sync(0xffffffffu, mn[a], o);
            mn[a] = y < mn[a] ? y : mn[a];
            O z = __shfl_xor_sync(0xffffffffu, mx[a], o);
            mx[a] = z > mx[a] ? z : mx[a];
        }
    }
    __shared__ O smn[32][3], smx[32][3];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0)
        for (int a = 0; a < 3; ++a) {
            smn[w][a] = mn[a];
            smx[w][a] = mx[a];
        }
    __syncthreads();
    if (threadIdx.x < 3) {
        int a = threadIdx.x;
        O m0 = smn[0][a], m1 = smx[0][a];
        for (int ww = 1; ww < (int)(blockDim.x >> 5); ++ww) {
            m0 = smn[ww][a] < m0 ? smn[ww][a] : m0;
            m1 = smx[ww][a] > m1 ? smx[ww][a] : m1;
        }
        atomicMin(&bb[6 * node + a], m0);
        atomicMax(&bb[6 * node + 3 + a], m1);
    }
}

// centre / half / radius of a node from its bounding box; true if it is a leaf
template <typename T>
__device__ __forceinline__ bool node_geometry(const T *mn, const T *mx, int n, int level, int leaf_size, int max_depth,
                                              typename Vec4<T>::type &cv, typename Vec4<T>::type &hv, bool &too_deep) {
    T c[3], h[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        c[a] = rn_mul((T)0.5, rn_add(mn[a], mx[a]));
        T hh = rn_mul((T)0.5, rn_sub(mx[a], mn[a]));
        h[a] = hh < (T)0 ? (T)0 : hh;
    }
    cv.x = c[0];
    cv.y = c[1];
    cv.z = c[2];
    cv.w = radius_of(h[0], h[1], h[2]);
    hv.x = h[0];
    hv.y = h[1];
    hv.z = h[2];
    hv.w = 0;  // expansion scale, filled after the root radius is known
    T hmax = h[0] > h[1] ? h[0] : h[1];
    hmax = hmax > h[2] ? hmax : h[2];
    const bool degenerate = (double)hmax < 1e-7;
    too_deep = level >= max_depth && n > leaf_size && !degenerate;
    return n <= leaf_size || level >= max_depth || degenerate;
}

// centre / half / radius / leaf decision for every node of the level
template <typename T>
__global__ void k_finalize(const typename OrdT<T>::type *bb, const int2 *rng, int K, int level, int leaf_size,
                           int max_depth, typename Vec4<T>::type *center, typename Vec4<T>::type *half,
                           uint8_t *is_leaf, int32_t *lev, BuildState *st) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= K) return;
    T mn[3], mx[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        mn[a] = from_ord(bb[6 * i + a]);
        mx[a] = from_ord(bb[6 * i + 3 + a]);
    }
    typename Vec4<T>::type cv, hv;
    bool deep;
    const bool leaf = node_geometry<T>(mn, mx, rng[i].y - rng[i].x, level, leaf_size, max_depth, cv, hv, deep);
    center[i] = cv;
    half[i] = hv;
    is_leaf[i] = leaf ? 1 : 0;
    lev[i] = level;
    if (leaf) atomicAdd(&st->leaves, 1);
    if (deep) atomicAdd(&st->warn, 1);
}

template <typename T>
__device__ __forceinline__ int octant_of(const typename Vec4<T>::type &p, const typename Vec4<T>::type &c) {
    return (p.x > c.x ? 1 : 0) + (p.y > c.y ? 2 : 0) + (p.z > c.z ? 4 : 0);
}

// per-chunk octant counts (chunks of split nodes only)
template <typename T>
__global__ void __launch_bounds__(kChunk) k_octant_counts(const typename Vec4<T>::type *__restrict__ xyz,
                                                          const int2 *rng, const int32_t *chunk_node,
                                                          const int32_t *chunk_off, const int64_t *n_chunks,
                                                          const typename Vec4<T>::type *center,
                                                          const uint8_t *is_leaf, int32_t *ccnt) {
    int q = blockIdx.x;
    if (q >= *n_chunks) return;
    int node = chunk_node[q];
    if (is_leaf[node]) return;
    __shared__ int cnt[8];
    if (threadIdx.x < 8) cnt[threadIdx.x] = 0;
    __syncthreads();
    int k = q - chunk_off[node];
    int s = rng[node].x + k * kChunk;
    int e = min(rng[node].y, s + kChunk);
    int i = s + threadIdx.x;
    if (i < e) atomicAdd(&cnt[octant_of<T>(xyz[i], center[node])], 1);
    __syncthreads();
    if (threadIdx.x < 8) ccnt[8 * q + threadIdx.x] = cnt[threadIdx.x];
}

// per split node: exclusive prefix of octant counts over its chunks, totals
__global__ void k_node_octants(const int2 *rng, int K, const int32_t *chunk_off, const uint8_t *is_leaf,
                               int32_t *ccnt, int32_t *oct_start, int32_t *oct_cnt, int32_t *n_children,
                               int32_t *max_child) {
    // all 32 lanes stay to the end: the shuffles below use the full mask
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    int i = t >> 3, o = t & 7;
    bool active = i < K && !is_leaf[i];
    int run = 0;
    if (active) {
        int n = rng[i].y - rng[i].x;
        int c = (n + kChunk - 1) / kChunk;
        int b = chunk_off[i];
        for (int k = 0; k < c; ++k) {
            int v = ccnt[8 * (b + k) + o];
            ccnt[8 * (b + k) + o] = run;
            run += v;
        }
    }
    // octant start = node start + counts of lower octants (the 8 lanes of one
    // node are consecutive lanes of one warp)
    int base = 0, nz = 0;
    for (int oo = 0; oo < 8; ++oo) {
        int v = __shfl_sync(0xffffffffu, run, (threadIdx.x & 31 & ~7) + oo);
        if (oo < o) base += v;
        nz += v > 0 ? 1 : 0;
    }
    if (i >= K) return;
    oct_cnt[8 * i + o] = run;
    oct_start[8 * i + o] = rng[i].x + base;
    if (o == 0) n_children[i] = nz;
    if (run > 0) atomicMax(max_child, run);
}

// a leaf's points to their final place (the buffer's positions are the tree's)
// or stable scatter of the chunk's points into their octant slots
template <typename T>
__global__ void __launch_bounds__(kChunk) k_scatter(const typename Vec4<T>::type *__restrict__ xyz,
                                                    const int32_t *__restrict__ perm, const int2 *rng,
                                                    const int32_t *chunk_node, const int32_t *chunk_off,
                                                    const int64_t *n_chunks, const typename Vec4<T>::type *center,
                                                    const uint8_t *is_leaf, const int32_t *ccnt,
                                                    const int32_t *oct_start, typename Vec4<T>::type *xyz_out,
                                                    int32_t *perm_out, typename Vec4<T>::type *pts, int32_t *index_map) {
    int q = blockIdx.x;
    if (q >= *n_chunks) return;
    int node = chunk_node[q];
    __shared__ int wcnt[32][8];
    int k = q - chunk_off[node];
    int s = rng[node].x + k * kChunk;
    int e = min(rng[node].y, s + kChunk);
    int i = s + threadIdx.x;
    bool valid = i < e;
    if (is_leaf[node]) {
        if (valid) {
            pts[i] = xyz[i];
            index_map[i] = perm[i];
        }
        return;
    }
    int o = -1;
    typename Vec4<T>::type v;
    if (valid) {
        v = xyz[i];
        o = octant_of<T>(v, center[node]);
    }
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned lt = (1u << lane) - 1u;
    int my_rank = 0;
#pragma unroll
    for (int oo = 0; oo < 8; ++oo) {
        unsigned m = __ballot_sync(0xffffffffu, o == oo);
        if (o == oo) my_rank = __popc(m & lt);
        if (lane == 0) wcnt[w][oo] = __popc(m);
    }
    __syncthreads();
    // exclusive scan over warps for each octant
    if (threadIdx.x < 8) {
        int run = 0;
        int nw = blockDim.x >> 5;
        for (int ww = 0; ww < nw; ++ww) {
            int c = wcnt[ww][threadIdx.x];
            wcnt[ww][threadIdx.x] = run;
            run += c;
        }
    }
    __syncthreads();
    if (valid) {
        int dest = oct_start[8 * node + o] + ccnt[8 * q + o] + wcnt[w][o] + my_rank;
        xyz_out[dest] = v;
        perm_out[dest] = perm[i];
    }
}

// A whole level whose nodes hold at most kChunk points each: one block per
// node does the bounding box, the node's geometry, its octants and the stable
// scatter with the points in registers (4 a thread).  Replaces 8 launches and
// three passes over the points.
constexpr int kSmallThreads = 256;
constexpr int kSmallTiles = kChunk / kSmallThreads;

template <typename T>
__global__ void __launch_bounds__(kSmallThreads) k_small_level(
    const typename Vec4<T>::type *__restrict__ xyz, const int32_t *__restrict__ perm, const int2 *rng, int level,
    int leaf_size, int max_depth, typename Vec4<T>::type *center, typename Vec4<T>::type *half, uint8_t *is_leaf,
    int32_t *lev, int32_t *oct_start, int32_t *oct_cnt, int32_t *n_children, typename Vec4<T>::type *xyz_out,
    int32_t *perm_out, typename Vec4<T>::type *pts, int32_t *index_map, BuildState *st) {
    using T4 = typename Vec4<T>::type;
    using O = typename OrdT<T>::type;
    constexpr int kWarps = kSmallThreads / 32;
    __shared__ O smn[kWarps][3], smx[kWarps][3];
    __shared__ T4 sc;
    __shared__ int sleaf;
    __shared__ int wcnt[kSmallTiles * kWarps][8], ostart[8];
    const int node = blockIdx.x;
    const int s = rng[node].x, e = rng[node].y;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T4 v[kSmallTiles];
    O mn[3] = {OrdT<T>::hi, OrdT<T>::hi, OrdT<T>::hi}, mx[3] = {OrdT<T>::lo, OrdT<T>::lo, OrdT<T>::lo};
#pragma unroll
    for (int t = 0; t < kSmallTiles; ++t) {
        const int i = s + t * kSmallThreads + threadIdx.x;
        if (i >= e) continue;
        v[t] = xyz[i];
        const O x = ord_of(v[t].x), y = ord_of(v[t].y), z = ord_of(v[t].z);
        mn[0] = x < mn[0] ? x : mn[0];
        mn[1] = y < mn[1] ? y : mn[1];
        mn[2] = z < mn[2] ? z : mn[2];
        mx[0] = x > mx[0] ? x : mx[0];
        mx[1] = y > mx[1] ? y : mx[1];
        mx[2] = z > mx[2] ? z : mx[2];
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const O y = __shfl_xor_sync(0xffffffffu, mn[a], o);
            mn[a] = y < mn[a] ? y : mn[a];
            const O z = __shfl_xor_sync(0xffffffffu, mx[a], o);
            mx[a] = z > mx[a] ? z : mx[a];
        }
    }
    if (lane == 0)
        for (int a = 0; a < 3; ++a) {
            smn[w][a] = mn[a];
            smx[w][a] = mx[a];
        }
    __syncthreads();
    if (threadIdx.x == 0) {
        T lo[3], hi[3];
        for (int a = 0; a < 3; ++a) {
            O m0 = smn[0][a], m1 = smx[0][a];
            for (int ww = 1; ww < kWarps; ++ww) {
                m0 = smn[ww][a] < m0 ? smn[ww][a] : m0;
                m1 = smx[ww][a] > m1 ? smx[ww][a] : m1;
            }
            lo[a] = from_ord(m0);
            hi[a] = from_ord(m1);
        }
        T4 cv, hv;
        bool deep;
        const bool leaf = node_geometry<T>(lo, hi, e - s, level, leaf_size, max_depth, cv, hv, deep);
        center[node] = cv;
        half[node] = hv;
        is_leaf[node] = leaf ? 1 : 0;
        lev[node] = level;
        if (leaf) {
            n_children[node] = 0;
            atomicAdd(&st->leaves, 1);
        }
        if (deep) atomicAdd(&st->warn, 1);
        sc = cv;
        sleaf = leaf ? 1 : 0;
    }
    __syncthreads();
    if (sleaf) {
#pragma unroll
        for (int t = 0; t < kSmallTiles; ++t) {
            const int i = s + t * kSmallThreads + threadIdx.x;
            if (i >= e) continue;
            pts[i] = v[t];
            index_map[i] = perm[i];
        }
        if (threadIdx.x < 8) oct_cnt[8 * node + threadIdx.x] = 0;
        return;
    }
    const T4 c = sc;
    const unsigned lt = (1u << lane) - 1u;
    int oct[kSmallTiles], rank[kSmallTiles];
#pragma unroll
    for (int t = 0; t < kSmallTiles; ++t) {
        const int i = s + t * kSmallThreads + threadIdx.x;
        oct[t] = i < e ? octant_of<T>(v[t], c) : -1;
        rank[t] = 0;
#pragma unroll
        for (int oo = 0; oo < 8; ++oo) {
            const unsigned m = __ballot_sync(0xffffffffu, oct[t] == oo);
            if (oct[t] == oo) rank[t] = __popc(m & lt);
            if (lane == 0) wcnt[t * kWarps + w][oo] = __popc(m);
        }
    }
    __syncthreads();
    if (threadIdx.x < 8) {
        int run = 0;
        for (int ww = 0; ww < kSmallTiles * kWarps; ++ww) {
            const int q = wcnt[ww][threadIdx.x];
            wcnt[ww][threadIdx.x] = run;
            run += q;
        }
        int base = 0, nz = 0;
        for (int oo = 0; oo < 8; ++oo) {
            const int q = __shfl_sync(0xffu, run, oo);
            if (oo < (int)threadIdx.x) base += q;
            nz += q > 0 ? 1 : 0;
        }
        oct_cnt[8 * node + threadIdx.x] = run;
        oct_start[8 * node + threadIdx.x] = s + base;
        ostart[threadIdx.x] = s + base;
        if (threadIdx.x == 0) n_children[node] = nz;
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < kSmallTiles; ++t) {
        if (oct[t] < 0) continue;
        const int dest = ostart[oct[t]] + wcnt[t * kWarps + w][oct[t]] + rank[t];
        xyz_out[dest] = v[t];
        perm_out[dest] = perm[s + t * kSmallThreads + threadIdx.x];
    }
}

// children of split nodes -> next level
__global__ void k_make_children(int K, const uint8_t *is_leaf, const int32_t *oct_start, const int32_t *oct_cnt,
                                const int32_t *child_off, int level_base, int next_base, int2 *next_rng,
                                int32_t *next_parent, int32_t *children_bfs, const int32_t *root,
                                int32_t *next_root) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= K) return;
    int j = child_off[i];
    for (int o = 0; o < 8; ++o) {
        int c = oct_cnt[8 * i + o];
        if (!is_leaf[i] && c > 0) {
            next_rng[j] = make_int2(oct_start[8 * i + o], oct_start[8 * i + o] + c);
            next_parent[j] = level_base + i;
            next_root[j] = root[i];
            children_bfs[8 * i + o] = next_base + j;
            ++j;
        } else {
            children_bfs[8 * i + o] = -1;
        }
    }
}

// DFS numbering
__global__ void k_dfs_marks(const int2 *rng, const int32_t *lev, int64_t M, int32_t *cnt_at, int32_t *minlev_at) {
    int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= M) return;
    int s = rng[b].x;
    atomicAdd(&cnt_at[s], 1);
    atomicMin(&minlev_at[s], lev[b]);
}

__global__ void k_dfs_ids(const int2 *rng, const int32_t *lev, int64_t M, const int32_t *base_at,
                          const int32_t *minlev_at, int32_t *dfs) {
    int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= M) return;
    int s = rng[b].x;
    dfs[b] = base_at[s] + lev[b] - minlev_at[s];
}

// Floor of the expansion scale of a tree: 2^-40 of its root's radius (1 for a
// root of radius 0).
template <typename T> __device__ __forceinline__ T scale_floor(T r) {
    return r > (T)0 ? (T)(r * (T)9.094947017729282e-13) : (T)1;
}

// Nodes into DFS order.  The expansion scale is the node's radius, but not
// below its tree's floor nor below 1/8 of the parent's scale: a node whose
// points coincide (radius 0, e.g. a single-point leaf) would otherwise get the
// global floor, and every M2L pair into it would have a source/target scale
// ratio far above the fast kernel's range.  Any positive scale is exact
// algebra; this one keeps the ratios O(10).  Multiplying by 1/8 rounds
// monotonically, so the largest of the ancestors' radii, each multiplied
// level by level, is what passing the scale down the levels gives.
template <typename T>
__global__ void k_permute_nodes(int64_t M, const int32_t *dfs, const int2 *rng, const int32_t *lev,
                                const int32_t *par_bfs, const int32_t *ch_bfs,
                                const typename Vec4<T>::type *cen, const typename Vec4<T>::type *hal,
                                const uint8_t *leaf, const int32_t *root, int2 *o_rng,
                                int32_t *o_lev, int32_t *o_par,
                                int32_t *o_ch, typename Vec4<T>::type *o_cen, typename Vec4<T>::type *o_hal,
                                uint8_t *o_leaf, int32_t *level_nodes, int32_t *flag) {
    int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= M) return;
    int d = dfs[b];
    o_rng[d] = rng[b];
    o_lev[d] = lev[b];
    o_par[d] = par_bfs[b] >= 0 ? dfs[par_bfs[b]] : -1;
    for (int o = 0; o < 8; ++o) {
        int c = ch_bfs[8 * b + o];
        o_ch[8 * d + o] = c >= 0 ? dfs[c] : -1;
    }
    o_cen[d] = cen[b];
    typename Vec4<T>::type h = hal[b];
    const T lo = scale_floor<T>(cen[root[b]].w);
    T a = cen[b].w;
    a = a > lo ? a : lo;
    int up = 0;  // levels between the node and the ancestor
    for (int q = par_bfs[b]; q >= 0; q = par_bfs[q]) {
        ++up;
        T r = cen[q].w;
        r = r > lo ? r : lo;
        for (int k = 0; k < up; ++k) r = rn_mul(r, (T)0.125);
        a = a > r ? a : r;
    }
    h.w = a;
    o_hal[d] = h;
    o_leaf[d] = leaf[b];
    level_nodes[b] = d;
    flag[d] = leaf[b];
}

__global__ void k_leaf_compact(const uint8_t *leaf, int64_t M, const int32_t *off, int32_t *leaves) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < M && leaf[i]) leaves[off[i]] = (int32_t)i;
}

inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

// The nodes of all levels so far, in BFS order.
template <typename T> struct BfsNodes {
    using T4 = typename Vec4<T>::type;
    DevBuf rng, parent, root, lev, center, half, leaf, children;
    int64_t cap = 0;
    // room for `want` nodes, at least doubled; the first `keep` nodes stay
    int ensure(int64_t want, int64_t keep, cudaStream_t s) {
        if (want <= cap) return EDFMM_OK;
        const int64_t nc = std::max<int64_t>(want, 2 * cap);
        DevBuf *bufs[] = {&rng, &parent, &root, &lev, &center, &half, &leaf, &children};
        const size_t sz[] = {sizeof(int2), 4, 4, 4, sizeof(T4), sizeof(T4), 1, 32};
        for (int i = 0; i < 8; ++i) {
            DevBuf nb;
            if (int rc = nb.reserve(sz[i] * (size_t)nc)) return rc;
            if (keep > 0)
                EDFMM_CUDA_TRY(cudaMemcpyAsync(nb.p, bufs[i]->p, sz[i] * (size_t)keep, cudaMemcpyDeviceToDevice, s));
            *bufs[i] = std::move(nb);  // the old block is reused in stream order, or freed behind the copy
        }
        cap = nc;
        return EDFMM_OK;
    }
};

__global__ void k_inst_node_off(const int32_t *level_nodes, int K, int32_t M, int32_t *off) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < K) off[k] = level_nodes[k];  // DFS id of root k
    if (k == K) off[K] = M;
}

// A forest when inst_off (host, n_inst + 1 point offsets) is given: level 0
// holds one root per instance over its rows, every later level the children
// of all instances' split nodes, so each level is one set of launches for
// the whole batch.  Each tree is the one a single build of its rows gives.
template <typename T>
int build_impl(const void *points_dev, int64_t n, int leaf_size, int max_depth, DevTree &tree, cudaStream_t s,
               const int64_t *inst_off, int n_inst) {
    using T4 = typename Vec4<T>::type;
    using O = typename OrdT<T>::type;
    int rc;
    tree.n_points = n;
    tree.dtype = sizeof(T) == 8 ? EDFMM_F64 : EDFMM_F32;
    tree.depth_warnings = 0;
    if (n == 0) {
        tree.n_nodes = tree.n_leaves = 0;
        tree.max_level = 0;
        tree.level_offsets.assign(1, 0);
        if ((rc = tree.pts.reserve(16)) || (rc = tree.index_map.reserve(16))) return rc;
        return EDFMM_OK;
    }
    if (n >= (int64_t)INT32_MAX) return fail(EDFMM_ERR_ARG, "n_points must be < 2^31");

    const int K0 = inst_off ? n_inst : 1;
    DevBuf xyz[2], perm[2], state, scan_tmp, chunks, d_off;
    BfsNodes<T> B;
    if ((rc = xyz[0].reserve(sizeof(T4) * n)) || (rc = xyz[1].reserve(sizeof(T4) * n)) ||
        (rc = perm[0].reserve(sizeof(int32_t) * n)) || (rc = perm[1].reserve(sizeof(int32_t) * n)) ||
        (rc = state.reserve(sizeof(BuildState))) || (rc = chunks.reserve(sizeof(int64_t))) ||
        (rc = tree.pts.reserve(sizeof(T4) * n)) || (rc = tree.index_map.reserve(sizeof(int32_t) * n)) ||
        (rc = B.ensure(std::max<int64_t>(1024, K0 + 4 * n / std::max(leaf_size, 2)), 0, s)))
        return rc;
    BuildState *st = dptr<BuildState>(state);
    EDFMM_CUDA_TRY(cudaMemsetAsync(st, 0, sizeof(BuildState), s));
    int64_t largest = n;  // points of the level's largest node
    if (inst_off) {
        if ((rc = d_off.reserve(sizeof(int64_t) * (K0 + 1)))) return rc;
        EDFMM_CUDA_TRY(cudaMemcpyAsync(d_off.p, inst_off, sizeof(int64_t) * (K0 + 1), cudaMemcpyHostToDevice, s));
        largest = 0;
        for (int k = 0; k < K0; ++k) largest = std::max(largest, inst_off[k + 1] - inst_off[k]);
    }
    k_init_points<T><<<nblk(std::max<int64_t>(n, K0), 256), 256, 0, s>>>(
        static_cast<const T *>(points_dev), n, dptr<T4>(xyz[0]), dptr<int32_t>(perm[0]), dptr<int64_t>(d_off), K0,
        dptr<int2>(B.rng), dptr<int32_t>(B.parent), dptr<int32_t>(B.root));
    EDFMM_LAUNCH_CHECK("k_init_points");

    DevBuf cnt, off, chunk_node, bb, ccnt, oct_start, oct_cnt, nchild, child_off;
    std::vector<int32_t> level_off(1, 0);  // BFS id of each level's first node
    int64_t total_nodes = K0;              // the roots
    BuildState h{};
    for (int lev = 0;; ++lev) {
        const int base = level_off[lev], K = (int)(total_nodes - base);
        level_off.push_back((int32_t)total_nodes);
        if ((rc = oct_start.reserve(sizeof(int32_t) * 8 * K)) || (rc = oct_cnt.reserve(sizeof(int32_t) * 8 * K)) ||
            (rc = nchild.reserve(sizeof(int32_t) * K)) || (rc = child_off.reserve(sizeof(int32_t) * K)) ||
            (rc = scan_tmp.reserve(scan_tmp_bytes(K))))
            return rc;
        const int2 *rng = dptr<int2>(B.rng) + base;
        T4 *center = dptr<T4>(B.center) + base, *half = dptr<T4>(B.half) + base;
        uint8_t *leaf = dptr<uint8_t>(B.leaf) + base;
        int32_t *blev = dptr<int32_t>(B.lev) + base;
        const T4 *in = dptr<T4>(xyz[lev & 1]);
        const int32_t *pin = dptr<int32_t>(perm[lev & 1]);
        T4 *out = dptr<T4>(xyz[(lev + 1) & 1]);
        int32_t *pout = dptr<int32_t>(perm[(lev + 1) & 1]);
        if (largest <= kChunk) {
            k_small_level<T><<<(unsigned)K, kSmallThreads, 0, s>>>(
                in, pin, rng, lev, leaf_size, max_depth, center, half, leaf, blev, dptr<int32_t>(oct_start),
                dptr<int32_t>(oct_cnt), dptr<int32_t>(nchild), out, pout, dptr<T4>(tree.pts),
                dptr<int32_t>(tree.index_map), st);
            EDFMM_LAUNCH_CHECK("k_small_level");
        } else {
            // chunks of the level's nodes: at most one short chunk a node
            const int64_t Q = n / kChunk + K;
            if ((rc = cnt.reserve(sizeof(int32_t) * K)) || (rc = off.reserve(sizeof(int32_t) * K)) ||
                (rc = bb.reserve(sizeof(O) * 6 * K)) || (rc = chunk_node.reserve(sizeof(int32_t) * Q)) ||
                (rc = ccnt.reserve(sizeof(int32_t) * 8 * Q)))
                return rc;
            const int64_t *nq = dptr<int64_t>(chunks);
            k_chunk_counts<T><<<nblk(K, 256), 256, 0, s>>>(rng, K, dptr<int32_t>(cnt), dptr<O>(bb));
            EDFMM_LAUNCH_CHECK("k_chunk_counts");
            if ((rc = scan_exclusive(dptr<int32_t>(cnt), dptr<int32_t>(off), K, dptr<int64_t>(chunks), scan_tmp.p, s)))
                return rc;
            k_chunk_fill<<<nblk(K, 256), 256, 0, s>>>(rng, K, dptr<int32_t>(off), dptr<int32_t>(chunk_node));
            EDFMM_LAUNCH_CHECK("k_chunk_fill");
            // bounding boxes and node geometry
            k_bbox<T><<<(unsigned)Q, kChunk, 0, s>>>(in, rng, dptr<int32_t>(chunk_node), dptr<int32_t>(off), nq, dptr<O>(bb));
            EDFMM_LAUNCH_CHECK("k_bbox");
            k_finalize<T><<<nblk(K, 256), 256, 0, s>>>(dptr<O>(bb), rng, K, lev, leaf_size, max_depth, center, half,
                                                         leaf, blev, st);
            EDFMM_LAUNCH_CHECK("k_finalize");
            // partition the points of split nodes
            k_octant_counts<T><<<(unsigned)Q, kChunk, 0, s>>>(in, rng, dptr<int32_t>(chunk_node), dptr<int32_t>(off), nq,
                                                              center, leaf, dptr<int32_t>(ccnt));
            EDFMM_LAUNCH_CHECK("k_octant_counts");
            k_node_octants<<<nblk((int64_t)K * 8, 256), 256, 0, s>>>(
                rng, K, dptr<int32_t>(off), leaf, dptr<int32_t>(ccnt), dptr<int32_t>(oct_start), dptr<int32_t>(oct_cnt),
                dptr<int32_t>(nchild), &st->max_child[lev + 1]);
            EDFMM_LAUNCH_CHECK("k_node_octants");
            k_scatter<T><<<(unsigned)Q, kChunk, 0, s>>>(in, pin, rng, dptr<int32_t>(chunk_node), dptr<int32_t>(off), nq,
                                                        center, leaf, dptr<int32_t>(ccnt), dptr<int32_t>(oct_start), out,
                                                        pout, dptr<T4>(tree.pts), dptr<int32_t>(tree.index_map));
            EDFMM_LAUNCH_CHECK("k_scatter");
        }
        // next level
        if ((rc = scan_exclusive(dptr<int32_t>(nchild), dptr<int32_t>(child_off), K, &st->next, scan_tmp.p, s))) return rc;
        EDFMM_CUDA_TRY(cudaMemcpyAsync(&h, st, sizeof(h), cudaMemcpyDeviceToHost, s));
        EDFMM_CUDA_TRY(cudaStreamSynchronize(s));
        const int64_t Kn = h.next;
        if (total_nodes + Kn >= (int64_t)INT32_MAX / 8) return fail(EDFMM_ERR_ARG, "octree too large");
        if ((rc = B.ensure(total_nodes + Kn, total_nodes, s))) return rc;
        const int next_base = (int)total_nodes;
        k_make_children<<<nblk(K, 256), 256, 0, s>>>(
            K, dptr<uint8_t>(B.leaf) + base, dptr<int32_t>(oct_start), dptr<int32_t>(oct_cnt), dptr<int32_t>(child_off),
            base, next_base, dptr<int2>(B.rng) + next_base, dptr<int32_t>(B.parent) + next_base,
            dptr<int32_t>(B.children) + 8 * (int64_t)base, dptr<int32_t>(B.root) + base, dptr<int32_t>(B.root) + next_base);
        EDFMM_LAUNCH_CHECK("k_make_children");
        if (Kn == 0) break;
        if (largest > kChunk) largest = h.max_child[lev + 1];
        total_nodes += Kn;
    }
    const int64_t M = total_nodes, nleaves = h.leaves;
    const int nlev = (int)level_off.size() - 1;
    tree.level_offsets = level_off;
    // DFS numbering
    DevBuf cnt_at, minlev_at, base_at, dfs;
    if ((rc = cnt_at.reserve(sizeof(int32_t) * n)) || (rc = minlev_at.reserve(sizeof(int32_t) * n)) ||
        (rc = base_at.reserve(sizeof(int32_t) * n)) || (rc = dfs.reserve(sizeof(int32_t) * M)) ||
        (rc = scan_tmp.reserve(scan_tmp_bytes(std::max<int64_t>(n, M)))))
        return rc;
    EDFMM_CUDA_TRY(cudaMemsetAsync(cnt_at.p, 0, sizeof(int32_t) * n, s));
    EDFMM_CUDA_TRY(cudaMemsetAsync(minlev_at.p, 0x7f, sizeof(int32_t) * n, s));
    k_dfs_marks<<<nblk(M, 256), 256, 0, s>>>(dptr<int2>(B.rng), dptr<int32_t>(B.lev), M, dptr<int32_t>(cnt_at),
                                             dptr<int32_t>(minlev_at));
    EDFMM_LAUNCH_CHECK("k_dfs_marks");
    if ((rc = scan_exclusive(dptr<int32_t>(cnt_at), dptr<int32_t>(base_at), n, nullptr, scan_tmp.p, s))) return rc;
    k_dfs_ids<<<nblk(M, 256), 256, 0, s>>>(dptr<int2>(B.rng), dptr<int32_t>(B.lev), M, dptr<int32_t>(base_at),
                                           dptr<int32_t>(minlev_at), dptr<int32_t>(dfs));
    EDFMM_LAUNCH_CHECK("k_dfs_ids");
    DevBuf flag, loff;
    if ((rc = tree.range.reserve(sizeof(int2) * M)) || (rc = tree.level.reserve(sizeof(int32_t) * M)) ||
        (rc = tree.parent.reserve(sizeof(int32_t) * M)) || (rc = tree.children.reserve(sizeof(int32_t) * 8 * M)) ||
        (rc = tree.center.reserve(sizeof(T4) * M)) || (rc = tree.half.reserve(sizeof(T4) * M)) ||
        (rc = tree.is_leaf.reserve(M)) || (rc = tree.level_nodes.reserve(sizeof(int32_t) * M)) ||
        (rc = tree.leaves.reserve(sizeof(int32_t) * nleaves)) || (rc = flag.reserve(sizeof(int32_t) * M)) ||
        (rc = loff.reserve(sizeof(int32_t) * M)))
        return rc;
    k_permute_nodes<T><<<nblk(M, 256), 256, 0, s>>>(
        M, dptr<int32_t>(dfs), dptr<int2>(B.rng), dptr<int32_t>(B.lev), dptr<int32_t>(B.parent),
        dptr<int32_t>(B.children), dptr<T4>(B.center), dptr<T4>(B.half), dptr<uint8_t>(B.leaf), dptr<int32_t>(B.root),
        dptr<int2>(tree.range), dptr<int32_t>(tree.level),
        dptr<int32_t>(tree.parent), dptr<int32_t>(tree.children), dptr<T4>(tree.center), dptr<T4>(tree.half),
        dptr<uint8_t>(tree.is_leaf), dptr<int32_t>(tree.level_nodes), dptr<int32_t>(flag));
    EDFMM_LAUNCH_CHECK("k_permute_nodes");
    // leaves
    if ((rc = scan_exclusive(dptr<int32_t>(flag), dptr<int32_t>(loff), M, nullptr, scan_tmp.p, s))) return rc;
    k_leaf_compact<<<nblk(M, 256), 256, 0, s>>>(dptr<uint8_t>(tree.is_leaf), M, dptr<int32_t>(loff), dptr<int32_t>(tree.leaves));
    EDFMM_LAUNCH_CHECK("k_leaf_compact");
    tree.n_nodes = M;
    tree.n_leaves = nleaves;
    tree.max_level = nlev - 1;
    tree.depth_warnings = h.warn;
    tree.n_inst = 0;
    if (inst_off) {
        // instance k owns the DFS range [root_k, root_{k+1}) (roots are BFS 0..K0-1)
        tree.n_inst = K0;
        if ((rc = tree.inst_node_off.reserve(sizeof(int32_t) * (K0 + 1)))) return rc;
        k_inst_node_off<<<nblk(K0 + 1, 256), 256, 0, s>>>(dptr<int32_t>(tree.level_nodes), K0, (int32_t)M,
                                                           dptr<int32_t>(tree.inst_node_off));
        EDFMM_LAUNCH_CHECK("k_inst_node_off");
    }
    return EDFMM_OK;
}

}  // namespace

int tree_build(const void *points_dev, int64_t n, int dtype, int leaf_size, int max_depth, DevTree &tree,
               cudaStream_t s) {
    if (dtype == EDFMM_F64) return build_impl<double>(points_dev, n, leaf_size, max_depth, tree, s, nullptr, 1);
    return build_impl<float>(points_dev, n, leaf_size, max_depth, tree, s, nullptr, 1);
}

int tree_build_forest(const void *points_dev, const int64_t *inst_off, int n_inst, int dtype, int leaf_size,
                      int max_depth, DevTree &tree, cudaStream_t s) {
    const int64_t n = inst_off[n_inst];
    if (dtype == EDFMM_F64) return build_impl<double>(points_dev, n, leaf_size, max_depth, tree, s, inst_off, n_inst);
    return build_impl<float>(points_dev, n, leaf_size, max_depth, tree, s, inst_off, n_inst);
}

}  // namespace edfmm
