// Internal declarations shared by the libedfmm translation units.
#pragma once

#include <algorithm>
#include <atomic>

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <vector>

#include "../../include/edfmm.h"

namespace edfmm {

// ---------------------------------------------------------------------------
// error plumbing
// ---------------------------------------------------------------------------
void set_error(const std::string &msg);
int fail(int code, const std::string &msg);
void count_launch(int n = 1);

#define EDFMM_CUDA_TRY(expr)                                                                  \
    do {                                                                                      \
        cudaError_t _e = (expr);                                                              \
        if (_e != cudaSuccess)                                                                \
            return ::edfmm::fail(EDFMM_ERR_CUDA, std::string(#expr " failed: ") +             \
                                                     cudaGetErrorString(_e));                 \
    } while (0)

#define EDFMM_LAUNCH_CHECK(name)                                                              \
    do {                                                                                      \
        ::edfmm::count_launch();                                                              \
        cudaError_t _e = cudaGetLastError();                                                  \
        if (_e != cudaSuccess)                                                                \
            return ::edfmm::fail(EDFMM_ERR_CUDA, std::string("launch of " name " failed: ") + \
                                                     cudaGetErrorString(_e));                 \
    } while (0)

// ---------------------------------------------------------------------------
// settings that belong to a device
// ---------------------------------------------------------------------------
// Runs `set` the first time it is asked for device `dev`: a kernel's attribute
// holds on the device that was current when it was set, and a process may use
// several.  A failure is not remembered; ordinals past the mask are set each time.
struct DeviceOnce {
    std::atomic<unsigned long long> done{0};
};
template <typename F> cudaError_t once_per_device(DeviceOnce &once, int dev, F &&set) {
    const unsigned long long bit = dev >= 0 && dev < 64 ? 1ull << dev : 0ull;
    if (once.done.load(std::memory_order_acquire) & bit) return cudaSuccess;
    const cudaError_t e = set();
    if (e == cudaSuccess && bit) once.done.fetch_or(bit, std::memory_order_release);
    return e;
}
// opt-in of a kernel to more than 48 KB of dynamic shared memory on the current device
template <typename K> cudaError_t allow_smem(DeviceOnce &once, K *kernel, size_t bytes) {
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    return once_per_device(once, dev, [&] {
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    });
}

// ---------------------------------------------------------------------------
// device buffer (owning)
// ---------------------------------------------------------------------------
// Blocks released while a BlockCacheScope is active on this thread are kept
// for the scope's later reserves instead of being freed: a build that runs on
// ONE stream then reuses its temporaries in stream order without a
// cudaMalloc / cudaFree (which synchronises the device) per temporary.  The
// scope frees what it still holds when it ends.
//
// A scope opened with a slab size also cuts blocks of up to half
// a slab from slabs of that size.  An allocation above about 2 MB costs 35 us
// whatever its size, and its cudaFree 35-60 us; the set-up of a plan of 100,000
// points took 137 blocks, 3.5 ms of its 6.3.  Slabs end with the scope, so what
// outlives it moves out first (pack_buffers, shrink_to_fit).
struct BlockCache;
BlockCache *block_cache();  // this thread's active cache or NULL
struct DevBlock {
    void *p = nullptr;
    size_t bytes = 0;
    BlockCache *slab = nullptr;  // the cache whose slab holds the block
};
// a held block of a fitting size, or a new one cut from a slab; p == NULL if neither
DevBlock block_cache_take(BlockCache *c, size_t nbytes);
void block_cache_put(BlockCache *c, const DevBlock &b);
// frees every block the cache holds (cudaFree waits for the device)
void block_cache_trim(BlockCache *c);
// cudaMalloc that, when it fails inside a cache scope, frees the cached
// blocks and tries once more (a held block may be what the device lacks)
cudaError_t malloc_or_trim(void **p, size_t nbytes);
struct BlockCacheScope {
    explicit BlockCacheScope(size_t slab_bytes = 0);
    ~BlockCacheScope();
    BlockCacheScope(const BlockCacheScope &) = delete;
    BlockCacheScope &operator=(const BlockCacheScope &) = delete;
    BlockCache *prev;
    BlockCache *cache;
};

struct DevBuf {
    void *p = nullptr;
    size_t bytes = 0;  // size of the block held
    size_t used = 0;   // size last asked for (a cached block may be larger)
    BlockCache *slab = nullptr;  // the block lies in a slab of this cache
    bool part = false;           // the block is a part of another buffer's (pack_buffers)
    DevBuf() = default;
    DevBuf(const DevBuf &) = delete;
    DevBuf &operator=(const DevBuf &) = delete;
    DevBuf(DevBuf &&o) noexcept { take(o); }
    DevBuf &operator=(DevBuf &&o) noexcept {
        if (this != &o) {
            release();
            take(o);
        }
        return *this;
    }
    ~DevBuf() { release(); }
    void take(DevBuf &o) {
        p = o.p;
        bytes = o.bytes;
        used = o.used;
        slab = o.slab;
        part = o.part;
        o.forget();
    }
    void forget() {
        p = nullptr;
        bytes = 0;
        used = 0;
        slab = nullptr;
        part = false;
    }
    void release() {
        if (p && !part) {
            BlockCache *c = block_cache();
            if (c && (!slab || slab == c)) block_cache_put(c, DevBlock{p, bytes, slab});
            else if (!slab) cudaFree(p);
        }
        forget();
    }
    // grows (never shrinks); contents are not preserved
    int reserve(size_t nbytes) {
        if (nbytes <= bytes && p) {
            used = nbytes;
            return EDFMM_OK;
        }
        release();
        size_t want = nbytes ? nbytes : 16;
        if (BlockCache *c = block_cache()) {
            const DevBlock b = block_cache_take(c, want);
            if (b.p) {
                p = b.p;
                bytes = b.bytes;
                slab = b.slab;
                used = want;
                return EDFMM_OK;
            }
        }
        cudaError_t e = malloc_or_trim(&p, want);
        if (e != cudaSuccess) {
            p = nullptr;
            return fail(EDFMM_ERR_ALLOC, std::string("cudaMalloc of ") + std::to_string(want) +
                                             " bytes failed: " + cudaGetErrorString(e));
        }
        bytes = want;
        used = want;
        return EDFMM_OK;
    }
    // A buffer that outlives its build (a plan's tree, lists, expansions)
    // and received a cached block well above its size, or one of a slab, moves
    // to a block of its own size (contents copied in stream order), so the
    // plan holds no slack for its lifetime.
    int shrink_to_fit(cudaStream_t s) {
        if (!p || part || (!slab && bytes <= used + used / 8 + 4096)) return EDFMM_OK;
        void *q = nullptr;
        cudaError_t e = malloc_or_trim(&q, used);
        if (e == cudaSuccess) e = cudaMemcpyAsync(q, p, used, cudaMemcpyDeviceToDevice, s);
        if (e != cudaSuccess) {
            if (q) cudaFree(q);
            return fail(EDFMM_ERR_ALLOC, std::string("exact-size copy of a plan buffer failed: ") +
                                             cudaGetErrorString(e));
        }
        const size_t keep = used;
        release();  // the cache frees it only after the device is done with it
        p = q;
        bytes = keep;
        used = keep;
        return EDFMM_OK;
    }
    template <class U> U *as() const { return static_cast<U *>(p); }
};

// Moves the buffers that lie in a slab into one exact block (one allocation
// and one copy kernel), of which they are then parts, and frees the others of
// slack; `fresh` buffers get parts of fresh_bytes each with no contents.
int pack_buffers(DevBuf *const *bufs, int n, DevBuf *const *fresh, int n_fresh, size_t fresh_bytes, DevBuf &block,
                 cudaStream_t s);

// typed view of a buffer (a free function, so no `template` keyword is needed
// inside templates)
template <class U> inline U *dptr(const DevBuf &b) { return static_cast<U *>(b.p); }

// ---------------------------------------------------------------------------
// primitives (scan.cu)
// ---------------------------------------------------------------------------
// Exclusive prefix sum of n int32 counts into int32 offsets; the grand total
// is written to *total_dev (int64) if non-null.  tmp must hold scan_tmp_bytes(n).
size_t scan_tmp_bytes(int64_t n);
int scan_exclusive(const int32_t *in, int32_t *out, int64_t n, int64_t *total_dev, void *tmp,
                   cudaStream_t s);

// Sort every CSR row of `vals` ascending (rows given by offsets[0..rows]; the
// values of a row are distinct, at least 0 and below `bound`).
int sort_csr_rows(const int32_t *offsets, int32_t *vals, int64_t rows, int64_t max_row_len, int64_t bound,
                  cudaStream_t s);

// ---------------------------------------------------------------------------
// tree + lists (tree.cu, lists.cu)
// ---------------------------------------------------------------------------
template <typename T> struct Vec4 {};
template <> struct Vec4<float> {
    using type = float4;
};
template <> struct Vec4<double> {
    using type = double4;
};

#ifdef __CUDACC__
// 1/sqrt(x) for a normal x > 0 (PTX rsqrt.approx.ftz.f32, relative error
// below 2^-22.9).  Callers clamp the argument well above the subnormal range,
// so flushing subnormals changes nothing and no range handling is needed.
__device__ __forceinline__ float rsqrt_normal(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
#endif

// Frame of an FP64 tree's split coordinates (gridpoint.cuh): the centre, 2^-k,
// 2^k, and the scaled r^2 below which a pair is evaluated in IEEE FP64; the
// largest x, y, z, -x, -y, -z while it is laid out (order-preserving integers).
struct GridInfo {
    double down, up;
    double center[3];
    float near2;
    long long ext[6];
};

// Device-resident tree in DFS pre-order (the reference's node numbering).
struct DevTree {
    int dtype = EDFMM_F32;
    int64_t n_points = 0;
    int64_t n_nodes = 0;
    int64_t n_leaves = 0;
    int max_level = 0;
    int depth_warnings = 0;
    DevBuf pts;        // T4 per point, tree order: (x, y, z, charge)
    DevBuf index_map;  // int32, tree position -> original index
    DevBuf center;     // T4 per node: (cx, cy, cz, radius)
    DevBuf half;       // T4 per node: (hx, hy, hz, expansion scale a)
    DevBuf range;      // int2 per node: [start, end)
    DevBuf parent;     // int32
    DevBuf children;   // int32 x 8
    DevBuf level;      // int32
    DevBuf is_leaf;    // uint8
    DevBuf leaves;     // int32 ids of leaf nodes (ascending)
    std::vector<int32_t> level_offsets;  // host: level l nodes = level_nodes[off[l], off[l+1])
    DevBuf level_nodes;                  // int32 node ids grouped by level
    // FP64 trees in two-float mode: per node (cx, cy, cz, expansion scale a)
    // split into FP32 (hi, lo) pairs
    DevBuf nodes_tf;
    // FP64 trees: per point the exact coordinate split of gridpoint.cuh and
    // the charge (three float4; the charge as a double, or as two floats in
    // two-float mode), and the split's scale (batched plans: one per instance)
    DevBuf pts_grid;
    DevBuf grid_info;
    bool grid_tf = false;
    // levels whose translations run a block per node (farfield.cu): what each
    // node's translation to and from its parent needs, level l's nodes from
    // frame_off[l] (-1: none)
    DevBuf shift_frames;
    std::vector<int64_t> frame_off;
    // batched plans: instance k owns nodes inst_node_off[k] .. inst_node_off[k+1]-1
    int n_inst = 0;
    DevBuf inst_node_off;  // int32 x (n_inst + 1)
};

// Per-instance activity of a batched plan's matvec: instance k is active
// when flags[k * stride] != 0 (a column of the batched GMRES state).  M2L
// rows and near-field leaves of inactive instances are skipped; their
// outputs are left unspecified (the batched solver does not read them).
struct InstMask {
    const int32_t *node_off = nullptr;  // NULL: no mask
    int n_inst = 0;
    const double *flags = nullptr;
    int stride = 0;
};
#ifdef __CUDACC__
// the instance of a node (0 when there is one tree, node_off NULL)
__device__ __forceinline__ int instance_of_node(const int32_t *node_off, int n_inst, int node) {
    if (!node_off) return 0;
    int lo = 0, hi = n_inst - 1;  // last instance whose first node <= node
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (node_off[mid] <= node) lo = mid; else hi = mid - 1;
    }
    return lo;
}
__device__ __forceinline__ bool inst_active(const InstMask &m, int node) {
    return !m.node_off || m.flags[(int64_t)instance_of_node(m.node_off, m.n_inst, node) * m.stride] != 0.0;
}
#endif

// Chains of small kernels (the far field of a small tree, the warm-start
// network): a kernel launched by
// chain_launch may start while its predecessor in the stream still runs.  It
// reads what the plan holds, calls chain_wait (all threads, before any return),
// and only then reads or writes what other kernels of the chain do; chain_next
// lets its own successor start.  A kernel that reads ahead what another may have
// written since the plan's set-up (the M2L) has an ordinary launch between them.
// Without the launch attribute both do nothing.
// What the chain writes is read through pointers that are neither const
// __restrict__ nor __ldg: those loads assume data that stay as they are for the
// kernel's whole life, which here begins before its predecessor's end.
#ifdef __CUDACC__
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <typename... K, typename... A>
cudaError_t chain_launch(bool chained, void (*kernel)(K...), unsigned grid, unsigned block, size_t smem, cudaStream_t s,
                         A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = chained ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<K>(args)...);
}
#endif
// outside a capture (a graph has its own order); small trees there
bool chain_stream(cudaStream_t s);
bool chain_tree(int64_t n_nodes, int dtype, cudaStream_t s);

int tree_build(const void *points_dev, int64_t n, int dtype, int leaf_size, int max_depth,
               DevTree &tree, cudaStream_t s);
// One tree per instance (rows inst_off[k] .. inst_off[k+1]-1, host offsets),
// built together level by level as one forest: nodes of instance k are the
// DFS range [inst_node_off[k], inst_node_off[k+1]), each tree equal to
// tree_build of its rows alone; nodes grouped by level across instances.
int tree_build_forest(const void *points_dev, const int64_t *inst_off, int n_inst, int dtype, int leaf_size,
                      int max_depth, DevTree &tree, cudaStream_t s);

struct DevLists {
    int64_t n_p2p = 0, n_m2l = 0;
    int64_t p2p_interactions = 0;
    int64_t max_p2p_row = 0, max_m2l_row = 0;
    DevBuf p2p_off, p2p_src;  // CSR by target, sources ascending
    DevBuf m2l_off, m2l_src;
    // the target tree's leaves in decreasing near-field work (sum over the
    // leaf's P2P sources of n_source * n_target): the near-field kernel takes
    // them in this order, so that its last wave holds the short leaves
    DevBuf p2p_leaves;
    // the target tree's nodes by decreasing M2L pair count: the M2L kernels
    // give warp w row m2l_rows[w], so that a block's warps (which run their
    // rounds of pairs together) hold rows of similar length
    DevBuf m2l_rows;
    // transposed M2L CSR (rows = listed sources), built on demand for the
    // reference's swapped pair order
    bool have_m2l_swapped = false;
    DevBuf m2l_swapped_off, m2l_swapped_src;
};

int lists_build(const DevTree &tree, double theta, DevLists &lists, cudaStream_t s);
int lists_build_swapped(const DevTree &tree, DevLists &lists, cudaStream_t s);
// lists between two trees: rows = target-tree nodes, sources = source-tree nodes
// (the reference's build_interaction_lists(source_tree, target_tree))
int lists_build_two(const DevTree &src_tree, const DevTree &tgt_tree, double theta, DevLists &lists, cudaStream_t s);

// ---------------------------------------------------------------------------
// FMM stages (farfield.cu, nearfield.cu)
// ---------------------------------------------------------------------------
inline int num_coeffs(int p) { return (p + 1) * (p + 2) / 2; }

// The FP32 and two-float kernels read the multipoles by columns: groups of 32
// nodes, word w (16 bytes) of node s at [(s / 32) * words * 32 + w * 32 + s % 32].
// The lanes of a warp hold consecutive sources of one target's row, which come
// in runs of siblings with consecutive node ids, so that a load takes a few
// 128-byte lines where rows take one line per lane.
constexpr int kColNodes = 32;
#ifdef __CUDACC__
__host__ __device__ __forceinline__ int64_t col_of(int64_t s, int words) {
    return (s / kColNodes) * ((int64_t)words * kColNodes) + s % kColNodes;
}
#endif
// nodes of an expansion buffer: whole groups
inline int64_t padded_nodes(int64_t n) { return (std::max<int64_t>(n, 1) + kColNodes - 1) / kColNodes * kColNodes; }

// M2L pairs whose source radius exceeds 256x the target radius, as CSR rows
// by target (FP32 plans only; empty for uniform trees).
struct ExtremeRows {
    bool built = false;
    int64_t n_pairs = 0, n_rows = 0;
    DevBuf off, src, rows;
};

struct FmmBuffers {
    int p = 8;
    int nc = 45;
    int nc_pad = 46;  // per-node stride in complex numbers (even: 16-byte rows for float)
    // rows of padded_nodes(n_nodes) nodes
    DevBuf multipoles;  // complex T, n_nodes x nc_pad
    DevBuf locals;      // complex T, n_nodes x nc_pad
    // complex T, n_nodes x nc_pad: each node's multipole moved to its parent's
    // centre (M2M), then, in FP32, the multipoles by columns (M2L)
    DevBuf translated;
    ExtremeRows extreme, extreme_swapped;
    InstMask mask;  // set around the steps of a batched solve
    // FP64 plans: EDFMM_ARITH_TWO_FLOAT runs M2L and the near field in
    // two-float arithmetic on the FP32 pipe (twofloat.cuh); mult_tf holds
    // the multipoles split into (hi, lo) pairs, by columns, for the two-float M2L
    int arith = EDFMM_ARITH_NATIVE;
    DevBuf mult_tf;
    // launch shapes the autotuner may change (edfmm_plan_set_launch)
    int m2l_tf_block = 128;  // two-float M2L threads per block (128 or 256, p = 8)
    int near_overlap = 1;    // full matvec: near field on a second stream beside the far field
    int m2l_packed = 1;      // two-float M2L: matrices on packed FP32x2 instructions
};

int set_charges(const DevTree &tree, const void *sigma, const void *areas, cudaStream_t s);
int run_p2m(const DevTree &tree, FmmBuffers &buf, cudaStream_t s);
int run_m2m(const DevTree &tree, FmmBuffers &buf, cudaStream_t s);
// alone: a stage of its own, not after this tree's M2M in a chain of launches.  The
// M2L reads its lists and the instances' flags ahead of its wait for its
// predecessor, and another kernel may have written them just before.
int run_m2l(const DevTree &tree, const DevLists &lists, FmmBuffers &buf, bool swapped, bool alone, cudaStream_t s);
// rotation-based M2L (m2l_rot.cu, kernels in m2l_rot.cuh), orders 1..8, FP32 and FP64
int launch_m2l_rot(int dtype, int p, int64_t M, const int32_t *off, const int32_t *src, const int32_t *rows,
                   const void *tcen,
                   const void *thal, const void *cen, const void *hal, const void *Mx, void *Lx, int nc_pad,
                   const InstMask &mask, cudaStream_t s);
// the same in two-float arithmetic for FP64 plans, orders 6..8
// (EDFMM_ERR_UNSUPPORTED for other orders, launching nothing): node geometry
// and multipoles split into (hi, lo) FP32 pairs (tnodes / snodes: 2 float4
// per node; Mx: one float4 per complex coefficient), locals written as FP64
int launch_m2l_rot_tf(int p, int64_t M, const int32_t *off, const int32_t *src, const int32_t *rows,
                      const void *tnodes, const void *thal,
                      const void *snodes, const void *hal, const void *Mx, void *Lx, int nc_pad, const InstMask &mask,
                      int block, bool packed, cudaStream_t s);
int run_m2l_two(const DevTree &tgt_tree, const DevTree &src_tree, const DevLists &lists, const FmmBuffers &src_buf,
                FmmBuffers &tgt_buf, bool alone, cudaStream_t s);
int run_l2l(const DevTree &tree, FmmBuffers &buf, cudaStream_t s);
// the same-tree extreme-pair rows of buf (built once; synchronises s)
int prepare_extreme_rows(const DevTree &tree, const DevLists &lists, FmmBuffers &buf, cudaStream_t s);
// two-float mode of an FP64 plan: split node geometry and the multipole
// buffer (sized for the current order); called when the mode is set and
// when the order changes
int prepare_two_float(DevTree &tree, FmmBuffers &buf, cudaStream_t s);

struct L2pArgs {
    const void *sigma = nullptr;     // original order (nullable)
    const void *areas = nullptr;     // original order (nullable)
    const void *self_int = nullptr;  // original order (nullable)
    double k_e = 1.0;
    void *out = nullptr;           // original order if scatter, else tree order
    bool scatter = false;          // write out[index_map[i]] with k_e, self term, clamp
    bool far = true;               // evaluate the local expansions
    const void *add_in = nullptr;  // near sums in tree order (nullable)
};
int run_targets_field(const DevTree &tree, const DevLists &lists, const FmmBuffers &buf, const DevTree &stree,
                      double k_e, bool near, bool far, void *out, cudaStream_t s);
// near sums in tree order; src_tree: the sources when they are another
// tree's points (targets evaluated against a source plan: no self exclusion)
int run_p2p(const DevTree &tree, const DevLists &lists, const FmmBuffers &buf, const DevTree *src_tree, void *out,
            cudaStream_t s);
int run_l2p(const DevTree &tree, const FmmBuffers &buf, const L2pArgs &args, cudaStream_t s);
int grid_prepare(DevTree &tree, cudaStream_t s);
// the tree's shift_frames (once per tree)
int shift_prepare(DevTree &tree, cudaStream_t s);
int upload_tables();

}  // namespace edfmm

struct edfmm_plan {
    edfmm::DevTree tree;
    edfmm::DevLists lists;
    bool lists_ok = true;  // false after a rebuild that failed
    edfmm::FmmBuffers fmm;
    double mac_theta = 0.5;
    int leaf_size = 64;
    int max_depth = 32;
    int device = 0;
    // matvec: the near field runs on a second stream beside the far-field
    // chain (fork / join events) into tree-order sums, created on first use
    cudaStream_t side = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    edfmm::DevBuf near_sum;
    edfmm::DevBuf block;  // the set-up's small buffers (pack_buffers)
    edfmm_plan() = default;
    edfmm_plan(const edfmm_plan &) = delete;
    edfmm_plan &operator=(const edfmm_plan &) = delete;
    ~edfmm_plan() {
        if (ev_fork) cudaEventDestroy(ev_fork);
        if (ev_join) cudaEventDestroy(ev_join);
        if (side) cudaStreamDestroy(side);
    }
};
