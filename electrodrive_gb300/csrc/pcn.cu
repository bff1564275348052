// Point-cloud warm-start network: per-panel features -> initial surface charge
// density for the GMRES start.  Inference and training kernels.
//
// Network (width 128, BF16 weights and activations, FP32 accumulation):
//   x_i  = 16 features of panel i (8 used, zero padded)
//   h1_i = relu(W1 x_i + b1)                          16 -> 128
//   g    = mean_i h1_i                                global context
//   h2_i = relu(W2 h1_i + V2 g + b2)                  128 -> 128
//   h3_i = relu(W3 h2_i + b3)                         128 -> 128
//   y_i  = w4 . h3_i + b4                             128 -> 1
// The three per-panel GEMMs and the weight gradients' partial products run
// on the tensor cores (mma.sync m16n8k16, BF16 inputs, FP32 accumulators);
// the context, output and bias reductions run on the FP32 pipe, and every
// reduction has a fixed order, so forward and backward are deterministic.
#include <cuda_bf16.h>

#include <algorithm>

#include "edfmm_internal.cuh"

namespace edfmm {
namespace {

constexpr int W = EDFMM_PCN_WIDTH;  // 128
constexpr int NIN = EDFMM_PCN_INPUTS;  // 16

// parameter block offsets (FP32)
constexpr int64_t O_W1 = 0;
constexpr int64_t O_B1 = O_W1 + W * NIN;
constexpr int64_t O_W2 = O_B1 + W;
constexpr int64_t O_V2 = O_W2 + W * W;
constexpr int64_t O_B2 = O_V2 + W * W;
constexpr int64_t O_W3 = O_B2 + W;
constexpr int64_t O_B3 = O_W3 + W * W;
constexpr int64_t O_W4 = O_B3 + W;
constexpr int64_t O_B4 = O_W4 + W;
constexpr int64_t NPARAM = O_B4 + 1;

inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }
inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// workspace layout for n panels
struct Ws {
    __nv_bfloat16 *x0, *h1, *h2, *h3, *dz, *dz2;  // activations / gradients (n x K)
    __nv_bfloat16 *w1b, *w2b, *w3b;          // weights (out x in)
    __nv_bfloat16 *w2t, *w3t;                // transposed (in x out) for the data gradients
    float *g, *c2, *dc, *dg, *part;          // context vectors, partial sums
    double *stats;
    size_t bytes;
};

constexpr int kColRows = 1024;  // rows per partial column sum

inline int64_t n_col_parts(int64_t n) { return std::max<int64_t>(1, (n + kColRows - 1) / kColRows); }

// Rows per weight-gradient partial.  It sets the order of the FP32 additions, and
// training amplifies a change of it (Adam scales gradients near zero up to the
// step size, and the weights are rounded to BF16), so the work is split over
// output rows instead of shorter partials: a training step of 30,000 panels took
// 221 us with it and 212 with partials of 256 rows, whose gradients had other
// last bits.
constexpr int kPartRows = 1024;
inline int64_t n_parts(int64_t n) { return std::max<int64_t>(1, (n + kPartRows - 1) / kPartRows); }

Ws carve(void *base, int64_t n) {
    Ws w{};
    size_t o = 0;
    auto take = [&](size_t b) {
        size_t at = o;
        o = align256(o + b);
        return at;
    };
    const size_t bf = sizeof(__nv_bfloat16);
    size_t a_x0 = take(n * NIN * bf), a_h1 = take(n * W * bf), a_h2 = take(n * W * bf), a_h3 = take(n * W * bf),
           a_dz = take(n * W * bf), a_dz2 = take(n * W * bf), a_w1 = take(W * NIN * bf), a_w2 = take(W * W * bf), a_w3 = take(W * W * bf),
           a_w2t = take(W * W * bf), a_w3t = take(W * W * bf), a_g = take(W * 4), a_c2 = take(W * 4), a_dc = take(W * 4),
           a_dg = take(W * 4), a_part = take(std::max((size_t)n_parts(n) * (W * W + W), (size_t)n_col_parts(n) * W) * 4), a_st = take(16 * 8);
    w.bytes = o + 255;  // the buffers start at the base rounded up to 256 bytes
    if (base) {
        char *b = reinterpret_cast<char *>((reinterpret_cast<uintptr_t>(base) + 255) & ~(uintptr_t)255);
        w.x0 = (__nv_bfloat16 *)(b + a_x0);
        w.h1 = (__nv_bfloat16 *)(b + a_h1);
        w.h2 = (__nv_bfloat16 *)(b + a_h2);
        w.h3 = (__nv_bfloat16 *)(b + a_h3);
        w.dz = (__nv_bfloat16 *)(b + a_dz);
        w.dz2 = (__nv_bfloat16 *)(b + a_dz2);
        w.w1b = (__nv_bfloat16 *)(b + a_w1);
        w.w2b = (__nv_bfloat16 *)(b + a_w2);
        w.w3b = (__nv_bfloat16 *)(b + a_w3);
        w.w2t = (__nv_bfloat16 *)(b + a_w2t);
        w.w3t = (__nv_bfloat16 *)(b + a_w3t);
        w.g = (float *)(b + a_g);
        w.c2 = (float *)(b + a_c2);
        w.dc = (float *)(b + a_dc);
        w.dg = (float *)(b + a_dg);
        w.part = (float *)(b + a_part);
        w.stats = (double *)(b + a_st);
    }
    return w;
}

// ---------------------------------------------------------------------------
// features
// ---------------------------------------------------------------------------
// stats: [0..2] mean centroid, [3] mean area, [4] rms rhs, [5] rms radius.
// Two passes of kStatBlocks blocks (grid-stride partial sums, then one small
// kernel that adds the blocks' partials in block order): the second pass
// needs the mean centroid of the first.  The partition is fixed, so the
// sums are deterministic.
constexpr int kStatBlocks = 152;

__global__ void __launch_bounds__(256) k_pcn_stats_part(const double *__restrict__ c, const double *__restrict__ a,
                                                        const double *__restrict__ b, int64_t n,
                                                        const double *__restrict__ mean, double *__restrict__ part) {
    __shared__ double red[5][8];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    double s[5] = {0, 0, 0, 0, 0};
    for (int64_t i = (int64_t)blockIdx.x * 256 + tid; i < n; i += (int64_t)gridDim.x * 256) {
        if (mean) {
            const double dx = c[3 * i] - mean[0], dy = c[3 * i + 1] - mean[1], dz = c[3 * i + 2] - mean[2];
            s[0] += dx * dx + dy * dy + dz * dz;
        } else {
            s[0] += c[3 * i];
            s[1] += c[3 * i + 1];
            s[2] += c[3 * i + 2];
            s[3] += a[i];
            s[4] += b[i] * b[i];
        }
    }
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        for (int o = 16; o > 0; o >>= 1) s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
        if (lane == 0) red[q][wid] = s[q];
    }
    __syncthreads();
    if (tid < 5) {
        double t = 0;
        for (int w = 0; w < 8; ++w) t += red[tid][w];
        part[(int64_t)blockIdx.x * 8 + tid] = t;
    }
}

// pass 0: stats[0..4] from the first partials; pass 1: stats[5]
__global__ void k_pcn_stats_fin(const double *__restrict__ part, int nb, int64_t n, int pass, double *stats) {
    const int q = threadIdx.x;
    if (pass == 0 && q < 5) {
        double t = 0;
        for (int k = 0; k < nb; ++k) t += part[(int64_t)k * 8 + q];
        const double inv = n > 0 ? 1.0 / (double)n : 0.0;
        stats[q] = q < 4 ? t * inv : sqrt(t * inv);
    } else if (pass == 1 && q == 0) {
        double t = 0;
        for (int k = 0; k < nb; ++k) t += part[(int64_t)k * 8];
        stats[5] = sqrt(t / (double)(n > 0 ? n : 1));
    }
}

__global__ void k_pcn_features(const double *__restrict__ c, const double *__restrict__ nrm,
                               const double *__restrict__ a, const double *__restrict__ b, int64_t n,
                               const double *__restrict__ stats, float *__restrict__ f) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double R = stats[5] > 0 ? stats[5] : 1.0, rb = stats[4] > 0 ? stats[4] : 1.0;
    float *o = f + i * NIN;
    o[0] = (float)((c[3 * i] - stats[0]) / R);
    o[1] = (float)((c[3 * i + 1] - stats[1]) / R);
    o[2] = (float)((c[3 * i + 2] - stats[2]) / R);
    o[3] = (float)nrm[3 * i];
    o[4] = (float)nrm[3 * i + 1];
    o[5] = (float)nrm[3 * i + 2];
    o[6] = (float)(a[i] > 0 ? log(a[i] / (R * R)) : 0.0);
    o[7] = (float)(b[i] / rb);
    for (int q = 8; q < NIN; ++q) o[q] = 0.0f;
}

// From here on all kernels but the loss are a chain of overlapped launches: they
// wait before their first access, and read through plain pointers (a step's
// parameters are written by the kernel before).  What it saves is the start of
// some 17 short kernels: a training step of 140 / 4,026 / 30,000 / 123,000 panels
// went from 117 / 170 / 208 / 424 to 92 / 148 / 194 / 409 us.

// ---------------------------------------------------------------------------
// weights: FP32 master -> BF16 (and transposed BF16 for the data gradients),
// and the features of all rows
// ---------------------------------------------------------------------------
__global__ void k_pcn_cast(const float *prm, __nv_bfloat16 *w1b, __nv_bfloat16 *w2b,
                           __nv_bfloat16 *w3b, __nv_bfloat16 *w2t, __nv_bfloat16 *w3t,
                           const float *f, int64_t nf, __nv_bfloat16 *x0) {
    chain_next();
    chain_wait();
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j < nf) x0[j] = __float2bfloat16_rn(f[j]);
    if (j >= W * W) return;
    const int i = (int)j;
    if (i < W * NIN) w1b[i] = __float2bfloat16_rn(prm[O_W1 + i]);
    const int r = i / W, c = i % W;
    const __nv_bfloat16 x2 = __float2bfloat16_rn(prm[O_W2 + i]), x3 = __float2bfloat16_rn(prm[O_W3 + i]);
    w2b[i] = x2;
    w3b[i] = x3;
    w2t[c * W + r] = x2;
    w3t[c * W + r] = x3;
}

// ---------------------------------------------------------------------------
// tensor-core linear layer: out[r][n] = epi(sum_k X[r][k] Wt[n][k])
// ---------------------------------------------------------------------------
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// four 8 x 8 BF16 matrices from shared memory; lane l gives row l % 8 of matrix l / 8
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const __nv_bfloat16 *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((unsigned)__cvta_generic_to_shared(p))
                 : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], const __nv_bfloat16 *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((unsigned)__cvta_generic_to_shared(p))
                 : "memory");
}
// 16 bytes to shared memory, zeros when !valid
__device__ __forceinline__ void cp16(__nv_bfloat16 *dst, const __nv_bfloat16 *src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(valid ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

enum Epi { EPI_RELU = 0, EPI_MASK = 1 };

constexpr int kLinRows = 128;  // rows per block, 16 per warp

// One warp computes 16 rows x 128 columns.  Wt (128 x K, K contiguous) and the
// block's rows of X are copied to shared memory 16 bytes at a time (padded
// rows: conflict-free ldmatrix), the results go back through the warp's rows of
// X.  EPI_RELU: out = relu(acc + bias[n]) and optionally y = w4 . out + b4;
// EPI_MASK: out = mask[r][n] > 0 ? acc + bias[n] : 0 (ReLU backward).  30,000
// rows of 128: 13 to 18 us with 4-byte loads of every fragment, 8 to 13 now (8
// MB in, 8 MB out).
template <int K> constexpr size_t lin_smem() { return (size_t)(W + kLinRows) * (K + 8) * sizeof(__nv_bfloat16); }
template <int K> constexpr size_t lin_smem_out() {  // the output rows take over the staging area
    return std::max(lin_smem<K>(), (size_t)kLinRows * (W + 8) * sizeof(__nv_bfloat16));
}

template <int K, int EPI, bool HEAD>
__global__ void __launch_bounds__(256) k_pcn_linear(const __nv_bfloat16 *X, const __nv_bfloat16 *Wt,
                                                    const float *bias, const __nv_bfloat16 *mask,
                                                    int64_t n, __nv_bfloat16 *out,
                                                    const float *prm, float *y) {
    chain_next();
    chain_wait();
    constexpr int LD = K + 8, LO = W + 8;  // padded row strides (bf16 elements)
    extern __shared__ __align__(16) __nv_bfloat16 lin_sm[];
    __nv_bfloat16 *sw = lin_sm, *sx = lin_sm + W * LD;
    const int64_t b0r = (int64_t)blockIdx.x * kLinRows;
    for (int i = threadIdx.x; i < W * K / 8; i += 256) cp16(sw + (i / (K / 8)) * LD + (i % (K / 8)) * 8, Wt + 8 * i, true);
    for (int i = threadIdx.x; i < kLinRows * K / 8; i += 256) {
        const int r = i / (K / 8), c = (i % (K / 8)) * 8;
        const bool ok = b0r + r < n;
        cp16(sx + r * LD + c, X + (ok ? (b0r + r) * K + c : 0), ok);
    }
    cp_wait();
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int64_t r0 = b0r + warp * 16;
    const int64_t ra = r0 + g, rb = r0 + g + 8;
    const bool va = ra < n, vb = rb < n;
    float acc[16][4];
#pragma unroll
    for (int j = 0; j < 16; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
    const int lr = lane & 7, lm = lane >> 3;
#pragma unroll
    for (int k0 = 0; k0 < K; k0 += 16) {
        uint32_t a[4];  // (rows 0-7, k 0-7), (8-15, 0-7), (0-7, 8-15), (8-15, 8-15)
        ldsm4(a, sx + (warp * 16 + (lm & 1) * 8 + lr) * LD + k0 + (lm >> 1) * 8);
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
            uint32_t b[4];  // column tiles j, j + 1, k halves 0, 1 of each
            ldsm4(b, sw + (8 * (j + (lm >> 1)) + lr) * LD + k0 + (lm & 1) * 8);
            mma_bf16(acc[j], a, b[0], b[1]);
            mma_bf16(acc[j + 1], a, b[2], b[3]);
        }
    }
    __syncthreads();  // the output rows overlay W and X
    __nv_bfloat16 *so = lin_sm + warp * 16 * LO;
    float ya = 0.0f, yb = 0.0f;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const int col = 8 * j + 2 * t;
        const float b0 = bias ? bias[col] : 0.0f, b1 = bias ? bias[col + 1] : 0.0f;
        float v[4] = {acc[j][0] + b0, acc[j][1] + b1, acc[j][2] + b0, acc[j][3] + b1};
        if (EPI == EPI_RELU) {
#pragma unroll
            for (int q = 0; q < 4; ++q) v[q] = fmaxf(v[q], 0.0f);
        } else {
            if (va) {
                const __nv_bfloat162 m = *reinterpret_cast<const __nv_bfloat162 *>(mask + ra * W + col);
                if (!(__bfloat162float(m.x) > 0.0f)) v[0] = 0.0f;
                if (!(__bfloat162float(m.y) > 0.0f)) v[1] = 0.0f;
            }
            if (vb) {
                const __nv_bfloat162 m = *reinterpret_cast<const __nv_bfloat162 *>(mask + rb * W + col);
                if (!(__bfloat162float(m.x) > 0.0f)) v[2] = 0.0f;
                if (!(__bfloat162float(m.y) > 0.0f)) v[3] = 0.0f;
            }
        }
        const __nv_bfloat162 oa = __floats2bfloat162_rn(v[0], v[1]), ob = __floats2bfloat162_rn(v[2], v[3]);
        *reinterpret_cast<__nv_bfloat162 *>(so + g * LO + col) = oa;
        *reinterpret_cast<__nv_bfloat162 *>(so + (g + 8) * LO + col) = ob;
        if (HEAD) {  // the head reads the stored (BF16-rounded) activations
            const float w0 = prm[O_W4 + col], w1 = prm[O_W4 + col + 1];
            ya += __bfloat162float(oa.x) * w0 + __bfloat162float(oa.y) * w1;
            yb += __bfloat162float(ob.x) * w0 + __bfloat162float(ob.y) * w1;
        }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i) {  // 16 rows of 256 bytes, two rows per step
        const int r = 2 * i + (lane >> 4), c = (lane & 15) * 8;
        if (r0 + r < n)
            *reinterpret_cast<uint4 *>(out + (r0 + r) * W + c) = *reinterpret_cast<const uint4 *>(so + r * LO + c);
    }
    if (HEAD) {
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            ya += __shfl_xor_sync(0xffffffffu, ya, o);
            yb += __shfl_xor_sync(0xffffffffu, yb, o);
        }
        if (t == 0) {
            const float b4 = prm[O_B4];
            if (va) y[ra] = ya + b4;
            if (vb) y[rb] = yb + b4;
        }
    }
}

template <int K, int EPI, bool HEAD>
int launch_linear(bool chained, const __nv_bfloat16 *X, const __nv_bfloat16 *Wt, const float *bias, const __nv_bfloat16 *mask,
                  int64_t n, __nv_bfloat16 *out, const float *prm, float *y, cudaStream_t s) {
    constexpr size_t smem = lin_smem_out<K>();
    static DeviceOnce once;
    EDFMM_CUDA_TRY(allow_smem(once, k_pcn_linear<K, EPI, HEAD>, smem));
    EDFMM_CUDA_TRY(chain_launch(chained, k_pcn_linear<K, EPI, HEAD>, nblk(n, kLinRows), 256, smem, s, X, Wt, bias, mask, n,
                                out, prm, y));
    EDFMM_LAUNCH_CHECK("k_pcn_linear");
    return EDFMM_OK;
}

// ---------------------------------------------------------------------------
// context: g = mean_i h1_i;  c2 = V2 g + b2
// ---------------------------------------------------------------------------
// per-part column sums of a BF16 (n x 128) matrix, optionally weighted by w[r],
// in row order.  Stages of 128 rows are copied to shared memory by the whole
// block, and one thread per column adds them: its chain of additions is the
// same as over device memory, without a load's latency in every few links
// (30,000 rows: 36 -> 12 us).
constexpr int kColStage = 128;
constexpr size_t kColSmem = 2 * kColStage * W * sizeof(__nv_bfloat16);
__global__ void __launch_bounds__(512) k_pcn_colsum_part(const __nv_bfloat16 *h, const float *w,
                                                         int64_t n, float *part) {
    chain_next();
    chain_wait();
    extern __shared__ __align__(16) __nv_bfloat16 stage[];  // two stages of kColStage rows
    __shared__ float tw[2][kColStage];
    const int c = threadIdx.x;
    const int64_t r0 = (int64_t)blockIdx.x * kColRows, r1 = (n < r0 + kColRows) ? n : r0 + kColRows;
    auto fetch = [&](int64_t rt, int buf) {  // the next stage's rows come while one is added
        if (rt < r1) {
            const int rows = (int)(r1 - rt < kColStage ? r1 - rt : kColStage);
            for (int i = threadIdx.x; i < rows * (W / 8); i += 512)
                cp16(stage + buf * kColStage * W + 8 * i, h + rt * W + 8 * i, true);
            if (w)
                for (int i = threadIdx.x; i < rows; i += 512) tw[buf][i] = w[rt + i];
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float s = 0.0f;
    fetch(r0, 0);
    int buf = 0;
    for (int64_t rt = r0; rt < r1; rt += kColStage, buf ^= 1) {
        const int rows = (int)(r1 - rt < kColStage ? r1 - rt : kColStage);
        fetch(rt + kColStage, buf ^ 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        if (c < W) {
            const __nv_bfloat16 *t = stage + buf * kColStage * W;
#pragma unroll 16
            for (int r = 0; r < rows; ++r) {
                const float v = __bfloat162float(t[r * W + c]);
                s += w ? tw[buf][r] * v : v;
            }
        }
        __syncthreads();
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (c < W) part[(int64_t)blockIdx.x * W + c] = s;
}

// out[c] = scale * sum_p part[p][c]  (fixed order)
__device__ __forceinline__ float reduce_cols(const float *part, int64_t np, int c) {
    float s = 0.0f;
#pragma unroll 16
    for (int64_t p = 0; p < np; ++p) s += part[p * W + c];
    return s;
}

// g = scale * column sums of h1, and the context c2 = b2 + V2 g: one block,
// since each is a chain of W adds that no second block shortens.  The matrix is staged by all threads (a thread per row that read its own words
// from memory took 10 us) while the first W add the sums; one thread a row then
// adds in column order
constexpr int kCtxLd = W + 1;
constexpr size_t kCtxSmem = (W * kCtxLd + W) * sizeof(float);
__global__ void __launch_bounds__(8 * W) k_pcn_context(const float *prm, const float *part,
                                                       int64_t np, float scale, float *g,
                                                       float *c2) {
    chain_next();
    chain_wait();
    extern __shared__ float ctx[];  // [W][W + 1], then g
#pragma unroll
    for (int i = 0; i < W / 8; ++i) {
        const int q = threadIdx.x + 8 * W * i;
        ctx[(q / W) * kCtxLd + q % W] = prm[O_V2 + q];
    }
    if (threadIdx.x < W) g[threadIdx.x] = ctx[W * kCtxLd + threadIdx.x] = reduce_cols(part, np, threadIdx.x) * scale;
    __syncthreads();
    if (threadIdx.x >= W) return;
    const int r = threadIdx.x;
    float s = prm[O_B2 + r];
#pragma unroll 32
    for (int k = 0; k < W; ++k) s += ctx[r * kCtxLd + k] * ctx[W * kCtxLd + k];
    c2[r] = s;
}

// ---------------------------------------------------------------------------
// backward
// ---------------------------------------------------------------------------
// Head of the network, three results of dy and h3 that need nothing of one
// another.  Block 0: db4 = sum dy; block 1: dw4 = sums of the column parts; the
// others: dz3[r][c] = (h3 > 0) ? dy[r] w4[c] : 0, eight columns (16 bytes) per
// thread.  The two reductions are latency chains of one block each, and run
// beside the rows instead of before them (with the casts in one launch and the
// context's sums in its kernel, a training step of 30,000 panels went from 221
// to 209 us).
constexpr int kHeadSums = 2;
__global__ void __launch_bounds__(256) k_pcn_head_grad(const __nv_bfloat16 *h3, const float *dy,
                                                       const float *prm, int64_t n,
                                                       const float *part, int64_t np,
                                                       float *grads, __nv_bfloat16 *dz) {
    chain_next();
    chain_wait();
    if (blockIdx.x == 0) {
        __shared__ float red[8];
        float s = 0.0f;
#pragma unroll 16
        for (int64_t i = threadIdx.x; i < n; i += 256) s += dy[i];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
        __syncthreads();
        if (threadIdx.x == 0) {
            float t = 0.0f;
            for (int w = 0; w < 8; ++w) t += red[w];
            grads[O_B4] = t;
        }
        return;
    }
    if (blockIdx.x == 1) {
        if (threadIdx.x < W) grads[O_W4 + threadIdx.x] = reduce_cols(part, np, threadIdx.x);
        return;
    }
    const int64_t i = (int64_t)(blockIdx.x - kHeadSums) * blockDim.x + threadIdx.x;
    if (i >= n * (W / 8)) return;
    const int c = (int)(i % (W / 8)) * 8;
    const float d = dy[i / (W / 8)];
    uint4 in = reinterpret_cast<const uint4 *>(h3)[i], o;
    const __nv_bfloat162 *x = reinterpret_cast<const __nv_bfloat162 *>(&in);
    __nv_bfloat162 *z = reinterpret_cast<__nv_bfloat162 *>(&o);
#pragma unroll
    for (int q = 0; q < 4; ++q)
        z[q] = __floats2bfloat162_rn(__bfloat162float(x[q].x) > 0.0f ? d * prm[O_W4 + c + 2 * q] : 0.0f,
                                     __bfloat162float(x[q].y) > 0.0f ? d * prm[O_W4 + c + 2 * q + 1] : 0.0f);
    reinterpret_cast<uint4 *>(dz)[i] = o;
}

// partial weight gradients over a block of rows, on the tensor cores:
//   part[p][o][k] = sum_{r in block p} D[r][o] X[r][k]     (o < 128, k < K)
//   part[p][128*K + o] = sum_r D[r][o]                   (bias gradient)
// The product D^T X has the rows r as its reduction dimension: stages of 64
// rows are copied to shared memory as they are (16 bytes at a time, padded
// rows, rows past the end zero) and ldmatrix transposes the fragments of both
// operands.  A block computes 32 of the 128 output rows (blockIdx.x % 4): a warp 16
// of them against up to 32 columns (mma.sync m16n8k16, BF16 in, FP32
// accumulate; fixed order), and one more warp the bias sums, in row order on
// the FP32 pipe.  Bound by the latency of the copies (a partial is a chain of
// 16 stages), so three stages are in flight; X is read four times, from L2.
constexpr int kWgStage = 64, kWgDepth = 4, kWgSlice = 32, kWgSlices = W / kWgSlice, kWgLdd = kWgSlice + 8;
template <int K>
struct Wg {
    static constexpr int groups = K > 32 ? K / 32 : 1, cols = K / groups, threads = (2 * groups + 1) * 32;
    static constexpr int ldx = K + 8;  // padded row strides (bf16 elements): odd multiples of 16 bytes
    static constexpr int stage = kWgStage * (kWgLdd + ldx);
    static constexpr size_t smem = kWgDepth * stage * sizeof(__nv_bfloat16);
};
template <int K>
__global__ void __launch_bounds__(Wg<K>::threads) k_pcn_wgrad_part(const __nv_bfloat16 *D,
                                                                   const __nv_bfloat16 *X, int64_t n,
                                                                   float *part) {
    chain_next();
    chain_wait();
    using G = Wg<K>;
    constexpr int LDX = G::ldx, NT = G::cols / 8;  // NT: n-tiles of 8 columns per warp
    extern __shared__ __align__(16) __nv_bfloat16 wg_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3, lr = lane & 7, lm = lane >> 3;
    const int slice = (int)(blockIdx.x % kWgSlices) * kWgSlice, o0 = 16 * (warp & 1), c0 = G::cols * (warp >> 1);
    const bool bias = warp == 2 * G::groups;
    float acc[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
    float bsum = 0.0f;
    const int64_t p = blockIdx.x / kWgSlices, r0 = p * kPartRows;
    const int rows = (int)((n - r0 < kPartRows) ? n - r0 : kPartRows), stages = (rows + kWgStage - 1) / kWgStage;
    auto fetch = [&](int q) {  // one group of copies per call, empty past the end
        if (q < stages) {
            __nv_bfloat16 *Dt = wg_smem + (q % kWgDepth) * G::stage, *Xt = Dt + kWgStage * kWgLdd;
            const int left = rows - q * kWgStage;
            const int64_t rq = r0 + q * kWgStage;
            for (int i = tid; i < kWgStage * (kWgSlice / 8); i += G::threads) {
                const int r = i / (kWgSlice / 8), c = (i % (kWgSlice / 8)) * 8;
                cp16(Dt + r * kWgLdd + c, D + (r < left ? (rq + r) * W + slice + c : 0), r < left);
            }
            for (int i = tid; i < kWgStage * (K / 8); i += G::threads) {
                const int r = i / (K / 8), c = (i % (K / 8)) * 8;
                cp16(Xt + r * LDX + c, X + (r < left ? (rq + r) * K + c : 0), r < left);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int q = 0; q < kWgDepth - 1; ++q) fetch(q);
    for (int q = 0; q < stages; ++q) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kWgDepth - 2) : "memory");
        __syncthreads();  // stage q is there, and stage q - 1 has been read
        fetch(q + kWgDepth - 1);
        const __nv_bfloat16 *Dt = wg_smem + (q % kWgDepth) * G::stage, *Xt = Dt + kWgStage * kWgLdd;
        if (bias) {
            const int left = rows - q * kWgStage, m = left < kWgStage ? left : kWgStage;
#pragma unroll 16
            for (int r = 0; r < m; ++r) bsum += __bfloat162float(Dt[r * kWgLdd + lane]);
        } else {
#pragma unroll
            for (int k0 = 0; k0 < kWgStage; k0 += 16) {
                uint32_t a[4];  // (o 0-7, r 0-7), (o 8-15, r 0-7), (o 0-7, r 8-15), (o 8-15, r 8-15)
                ldsm4t(a, Dt + (k0 + (lm >> 1) * 8 + lr) * kWgLdd + o0 + (lm & 1) * 8);
#pragma unroll
                for (int j = 0; j < NT; j += 2) {
                    uint32_t b[4];  // column tiles j, j + 1, row halves 0, 1 of each
                    ldsm4t(b, Xt + (k0 + (lm & 1) * 8 + lr) * LDX + c0 + 8 * (j + (lm >> 1)));
                    mma_bf16(acc[j], a, b[0], b[1]);
                    mma_bf16(acc[j + 1], a, b[2], b[3]);
                }
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    float *pp = part + p * (W * K + W);
    if (bias) {
        pp[W * K + slice + lane] = bsum;
        return;
    }
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        const int col = c0 + 8 * j + 2 * t;
        *reinterpret_cast<float2 *>(pp + (slice + o0 + g) * K + col) = make_float2(acc[j][0], acc[j][1]);
        *reinterpret_cast<float2 *>(pp + (slice + o0 + g + 8) * K + col) = make_float2(acc[j][2], acc[j][3]);
    }
}
template <int K>
cudaError_t launch_wgrad(bool chained, const __nv_bfloat16 *D, const __nv_bfloat16 *X, int64_t n, float *part, cudaStream_t s) {
    return chain_launch(chained, k_pcn_wgrad_part<K>, (unsigned)(n_parts(n) * kWgSlices), Wg<K>::threads, Wg<K>::smem, s, D, X,
                        n, part);
}

// grads[off + i] = sum_p part[p][i] (i < W*K), grads[boff + o] = sum_p part[p][W*K + o]
__global__ void k_pcn_wgrad_reduce(const float *part, int64_t np, int K, float *grads,
                                   int64_t off, int64_t boff) {
    chain_next();
    chain_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int stride = W * K + W;
    if (i >= stride) return;
    float s = 0.0f;
#pragma unroll 16
    for (int64_t p = 0; p < np; ++p) s += part[p * stride + i];
    if (i < W * K)
        grads[off + i] = s;
    else
        grads[boff + (i - W * K)] = s;
}

// context backward: dV2 = dc2 g^T, db2 = dc2, dg = V2^T dc2 / n  (dc2 = column
// sum of dz2); block r < 128 writes row r of dV2, block 128 dg
__global__ void __launch_bounds__(W) k_pcn_context_grad(const float *prm, const float *g,
                                                        const float *dc, int64_t n, float *grads,
                                                        float *dg) {
    chain_next();
    chain_wait();
    const int k = threadIdx.x, r = blockIdx.x;
    if (r < W) {
        grads[O_V2 + r * W + k] = dc[r] * g[k];
        return;
    }
    float s = 0.0f;
#pragma unroll 32
    for (int o = 0; o < W; ++o) s += prm[O_V2 + o * W + k] * dc[o];
    dg[k] = s / (float)(n > 0 ? n : 1);
}

int staged_smem() {  // dynamic shared memory above 48 KB
    static DeviceOnce once[3];
    EDFMM_CUDA_TRY(allow_smem(once[0], k_pcn_wgrad_part<W>, Wg<W>::smem));
    EDFMM_CUDA_TRY(allow_smem(once[1], k_pcn_context, kCtxSmem));
    EDFMM_CUDA_TRY(allow_smem(once[2], k_pcn_colsum_part, kColSmem));
    return EDFMM_OK;
}

// ---------------------------------------------------------------------------
// loss: L = sum A (s (1 + y) - sigma)^2 / sum A sigma^2, dL/dy.  One cluster of
// eight blocks: dL/dy needs the whole denominator, and the blocks exchange
// their sums through distributed shared memory (added in block order), so the
// call needs no scratch.  30,000 panels: one block took 189 us, the cluster
// 24, 18 with the products of a thread's first elements kept for dL/dy (about
// 13 FP64 operations an element on eight SMs' pipes).
// ---------------------------------------------------------------------------
constexpr int kLossBlocks = 8, kLossKept = 4;
__global__ void __cluster_dims__(kLossBlocks, 1, 1) __launch_bounds__(1024)
    k_pcn_loss(const float *__restrict__ y, const double *__restrict__ s, const double *__restrict__ sigma,
               const double *__restrict__ a, int64_t n, float *__restrict__ dy, double *__restrict__ loss) {
    __shared__ double red[2][32];
    __shared__ double sums[2], inv_s;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, rank = blockIdx.x;
    double num = 0, den = 0, kept[kLossKept];  // a e s of the thread's first elements
    int k = 0;
    for (int64_t i = rank * 1024 + tid; i < n; i += kLossBlocks * 1024, ++k) {
        const double si = s[i], gi = sigma[i], e = si * (1.0 + (double)y[i]) - gi, ae = a[i] * e;
        num += ae * e;
        den += a[i] * gi * gi;
#pragma unroll
        for (int q = 0; q < kLossKept; ++q)
            if (q == k) kept[q] = ae * si;
    }
    for (int o = 16; o > 0; o >>= 1) {
        num += __shfl_xor_sync(0xffffffffu, num, o);
        den += __shfl_xor_sync(0xffffffffu, den, o);
    }
    if (lane == 0) {
        red[0][wid] = num;
        red[1][wid] = den;
    }
    __syncthreads();
    if (tid < 2) {
        double t = 0;
        for (int w = 0; w < 32; ++w) t += red[tid][w];
        sums[tid] = t;
    }
    auto cluster_sync = [] {
        asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    };
    cluster_sync();
    if (tid == 0) {
        double t[2] = {0, 0};
        for (int r = 0; r < kLossBlocks; ++r) {
            for (int q = 0; q < 2; ++q) {
                unsigned at;
                double v;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                             : "=r"(at)
                             : "r"((unsigned)__cvta_generic_to_shared(&sums[q])), "r"(r));
                asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(at) : "memory");
                t[q] += v;
            }
        }
        const double d = t[1] > 0 ? t[1] : 1.0;
        if (rank == 0) *loss = t[0] / d;
        inv_s = 2.0 / d;
    }
    cluster_sync();  // the sums have been read (and the block sees inv_s)
    const double f = inv_s;
    int64_t i = rank * 1024 + tid;
#pragma unroll
    for (int q = 0; q < kLossKept; ++q, i += kLossBlocks * 1024)
        if (i < n) dy[i] = (float)(kept[q] * f);
    for (; i < n; i += kLossBlocks * 1024) {
        const double e = s[i] * (1.0 + (double)y[i]) - sigma[i];
        dy[i] = (float)(a[i] * e * s[i] * f);
    }
}

__global__ void k_pcn_adam(float *p, const float *gr, float *m,
                           float *v, int64_t count, float lr, float b1, float b2, float eps, float c1,
                           float c2) {
    chain_next();
    chain_wait();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const float gi = gr[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

}  // namespace
}  // namespace edfmm

using namespace edfmm;

extern "C" EDFMM_API int64_t edfmm_pcn_num_params(void) { return NPARAM; }

extern "C" EDFMM_API size_t edfmm_pcn_workspace_bytes(int64_t n) { return carve(nullptr, std::max<int64_t>(n, 1)).bytes; }

extern "C" EDFMM_API int edfmm_pcn_features(const double *centroids_dev, const double *normals_dev,
                                            const double *areas_dev, const double *rhs_dev, int64_t n,
                                            float *features_dev, void *ws_dev, size_t ws_bytes, void *stream) {
    if (n <= 0 || !centroids_dev || !normals_dev || !areas_dev || !rhs_dev || !features_dev || !ws_dev)
        return fail(EDFMM_ERR_ARG, "edfmm_pcn_features: bad arguments");
    Ws w = carve(ws_dev, n);
    if (ws_bytes < w.bytes) return fail(EDFMM_ERR_ARG, "edfmm_pcn_features: workspace too small");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // the stats partials borrow the weight-gradient partial buffer (at least
    // W * W + W floats, far more than kStatBlocks * 8 doubles; not in use here)
    double *sp = reinterpret_cast<double *>(w.part);
    k_pcn_stats_part<<<kStatBlocks, 256, 0, s>>>(centroids_dev, areas_dev, rhs_dev, n, nullptr, sp);
    EDFMM_LAUNCH_CHECK("k_pcn_stats_part");
    k_pcn_stats_fin<<<1, 32, 0, s>>>(sp, kStatBlocks, n, 0, w.stats);
    EDFMM_LAUNCH_CHECK("k_pcn_stats_fin");
    k_pcn_stats_part<<<kStatBlocks, 256, 0, s>>>(centroids_dev, areas_dev, rhs_dev, n, w.stats, sp);
    EDFMM_LAUNCH_CHECK("k_pcn_stats_part");
    k_pcn_stats_fin<<<1, 32, 0, s>>>(sp, kStatBlocks, n, 1, w.stats);
    EDFMM_LAUNCH_CHECK("k_pcn_stats_fin");
    k_pcn_features<<<nblk(n, 256), 256, 0, s>>>(centroids_dev, normals_dev, areas_dev, rhs_dev, n, w.stats,
                                                 features_dev);
    EDFMM_LAUNCH_CHECK("k_pcn_features");
    return EDFMM_OK;
}

extern "C" EDFMM_API int edfmm_pcn_forward(const float *params_dev, const float *features_dev, int64_t n,
                                           float *y_dev, void *ws_dev, size_t ws_bytes, void *stream) {
    if (n <= 0 || !params_dev || !features_dev || !y_dev || !ws_dev)
        return fail(EDFMM_ERR_ARG, "edfmm_pcn_forward: bad arguments");
    Ws w = carve(ws_dev, n);
    if (ws_bytes < w.bytes) return fail(EDFMM_ERR_ARG, "edfmm_pcn_forward: workspace too small");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (int rc = staged_smem()) return rc;
    const bool chained = chain_stream(s);
    const int64_t np = n_col_parts(n);
    const int64_t nf = n * NIN;
    EDFMM_CUDA_TRY(chain_launch(chained, k_pcn_cast, nblk(nf > W * W ? nf : W * W, 256), 256, 0, s, params_dev, w.w1b,
                                w.w2b, w.w3b, w.w2t, w.w3t, features_dev, nf, w.x0));
    EDFMM_LAUNCH_CHECK("k_pcn_cast");
    if (int rc = launch_linear<NIN, EPI_RELU, false>(chained, w.x0, w.w1b, params_dev + O_B1, nullptr, n, w.h1, params_dev, nullptr, s))
        return rc;
    EDFMM_CUDA_TRY(chain_launch(chained, k_pcn_colsum_part, (unsigned)np, 512, kColSmem, s, w.h1, nullptr, n, w.part));
    EDFMM_LAUNCH_CHECK("k_pcn_colsum_part");
    EDFMM_CUDA_TRY(chain_launch(chained, k_pcn_context, 1, 8 * W, kCtxSmem, s, params_dev, w.part, np, 1.0f / (float)n,
                                w.g, w.c2));
    EDFMM_LAUNCH_CHECK("k_pcn_context");
    if (int rc = launch_linear<W, EPI_RELU, false>(chained, w.h1, w.w2b, w.c2, nullptr, n, w.h2, params_dev, nullptr, s)) return rc;
    return launch_linear<W, EPI_RELU, true>(chained, w.h2, w.w3b, params_dev + O_B3, nullptr, n, w.h3, params_dev, y_dev, s);
}

extern "C" EDFMM_API int edfmm_pcn_backward(const float *params_dev, int64_t n, const float *dy_dev, float *grads_dev,
                                            void *ws_dev, size_t ws_bytes, void *stream) {
    if (n <= 0 || !params_dev || !dy_dev || !grads_dev || !ws_dev)
        return fail(EDFMM_ERR_ARG, "edfmm_pcn_backward: bad arguments");
    Ws w = carve(ws_dev, n);
    if (ws_bytes < w.bytes) return fail(EDFMM_ERR_ARG, "edfmm_pcn_backward: workspace too small");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (int rc = staged_smem()) return rc;
    const bool chained = chain_stream(s);
    const int64_t np = n_parts(n), nc = n_col_parts(n);
    // head: dw4 = sum_r dy_r h3_r, db4 = sum dy, dz3 = (h3 > 0) dy w4
    EDFMM_CUDA_TRY(chain_launch(chained, k_pcn_colsum_part, (unsigned)nc, 512, kColSmem, s, w.h3, dy_dev, n, w.part));
    EDFMM_LAUNCH_CHECK("k_pcn_colsum_part");
    EDFMM_CUDA_TRY(chain_launch(chained, k_pcn_head_grad, kHeadSums + nblk(n * (W / 8), 256), 256, 0, s, w.h3, dy_dev,
                                params_dev, n, w.part, nc, grads_dev, w.dz));
    EDFMM_LAUNCH_CHECK("k_pcn_head_grad");
    // layer 3: dW3 = dz3^T h2;  dz2 = (h2 > 0) dz3 W3
    EDFMM_CUDA_TRY(launch_wgrad<W>(chained, w.dz, w.h2, n, w.part, s));
    EDFMM_LAUNCH_CHECK("k_pcn_wgrad_part");
    EDFMM_CUDA_TRY(chain_launch(chained, k_pcn_wgrad_reduce, nblk(W * W + W, 256), 256, 0, s, w.part, np, W, grads_dev,
                                O_W3, O_B3));
    EDFMM_LAUNCH_CHECK("k_pcn_wgrad_reduce");
    if (int rc = launch_linear<W, EPI_MASK, false>(chained, w.dz, w.w3t, nullptr, w.h2, n, w.dz2, params_dev, nullptr, s)) return rc;
    // layer 2: dW2 = dz2^T h1, dc2 = colsum(dz2) -> dV2, db2, dg
    EDFMM_CUDA_TRY(launch_wgrad<W>(chained, w.dz2, w.h1, n, w.part, s));
    EDFMM_LAUNCH_CHECK("k_pcn_wgrad_part");
    EDFMM_CUDA_TRY(chain_launch(chained, k_pcn_wgrad_reduce, nblk(W * W + W, 256), 256, 0, s, w.part, np, W, grads_dev,
                                O_W2, O_B2));
    EDFMM_LAUNCH_CHECK("k_pcn_wgrad_reduce");
    EDFMM_CUDA_TRY(chain_launch(chained, k_pcn_context_grad, W + 1, W, 0, s, params_dev, w.g, grads_dev + O_B2, n,
                                grads_dev, w.dg));
    EDFMM_LAUNCH_CHECK("k_pcn_context_grad");
    // layer 1: dz1 = (h1 > 0) (dz2 W2 + dg / n);  dW1 = dz1^T x0
    if (int rc = launch_linear<W, EPI_MASK, false>(chained, w.dz2, w.w2t, w.dg, w.h1, n, w.dz, params_dev, nullptr, s)) return rc;
    EDFMM_CUDA_TRY(launch_wgrad<NIN>(chained, w.dz, w.x0, n, w.part, s));
    EDFMM_LAUNCH_CHECK("k_pcn_wgrad_part");
    EDFMM_CUDA_TRY(chain_launch(chained, k_pcn_wgrad_reduce, nblk(W * NIN + W, 256), 256, 0, s, w.part, np, NIN, grads_dev,
                                O_W1, O_B1));
    EDFMM_LAUNCH_CHECK("k_pcn_wgrad_reduce");
    return EDFMM_OK;
}

extern "C" EDFMM_API int edfmm_pcn_loss(const float *y_dev, const double *scale_dev, const double *sigma_dev,
                                        const double *areas_dev, int64_t n, float *dy_dev, double *loss_dev,
                                        void *stream) {
    if (n <= 0 || !y_dev || !scale_dev || !sigma_dev || !areas_dev || !dy_dev || !loss_dev)
        return fail(EDFMM_ERR_ARG, "edfmm_pcn_loss: bad arguments");
    k_pcn_loss<<<kLossBlocks, 1024, 0, static_cast<cudaStream_t>(stream)>>>(y_dev, scale_dev, sigma_dev, areas_dev, n, dy_dev,
                                                                   loss_dev);
    EDFMM_LAUNCH_CHECK("k_pcn_loss");
    return EDFMM_OK;
}

extern "C" EDFMM_API int edfmm_pcn_adam(float *params_dev, const float *grads_dev, float *m_dev, float *v_dev,
                                        int64_t count, float lr, float beta1, float beta2, float eps, int step,
                                        void *stream) {
    if (count <= 0 || step <= 0 || !params_dev || !grads_dev || !m_dev || !v_dev)
        return fail(EDFMM_ERR_ARG, "edfmm_pcn_adam: bad arguments");
    const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
    const bool chained = chain_stream(static_cast<cudaStream_t>(stream));
    EDFMM_CUDA_TRY(chain_launch(chained, k_pcn_adam, nblk(count, 256), 256, 0, static_cast<cudaStream_t>(stream),
                                params_dev, grads_dev, m_dev, v_dev, count, lr, beta1, beta2, eps, c1, c2));
    EDFMM_LAUNCH_CHECK("k_pcn_adam");
    return EDFMM_OK;
}
