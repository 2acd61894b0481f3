// mlp_kernel.cu -- the learned tracklet scorer: a 16-64-64-1 MLP with BF16
// weights and activations, FP32 accumulation and a sigmoid output.
//
//   mlp_score_kernel   inference on the 5th-generation tensor cores: tiles
//                      of 128 tracklets; tcgen05.mma (kind::f16, BF16 x BF16
//                      -> FP32 in tensor memory) for both hidden layers,
//                      operands in shared memory in the no-swizzle K-major
//                      core-matrix layout, completion through an mbarrier,
//                      accumulators read back with tcgen05.ld; bias, ReLU
//                      and the 64 -> 1 output layer on the CUDA cores.
//   mlp_train_kernel   one mini-batch: forward and backward on the CUDA
//                      cores with the same rounding points (input and first
//                      hidden layer rounded to BF16, weights BF16, FP32
//                      sums), weighted binary cross-entropy; per-block
//                      partial gradients (no atomics: the Adam kernel sums
//                      them in block order, so training is deterministic).
//   mlp_adam_kernel    Adam on the FP32 master parameters, then the BF16
//                      copies the forward passes read.
#include <cstddef>
#include <cuda_bf16.h>

#include "../../include/or_gb300.h"
#include "or_device.cuh"

namespace orgpu {

constexpr int MLP_IN = OR_NFEAT, MLP_H = OR_MLP_H;
constexpr uint32_t MLP_WAIT_LIMIT = 1u << 22;  // bounded mbarrier polls per wait

__device__ __forceinline__ float bf16_bits_to_float(uint16_t b) { return __uint_as_float((uint32_t)b << 16); }
__device__ __forceinline__ uint16_t float_to_bf16_bits(float f) {
    return __bfloat16_as_ushort(__float2bfloat16_rn(f));
}
__device__ __forceinline__ float round_bf16(float f) { return bf16_bits_to_float(float_to_bf16_bits(f)); }

// ---------------------------------------------------------------------------
// tcgen05 helpers
// ---------------------------------------------------------------------------
// byte offset of element (row, k) of a K-major operand with K columns in the
// no-swizzle core-matrix layout: 8 rows x 16 bytes per core matrix, core
// matrices along K adjacent (128 B apart), row groups K/8 core matrices apart
__device__ __forceinline__ uint32_t cm_offset(int row, int k, int K) {
    return (uint32_t)(((row >> 3) * (K >> 3) + (k >> 3)) * 128 + (row & 7) * 16 + (k & 7) * 2);
}
// shared-memory matrix descriptor (no swizzle): start, leading-dimension
// (K direction) and stride-dimension (row-group) byte offsets, version 1
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46);
}
// instruction descriptor, kind::f16: D = F32, A = B = BF16, both K-major
__host__ __device__ constexpr uint32_t idesc_bf16_f32(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// 16 consecutive FP32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float *v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

constexpr int MS_ROWS = 128;       // tracklets per tile = MMA M
constexpr int MS_TMEM_COLS = 64;   // D1, then D2: D1 is read before the second layer's MMAs
constexpr int MS_CTAS = 7;         // per SM: 32 KB of shared memory and 64 TMEM columns each

struct __align__(1024) MlpSmem {
    uint8_t a1[MS_ROWS * MLP_IN * 2];  // x tile, K = 16
    uint8_t a2[MS_ROWS * MLP_H * 2];   // h1 tile, K = 64
    uint8_t b1[MLP_H * MLP_IN * 2];    // W1 [64][16]
    uint8_t b2[MLP_H * MLP_H * 2];     // W2 [64][64]
    alignas(16) float mean[MLP_IN], inv_std[MLP_IN], bias1[MLP_H], bias2[MLP_H], w3[MLP_H];
    float b3;
    uint32_t tmem_base;
    uint64_t bar;
};
static_assert(MS_CTAS * (sizeof(MlpSmem) + 1024) <= 228 * 1024, "an SM holds them, with the 1 KB each that CUDA takes");
static_assert(MS_CTAS * MS_TMEM_COLS <= 512, "and their tensor memory");

// A tile's time is its two MMA round trips and the epilogues between them, so
// the CTAs of an SM overlap their tiles: seven of them at 72 registers (the
// epilogues hold 16 accumulator columns at a time, both layers' accumulators
// take the same 64), each loading its next rows while its first layer runs.
// Weights come in four bytes at a time, whatever the model's address (100,000
// rows 17 us; in 16 bytes, where the address allows it, the same; in two 29).
// Bound: issue of the epilogues.  With four CTAs, 2-byte weight loads and
// all 64 columns in registers 1,000,003 and 4,000,000 rows took 66 and 197 us;
// with six CTAs (a seventh did not fit beside 1 KB of unused shared memory
// each, and its share of the tiles ran after the others) 56 and 187 us; this
// takes 50 and 154 us (floor: 10 us for 68 bytes a row, and 40).
__device__ __forceinline__ void mlp_load_row(const float *__restrict__ feat, long row, long n_rows, const float *mean,
                                             float4 x[MLP_IN / 4]) {
    const float4 *src = reinterpret_cast<const float4 *>(row < n_rows ? feat + row * MLP_IN : mean);
#pragma unroll
    for (int q = 0; q < MLP_IN / 4; ++q) x[q] = src[q];
}

__global__ void __launch_bounds__(MS_ROWS, MS_CTAS)
    mlp_score_kernel(const or_mlp_t *__restrict__ model, const float *__restrict__ feat, long max_rows,
                     const int32_t *__restrict__ n_rows_dev, float *__restrict__ score, uint32_t *__restrict__ errw) {
    // rows to score: max_rows, or fewer when the count is on the device
    const long n_rows = n_rows_dev ? min(max_rows, (long)*n_rows_dev) : max_rows;
    const long ntiles = (n_rows + MS_ROWS - 1) / MS_ROWS;
    if ((long)blockIdx.x >= ntiles) return;  // no tile for this CTA: nothing allocated yet
    extern __shared__ __align__(1024) uint8_t ms_raw[];
    MlpSmem &S = *reinterpret_cast<MlpSmem *>(ms_raw);
    const int t = threadIdx.x, w = t >> 5;
    // weights into the B operand layouts, two at a time (their address in the
    // model is that of its floats), small vectors as floats
    {
        static_assert(alignof(or_mlp_t) >= 4 && offsetof(or_mlp_t, w1) % 4 == 0 && offsetof(or_mlp_t, w2) % 4 == 0,
                      "4-byte weight loads");
        const uint32_t *w1 = reinterpret_cast<const uint32_t *>(model->w1);
        const uint32_t *w2 = reinterpret_cast<const uint32_t *>(model->w2);
#pragma unroll
        for (int i = t; i < MLP_H * MLP_IN / 2; i += MS_ROWS)
            *reinterpret_cast<uint32_t *>(S.b1 + cm_offset(i * 2 / MLP_IN, i * 2 % MLP_IN, MLP_IN)) = w1[i];
#pragma unroll
        for (int i = t; i < MLP_H * MLP_H / 2; i += MS_ROWS)
            *reinterpret_cast<uint32_t *>(S.b2 + cm_offset(i * 2 / MLP_H, i * 2 % MLP_H, MLP_H)) = w2[i];
    }
    if (t < MLP_IN) {
        S.mean[t] = model->mean[t];
        S.inv_std[t] = model->inv_std[t];
    }
    if (t < MLP_H) {
        S.bias1[t] = model->b1[t];
        S.bias2[t] = model->b2[t];
        S.w3[t] = model->w3[t];
    }
    if (t == 0) {
        S.b3 = model->b3;
        mbar_init(&S.bar, 1);
    }
    if (w == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem_base)),
                     "r"(MS_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_proxy_async_smem();  // weights written by threads, read by the tensor core
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = S.tmem_base;
    const uint32_t lane_base = (uint32_t)(32 * w) << 16;  // this warp's quarter of the 128 lanes
    const uint32_t sa1 = smem_u32(S.a1), sa2 = smem_u32(S.a2), sb1 = smem_u32(S.b1), sb2 = smem_u32(S.b2);
    const uint32_t id = idesc_bf16_f32(MS_ROWS, MLP_H);
    uint32_t phase = 0;
    bool timed_out = false;

    float4 x[MLP_IN / 4];
    mlp_load_row(feat, (long)blockIdx.x * MS_ROWS + t, n_rows, S.mean, x);
    for (long tile = blockIdx.x; tile < ntiles && !timed_out; tile += gridDim.x) {
        const long row = tile * MS_ROWS + t;
        // ---- x row -> A1 (normalised, BF16) ----------------------------------
        {
            uint32_t pk[MLP_IN / 2];
#pragma unroll
            for (int q = 0; q < MLP_IN / 4; ++q) {
                const float4 m = reinterpret_cast<const float4 *>(S.mean)[q];
                const float4 d = reinterpret_cast<const float4 *>(S.inv_std)[q];
                pk[2 * q] = (uint32_t)float_to_bf16_bits((x[q].x - m.x) * d.x) |
                            ((uint32_t)float_to_bf16_bits((x[q].y - m.y) * d.y) << 16);
                pk[2 * q + 1] = (uint32_t)float_to_bf16_bits((x[q].z - m.z) * d.z) |
                                ((uint32_t)float_to_bf16_bits((x[q].w - m.w) * d.w) << 16);
            }
            *reinterpret_cast<uint4 *>(S.a1 + cm_offset(t, 0, MLP_IN)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            *reinterpret_cast<uint4 *>(S.a1 + cm_offset(t, 8, MLP_IN)) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
        }
        fence_proxy_async_smem();
        tc_fence_before();
        __syncthreads();  // A1 written, the previous tile's D2 read
        if (t == 0) {
            tc_fence_after();
            umma_bf16(tmem, umma_desc(sa1, 128, 256), umma_desc(sb1, 128, 256), id, 0u);
            umma_commit(&S.bar);
        }
        if (tile + gridDim.x < ntiles) mlp_load_row(feat, row + (long)gridDim.x * MS_ROWS, n_rows, S.mean, x);
        bool ok = mbar_wait_bounded(&S.bar, phase, MLP_WAIT_LIMIT);
        phase ^= 1u;
        if (__syncthreads_or(!ok)) {
            timed_out = true;
            break;
        }
        tc_fence_after();
        // ---- D1 -> h1 = bf16(relu(D1 + b1)) -> A2 --------------------------
#pragma unroll
        for (int c = 0; c < MLP_H; c += 16) {
            float d[16];
            tmem_ld16(tmem + lane_base + (uint32_t)c, d);
            tmem_ld_wait();
#pragma unroll
            for (int g = 0; g < 16; g += 8) {
                uint32_t pk[4];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const float4 b = reinterpret_cast<const float4 *>(S.bias1)[(c + g) / 4 + q];
                    const float *v = d + g + 4 * q;
                    pk[2 * q] = (uint32_t)float_to_bf16_bits(fmaxf(v[0] + b.x, 0.f)) |
                                ((uint32_t)float_to_bf16_bits(fmaxf(v[1] + b.y, 0.f)) << 16);
                    pk[2 * q + 1] = (uint32_t)float_to_bf16_bits(fmaxf(v[2] + b.z, 0.f)) |
                                    ((uint32_t)float_to_bf16_bits(fmaxf(v[3] + b.w, 0.f)) << 16);
                }
                *reinterpret_cast<uint4 *>(S.a2 + cm_offset(t, c + g, MLP_H)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            }
        }
        fence_proxy_async_smem();
        tc_fence_before();
        __syncthreads();  // A2 written, D1 read
        if (t == 0) {
            tc_fence_after();
#pragma unroll
            for (int s = 0; s < MLP_H / 16; ++s)
                umma_bf16(tmem, umma_desc(sa2 + 256u * s, 128, 1024), umma_desc(sb2 + 256u * s, 128, 1024), id,
                          s > 0 ? 1u : 0u);
            umma_commit(&S.bar);
        }
        ok = mbar_wait_bounded(&S.bar, phase, MLP_WAIT_LIMIT);
        phase ^= 1u;
        if (__syncthreads_or(!ok)) {
            timed_out = true;
            break;
        }
        tc_fence_after();
        // ---- D2 -> h2 = relu(D2 + b2); z = w3 . h2 + b3; sigmoid -------------
        float z = S.b3;
#pragma unroll
        for (int c = 0; c < MLP_H; c += 16) {
            float d[16];
            tmem_ld16(tmem + lane_base + (uint32_t)c, d);
            tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 b = reinterpret_cast<const float4 *>(S.bias2)[c / 4 + q];
                const float4 v = reinterpret_cast<const float4 *>(S.w3)[c / 4 + q];
                z += v.x * fmaxf(d[4 * q] + b.x, 0.f);
                z += v.y * fmaxf(d[4 * q + 1] + b.y, 0.f);
                z += v.z * fmaxf(d[4 * q + 2] + b.z, 0.f);
                z += v.w * fmaxf(d[4 * q + 3] + b.w, 0.f);
            }
        }
        if (row < n_rows) score[row] = 1.f / (1.f + expf(-z));
    }
    if (timed_out) {
        if (t == 0) atomicOr(errw, ERRW_TMA_TIMEOUT);
        // let the MMA in flight finish (bounded) before the columns are freed
        mbar_wait_bounded(&S.bar, phase ^ 1u, MLP_WAIT_LIMIT);
    }
    tc_fence_before();
    __syncthreads();
    if (w == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(MS_TMEM_COLS)
                     : "memory");
    }
}

// ---------------------------------------------------------------------------
// training
// ---------------------------------------------------------------------------
constexpr int TR_ROWS = 128;     // samples per block (a partial gradient each)
constexpr int TR_THREADS = 512;
constexpr int TR_LD = MLP_H + 4;  // row stride: rows stay 16-byte aligned

// parameter offsets in the FP32 vector
constexpr int P_W1 = 0, P_B1 = P_W1 + MLP_H * MLP_IN, P_W2 = P_B1 + MLP_H, P_B2 = P_W2 + MLP_H * MLP_H,
              P_W3 = P_B2 + MLP_H, P_B3 = P_W3 + MLP_H, P_N = P_B3 + 1;
static_assert(P_N == OR_MLP_NPARAM, "parameter vector layout");

struct TrainSmem {
    float w1[MLP_H * MLP_IN];        // [out][in]
    float w2[MLP_H][TR_LD];          // [out][in]
    float w2t[MLP_H][TR_LD];         // [in][out]
    float b1[MLP_H], b2[MLP_H], w3[MLP_H];
    float mean[MLP_IN], inv_std[MLP_IN];
    float x[TR_ROWS][MLP_IN + 4];
    float h1[TR_ROWS][TR_LD];        // first hidden layer; kept where a1 <= 0: 0
    float a2[TR_ROWS][TR_LD];        // second layer before the ReLU, then its gradient
    float dh1[TR_ROWS][TR_LD];
    float dz[TR_ROWS], loss[TR_ROWS];
    float b3;
};
// the arrays read 8 and 16 bytes at a time
static_assert(offsetof(TrainSmem, w2) % 16 == 0 && offsetof(TrainSmem, w2t) % 16 == 0 &&
                  offsetof(TrainSmem, x) % 16 == 0 && offsetof(TrainSmem, h1) % 16 == 0 &&
                  offsetof(TrainSmem, a2) % 16 == 0 && sizeof(float) * TR_LD % 16 == 0 &&
                  sizeof(float) * (MLP_IN + 4) % 16 == 0,
              "vector accesses are aligned");
static_assert(sizeof(TrainSmem) <= 227 * 1024, "one block per SM");

__device__ __forceinline__ float softplus(float a) { return fmaxf(a, 0.f) + log1pf(expf(-fabsf(a))); }

// Forward (and backward when grad_part != nullptr) of the samples
// idx[blockIdx.x*128 ...] of one batch of `batch` samples.  Loss: mean over
// the batch of pos_weight*y*softplus(-z) + (1-y)*softplus(z).  prob
// (optional) receives the sigmoid output per batch position.
//
// 512 threads per block: the 64x64 layers and their gradients are tiles of
// 4x4 outputs per thread over operands in shared memory, 16 bytes at a time.
// Every sum runs over its inputs (or samples) in order, one rounding per
// operation, so the results are those of one thread per output.  Bound: FP32
// issue, on one SM per 128 samples.  With one thread per sample (hidden
// vectors in local memory, weights read one word at a time) a batch of 8,192
// took 76 us; this takes 33 us.
__global__ void __launch_bounds__(TR_THREADS)
    mlp_train_kernel(const or_mlp_t *__restrict__ model, const float *__restrict__ feat,
                     const uint8_t *__restrict__ label, const int64_t *__restrict__ idx, int batch, float pos_weight,
                     float *__restrict__ grad_part, float *__restrict__ loss_part, float *__restrict__ prob) {
    extern __shared__ __align__(16) uint8_t tr_raw[];
    TrainSmem &S = *reinterpret_cast<TrainSmem *>(tr_raw);
    const int t = threadIdx.x;
    for (int i = t; i < MLP_H * MLP_IN; i += TR_THREADS) S.w1[i] = bf16_bits_to_float(model->w1[i]);
    for (int i = t; i < MLP_H * MLP_H; i += TR_THREADS) {
        const float v = bf16_bits_to_float(model->w2[i]);
        S.w2[i / MLP_H][i % MLP_H] = v;
        S.w2t[i % MLP_H][i / MLP_H] = v;
    }
    if (t < MLP_H) {
        S.b1[t] = model->b1[t];
        S.b2[t] = model->b2[t];
        S.w3[t] = model->w3[t];
    }
    if (t < MLP_IN) {
        S.mean[t] = model->mean[t];
        S.inv_std[t] = model->inv_std[t];
    }
    if (t == 0) S.b3 = model->b3;
    __syncthreads();
    const int base = blockIdx.x * TR_ROWS;
    for (int i = t; i < TR_ROWS * MLP_IN; i += TR_THREADS) {
        const int r = i / MLP_IN, k = i % MLP_IN;
        const bool valid = base + r < batch;
        const long row = valid ? idx[base + r] : 0;
        S.x[r][k] = round_bf16((feat[row * MLP_IN + k] - S.mean[k]) * S.inv_std[k]);
    }
    __syncthreads();
    // first layer: thread = one output column j of 16 samples
    {
        const int j = t % MLP_H, r0 = t / MLP_H;
        float w[MLP_IN];
#pragma unroll
        for (int k = 0; k < MLP_IN; ++k) w[k] = S.w1[j * MLP_IN + k];
        const float b = S.b1[j];
#pragma unroll 4
        for (int r = r0; r < TR_ROWS; r += TR_THREADS / MLP_H) {
            float sum = 0.f;
#pragma unroll
            for (int k = 0; k < MLP_IN; ++k) sum += w[k] * S.x[r][k];
            const float a = sum + b;
            S.h1[r][j] = round_bf16(fmaxf(a, 0.f));
            S.dh1[r][j] = a;  // its sign, for the way back
        }
    }
    __syncthreads();
    const int cj = (t % 16) * 4, cr = (t / 16) * 4;  // 4 columns, 4 samples
    // second layer: a2[r][j] = sum over k of w2[j][k] h1[r][k], k in order
    {
        float s[4][4] = {};
#pragma unroll 4
        for (int k = 0; k < MLP_H; ++k) {
            const float4 w = *reinterpret_cast<const float4 *>(&S.w2t[k][cj]);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float h = S.h1[cr + r][k];
                s[r][0] += w.x * h;
                s[r][1] += w.y * h;
                s[r][2] += w.z * h;
                s[r][3] += w.w * h;
            }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int j = 0; j < 4; ++j) S.a2[cr + r][cj + j] = s[r][j] + S.b2[cj + j];
    }
    __syncthreads();
    // output layer and the loss's derivative, one thread per sample
    if (t < TR_ROWS) {
        const int pos = base + t;
        const bool valid = pos < batch;
        const long r = valid ? idx[pos] : 0;
        float z = S.b3;
#pragma unroll 4
        for (int j = 0; j < MLP_H; ++j) z += S.w3[j] * fmaxf(S.a2[t][j], 0.f);
        const float p = 1.f / (1.f + expf(-z));
        if (prob && valid) prob[pos] = p;
        if (grad_part) {
            const float y = valid ? (float)label[r] : 0.f;
            const float inv_b = 1.f / (float)batch;
            S.dz[t] = valid ? (p * (pos_weight * y + 1.f - y) - pos_weight * y) * inv_b : 0.f;
            S.loss[t] = valid ? (pos_weight * y * softplus(-z) + (1.f - y) * softplus(z)) * inv_b : 0.f;
        }
    }
    if (!grad_part) return;
    __syncthreads();
    for (int i = t; i < TR_ROWS * MLP_IN; i += TR_THREADS)
        if (base + i / MLP_IN >= batch) S.x[i / MLP_IN][i % MLP_IN] = 0.f;
    float *gp = grad_part + (long)blockIdx.x * P_N;
    // gradients of w3, b3 and the loss while a2 stands
    if (t < MLP_H) {
        float g = 0.f;
#pragma unroll 4
        for (int i = 0; i < TR_ROWS; ++i) g += S.dz[i] * fmaxf(S.a2[i][t], 0.f);
        gp[P_W3 + t] = g;
    } else if (t == MLP_H) {
        float g = 0.f;
        for (int i = 0; i < TR_ROWS; ++i) g += S.dz[i];
        gp[P_B3] = g;
    } else if (t == MLP_H + 32) {
        float l = 0.f;
        for (int i = 0; i < TR_ROWS; ++i) l += S.loss[i];
        loss_part[blockIdx.x] = l;
    }
    __syncthreads();
    // a2 -> its gradient
#pragma unroll 4
    for (int i = t; i < TR_ROWS * MLP_H; i += TR_THREADS) {
        const int r = i / MLP_H, j = i % MLP_H;
        S.a2[r][j] = S.a2[r][j] > 0.f ? S.dz[r] * S.w3[j] : 0.f;
    }
    __syncthreads();
    // back through w2: dh1[r][k] = sum over j of w2[j][k] dh2[r][j], j in order
    {
        float s[4][4] = {};
#pragma unroll 4
        for (int j = 0; j < MLP_H; ++j) {
            const float4 w = *reinterpret_cast<const float4 *>(&S.w2[j][cj]);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float g = S.a2[cr + r][j];
                s[r][0] += w.x * g;
                s[r][1] += w.y * g;
                s[r][2] += w.z * g;
                s[r][3] += w.w * g;
            }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float &d = S.dh1[cr + r][cj + k];  // holds a1: the thread's own outputs only
                d = d > 0.f ? s[r][k] : 0.f;
            }
    }
    __syncthreads();
    // weight gradients, samples in order: w2 as 64x64 outputs of 8 a thread,
    // w1 as 64x16 of 2
    {
        const int j = (t / 16) * 2, k = (t % 16) * 4;
        float s[2][4] = {};
#pragma unroll 4
        for (int i = 0; i < TR_ROWS; ++i) {
            const float4 h = *reinterpret_cast<const float4 *>(&S.h1[i][k]);
            const float2 d = *reinterpret_cast<const float2 *>(&S.a2[i][j]);
            s[0][0] += d.x * h.x;
            s[0][1] += d.x * h.y;
            s[0][2] += d.x * h.z;
            s[0][3] += d.x * h.w;
            s[1][0] += d.y * h.x;
            s[1][1] += d.y * h.y;
            s[1][2] += d.y * h.z;
            s[1][3] += d.y * h.w;
        }
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) gp[P_W2 + (j + a) * MLP_H + k + b] = s[a][b];
    }
    {
        const int j = t / 8, k = (t % 8) * 2;
        float s0 = 0.f, s1 = 0.f;
#pragma unroll 4
        for (int i = 0; i < TR_ROWS; ++i) {
            const float d = S.dh1[i][j];
            const float2 x = *reinterpret_cast<const float2 *>(&S.x[i][k]);
            s0 += d * x.x;
            s1 += d * x.y;
        }
        gp[P_W1 + j * MLP_IN + k] = s0;
        gp[P_W1 + j * MLP_IN + k + 1] = s1;
    }
    if (t < 2 * MLP_H) {
        const int j = t % MLP_H;
        float g = 0.f;
#pragma unroll 4
        for (int i = 0; i < TR_ROWS; ++i) g += t < MLP_H ? S.dh1[i][j] : S.a2[i][j];
        gp[(t < MLP_H ? P_B1 : P_B2) + j] = g;
    }
}

// Adam on the FP32 parameters (gradient = sum of the blocks' partials, in
// block order), then the model copy the forward passes read.
__global__ void mlp_adam_kernel(float *__restrict__ param, float *__restrict__ m1, float *__restrict__ m2,
                                const float *__restrict__ grad_part, int nblocks, int step, float lr, float beta1,
                                float beta2, float eps, or_mlp_t *__restrict__ model) {
    const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < P_N; q += gridDim.x * blockDim.x) {
        float g = 0.f;
        for (int b = 0; b < nblocks; ++b) g += grad_part[(long)b * P_N + q];
        const float a = beta1 * m1[q] + (1.f - beta1) * g;
        const float v = beta2 * m2[q] + (1.f - beta2) * g * g;
        m1[q] = a;
        m2[q] = v;
        const float w = param[q] - lr * (a / c1) / (sqrtf(v / c2) + eps);
        param[q] = w;
        if (q < P_B1) model->w1[q - P_W1] = float_to_bf16_bits(w);
        else if (q < P_W2) model->b1[q - P_B1] = w;
        else if (q < P_B2) model->w2[q - P_W2] = float_to_bf16_bits(w);
        else if (q < P_W3) model->b2[q - P_B2] = w;
        else if (q < P_B3) model->w3[q - P_W3] = w;
        else model->b3 = w;
    }
}

size_t mlp_score_smem() { return sizeof(MlpSmem); }
size_t mlp_train_smem() { return sizeof(TrainSmem); }

cudaError_t launch_mlp_score(const or_mlp_t *model, const float *feat, long n_rows, const int32_t *n_rows_dev,
                             float *score, uint32_t *errw, cudaStream_t stream, int sm_count) {
    if (n_rows <= 0) return cudaSuccess;
    const size_t smem = mlp_score_smem();
    cudaError_t err = smem_attr_once((const void *)mlp_score_kernel, (int)smem);
    if (err != cudaSuccess) return err;
    const long ntiles = (n_rows + MS_ROWS - 1) / MS_ROWS;
    long blocks = ntiles;
    const long cap = (long)sm_count * MS_CTAS;
    if (blocks > cap) blocks = cap;
    mlp_score_kernel<<<(unsigned)blocks, MS_ROWS, smem, stream>>>(model, feat, n_rows, n_rows_dev, score, errw);
    return cudaGetLastError();
}

int mlp_train_blocks(int batch) { return (batch + TR_ROWS - 1) / TR_ROWS; }

cudaError_t launch_mlp_train(const or_mlp_t *model, const float *feat, const uint8_t *label, const int64_t *idx,
                             int batch, float pos_weight, float *grad_part, float *loss_part, float *prob,
                             cudaStream_t stream) {
    if (batch <= 0) return cudaSuccess;
    const size_t smem = mlp_train_smem();
    cudaError_t err = smem_attr_once((const void *)mlp_train_kernel, (int)smem);
    if (err != cudaSuccess) return err;
    mlp_train_kernel<<<(unsigned)mlp_train_blocks(batch), TR_THREADS, smem, stream>>>(
        model, feat, label, idx, batch, pos_weight, grad_part, loss_part, prob);
    return cudaGetLastError();
}

cudaError_t launch_mlp_adam(float *param, float *m1, float *m2, const float *grad_part, int nblocks, int step,
                            float lr, float beta1, float beta2, float eps, or_mlp_t *model, cudaStream_t stream) {
    mlp_adam_kernel<<<(P_N + 255) / 256, 256, 0, stream>>>(param, m1, m2, grad_part, nblocks, step, lr, beta1, beta2,
                                                          eps, model);
    return cudaGetLastError();
}

}  // namespace orgpu
