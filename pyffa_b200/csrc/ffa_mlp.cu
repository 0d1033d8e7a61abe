// ffa_mlp.cu -- the learned sector map: a residual MLP on the tensor cores.
//
// y = x + x Ws + bs + f(x),  f = L4 . SiLU . L3 . SiLU . L2 . SiLU . L1,
// widths 6 -> 256 -> 256 -> 256 -> 6.  Weights are float32 masters, rounded to
// bfloat16 where they enter an MMA; products accumulate in float32.  The skip layer (Ws, bs) stays float32.
//
// Training: one fused kernel per 64 samples runs forward and backward, one more
// forms the weight gradients, one sums them and takes the Adam step.
// Inference: one fused kernel per 128 particles applies the map n_apply times
// in a row.  Both run on tcgen05 with accumulators in tensor memory.  A general
// product (op(A) op(B) + bias, float32 in and out) is exported beside them.
#include <cuda_bf16.h>

#include "ffa_internal.cuh"

namespace {

// ----------------------------------------------------------- parameters
constexpr int H = FFA_MLP_HIDDEN;      // 256
constexpr int KIN = 16;                // input width padded to one k tile
constexpr int NOUT = 8;                // output width padded to one n tile
// float32 parameter block (offsets in floats)
constexpr int64_t P_W1 = 0;                       // [KIN][H]
constexpr int64_t P_B1 = P_W1 + KIN * H;
constexpr int64_t P_W2 = P_B1 + H;                // [H][H]
constexpr int64_t P_B2 = P_W2 + H * H;
constexpr int64_t P_W3 = P_B2 + H;                // [H][H]
constexpr int64_t P_B3 = P_W3 + H * H;
constexpr int64_t P_W4 = P_B3 + H;                // [H][NOUT]
constexpr int64_t P_B4 = P_W4 + H * NOUT;
constexpr int64_t P_WS = P_B4 + NOUT;             // [NOUT][NOUT] (6 x 6 used)
constexpr int64_t P_BS = P_WS + NOUT * NOUT;
constexpr int64_t P_WQ = P_BS + NOUT;             // [16][NOUT] (15 x 6 used)
constexpr int64_t P_TOTAL = P_WQ + 16 * NOUT;
// the 15 quadratic skip features s_i s_j, i <= j < 5, of a register-resident
// state, in the order (0, 0), (0, 1) .. (0, 4), (1, 1) .. (4, 4)
__device__ __forceinline__ void quad_features(const float *x, float *q)
{
    q[0] = x[0] * x[0]; q[1] = x[0] * x[1]; q[2] = x[0] * x[2]; q[3] = x[0] * x[3]; q[4] = x[0] * x[4];
    q[5] = x[1] * x[1]; q[6] = x[1] * x[2]; q[7] = x[1] * x[3]; q[8] = x[1] * x[4];
    q[9] = x[2] * x[2]; q[10] = x[2] * x[3]; q[11] = x[2] * x[4];
    q[12] = x[3] * x[3]; q[13] = x[3] * x[4];
    q[14] = x[4] * x[4];
}
static_assert(P_TOTAL == FFA_MLP_PARAMS, "parameter block layout");

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}

__device__ __forceinline__ void mma_bf16(float c[4], const uint32_t a[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ float tanh_approx(float x)
{
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// SiLU(z) = z sigmoid(z) = h + h tanh(h), h = z / 2 (training and inference
// evaluate it the same way)
__device__ __forceinline__ float silu(float z)
{
    const float h = 0.5f * z;
    return fmaf(h, tanh_approx(h), h);
}

// d SiLU / dz = sigmoid(z) (1 + z (1 - sigmoid(z))) = (1 + t)(1 + h (1 - t)) / 2
__device__ __forceinline__ float dsilu(float z)
{
    const float h = 0.5f * z, t = tanh_approx(h);
    return 0.5f * (1.0f + t) * fmaf(h, 1.0f - t, 1.0f);
}

// ------------------------------------------------------------- GEMM, narrow
// C[M][N] = op(A)[M][K] op(B)[K][N] (+ bias[N]); op(A)[m][k] = A[m*lda + k]
// or, with transA, A[k*lda + m]; op(B)[k][n] = B[k*ldb + n] or, with transB,
// B[n*ldb + k].  64 x 64 block tile, K staged 32 at a time as bf16 in shared
// memory (A row-major in k, B n-major in k: both fragment loads are 32-bit
// words), four warps of 32 x 32.
constexpr int GT_M = 64, GT_N = 64, GT_K = 32, GT_PAD = 8;

__global__ void __launch_bounds__(128) gemm_tc(const float *__restrict__ A, int lda, int transA,
                                               const float *__restrict__ B, int ldb, int transB,
                                               float *__restrict__ C, int ldc, int M, int N, int K,
                                               const float *__restrict__ bias)
{
    __shared__ __align__(16) __nv_bfloat16 sA[GT_M][GT_K + GT_PAD];
    __shared__ __align__(16) __nv_bfloat16 sB[GT_N][GT_K + GT_PAD];
    const int m0 = blockIdx.y * GT_M, n0 = blockIdx.x * GT_N;
    const int kb = 0, ke = K;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
    const int r = lane >> 2, c2 = (lane & 3) * 2;
    float acc[2][4][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.0f;
    for (int k0 = kb; k0 < ke; k0 += GT_K) {
        // staging: the index that is contiguous in global memory runs fastest
        // across threads (coalesced loads), converted to bfloat16
        // fixed trip counts (128 threads): the loads of a stage are issued together
        if (!transA) {
#pragma unroll
            for (int it = 0; it < GT_M * GT_K / 128; ++it) {
                const int e = threadIdx.x + 128 * it;
                const int mm = e / GT_K, kk = e - mm * GT_K;
                const int gm = m0 + mm, gk = k0 + kk;
                sA[mm][kk] = __float2bfloat16_rn((gm < M && gk < ke) ? A[(int64_t)gm * lda + gk] : 0.0f);
            }
        } else {
#pragma unroll
            for (int it = 0; it < GT_M * GT_K / 128; ++it) {
                const int e = threadIdx.x + 128 * it;
                const int kk = e / GT_M, mm = e - kk * GT_M;
                const int gm = m0 + mm, gk = k0 + kk;
                sA[mm][kk] = __float2bfloat16_rn((gm < M && gk < ke) ? A[(int64_t)gk * lda + gm] : 0.0f);
            }
        }
        if (transB) {
#pragma unroll
            for (int it = 0; it < GT_N * GT_K / 128; ++it) {
                const int e = threadIdx.x + 128 * it;
                const int nn = e / GT_K, kk = e - nn * GT_K;
                const int gn = n0 + nn, gk = k0 + kk;
                sB[nn][kk] = __float2bfloat16_rn((gn < N && gk < ke) ? B[(int64_t)gn * ldb + gk] : 0.0f);
            }
        } else {
#pragma unroll
            for (int it = 0; it < GT_N * GT_K / 128; ++it) {
                const int e = threadIdx.x + 128 * it;
                const int kk = e / GT_N, nn = e - kk * GT_N;
                const int gn = n0 + nn, gk = k0 + kk;
                sB[nn][kk] = __float2bfloat16_rn((gn < N && gk < ke) ? B[(int64_t)gk * ldb + gn] : 0.0f);
            }
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < GT_K; kk += 16) {
            uint32_t a[2][4];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int row = wm + i * 16 + r;
                a[i][0] = *reinterpret_cast<const uint32_t *>(&sA[row][kk + c2]);
                a[i][1] = *reinterpret_cast<const uint32_t *>(&sA[row + 8][kk + c2]);
                a[i][2] = *reinterpret_cast<const uint32_t *>(&sA[row][kk + c2 + 8]);
                a[i][3] = *reinterpret_cast<const uint32_t *>(&sA[row + 8][kk + c2 + 8]);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int col = wn + j * 8 + r;
                const uint32_t b0 = *reinterpret_cast<const uint32_t *>(&sB[col][kk + c2]);
                const uint32_t b1 = *reinterpret_cast<const uint32_t *>(&sB[col][kk + c2 + 8]);
#pragma unroll
                for (int i = 0; i < 2; ++i) mma_bf16(acc[i][j], a[i], b0, b1);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int gm = m0 + wm + i * 16 + r + ((q & 2) ? 8 : 0);
                const int gn = n0 + wn + j * 8 + c2 + (q & 1);
                if (gm < M && gn < N) C[(int64_t)gm * ldc + gn] = acc[i][j][q] + (bias ? bias[gn] : 0.0f);
            }
}

constexpr int64_t SPLIT_WORK = FFA_MLP_SPLIT_WORK;   // floats of the training work area beside those per sample

// ------------------------------------------------------- fused inference
// tcgen05 tensor cores, one 128-state tile per CTA at a time (persistent grid,
// one CTA per SM).  Every layer is one 128 x N accumulator in tensor memory:
// D0 = columns 0..255, D1 = columns 256..511, layers 1..4 alternate D0, D1.
// Warp roles: warp 0 streams W2 / W3 from global (L2-resident) into a ring
// of three 32 KB shared-memory slots with cp.async.bulk; warp 1 owns tensor
// memory and issues the MMAs (one thread); warps 2..17 are the epilogue, four
// threads per state (its tensor-memory lane), one per 16-column quarter of
// each 64-column chunk.  They read the accumulator row, add the bias, apply
// SiLU, round to bfloat16 and write the next layer's A operand one chunk at
// a time (the next chunk's tensor-memory load in flight meanwhile), so the
// next layer's MMAs on chunk c start while chunk c + 1 is still being
// written.  The state, the domain check and the float32 skip connection stay
// in the registers of the quarter-0 thread for all n_apply maps.
//
// Shared-memory operand layouts (K-major):
//  - A (activations, 128 x 256) and W2 / W3 / W4 (B operand, N x 256): four
//    64-column chunks, each row 128 B with the 128-byte swizzle (16-byte
//    unit j of row m stored at unit j ^ (m mod 8)), rows consecutive,
//    chunk bases 1024-aligned; descriptor SBO = 1024 B; the K = 16 slices of
//    a chunk start 32 B apart;
//  - X (layer-1 input, 128 x 16) and W1 (256 x 16): no swizzle, 8 x 8 core
//    matrices of 128 B, the two K halves 128 B apart (LBO) and 8-row groups
//    256 B apart (SBO).
// The inference weight pack in global memory holds W1, W4, W2, W3 in exactly
// these layouts, so each ring slot is one linear bulk copy.
constexpr int TC_M = 128;
constexpr int TC_CHUNK = 64;                                 // K columns per chunk
constexpr uint32_t A_CHUNK_BYTES = TC_M * 128;               // 16 KB
constexpr uint32_t W_CHUNK_BYTES = H * 128;                  // 32 KB
constexpr uint32_t W4_CHUNK_BYTES = 16 * 128;                // 2 KB
constexpr int RING = 3;
// weight pack (bytes)
constexpr uint32_t PK_W1 = 0;                                // 256 x 16 bf16, core matrices
constexpr uint32_t PK_W4 = PK_W1 + H * KIN * 2;              // 4 chunks x 16 rows
constexpr uint32_t PK_W2 = PK_W4 + 4 * W4_CHUNK_BYTES;       // 4 chunks x 256 rows
constexpr uint32_t PK_W3 = PK_W2 + 4 * W_CHUNK_BYTES;
constexpr uint32_t PK_TOTAL = PK_W3 + 4 * W_CHUNK_BYTES;
// shared memory (bytes from the 1024-aligned base)
constexpr uint32_t SM_A = 0;
constexpr uint32_t SM_RING = SM_A + 4 * A_CHUNK_BYTES;
constexpr uint32_t SM_W4 = SM_RING + RING * W_CHUNK_BYTES;
constexpr uint32_t SM_W1 = SM_W4 + 4 * W4_CHUNK_BYTES;
constexpr uint32_t SM_X = SM_W1 + H * KIN * 2;
constexpr uint32_t SM_BIAS = SM_X + TC_M * KIN * 2;          // b1 b2 b3 (halved), float
constexpr uint32_t SM_TAIL = SM_BIAS + 3 * H * 4;            // b4[8] Ws[64] bs[8] Wq[128]
constexpr uint32_t SM_BAR = SM_TAIL + 208 * 4;               // mbarriers (8 B each)
constexpr int NBAR = 1 + 4 + 1 + 2 * RING + 1;               // x_ready, a_ready[4], d_full, full[], empty[], drain
constexpr uint32_t SM_MISC = SM_BAR + NBAR * 8;              // tmem base, abort flag
constexpr uint32_t SM_TOTAL = SM_MISC + 16;
constexpr size_t TC_SMEM = SM_TOTAL + 1024;                  // + alignment slack
constexpr uint64_t WAIT_NS = 2000000000ull;                  // a pipeline wait gives up after 2 s

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t global_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// Waits for the phase of `bar` with `parity` for at most WAIT_NS, whatever
// the abort flag says (teardown: copies and MMAs in flight must land).
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity)
{
    const uint64_t t0 = global_ns();
    while (!mbar_test(bar, parity))
        if (global_ns() - t0 > WAIT_NS) return false;
    return true;
}

// Waits for the phase of `bar` with `parity`; gives up (and raises the
// block's abort flag) after WAIT_NS or when another thread has raised it.
// try_wait suspends the thread for a while by itself; the clock and the flag
// are read once every 64 polls.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag)
{
    if (mbar_test(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    while (true) {
#pragma unroll 1
        for (int i = 0; i < 64; ++i)
            if (mbar_test(bar, parity)) return true;
        if (*abort_flag) return false;
        if (global_ns() - t0 > WAIT_NS) {
            *abort_flag = 1;
            return false;
        }
    }
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// smem matrix descriptor: start, leading / stride byte offsets, layout
// (0: no swizzle, 2: 128-byte swizzle), version 1
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo, uint32_t layout)
{
    return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46) | ((uint64_t)layout << 61);
}

// instruction descriptor, kind::f16: bfloat16 A and B (K-major), float32 D
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void umma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void umma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

#define TMEM_LD32(taddr, v)                                                                                  \
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15," \
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"              \
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),      \
                   "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),  \
                   "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),             \
                   "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]),             \
                   "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])              \
                 : "r"(taddr))

#define TMEM_LD16(taddr, v)                                                                                  \
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}," \
                 " [%16];"                                                                                   \
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),      \
                   "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),  \
                   "=r"(v[14]), "=r"(v[15])                                                                  \
                 : "r"(taddr))

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// keeps the compiler from moving uses of tcgen05.ld results above the wait
#define REG_FENCE16(v)                                                                                       \
    asm volatile("" : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]),   \
                 "+r"(v[7]), "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]),      \
                 "+r"(v[14]), "+r"(v[15]))
#define REG_FENCE32(v)  \
    REG_FENCE16(v);     \
    REG_FENCE16((v + 16))

// byte offset of element (row, k) in a 128-byte-swizzled chunked operand
// with `rows` rows per chunk
__host__ __device__ __forceinline__ uint32_t swz_off(int row, int k, int rows)
{
    return (uint32_t)((k >> 6) * rows * 128 + row * 128 + ((((k & 63) >> 3) ^ (row & 7)) << 4) + ((k & 7) << 1));
}

// byte offset of element (row, k) of a no-swizzle K = 16 operand
__host__ __device__ __forceinline__ uint32_t core_off(int row, int k)
{
    return (uint32_t)((((row >> 3) * 2 + (k >> 3)) << 7) + ((row & 7) << 4) + ((k & 7) << 1));
}

// float32 parameters -> the inference weight pack (bfloat16, layouts above)
__global__ void pack_weights_kernel(const float *__restrict__ P, unsigned char *__restrict__ wp)
{
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    if (tid < H * H) {
        const int n = tid / H, k = tid % H;
        *reinterpret_cast<__nv_bfloat16 *>(wp + PK_W2 + swz_off(n, k, H)) = __float2bfloat16_rn(P[P_W2 + k * H + n]);
        *reinterpret_cast<__nv_bfloat16 *>(wp + PK_W3 + swz_off(n, k, H)) = __float2bfloat16_rn(P[P_W3 + k * H + n]);
    }
    if (tid < H * KIN) {
        // columns 0..5 and 6..11 both hold W1 rows 0..5 (high / low input parts)
        const int n = tid / KIN, k = tid % KIN;
        const float v = k < 12 ? P[P_W1 + (k % 6) * H + n] : 0.0f;
        *reinterpret_cast<__nv_bfloat16 *>(wp + PK_W1 + core_off(n, k)) = __float2bfloat16_rn(v);
    }
    if (tid < 16 * H) {
        const int n = tid / H, k = tid % H;
        const float v = n < NOUT ? P[P_W4 + k * NOUT + n] : 0.0f;
        *reinterpret_cast<__nv_bfloat16 *>(wp + PK_W4 + swz_off(n, k, 16)) = __float2bfloat16_rn(v);
    }
}

// SiLU of 8 accumulator values (bias pre-halved), packed to 4 bfloat16 pairs
__device__ __forceinline__ uint4 silu8(const uint32_t *v, const float *hb)
{
    float h[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) h[i] = fmaf(__uint_as_float(v[i]), 0.5f, hb[i]);
    uint4 o;
    o.x = pack_bf16(fmaf(h[0], tanh_approx(h[0]), h[0]), fmaf(h[1], tanh_approx(h[1]), h[1]));
    o.y = pack_bf16(fmaf(h[2], tanh_approx(h[2]), h[2]), fmaf(h[3], tanh_approx(h[3]), h[3]));
    o.z = pack_bf16(fmaf(h[4], tanh_approx(h[4]), h[4]), fmaf(h[5], tanh_approx(h[5]), h[5]));
    o.w = pack_bf16(fmaf(h[6], tanh_approx(h[6]), h[6]), fmaf(h[7], tanh_approx(h[7]), h[7]));
    return o;
}

constexpr int TC_THREADS = 32 * (2 + 16);

__global__ void __launch_bounds__(TC_THREADS, 1)
    mlp_infer_tc_kernel(const float *__restrict__ P, const unsigned char *__restrict__ wp, float *__restrict__ state,
                        int32_t *__restrict__ applied, int32_t *__restrict__ error, int64_t n, int n_apply,
                        float radius2)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char *sm = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t s0 = smem_u32(sm);
    float *sbias = reinterpret_cast<float *>(sm + SM_BIAS);
    float *stail = reinterpret_cast<float *>(sm + SM_TAIL);   // b4[0..7], Ws[8..71], bs[72..79], Wq[80..207]
    const uint32_t bar0 = s0 + SM_BAR;
    const uint32_t BAR_X = bar0, BAR_A = bar0 + 8, BAR_D = bar0 + 40, BAR_FULL = bar0 + 48,
                   BAR_EMPTY = bar0 + 48 + 8 * RING, BAR_DRAIN = bar0 + 48 + 16 * RING;
    uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(sm + SM_MISC);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(sm + SM_MISC + 4);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t ntiles = (n + TC_M - 1) / TC_M;

    // resident operands and constants
    for (int i = threadIdx.x; i < (int)(H * KIN * 2 / 16); i += blockDim.x)
        reinterpret_cast<uint4 *>(sm + SM_W1)[i] = reinterpret_cast<const uint4 *>(wp + PK_W1)[i];
    for (int i = threadIdx.x; i < (int)(4 * W4_CHUNK_BYTES / 16); i += blockDim.x)
        reinterpret_cast<uint4 *>(sm + SM_W4)[i] = reinterpret_cast<const uint4 *>(wp + PK_W4)[i];
    for (int i = threadIdx.x; i < 3 * H; i += blockDim.x) sbias[i] = 0.5f * P[(i < H ? P_B1 : i < 2 * H ? P_B2 : P_B3) + (i % H)];
    for (int i = threadIdx.x; i < 208; i += blockDim.x)
        stail[i] = i < 8 ? P[P_B4 + i] : i < 72 ? P[P_WS + (i - 8)] : i < 80 ? P[P_BS + (i - 72)] : P[P_WQ + (i - 80)];
    if (threadIdx.x == 0) {
        mbar_init(BAR_X, 4);
        for (int c = 0; c < 4; ++c) mbar_init(BAR_A + 8 * c, 16);
        mbar_init(BAR_D, 1);
        for (int s = 0; s < RING; ++s) {
            mbar_init(BAR_FULL + 8 * s, 1);
            mbar_init(BAR_EMPTY + 8 * s, 1);
        }
        mbar_init(BAR_DRAIN, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)),
                     "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_async_smem();
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    const uint32_t tmem = *tmem_holder;

    if (warp == 0) {
        // ---------------------------------------------------- weight stream
        if (lane == 0) {
            uint32_t q = 0;
            for (int64_t tile = blockIdx.x; tile < ntiles && !*abort_flag; tile += gridDim.x)
                for (int it = 0; it < n_apply && !*abort_flag; ++it)
                    for (int l = 0; l < 2; ++l)
                        for (int c = 0; c < 4; ++c, ++q) {
                            const uint32_t slot = q % RING, use = q / RING;
                            if (!mbar_wait(BAR_EMPTY + 8 * slot, (use & 1) ^ 1, abort_flag)) break;
                            mbar_expect_tx(BAR_FULL + 8 * slot, W_CHUNK_BYTES);
                            bulk_load(s0 + SM_RING + slot * W_CHUNK_BYTES,
                                      wp + (l == 0 ? PK_W2 : PK_W3) + c * W_CHUNK_BYTES, W_CHUNK_BYTES,
                                      BAR_FULL + 8 * slot);
                        }
            // drain: every issued copy has landed before the block exits
            const uint32_t issued = q;
            for (uint32_t r = issued > RING ? issued - RING : 0; r < issued; ++r)
                if (!mbar_wait_bounded(BAR_FULL + 8 * (r % RING), (r / RING) & 1)) *abort_flag = 1;
        }
    } else if (warp == 1) {
        // ---------------------------------------------------- MMA issue
        if (lane == 0) {
            const uint32_t ID256 = idesc_bf16(TC_M, H), ID16 = idesc_bf16(TC_M, 16);
            const uint32_t D0 = tmem, D1 = tmem + 256;
            uint32_t q = 0, nx = 0, na = 0;
            bool ok = true;
            for (int64_t tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x)
                for (int it = 0; it < n_apply && ok; ++it) {
                    // layer 1: X (128 x 16) x W1^T -> D0
                    ok = mbar_wait(BAR_X, nx++ & 1, abort_flag);
                    if (!ok) break;
                    tc_after_sync();
                    umma(D0, sdesc(s0 + SM_X, 128, 256, 0), sdesc(s0 + SM_W1, 128, 256, 0), ID256, 0);
                    umma_commit(BAR_D);
                    // layers 2, 3: A (128 x 256) x W^T (streamed) -> D1, D0
                    for (int l = 0; l < 2 && ok; ++l) {
                        const uint32_t D = l == 0 ? D1 : D0;
                        for (int c = 0; c < 4; ++c, ++q) {
                            const uint32_t slot = q % RING, use = q / RING;
                            ok = mbar_wait(BAR_A + 8 * c, na & 1, abort_flag) &&
                                 mbar_wait(BAR_FULL + 8 * slot, use & 1, abort_flag);
                            if (!ok) break;
                            tc_after_sync();
                            const uint32_t a0 = s0 + SM_A + c * A_CHUNK_BYTES;
                            const uint32_t b0 = s0 + SM_RING + slot * W_CHUNK_BYTES;
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk)
                                umma(D, sdesc(a0 + 32 * kk, 16, 1024, 2), sdesc(b0 + 32 * kk, 16, 1024, 2), ID256,
                                     (c | kk) != 0);
                            umma_commit(BAR_EMPTY + 8 * slot);
                        }
                        ++na;
                        if (ok) umma_commit(BAR_D);
                    }
                    if (!ok) break;
                    // layer 4: A (128 x 256) x W4^T (16 x 256, resident) -> D1 columns 0..15
                    for (int c = 0; c < 4; ++c) {
                        ok = mbar_wait(BAR_A + 8 * c, na & 1, abort_flag);
                        if (!ok) break;
                        tc_after_sync();
                        const uint32_t a0 = s0 + SM_A + c * A_CHUNK_BYTES;
                        const uint32_t b0 = s0 + SM_W4 + c * W4_CHUNK_BYTES;
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
                            umma(D1, sdesc(a0 + 32 * kk, 16, 1024, 2), sdesc(b0 + 32 * kk, 16, 1024, 2), ID16,
                                 (c | kk) != 0);
                    }
                    ++na;
                    if (ok) umma_commit(BAR_D);
                }
            // drain: every MMA issued has completed before tensor memory is freed
            umma_commit(BAR_DRAIN);
            if (!mbar_wait_bounded(BAR_DRAIN, 0)) *abort_flag = 1;
        }
    } else {
        // ---------------------------------------------------- epilogue
        // warps 2..17: tensor-memory lane quarter warp % 4, column quarter
        // (warp - 2) / 4 of every 64-column chunk; the quarter-0 thread of a
        // row owns that state
        const int quarter = warp & 3;
        const int half = (warp - 2) >> 2;          // column quarter 0..3
        const int row = quarter * 32 + lane;
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16) + 16 * half;
        uint32_t nd = 0;
        bool ok = true;
        for (int64_t tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
            const int64_t p = tile * TC_M + row;
            float x[NOUT];
            if (p < n) {
                const float4 u = reinterpret_cast<const float4 *>(state)[2 * p];
                const float4 w = reinterpret_cast<const float4 *>(state)[2 * p + 1];
                x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w; x[4] = w.x; x[5] = w.y; x[6] = w.z; x[7] = w.w;
            } else {
#pragma unroll
                for (int i = 0; i < NOUT; ++i) x[i] = 0.0f;
            }
            bool act = p < n;
            int cnt = 0;
            for (int it = 0; it < n_apply && ok; ++it) {
                if (half == 0) {
                    if (radius2 > 0.0f)
                        act = act && (x[0] * x[0] + x[1] * x[1] <= radius2) &&
                              (x[2] * x[2] + x[3] * x[3] <= radius2) && (fabsf(x[4]) <= 1.0f);
                    // layer-1 input row: s0..s5 split into bfloat16 high and low
                    // parts (columns 0..5 and 6..11; W1 is stacked twice), so
                    // the product sees the float32 state, zero padding to 16
                    float xl[6];
#pragma unroll
                    for (int k = 0; k < 6; ++k) xl[k] = x[k] - __bfloat162float(__float2bfloat16_rn(x[k]));
                    uint4 lo, hi;
                    lo.x = pack_bf16(x[0], x[1]);
                    lo.y = pack_bf16(x[2], x[3]);
                    lo.z = pack_bf16(x[4], x[5]);
                    lo.w = pack_bf16(xl[0], xl[1]);
                    hi.x = pack_bf16(xl[2], xl[3]);
                    hi.y = pack_bf16(xl[4], xl[5]);
                    hi.z = 0u;
                    hi.w = 0u;
                    *reinterpret_cast<uint4 *>(sm + SM_X + core_off(row, 0)) = lo;
                    *reinterpret_cast<uint4 *>(sm + SM_X + core_off(row, 8)) = hi;
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(BAR_X);
                }
                // hidden layers: D0 (layer 1), D1 (layer 2), D0 (layer 3)
                for (int l = 0; l < 3 && ok; ++l) {
                    ok = __all_sync(0xffffffffu, mbar_wait(BAR_D, nd++ & 1, abort_flag));
                    if (!ok) break;
                    tc_after_sync();
                    const uint32_t src = lane_base + ((l == 1) ? 256u : 0u);
                    const float *hb = sbias + l * H + 16 * half;
                    unsigned char *arow = sm + SM_A + row * 128;
                    uint32_t va[16], vb[16];
                    TMEM_LD16(src, va);
                    tmem_wait_ld();
                    REG_FENCE16(va);
                    // chunk c is converted while chunk c + 1 is in flight
#define EPI_CHUNK(c, cur, nxt)                                                                           \
    {                                                                                                    \
        if ((c) < 3) TMEM_LD16(src + ((c) + 1) * TC_CHUNK, nxt);                                         \
        _Pragma("unroll") for (int j = 0; j < 2; ++j)                                                    \
        {                                                                                                \
            const uint4 o = silu8(cur + 8 * j, hb + (c) * TC_CHUNK + 8 * j);                            \
            *reinterpret_cast<uint4 *>(arow + (c) * A_CHUNK_BYTES + (((2 * half + j) ^ (row & 7)) << 4)) = o; \
        }                                                                                                \
        fence_async_smem();                                                                              \
        if ((c) < 3) {                                                                                   \
            tmem_wait_ld();                                                                              \
            REG_FENCE16(nxt);                                                                            \
        }                                                                                                \
        tc_before_sync();                                                                                \
        __syncwarp();                                                                                    \
        if (lane == 0) mbar_arrive(BAR_A + 8 * (c));                                                     \
    }
                    EPI_CHUNK(0, va, vb)
                    EPI_CHUNK(1, vb, va)
                    EPI_CHUNK(2, va, vb)
                    EPI_CHUNK(3, vb, va)
#undef EPI_CHUNK
                }
                if (!ok) break;
                // layer 4 and the residual update
                ok = __all_sync(0xffffffffu, mbar_wait(BAR_D, nd++ & 1, abort_flag));
                if (!ok) break;
                if (half == 0) {
                    tc_after_sync();
                    uint32_t f[16];
                    TMEM_LD16(lane_base + 256, f);
                    tmem_wait_ld();
                    REG_FENCE16(f);
                    tc_before_sync();
                    if (act) {
                        float y[4], q[15];
                        quad_features(x, q);
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            float lin = stail[72 + c];
#pragma unroll
                            for (int k = 0; k < 6; ++k) lin = fmaf(x[k], stail[8 + k * NOUT + c], lin);
#pragma unroll
                            for (int m = 0; m < 15; ++m) lin = fmaf(q[m], stail[80 + m * NOUT + c], lin);
                            y[c] = x[c] + (lin + (__uint_as_float(f[c]) + stail[c]));
                        }
#pragma unroll
                        for (int c = 0; c < 4; ++c) x[c] = y[c];
                        ++cnt;
                    }
                }
            }
            if (half == 0 && p < n && ok) {
                reinterpret_cast<float4 *>(state)[2 * p] = make_float4(x[0], x[1], x[2], x[3]);
                reinterpret_cast<float4 *>(state)[2 * p + 1] = make_float4(x[4], x[5], x[6], x[7]);
                if (applied) applied[p] = cnt;
            }
        }
    }
    // teardown: the MMA thread has drained its MMAs, the epilogue its loads
    tc_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
    }
    if (threadIdx.x == 0 && *abort_flag && error) atomicExch(error, 1);
}

// ------------------------------------------------ paired-tile inference
// Two 128-state tiles per CTA in flight (slots 0 and 1), each with one
// 256-column accumulator (D_s = tensor-memory columns 256 s .. 256 s + 255),
// its own activation operand A_s and layer-1 input X_s in shared memory.
// The epilogue warps alternate between the slots layer by layer,
//   E(0, l)  E(1, l)  E(0, l + 1)  E(1, l + 1) ...
// and the MMA thread issues in the same order, so the tensor cores run one
// slot's layer while the epilogue converts the other slot's.  The MMAs of a
// slot's next layer overwrite its accumulator: they wait for d_free[s], which
// the epilogue warps signal once their last tensor-memory load of D_s has
// completed (before the last chunk is converted), besides the A_s chunks.
// W2 / W3 stream through a ring of two 32 KB slots, once per slot and layer.
// A CTA's tiles are t, t + G (a pair), t + 2G, t + 3G, ... (G = grid size);
// an unpaired last tile runs in slot 0 alone.
constexpr int RING2 = 2;
constexpr uint32_t S2_A = 0;                                   // A_0, A_1: 64 KB each
constexpr uint32_t S2_RING = S2_A + 2 * 4 * A_CHUNK_BYTES;
constexpr uint32_t S2_W4 = S2_RING + RING2 * W_CHUNK_BYTES;
constexpr uint32_t S2_W1 = S2_W4 + 4 * W4_CHUNK_BYTES;
constexpr uint32_t S2_X = S2_W1 + H * KIN * 2;                 // X_0, X_1: 4 KB each
constexpr uint32_t S2_XB = TC_M * KIN * 2;
constexpr uint32_t S2_BIAS = S2_X + 2 * S2_XB;
constexpr uint32_t S2_TAIL = S2_BIAS + 3 * H * 4;
constexpr uint32_t S2_BAR = S2_TAIL + 208 * 4;
// x_ready[2], a_ready[2][4], d_full[2], d_free[2], full[RING2], empty[RING2], drain
constexpr int NBAR2 = 2 + 8 + 2 + 2 + 2 * RING2 + 1;
constexpr uint32_t S2_MISC = S2_BAR + NBAR2 * 8;
constexpr uint32_t S2_TOTAL = S2_MISC + 16;
constexpr size_t TC2_SMEM = S2_TOTAL + 1024;
static_assert(TC2_SMEM <= 232448, "paired inference: shared memory per block");

__global__ void __launch_bounds__(TC_THREADS, 1)
    mlp_infer_tc2_kernel(const float *__restrict__ P, const unsigned char *__restrict__ wp, float *__restrict__ state,
                         int32_t *__restrict__ applied, int32_t *__restrict__ error, int64_t n, int n_apply,
                         float radius2)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char *sm = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t s0 = smem_u32(sm);
    float *sbias = reinterpret_cast<float *>(sm + S2_BIAS);
    float *stail = reinterpret_cast<float *>(sm + S2_TAIL);   // b4[0..7], Ws[8..71], bs[72..79], Wq[80..207]
    const uint32_t bar0 = s0 + S2_BAR;
    const uint32_t BAR_X = bar0, BAR_A = bar0 + 16, BAR_D = bar0 + 80, BAR_F = bar0 + 96, BAR_FULL = bar0 + 112,
                   BAR_EMPTY = BAR_FULL + 8 * RING2, BAR_DRAIN = BAR_EMPTY + 8 * RING2;
    uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(sm + S2_MISC);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(sm + S2_MISC + 4);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t ntiles = (n + TC_M - 1) / TC_M, G = gridDim.x;

    for (int i = threadIdx.x; i < (int)(H * KIN * 2 / 16); i += blockDim.x)
        reinterpret_cast<uint4 *>(sm + S2_W1)[i] = reinterpret_cast<const uint4 *>(wp + PK_W1)[i];
    for (int i = threadIdx.x; i < (int)(4 * W4_CHUNK_BYTES / 16); i += blockDim.x)
        reinterpret_cast<uint4 *>(sm + S2_W4)[i] = reinterpret_cast<const uint4 *>(wp + PK_W4)[i];
    for (int i = threadIdx.x; i < 3 * H; i += blockDim.x) sbias[i] = 0.5f * P[(i < H ? P_B1 : i < 2 * H ? P_B2 : P_B3) + (i % H)];
    for (int i = threadIdx.x; i < 208; i += blockDim.x)
        stail[i] = i < 8 ? P[P_B4 + i] : i < 72 ? P[P_WS + (i - 8)] : i < 80 ? P[P_BS + (i - 72)] : P[P_WQ + (i - 80)];
    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(BAR_X + 8 * s, 4);
            for (int c = 0; c < 4; ++c) mbar_init(BAR_A + 8 * (4 * s + c), 16);
            mbar_init(BAR_D + 8 * s, 1);
            mbar_init(BAR_F + 8 * s, 16);
        }
        for (int r = 0; r < RING2; ++r) {
            mbar_init(BAR_FULL + 8 * r, 1);
            mbar_init(BAR_EMPTY + 8 * r, 1);
        }
        mbar_init(BAR_DRAIN, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)),
                     "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_async_smem();
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    const uint32_t tmem = *tmem_holder;

    if (warp == 0) {
        // ---------------------------------------------------- weight stream
        // consumption order of the MMA thread: per map, W2 for slot 0, W2 for
        // slot 1, W3 for slot 0, W3 for slot 1, four chunks each
        if (lane == 0) {
            uint32_t q = 0;
            for (int64_t t0 = blockIdx.x; t0 < ntiles && !*abort_flag; t0 += 2 * G) {
                const int ns = t0 + G < ntiles ? 2 : 1;
                for (int it = 0; it < n_apply && !*abort_flag; ++it)
                    for (int l = 0; l < 2; ++l)
                        for (int s = 0; s < ns; ++s)
                            for (int c = 0; c < 4; ++c, ++q) {
                                const uint32_t slot = q % RING2, use = q / RING2;
                                if (!mbar_wait(BAR_EMPTY + 8 * slot, (use & 1) ^ 1, abort_flag)) break;
                                mbar_expect_tx(BAR_FULL + 8 * slot, W_CHUNK_BYTES);
                                bulk_load(s0 + S2_RING + slot * W_CHUNK_BYTES,
                                          wp + (l == 0 ? PK_W2 : PK_W3) + c * W_CHUNK_BYTES, W_CHUNK_BYTES,
                                          BAR_FULL + 8 * slot);
                            }
            }
            // drain: every issued copy has landed before the block exits
            const uint32_t issued = q;
            for (uint32_t r = issued > RING2 ? issued - RING2 : 0; r < issued; ++r)
                if (!mbar_wait_bounded(BAR_FULL + 8 * (r % RING2), (r / RING2) & 1)) *abort_flag = 1;
        }
    } else if (warp == 1) {
        // ---------------------------------------------------- MMA issue
        if (lane == 0) {
            const uint32_t ID256 = idesc_bf16(TC_M, H), ID16 = idesc_bf16(TC_M, 16);
            uint32_t q = 0, nx[2] = {0, 0}, na[2] = {0, 0}, nb[2] = {0, 0};
            bool ok = true;
            for (int64_t t0 = blockIdx.x; t0 < ntiles && ok; t0 += 2 * G) {
                const int ns = t0 + G < ntiles ? 2 : 1;
                for (int it = 0; it < n_apply && ok; ++it)
                    for (int layer = 0; layer < 4 && ok; ++layer)
                        for (int s = 0; s < ns && ok; ++s) {
                            const uint32_t D = tmem + 256 * s;
                            // the accumulator's previous contents have been read
                            if (nb[s] > 0) ok = mbar_wait(BAR_F + 8 * s, (nb[s] - 1) & 1, abort_flag);
                            ++nb[s];
                            if (!ok) break;
                            if (layer == 0) {
                                // layer 1: X_s (128 x 16) x W1^T -> D_s
                                ok = mbar_wait(BAR_X + 8 * s, nx[s]++ & 1, abort_flag);
                                if (!ok) break;
                                tc_after_sync();
                                umma(D, sdesc(s0 + S2_X + s * S2_XB, 128, 256, 0), sdesc(s0 + S2_W1, 128, 256, 0), ID256, 0);
                            } else if (layer < 3) {
                                // layers 2, 3: A_s (128 x 256) x W^T (streamed) -> D_s
                                for (int c = 0; c < 4; ++c, ++q) {
                                    const uint32_t slot = q % RING2, use = q / RING2;
                                    ok = mbar_wait(BAR_A + 8 * (4 * s + c), na[s] & 1, abort_flag) &&
                                         mbar_wait(BAR_FULL + 8 * slot, use & 1, abort_flag);
                                    if (!ok) break;
                                    tc_after_sync();
                                    const uint32_t a0 = s0 + S2_A + (4 * s + c) * A_CHUNK_BYTES;
                                    const uint32_t b0 = s0 + S2_RING + slot * W_CHUNK_BYTES;
#pragma unroll
                                    for (int kk = 0; kk < 4; ++kk)
                                        umma(D, sdesc(a0 + 32 * kk, 16, 1024, 2), sdesc(b0 + 32 * kk, 16, 1024, 2),
                                             ID256, (c | kk) != 0);
                                    umma_commit(BAR_EMPTY + 8 * slot);
                                }
                                ++na[s];
                            } else {
                                // layer 4: A_s x W4^T (16 x 256, resident) -> D_s columns 0..15
                                for (int c = 0; c < 4; ++c) {
                                    ok = mbar_wait(BAR_A + 8 * (4 * s + c), na[s] & 1, abort_flag);
                                    if (!ok) break;
                                    tc_after_sync();
                                    const uint32_t a0 = s0 + S2_A + (4 * s + c) * A_CHUNK_BYTES;
                                    const uint32_t b0 = s0 + S2_W4 + c * W4_CHUNK_BYTES;
#pragma unroll
                                    for (int kk = 0; kk < 4; ++kk)
                                        umma(D, sdesc(a0 + 32 * kk, 16, 1024, 2), sdesc(b0 + 32 * kk, 16, 1024, 2),
                                             ID16, (c | kk) != 0);
                                }
                                ++na[s];
                            }
                            if (ok) umma_commit(BAR_D + 8 * s);
                        }
            }
            // drain: every MMA issued has completed before tensor memory is freed
            umma_commit(BAR_DRAIN);
            if (!mbar_wait_bounded(BAR_DRAIN, 0)) *abort_flag = 1;
        }
    } else {
        // ---------------------------------------------------- epilogue
        // warps 2..17: tensor-memory lane quarter warp % 4, column quarter
        // (warp - 2) / 4 of every 64-column chunk; the quarter-0 thread of a
        // row owns that row's state in both slots
        const int quarter = warp & 3;
        const int half = (warp - 2) >> 2;          // column quarter 0..3
        const int row = quarter * 32 + lane;
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16) + 16 * half;
        uint32_t nd[2] = {0, 0};
        bool ok = true;
        // layer-1 input row of slot s (quarter-0 threads): the domain test, then
        // s0..s5 split into bfloat16 high and low parts (columns 0..5 and 6..11;
        // W1 is stacked twice), zero padding to 16
        auto write_x = [&](const float *x, bool &act, int s) {
            if (radius2 > 0.0f)
                act = act && (x[0] * x[0] + x[1] * x[1] <= radius2) && (x[2] * x[2] + x[3] * x[3] <= radius2) &&
                      (fabsf(x[4]) <= 1.0f);
            float xl[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) xl[k] = x[k] - __bfloat162float(__float2bfloat16_rn(x[k]));
            uint4 lo, hi;
            lo.x = pack_bf16(x[0], x[1]);
            lo.y = pack_bf16(x[2], x[3]);
            lo.z = pack_bf16(x[4], x[5]);
            lo.w = pack_bf16(xl[0], xl[1]);
            hi.x = pack_bf16(xl[2], xl[3]);
            hi.y = pack_bf16(xl[4], xl[5]);
            hi.z = 0u;
            hi.w = 0u;
            unsigned char *xb = sm + S2_X + s * S2_XB;
            *reinterpret_cast<uint4 *>(xb + core_off(row, 0)) = lo;
            *reinterpret_cast<uint4 *>(xb + core_off(row, 8)) = hi;
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(BAR_X + 8 * s);
        };
        // layer 4 of slot s: the fitted outputs, the float32 skip connection
        auto update = [&](float *x, bool act, int &cnt, const uint32_t *f) {
            if (!act) return;
            float y[4], q[15];
            quad_features(x, q);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                float lin = stail[72 + c];
#pragma unroll
                for (int k = 0; k < 6; ++k) lin = fmaf(x[k], stail[8 + k * NOUT + c], lin);
#pragma unroll
                for (int m = 0; m < 15; ++m) lin = fmaf(q[m], stail[80 + m * NOUT + c], lin);
                y[c] = x[c] + (lin + (__uint_as_float(f[c]) + stail[c]));
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) x[c] = y[c];
            ++cnt;
        };
        for (int64_t t0 = blockIdx.x; t0 < ntiles && ok; t0 += 2 * G) {
            const int ns = t0 + G < ntiles ? 2 : 1;
            const int64_t p0 = t0 * TC_M + row, p1 = (t0 + G) * TC_M + row;
            float x0[NOUT], x1[NOUT];
            bool act0 = p0 < n, act1 = ns == 2 && p1 < n;
            int cnt0 = 0, cnt1 = 0;
            if (half == 0) {
#pragma unroll
                for (int i = 0; i < NOUT; ++i) x0[i] = x1[i] = 0.0f;
                if (act0) {
                    const float4 u = reinterpret_cast<const float4 *>(state)[2 * p0];
                    const float4 w = reinterpret_cast<const float4 *>(state)[2 * p0 + 1];
                    x0[0] = u.x; x0[1] = u.y; x0[2] = u.z; x0[3] = u.w; x0[4] = w.x; x0[5] = w.y; x0[6] = w.z; x0[7] = w.w;
                }
                if (act1) {
                    const float4 u = reinterpret_cast<const float4 *>(state)[2 * p1];
                    const float4 w = reinterpret_cast<const float4 *>(state)[2 * p1 + 1];
                    x1[0] = u.x; x1[1] = u.y; x1[2] = u.z; x1[3] = u.w; x1[4] = w.x; x1[5] = w.y; x1[6] = w.z; x1[7] = w.w;
                }
                write_x(x0, act0, 0);
                if (ns == 2) write_x(x1, act1, 1);
            }
            for (int it = 0; it < n_apply && ok; ++it) {
                // hidden layers 1..3 of slot 0, then slot 1
                for (int l = 0; l < 3 && ok; ++l)
                    for (int s = 0; s < ns && ok; ++s) {
                        ok = __all_sync(0xffffffffu, mbar_wait(BAR_D + 8 * s, nd[s]++ & 1, abort_flag));
                        if (!ok) break;
                        tc_after_sync();
                        const uint32_t src = lane_base + 256u * s;
                        const float *hb = sbias + l * H + 16 * half;
                        unsigned char *arow = sm + S2_A + s * (4 * A_CHUNK_BYTES) + row * 128;
                        const uint32_t bar_a = BAR_A + 8 * (4 * s), bar_f = BAR_F + 8 * s;
                        uint32_t va[16], vb[16];
                        TMEM_LD16(src, va);
                        tmem_wait_ld();
                        REG_FENCE16(va);
                        // chunk c is converted while chunk c + 1 is in flight; once
                        // chunk 3 has landed, D_s is free for the next layer's MMAs
#define EPI2_CHUNK(c, cur, nxt)                                                                          \
    {                                                                                                    \
        if ((c) < 3) TMEM_LD16(src + ((c) + 1) * TC_CHUNK, nxt);                                         \
        _Pragma("unroll") for (int j = 0; j < 2; ++j)                                                    \
        {                                                                                                \
            const uint4 o = silu8(cur + 8 * j, hb + (c) * TC_CHUNK + 8 * j);                            \
            *reinterpret_cast<uint4 *>(arow + (c) * A_CHUNK_BYTES + (((2 * half + j) ^ (row & 7)) << 4)) = o; \
        }                                                                                                \
        fence_async_smem();                                                                              \
        if ((c) < 3) {                                                                                   \
            tmem_wait_ld();                                                                              \
            REG_FENCE16(nxt);                                                                            \
        }                                                                                                \
        tc_before_sync();                                                                                \
        __syncwarp();                                                                                    \
        if (lane == 0) {                                                                                 \
            mbar_arrive(bar_a + 8 * (c));                                                                \
            if ((c) == 2) mbar_arrive(bar_f);                                                            \
        }                                                                                                \
    }
                        EPI2_CHUNK(0, va, vb)
                        EPI2_CHUNK(1, vb, va)
                        EPI2_CHUNK(2, va, vb)
                        EPI2_CHUNK(3, vb, va)
#undef EPI2_CHUNK
                    }
                if (!ok) break;
                // layer 4 and the residual update per slot, then that slot's
                // layer-1 input of the next map
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    if (s >= ns || !ok) break;
                    ok = __all_sync(0xffffffffu, mbar_wait(BAR_D + 8 * s, nd[s]++ & 1, abort_flag));
                    if (!ok) break;
                    uint32_t f[16];
                    if (half == 0) {
                        tc_after_sync();
                        TMEM_LD16(lane_base + 256u * s, f);
                        tmem_wait_ld();
                        REG_FENCE16(f);
                    }
                    tc_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(BAR_F + 8 * s);
                    if (half == 0) {
                        if (s == 0) {
                            update(x0, act0, cnt0, f);
                            if (it + 1 < n_apply) write_x(x0, act0, 0);
                        } else {
                            update(x1, act1, cnt1, f);
                            if (it + 1 < n_apply) write_x(x1, act1, 1);
                        }
                    }
                }
            }
            if (half == 0 && ok) {
                if (p0 < n) {
                    reinterpret_cast<float4 *>(state)[2 * p0] = make_float4(x0[0], x0[1], x0[2], x0[3]);
                    reinterpret_cast<float4 *>(state)[2 * p0 + 1] = make_float4(x0[4], x0[5], x0[6], x0[7]);
                    if (applied) applied[p0] = cnt0;
                }
                if (ns == 2 && p1 < n) {
                    reinterpret_cast<float4 *>(state)[2 * p1] = make_float4(x1[0], x1[1], x1[2], x1[3]);
                    reinterpret_cast<float4 *>(state)[2 * p1 + 1] = make_float4(x1[4], x1[5], x1[6], x1[7]);
                    if (applied) applied[p1] = cnt1;
                }
            }
        }
    }
    // teardown: the MMA thread has drained its MMAs, the epilogue its loads
    tc_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
    }
    if (threadIdx.x == 0 && *abort_flag && error) atomicExch(error, 1);
}

// ------------------------------------------------------------ GEMM, tcgen05
// Products of at least 128 x 128 x 64 on the 5th-generation tensor cores:
// C[M][N] = op(A) op(B) (+ bias) with the operands and the meaning of transA /
// transB of gemm_tc.  One CTA of sixteen warps per 128 x 128 output tile; K is
// staged 64 at a time: every thread loads its 16 + 16 float32 of the step
// from global memory along the index that is contiguous there (into
// registers, one step ahead), rounds to bfloat16 (as gemm_tc does) and
// stores into a 128-byte-swizzled K-major tile (A: 128 m-rows, B: 128
// n-rows, 128 bytes of k each), two stages; one thread issues the four
// K = 16 MMAs of a stage into a 128-column TMEM accumulator and commits them
// to that stage's mbarrier, which frees the stage for the store two steps
// later.  Epilogue: warp w reads TMEM lanes 32 (w % 4) .. + 31 (its 32 output
// rows) and 32 columns, adds the bias and stores float32.  Waits are
// bounded: on a timeout the tile is written as NaN and g_gemm_timeouts is
// counted.
constexpr int G5_BM = 128, G5_BN = 128, G5_BK = 64, G5_STAGES = 2, G5_THREADS = 512;
constexpr uint32_t G5_TILE = 128 * 128;                               // one operand stage: 16 KB
constexpr uint32_t G5_SM_A = 0;
constexpr uint32_t G5_SM_B = G5_SM_A + G5_STAGES * G5_TILE;
constexpr uint32_t G5_SM_BAR = G5_SM_B + G5_STAGES * G5_TILE;        // one mbarrier per stage
constexpr uint32_t G5_SM_MISC = G5_SM_BAR + 8 * G5_STAGES;            // tmem base, abort flag
constexpr size_t G5_SMEM = G5_SM_MISC + 16 + 1024;                    // + alignment slack
constexpr uint32_t G5_TMEM_COLS = 128;
constexpr int G5_PER = G5_BM * G5_BK / G5_THREADS;                    // floats per thread per operand: 16
static_assert(G5_PER == 16, "staging split");

__device__ int g_gemm_timeouts;

// This thread's share of rows [r0, r0 + 128) x k [k0, k0 + 64) of op(X)
// (X[r ld + k] when kcont, else X[k ld + r]) into registers; rows >= nrows
// and k >= kend read as 0.  kcont: 8 threads per row, two runs of 8
// consecutive k each (a row's 256 bytes over 8 lanes); otherwise one row per
// thread and 16 consecutive k (every load 32 consecutive rows of one k).
__device__ __forceinline__ void g5_load(float v[G5_PER], const float *__restrict__ X, int ld, bool kcont, bool vec,
                                        int r0, int nrows, int k0, int kend)
{
    const int t = threadIdx.x;
    if (kcont) {
#pragma unroll
        for (int it = 0; it < 2; ++it) {
            const int id = t + G5_THREADS * it;
            const int gr = r0 + (id >> 3), gk = k0 + 8 * (id & 7);
            if (gr < nrows && vec && gk + 8 <= kend) {
                const float4 *src = reinterpret_cast<const float4 *>(X + (int64_t)gr * ld + gk);
                const float4 a = __ldg(src), b = __ldg(src + 1);
                v[8 * it + 0] = a.x; v[8 * it + 1] = a.y; v[8 * it + 2] = a.z; v[8 * it + 3] = a.w;
                v[8 * it + 4] = b.x; v[8 * it + 5] = b.y; v[8 * it + 6] = b.z; v[8 * it + 7] = b.w;
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    v[8 * it + j] = (gr < nrows && gk + j < kend) ? __ldg(X + (int64_t)gr * ld + gk + j) : 0.0f;
            }
        }
    } else {
        const int gr = r0 + (t & 127), kq = k0 + 16 * (t >> 7);
        const bool rok = gr < nrows;
#pragma unroll
        for (int j = 0; j < G5_PER; ++j) v[j] = (rok && kq + j < kend) ? __ldg(X + (int64_t)(kq + j) * ld + gr) : 0.0f;
    }
}

// the registers of g5_load as bfloat16 into a 128-byte-swizzled K-major stage
__device__ __forceinline__ void g5_store(unsigned char *dst, const float v[G5_PER], bool kcont)
{
    const int t = threadIdx.x;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        int row, c;
        if (kcont) {
            const int id = t + G5_THREADS * h;
            row = id >> 3;
            c = id & 7;
        } else {
            row = t & 127;
            c = 2 * (t >> 7) + h;
        }
        *reinterpret_cast<uint4 *>(dst + row * 128 + ((c ^ (row & 7)) << 4)) =
            make_uint4(pack_bf16(v[8 * h], v[8 * h + 1]), pack_bf16(v[8 * h + 2], v[8 * h + 3]),
                       pack_bf16(v[8 * h + 4], v[8 * h + 5]), pack_bf16(v[8 * h + 6], v[8 * h + 7]));
    }
}

__global__ void __launch_bounds__(G5_THREADS) gemm_tc05(const float *__restrict__ A, int lda, int transA,
                                                        const float *__restrict__ B, int ldb, int transB,
                                                        float *__restrict__ C, int ldc, int M, int N, int K,
                                                        const float *__restrict__ bias, int vecA, int vecB)
{
    extern __shared__ unsigned char g5_raw[];
    unsigned char *sm = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(g5_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t s0 = smem_u32(sm);
    uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(sm + G5_SM_MISC);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(sm + G5_SM_MISC + 4);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.y * G5_BM, n0 = blockIdx.x * G5_BN;
    const int kb = 0, ke = K;
    if (threadIdx.x == 0) {
        for (int s = 0; s < G5_STAGES; ++s) mbar_init(s0 + G5_SM_BAR + 8 * s, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)),
                     "r"(G5_TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    const int nk = ke > kb ? (ke - kb + G5_BK - 1) / G5_BK : 0;
    const bool kcA = !transA, kcB = transB != 0;
    float va[G5_PER], vb[G5_PER];
    if (nk > 0) {                                  // the first K step's loads overlap the set-up barrier
        g5_load(va, A, lda, kcA, vecA != 0, m0, M, kb, ke);
        g5_load(vb, B, ldb, kcB, vecB != 0, n0, N, kb, ke);
    }
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    const uint32_t tmem = *tmem_holder;
    constexpr uint32_t IDESC = idesc_bf16(G5_BM, G5_BN);
    int issued = 0;                                // commits made (thread 0)
    for (int kt = 0; kt < nk; ++kt) {
        const int s = kt % G5_STAGES;
        const uint32_t bar = s0 + G5_SM_BAR + 8 * s;
        if (kt >= G5_STAGES) {
            // the MMAs that read this stage two steps ago have completed
            if (threadIdx.x == 0) mbar_wait(bar, ((kt / G5_STAGES) - 1) & 1, abort_flag);
            __syncthreads();
            if (*abort_flag) break;                // read by every thread after the barrier
        }
        g5_store(sm + G5_SM_A + s * G5_TILE, va, kcA);
        g5_store(sm + G5_SM_B + s * G5_TILE, vb, kcB);
        if (kt + 1 < nk) {                         // next K step in flight during the MMAs
            const int k1 = kb + (kt + 1) * G5_BK;
            g5_load(va, A, lda, kcA, vecA != 0, m0, M, k1, ke);
            g5_load(vb, B, ldb, kcB, vecB != 0, n0, N, k1, ke);
        }
        fence_async_smem();
        __syncthreads();
        if (threadIdx.x == 0) {
            tc_after_sync();
            const uint32_t a0 = s0 + G5_SM_A + s * G5_TILE, b0 = s0 + G5_SM_B + s * G5_TILE;
#pragma unroll
            for (int kk = 0; kk < G5_BK / 16; ++kk)
                umma(tmem, sdesc(a0 + 32 * kk, 16, 1024, 2), sdesc(b0 + 32 * kk, 16, 1024, 2), IDESC, (kt | kk) != 0);
            umma_commit(bar);
            ++issued;
        }
    }
    // the last commit covers every MMA of the tile
    if (threadIdx.x == 0 && issued > 0) {
        const int last = issued - 1;
        const uint32_t bar = s0 + G5_SM_BAR + 8 * (last % G5_STAGES);
        if (*abort_flag) mbar_wait_bounded(bar, (last / G5_STAGES) & 1);   // drain what is in flight
        else mbar_wait(bar, (last / G5_STAGES) & 1, abort_flag);
    }
    __syncthreads();
    tc_after_sync();
    const bool failed = *abort_flag != 0;
    // warp w: TMEM lanes 32 (w % 4) .. + 31 (its output rows), columns 32 (w / 4) .. + 31
    const int quarter = warp & 3, cg = warp >> 2;
    const int row = m0 + 32 * quarter + lane;
    const bool vecC = ((ldc & 3) == 0) && ((reinterpret_cast<uintptr_t>(C) & 15) == 0);
    uint32_t v[32];
    if (nk > 0 && !failed) {
        TMEM_LD32(tmem + ((uint32_t)(32 * quarter) << 16) + 32 * cg, v);
        tmem_wait_ld();
        REG_FENCE32(v);
    } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = failed ? 0x7FC00000u : 0u;
    }
    const int gn0 = n0 + 32 * cg;
    if (row < M && gn0 < N) {
        float *dst = C + (int64_t)row * ldc + gn0;
        if (vecC && gn0 + 32 <= N) {
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                float4 o = make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]), __uint_as_float(v[j + 2]),
                                       __uint_as_float(v[j + 3]));
                if (bias) {
                    o.x += bias[gn0 + j]; o.y += bias[gn0 + j + 1]; o.z += bias[gn0 + j + 2]; o.w += bias[gn0 + j + 3];
                }
                *reinterpret_cast<float4 *>(dst + j) = o;
            }
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
                if (gn0 + j < N) dst[j] = __uint_as_float(v[j]) + (bias ? bias[gn0 + j] : 0.0f);
        }
    }
    tc_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(G5_TMEM_COLS));
    }
    if (threadIdx.x == 0 && failed) atomicAdd(&g_gemm_timeouts, 1);
}

// -------------------------------------------------- training step (fused)
// One optimiser step in four launches (the plain sequence of products and
// element-wise passes took about 37 and spent its time between them: 254 us for
// 8192 samples against 5 us of tensor-core work):
//   train_pack_kernel   W2 / W3 rounded to bfloat16 as B operands, both ways
//                       round (forward and backward products)
//   train_tile_kernel   forward and backward of 64 samples per CTA without
//                       leaving the SM: activations and deltas as bfloat16 A
//                       operands in shared memory, the pre-activations z2, z3
//                       and the products in the two 256-column halves of tensor
//                       memory, z1 formed again from the input where the
//                       backward pass needs it.  A tile's 64 samples fill the
//                       128 rows of its products twice: a thread reaches only
//                       its own rows of tensor memory, so the copy lets eight
//                       threads instead of four share a sample's epilogues,
//                       which are the kernel's time (the doubled products
//                       are not)
//   train_wgrad_kernel  weight gradients over the batch: the tiles that the
//                       kernel above left in global memory are MN-major
//                       operands as they stand (K = the sample), split over
//                       CTAs
//   train_update_kernel sums of the splits in a fixed order, Adam
// The roundings are those of separate products on bfloat16 operands with
// float32 accumulation: h, delta, x, dd and W rounded where they enter a
// product, bias sums and the skip layer in float32 from unrounded deltas.
// 8192 samples: 254 -> 69 us a step (graph replay); the tile kernel is 28 us of it,
// bound by the latency of its epilogues (5 of them, SiLU and its derivative on
// 128 columns each way per thread), the products about 6 us.
constexpr int TT_THREADS = TC_THREADS;                          // weight stream, MMA, 16 epilogue warps
constexpr int TT_EPI = TT_THREADS - 64;                         // epilogue threads
constexpr int TS = 64;                                          // samples per tile
constexpr uint32_t TS_CHUNK = TS * 128;                         // 64 samples x 64 columns, bfloat16
constexpr int TT_IMG = 4 * (int)TS_CHUNK;                       // a tile in global memory: four swizzled chunks
constexpr int TT_SMALL = (int)TS_CHUNK;                         // 16 columns in one chunk (x, dd)
constexpr uint32_t T_A = 0;                                     // two activation buffers, 128 rows
constexpr uint32_t T_BUF = 4 * A_CHUNK_BYTES;
constexpr uint32_t T_RING = T_A + 2 * T_BUF;
constexpr uint32_t T_W1 = T_RING + 2 * W_CHUNK_BYTES;           // float [6][256], rounded to bfloat16
constexpr uint32_t T_W4 = T_W1 + 6 * H * 4;                     // float [256][8], rounded to bfloat16
constexpr uint32_t T_BIAS = T_W4 + H * NOUT * 4;                // b1, b2, b3
constexpr uint32_t T_F = T_BIAS + 3 * H * 4;                    // partial outputs [8][6][64], then skip features [22][64 + 1]
constexpr uint32_t T_SKIP = T_F + 8 * 6 * TS * 4;               // b4[8] Ws[64] bs[8] Wq[128]
constexpr uint32_t T_DD = T_SKIP + 208 * 4;                     // output gradients [6][64 + 1]
constexpr uint32_t T_BAR = T_DD + 6 * (TS + 1) * 4;             // a_ready[2][4], d_full, f_ready, full[2], empty[2], drain
constexpr uint32_t T_MISC = T_BAR + 15 * 8;
constexpr size_t TT_SMEM = T_MISC + 16 + 1024;
static_assert(TT_SMEM <= 232448, "training tile: shared memory per block");
static_assert(22 * (TS + 1) <= 8 * 6 * TS, "training tile: skip features");
static_assert(T_BAR % 8 == 0 && T_SKIP % 16 == 0, "training tile: alignment");

constexpr int SKIP_SUMS = 22 * 6;                               // skip-layer sums: x0..x5, the 15 products, 1, times dd
constexpr int TG_SPLITS = 16, TG_SMALL_SPLITS = 8;

// the step's scratch inside the caller's work area
struct TrainWork {
    int64_t T;                  // tiles
    int S, SS;                  // splits of the large and small weight gradients
    unsigned char *img;         // h1 h2 h3 dz1 dz2 dz3: [6][T] tiles
    unsigned char *small;       // x, dd: [2][T] small tiles
    unsigned char *wpk;         // W2, W3 forward, W2, W3 backward: 4 x 128 KB
    float *part;                // [2][S] partial gW2, gW3: [n / 4][k][4]
    float *part16;              // [2][SS] partial gW1, gW4: [16][256]
    float *bias;                // [3][2 T][256] sums of dz1, dz2, dz3
    float *skip;                // [T][SKIP_SUMS]
    double *loss;               // [2 T]
    int32_t *ticket;
    // FFA_MLP_STEP_FAILED from a block whose pipeline waits ran out until the
    // update has seen it: what that block did not write is another step's
    unsigned long long *failed;
};

__host__ __device__ inline unsigned char *tile_img(const TrainWork &w, int arr, int64_t t)
{
    return w.img + ((int64_t)arr * w.T + t) * TT_IMG;
}

__device__ __forceinline__ void train_gave_up(const TrainWork &w)
{
    *w.failed = FFA_MLP_STEP_FAILED;
    atomicAdd(&g_gemm_timeouts, 1);
}

__global__ void __launch_bounds__(256) train_pack_kernel(const float *__restrict__ P, TrainWork w)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;       // H * H / 4 threads
    if (t == 0) *w.ticket = 0;
    const int k = t / (H / 4), n = 4 * (t % (H / 4));
#pragma unroll
    for (int l = 0; l < 2; ++l) {
        const float *W = P + (l == 0 ? P_W2 : P_W3) + k * H + n;
        const float v[4] = {W[0], W[1], W[2], W[3]};
        unsigned char *f = w.wpk + l * 4 * W_CHUNK_BYTES, *b = w.wpk + (2 + l) * 4 * W_CHUNK_BYTES;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            *reinterpret_cast<__nv_bfloat16 *>(f + swz_off(n + i, k, H)) = __float2bfloat16_rn(v[i]);
        *reinterpret_cast<uint2 *>(b + swz_off(k, n, H)) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
    }
}

__device__ __forceinline__ void bulk_store(void *dst, uint32_t src, uint32_t bytes)
{
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// Sums over the warp's 32 rows of 8 columns: lane l ends with column l & 7.
// Each of the first three exchanges halves the columns a lane keeps: nine
// shuffles in all.
__device__ __forceinline__ float warp_colsum8(float (&v)[8])
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int s = 4; s >= 1; s >>= 1) {
        const bool up = (lane & s) != 0;
#pragma unroll
        for (int i = 0; i < s; ++i) {
            const float mine = up ? v[i + s] : v[i], theirs = up ? v[i] : v[i + s];
            v[i] = mine + __shfl_xor_sync(0xffffffffu, theirs, s);
        }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 8);
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 16);
}

__device__ __forceinline__ void tmem_load8(uint32_t addr, float (&v)[8])
{
    uint32_t u[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                 : "r"(addr));
    tmem_wait_ld();
    asm volatile("" : "+r"(u[0]), "+r"(u[1]), "+r"(u[2]), "+r"(u[3]), "+r"(u[4]), "+r"(u[5]), "+r"(u[6]), "+r"(u[7]));
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(u[j]);
}

__device__ __forceinline__ void tmem_load8x2(uint32_t a, uint32_t b, float (&v)[8], float (&y)[8])
{
    uint32_t u[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                 : "r"(a));
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
                 : "r"(b));
    tmem_wait_ld();
    REG_FENCE16(u);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        v[j] = __uint_as_float(u[j]);
        y[j] = __uint_as_float(u[8 + j]);
    }
}

__device__ __forceinline__ uint4 pack8(const float (&v)[8])
{
    return make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
}

__device__ __forceinline__ void load8(const float *p, float (&v)[8])       // 16-byte aligned
{
    const float4 a = reinterpret_cast<const float4 *>(p)[0], b = reinterpret_cast<const float4 *>(p)[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

// NO: outputs evaluated, 4 (n_fit <= 4) or 6.
// Of its threads only the weight stream waits for the kernel before
// (train_pack_kernel, whose packed weights it loads).  The others read what that
// kernel only reads and write what it does not touch; all that came before the
// step is complete, because train_pack_kernel is an ordinary launch.  If that one
// is ever chained too, every thread here has to wait.
template <int NO>
__global__ void __launch_bounds__(TT_THREADS, 1)
    train_tile_kernel(const float *__restrict__ P, const float *__restrict__ X, const float *__restrict__ Y, TrainWork w,
                      int64_t B, int n_fit)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char *sm = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t s0 = smem_u32(sm);
    float *sw1 = reinterpret_cast<float *>(sm + T_W1), *sw4 = reinterpret_cast<float *>(sm + T_W4);
    float *sbias = reinterpret_cast<float *>(sm + T_BIAS), *sf = reinterpret_cast<float *>(sm + T_F);
    float *stail = reinterpret_cast<float *>(sm + T_SKIP);      // b4[0..7], Ws[8..71], bs[72..79], Wq[80..207]
    float *sdd = reinterpret_cast<float *>(sm + T_DD);
    const uint32_t BAR_A = s0 + T_BAR, BAR_D = BAR_A + 64, BAR_FR = BAR_A + 72, BAR_FULL = BAR_A + 80,
                   BAR_EMPTY = BAR_A + 96, BAR_DRAIN = BAR_A + 112;
    uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(sm + T_MISC);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(sm + T_MISC + 4);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int c = 0; c < 8; ++c) mbar_init(BAR_A + 8 * c, 16);
        mbar_init(BAR_D, 1);
        mbar_init(BAR_FR, 16);
        for (int r = 0; r < 2; ++r) {
            mbar_init(BAR_FULL + 8 * r, 1);
            mbar_init(BAR_EMPTY + 8 * r, 1);
        }
        mbar_init(BAR_DRAIN, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = threadIdx.x; i < 6 * H; i += blockDim.x) sw1[i] = __bfloat162float(__float2bfloat16_rn(P[P_W1 + i]));
    for (int i = threadIdx.x; i < H * NOUT; i += blockDim.x) sw4[i] = __bfloat162float(__float2bfloat16_rn(P[P_W4 + i]));
    for (int i = threadIdx.x; i < 3 * H; i += blockDim.x) sbias[i] = P[(i < H ? P_B1 : i < 2 * H ? P_B2 : P_B3) + (i % H)];
    for (int i = threadIdx.x; i < 208; i += blockDim.x)
        stail[i] = i < 8 ? P[P_B4 + i] : i < 72 ? P[P_WS + (i - 8)] : i < 80 ? P[P_BS + (i - 72)] : P[P_WQ + (i - 80)];
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)),
                     "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    const uint32_t tmem = *tmem_holder;
    // products in order: h1 W2 -> D0 (z2), h2 W3 -> D1 (z3), dz3 W3^T -> D1, dz2 W2^T -> D1;
    // operand buffers: h1 0, h2 1, h3 0, dz3 1, dz2 0, dz1 1

    if (warp == 0) {
        // ---------------------------------------------------- weight stream
        if (lane == 0) {
            const int mat[4] = {0, 1, 3, 2};
            uint32_t q = 0;
            ffa::chain_wait();                                  // the packed weights
            for (int64_t t = blockIdx.x; t < w.T && !*abort_flag; t += gridDim.x)
                for (int l = 0; l < 4; ++l)
                    for (int c = 0; c < 4; ++c, ++q) {
                        const uint32_t slot = q & 1;
                        if (!mbar_wait(BAR_EMPTY + 8 * slot, ((q >> 1) & 1) ^ 1, abort_flag)) goto stream_end;
                        mbar_expect_tx(BAR_FULL + 8 * slot, W_CHUNK_BYTES);
                        bulk_load(s0 + T_RING + slot * W_CHUNK_BYTES, w.wpk + (4 * mat[l] + c) * W_CHUNK_BYTES,
                                  W_CHUNK_BYTES, BAR_FULL + 8 * slot);
                    }
        stream_end:
            // every issued copy has landed before the block exits
            for (uint32_t r = q > 2 ? q - 2 : 0; r < q; ++r)
                if (!mbar_wait_bounded(BAR_FULL + 8 * (r & 1), (r >> 1) & 1)) *abort_flag = 1;
        }
    } else if (warp == 1) {
        // ------------------------------------------- MMA issue, tile stores
        if (lane == 0) {
            constexpr uint32_t ID = idesc_bf16(TC_M, H);
            const int arr[6] = {0, 1, 2, 5, 4, 3};              // h1 h2 h3 dz3 dz2 dz1
            uint32_t q = 0, na[2] = {0, 0};
            bool ok = true;
            for (int64_t t = blockIdx.x; t < w.T && ok; t += gridDim.x)
                for (int l = 0; l < 6 && ok; ++l) {
                    // a buffer's barriers: its next writer waits for a d_full
                    // that is committed after this use, so they are never two
                    // phases ahead
                    const uint32_t a0 = s0 + T_A + (l & 1) * T_BUF, bar_a = BAR_A + 32 * (l & 1), ph = na[l & 1]++ & 1;
                    const bool product = l != 2 && l != 5;
                    const uint32_t D = tmem + (l == 0 ? 0u : 256u);
                    // the backward products overwrite the half that the
                    // epilogue reads up to its last chunk
                    if (l >= 3)
                        for (int c = 0; c < 4 && ok; ++c) ok = mbar_wait(bar_a + 8 * c, ph, abort_flag);
                    for (int c = 0; c < 4 && ok; ++c) {
                        ok = mbar_wait(bar_a + 8 * c, ph, abort_flag);
                        if (ok && product) ok = mbar_wait(BAR_FULL + 8 * (q & 1), (q >> 1) & 1, abort_flag);
                        if (!ok) break;
                        bulk_store(tile_img(w, arr[l], t) + c * TS_CHUNK, a0 + c * A_CHUNK_BYTES, TS_CHUNK);
                        if (product) {
                            tc_after_sync();
                            const uint32_t ac = a0 + c * A_CHUNK_BYTES, bc = s0 + T_RING + (q & 1) * W_CHUNK_BYTES;
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk)
                                umma(D, sdesc(ac + 32 * kk, 16, 1024, 2), sdesc(bc + 32 * kk, 16, 1024, 2), ID, (c | kk) != 0);
                            umma_commit(BAR_EMPTY + 8 * (q & 1));
                            ++q;
                        }
                    }
                    if (!ok) break;
                    bulk_commit();
                    // the stores have read a buffer before the d_full that lets
                    // its next writer go on
                    bulk_wait_read<0>();
                    if (product) umma_commit(BAR_D);
                }
            umma_commit(BAR_DRAIN);
            if (!mbar_wait_bounded(BAR_DRAIN, 0)) *abort_flag = 1;
            bulk_wait_all();
        }
    } else {
        // ---------------------------------------------------- epilogue
        // this thread: sample `smp` of the tile (row `row` of the products, and
        // its copy 64 rows on or back), columns 8 u .. 8 u + 7 of each chunk
        const int quarter = warp & 3, u = 2 * ((warp - 2) >> 2) + (quarter >> 1);
        const int row = quarter * 32 + lane, smp = row & (TS - 1), group = quarter & 1;
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16) + 8 * u;
        uint32_t nd = 0, nf = 0;
        bool ok = true;
        for (int64_t t = blockIdx.x; t < w.T && ok; t += gridDim.x) {
            const int64_t p = t * TS + smp;
            const bool in = p < B;
            float x[6], tg[NO];
#pragma unroll
            for (int k = 0; k < 6; ++k) x[k] = in ? X[p * NOUT + k] : 0.0f;
#pragma unroll
            for (int c = 0; c < NO; ++c) tg[c] = in ? Y[p * NOUT + c] : 0.0f;
            auto z1_of = [&](int c, float (&z)[8]) {            // layer 1: float32 x, bfloat16-rounded W1
                const int n0 = c * TC_CHUNK + 8 * u;
                load8(sbias + n0, z);
#pragma unroll
                for (int k = 0; k < 6; ++k) {
                    float wk[8];
                    load8(sw1 + k * H + n0, wk);
#pragma unroll
                    for (int j = 0; j < 8; ++j) z[j] = fmaf(x[k], wk[j], z[j]);
                }
            };
            auto put = [&](int buf, int c, const float (&v)[8]) {   // both copies of the sample's row
                const uint4 o = pack8(v);
                unsigned char *a = sm + T_A + buf * T_BUF + c * A_CHUNK_BYTES + smp * 128 + ((u ^ (smp & 7)) << 4);
                *reinterpret_cast<uint4 *>(a) = o;
                *reinterpret_cast<uint4 *>(a + TS * 128) = o;
                fence_async_smem();
                tc_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(BAR_A + 32 * buf + 8 * c);
            };
            auto wait_d = [&]() {
                ok = __all_sync(0xffffffffu, mbar_wait(BAR_D, nd++ & 1, abort_flag));
                if (ok) tc_after_sync();
                return ok;
            };
            auto bias_sum = [&](int l, int c, float (&v)[8]) {  // column sums of dz_(l + 1)
                const float s = warp_colsum8(v);
                if (lane < 8) w.bias[((int64_t)l * 2 * w.T + 2 * t + group) * H + c * TC_CHUNK + 8 * u + lane] = s;
            };
            float z[8], bz[8];
            // h1 -> buffer 0
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
                z1_of(c, z);
#pragma unroll
                for (int j = 0; j < 8; ++j) z[j] = silu(z[j]);
                put(0, c, z);
            }
            // h2 -> buffer 1
            if (!wait_d()) break;
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
                tmem_load8(lane_base + c * TC_CHUNK, z);
                load8(sbias + H + c * TC_CHUNK + 8 * u, bz);
#pragma unroll
                for (int j = 0; j < 8; ++j) z[j] = silu(z[j] + bz[j]);
                put(1, c, z);
            }
            // h3 -> buffer 0 (stored only), and this thread's share of h3 W4
            if (!wait_d()) break;
            float f[NO];
#pragma unroll
            for (int c = 0; c < NO; ++c) f[c] = 0.0f;
            auto w4_row = [&](int n, float (&v)[NO]) {
                const float4 wa = *reinterpret_cast<const float4 *>(sw4 + n * NOUT);
                v[0] = wa.x; v[1] = wa.y; v[2] = wa.z; v[3] = wa.w;
                if constexpr (NO > 4) {
                    const float2 wb = *reinterpret_cast<const float2 *>(sw4 + n * NOUT + 4);
                    v[4] = wb.x; v[5] = wb.y;
                }
            };
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
                tmem_load8(lane_base + 256 + c * TC_CHUNK, z);
                load8(sbias + 2 * H + c * TC_CHUNK + 8 * u, bz);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    z[j] = silu(z[j] + bz[j]);
                    const float hb = __bfloat162float(__float2bfloat16_rn(z[j]));
                    float wv[NO];
                    w4_row(c * TC_CHUNK + 8 * u + j, wv);
#pragma unroll
                    for (int o = 0; o < NO; ++o) f[o] = fmaf(hb, wv[o], f[o]);
                }
                put(0, c, z);
            }
#pragma unroll
            for (int c = 0; c < NO; ++c) sf[(u * 6 + c) * TS + smp] = f[c];
            __syncwarp();
            if (lane == 0) mbar_arrive(BAR_FR);
            ok = __all_sync(0xffffffffu, mbar_wait(BAR_FR, nf++ & 1, abort_flag));
            if (!ok) break;
            // outputs, loss and its gradient (every thread of a sample alike)
            float dd[NO], q[15];
            quad_features(x, q);
            double loss = 0.0;
#pragma unroll
            for (int c = 0; c < NO; ++c) {
                float fc = 0.0f;
#pragma unroll
                for (int g = 0; g < 8; ++g) fc += sf[(g * 6 + c) * TS + smp];
                float v = x[c] + (fc + stail[c]) + stail[72 + c];
#pragma unroll
                for (int k = 0; k < 6; ++k) v += x[k] * stail[8 + k * NOUT + c];
#pragma unroll
                for (int m = 0; m < 15; ++m) v += q[m] * stail[80 + m * NOUT + c];
                dd[c] = 0.0f;
                if (in && c < n_fit) {
                    const float e = v - tg[c];
                    loss += (double)e * (double)e;
                    dd[c] = 2.0f * e / (float)(B * n_fit);
                }
            }
            if (u == 0) {
                // x and dd as operands of the weight gradients, 16 columns
                unsigned char *sx = w.small + t * TT_SMALL + smp * 128, *sd = w.small + (w.T + t) * TT_SMALL + smp * 128;
                const float xv[8] = {x[0], x[1], x[2], x[3], x[4], x[5]};
                float dv[8] = {};
#pragma unroll
                for (int c = 0; c < NO; ++c) dv[c] = dd[c];
                const int s7 = smp & 7;
                *reinterpret_cast<uint4 *>(sx + ((0 ^ s7) << 4)) = pack8(xv);
                *reinterpret_cast<uint4 *>(sx + ((1 ^ s7) << 4)) = make_uint4(0, 0, 0, 0);
                *reinterpret_cast<uint4 *>(sd + ((0 ^ s7) << 4)) = pack8(dv);
                *reinterpret_cast<uint4 *>(sd + ((1 ^ s7) << 4)) = make_uint4(0, 0, 0, 0);
            } else if (u == 2) {
                for (int off = 16; off > 0; off >>= 1) loss += __shfl_down_sync(0xffffffffu, loss, off);
                if (lane == 0) w.loss[2 * t + group] = loss;
            } else if (u == 4) {
#pragma unroll
                for (int c = 0; c < 6; ++c) sdd[c * (TS + 1) + smp] = c < NO ? dd[c < NO ? c : 0] : 0.0f;
            }
#pragma unroll
            for (int c = 0; c < NO; ++c) dd[c] = __bfloat162float(__float2bfloat16_rn(dd[c]));
            // dz3 = (dd W4^T) SiLU'(z3) -> buffer 1
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
                tmem_load8(lane_base + 256 + c * TC_CHUNK, z);
                load8(sbias + 2 * H + c * TC_CHUNK + 8 * u, bz);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    float wv[NO];
                    w4_row(c * TC_CHUNK + 8 * u + j, wv);
                    float dh = dd[0] * wv[0];
#pragma unroll
                    for (int o = 1; o < NO; ++o) dh = fmaf(dd[o], wv[o], dh);
                    z[j] = dh * dsilu(z[j] + bz[j]);
                }
                put(1, c, z);
                bias_sum(2, c, z);
            }
            // dz2 = (dz3 W3^T) SiLU'(z2) -> buffer 0
            if (!wait_d()) break;
            // (every warp has read the partial outputs: their place takes the
            // skip layer's features)
            if (u == 6) {
                float q[15];
                quad_features(x, q);
#pragma unroll
                for (int k = 0; k < 6; ++k) sf[k * (TS + 1) + smp] = x[k];
#pragma unroll
                for (int k = 0; k < 15; ++k) sf[(6 + k) * (TS + 1) + smp] = q[k];
                sf[21 * (TS + 1) + smp] = 1.0f;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(BAR_FR);
            float dh[8];
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
                tmem_load8x2(lane_base + c * TC_CHUNK, lane_base + 256 + c * TC_CHUNK, z, dh);
                load8(sbias + H + c * TC_CHUNK + 8 * u, bz);
#pragma unroll
                for (int j = 0; j < 8; ++j) dh[j] *= dsilu(z[j] + bz[j]);
                put(0, c, dh);
                bias_sum(1, c, dh);
            }
            // dz1 = (dz2 W2^T) SiLU'(z1) -> buffer 1 (stored only)
            if (!wait_d()) break;
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
                tmem_load8(lane_base + 256 + c * TC_CHUNK, dh);
                z1_of(c, z);
#pragma unroll
                for (int j = 0; j < 8; ++j) dh[j] *= dsilu(z[j]);
                put(1, c, dh);
                bias_sum(0, c, dh);
            }
            // skip-layer sums: four threads a sum, 16 samples each
            ok = __all_sync(0xffffffffu, mbar_wait(BAR_FR, nf++ & 1, abort_flag));
            if (!ok) break;
            const int et = threadIdx.x - 64;
            for (int e0 = 0; e0 < SKIP_SUMS; e0 += TT_EPI / 4) {
                const int e = min(e0 + (et >> 2), SKIP_SUMS - 1);
                const float *fx = sf + (e / 6) * (TS + 1) + 16 * (et & 3), *fd = sdd + (e % 6) * (TS + 1) + 16 * (et & 3);
                float s = 0.0f;
#pragma unroll
                for (int i = 0; i < 16; ++i) s = fmaf(fx[i], fd[i], s);
                s += __shfl_xor_sync(0xffffffffu, s, 1);
                s += __shfl_xor_sync(0xffffffffu, s, 2);
                if ((et & 3) == 0 && e0 + (et >> 2) < SKIP_SUMS) w.skip[t * SKIP_SUMS + e] = s;
            }
        }
    }
    tc_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
    }
    if (threadIdx.x == 0 && *abort_flag) train_gave_up(w);
}

// Weight gradients.  Blocks 0 .. 8 S - 1: (product, quadrant, split): 128 x 128
// of gW2 = h1^T dz2 or gW3 = h2^T dz3 over the split's tiles; the next 2 SS
// blocks: (dz1^T x, h3^T dd: 256 x 16, two accumulators).  Each tile
// (K = 64 samples) is a stage of bulk copies, four stages; operands are MN-major: 64 columns of a row
// contiguous (128 B, swizzled), 8 rows per 1024 B (SBO), the next 64 columns one
// chunk on (LBO).
constexpr int TG_THREADS = 128, TG_STAGES = 4;
constexpr uint32_t TG_STAGE = 5 * TS_CHUNK;                     // 2 + 2 chunks, or 4 + 1
constexpr uint32_t TG_BAR = TG_STAGES * TG_STAGE;               // full[], empty[]
constexpr uint32_t TG_MISC = TG_BAR + 16 * TG_STAGES;
constexpr size_t TG_SMEM = TG_MISC + 16 + 1024;

__global__ void __launch_bounds__(TG_THREADS, 1) train_wgrad_kernel(TrainWork w)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char *sm = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t s0 = smem_u32(sm), FULL = s0 + TG_BAR, EMPTY = FULL + 8 * TG_STAGES;
    uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(sm + TG_MISC);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(sm + TG_MISC + 4);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool large = (int)blockIdx.x < 8 * w.S;
    const int id = large ? blockIdx.x : blockIdx.x - 8 * w.S;
    const int prod = large ? (id >> 2) & 1 : id & 1, kh = id & 1, nh = (id >> 1) & 1;
    const int split = large ? id >> 3 : id >> 1, splits = large ? w.S : w.SS;
    const int64_t t0 = w.T * split / splits, t1 = w.T * (split + 1) / splits;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2 * TG_STAGES; ++i) mbar_init(FULL + 8 * i, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)),
                     "r"(128));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    const uint32_t tmem = *tmem_holder;
    ffa::chain_wait();
    if (threadIdx.x == 0) {
        auto fill = [&](int64_t t, uint32_t q) {                // use q of the ring: tile t
            const uint32_t sl = q % TG_STAGES, st = s0 + sl * TG_STAGE, bar = FULL + 8 * sl;
            if (!mbar_wait(EMPTY + 8 * sl, ((q / TG_STAGES) & 1) ^ 1, abort_flag)) return false;
            if (large) {
                mbar_expect_tx(bar, 4 * TS_CHUNK);
                bulk_load(st, tile_img(w, prod, t) + 2 * kh * TS_CHUNK, 2 * TS_CHUNK, bar);
                bulk_load(st + 2 * TS_CHUNK, tile_img(w, 4 + prod, t) + 2 * nh * TS_CHUNK, 2 * TS_CHUNK, bar);
            } else {
                mbar_expect_tx(bar, 5 * TS_CHUNK);
                bulk_load(st, tile_img(w, prod == 0 ? 3 : 2, t), 4 * TS_CHUNK, bar);
                bulk_load(st + 4 * TS_CHUNK, w.small + (prod * w.T + t) * TT_SMALL, TS_CHUNK, bar);
            }
            return true;
        };
        constexpr uint32_t MN = (1u << 15) | (1u << 16);        // both operands MN-major
        constexpr uint32_t ID_L = idesc_bf16(TC_M, 128) | MN, ID_S = idesc_bf16(TC_M, 16) | MN;
        uint32_t filled = 0, used = 0;
        bool ok = true;
        for (int64_t t = t0; t < t1 && ok; ++t) {
            while (ok && filled < used + TG_STAGES && t0 + filled < t1) {
                ok = fill(t0 + filled, filled);
                if (ok) ++filled;
            }
            if (!ok) break;
            const uint32_t sl = used % TG_STAGES, st = s0 + sl * TG_STAGE;
            ok = mbar_wait(FULL + 8 * sl, (used / TG_STAGES) & 1, abort_flag);
            if (!ok) break;
            tc_after_sync();
#pragma unroll
            for (int kk = 0; kk < TS / 16; ++kk) {              // 16 samples a product
                const uint32_t off = 2048 * kk, acc = t > t0 || kk > 0;
                if (large) {
                    umma(tmem, sdesc(st + off, TS_CHUNK, 1024, 2), sdesc(st + 2 * TS_CHUNK + off, TS_CHUNK, 1024, 2), ID_L,
                         acc);
                } else {
                    const uint64_t b = sdesc(st + 4 * TS_CHUNK + off, TS_CHUNK, 1024, 2);
                    umma(tmem, sdesc(st + off, TS_CHUNK, 1024, 2), b, ID_S, acc);
                    umma(tmem + 16, sdesc(st + 2 * TS_CHUNK + off, TS_CHUNK, 1024, 2), b, ID_S, acc);
                }
            }
            umma_commit(EMPTY + 8 * sl);
            ++used;
        }
        // every copy has landed and every product is complete
        for (uint32_t r = used; r < filled; ++r)
            if (!mbar_wait_bounded(FULL + 8 * (r % TG_STAGES), (r / TG_STAGES) & 1)) *abort_flag = 1;
        if (used > 0 && !mbar_wait_bounded(EMPTY + 8 * ((used - 1) % TG_STAGES), ((used - 1) / TG_STAGES) & 1)) *abort_flag = 1;
    }
    __syncthreads();
    tc_after_sync();
    const int row = 32 * warp + lane;                           // accumulator row
    const uint32_t base = tmem + ((uint32_t)(32 * warp) << 16);
    if (large) {
        float4 *out = reinterpret_cast<float4 *>(w.part) + ((int64_t)prod * w.S + split) * (H * H / 4) +
                      (int64_t)(32 * nh) * H + 128 * kh + row;
#pragma unroll 1
        for (int n = 0; n < 128; n += 32) {
            uint32_t v[32];
            TMEM_LD32(base + n, v);
            tmem_wait_ld();
            REG_FENCE32(v);
#pragma unroll
            for (int j = 0; j < 32; j += 4)
                out[(int64_t)((n + j) / 4) * H] = make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]),
                                                              __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
        }
    } else {
        uint32_t v[32];                                         // 16 columns of rows `row` and 128 + row
        TMEM_LD32(base, v);
        tmem_wait_ld();
        REG_FENCE32(v);
        float *out = w.part16 + ((int64_t)prod * w.SS + split) * (16 * H);
#pragma unroll
        for (int j = 0; j < 32; ++j)
            out[(j & 15) * H + 128 * (j >> 4) + row] = __uint_as_float(v[j]);
    }
    tc_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(128));
    }
    if (threadIdx.x == 0 && *abort_flag) train_gave_up(w);
}

struct AdamArgs {
    float *P, *G, *m, *v;
    const uint8_t *mask;
    float lr, b1, b2, eps, c1, c2;
    const float *lr_table;      // device schedule, or NULL
    int32_t *counter;
    int update;
};

__device__ __forceinline__ void adam_one(const AdamArgs &a, int i, float g, float lr, float c1, float c2, bool failed)
{
    a.G[i] = failed ? __uint_as_float(0x7FC00000u) : g;
    if (failed || !a.update || (a.mask && !a.mask[i])) return;
    const float mi = a.b1 * a.m[i] + (1.0f - a.b1) * g;
    const float vi = a.b2 * a.v[i] + (1.0f - a.b2) * g * g;
    a.m[i] = mi;
    a.v[i] = vi;
    a.P[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + a.eps);
}

// Every parameter's gradient from the partial sums, in a fixed order, then Adam.
// A step that failed gives NaN gradients and loss, and updates nothing.
// Blocks 0 .. 255: 32 k x 16 n of W2 and W3 (summed along k, which is contiguous
// in the partial products, updated along n); then 32 parameters a block, the
// partial sums of each over eight warps; the loss in the last block.
constexpr int TU_TILES = 2 * (H / 32) * (H / 16);
constexpr int TU_REST = (int)(P_TOTAL - 2 * H * H), TU_BLOCKS = TU_TILES + (TU_REST + 31) / 32 + 1;

__global__ void __launch_bounds__(256) train_update_kernel(TrainWork w, AdamArgs a, double *__restrict__ loss_part)
{
    __shared__ float sh[32][33];
    ffa::chain_wait();
    const bool failed = *w.failed == FFA_MLP_STEP_FAILED;
    float lr = a.lr, c1 = a.c1, c2 = a.c2;
    if (a.lr_table) {
        const int k = *a.counter;
        const float t = (float)(k + 1);
        lr = a.lr_table[k];
        c1 = 1.0f - powf(a.b1, t);
        c2 = 1.0f - powf(a.b2, t);
    }
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    if ((int)blockIdx.x < TU_TILES) {
        const int prod = blockIdx.x / (TU_TILES / 2), tile = blockIdx.x % (TU_TILES / 2);
        const int k0 = 32 * (tile / (H / 16)), n0 = 16 * (tile % (H / 16));
        // warp wp: columns n0 + 4 (wp & 3) .., the splits of one parity
        const float4 *src = reinterpret_cast<const float4 *>(w.part) + (int64_t)prod * w.S * (H * H / 4) +
                            (int64_t)(n0 / 4 + (wp & 3)) * H + k0 + lane;
        float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 8
        for (int z = wp >> 2; z < w.S; z += 2) {
            const float4 v = __ldg(src + (int64_t)z * (H * H / 4));
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        float *d = &sh[lane][16 * (wp >> 2) + 4 * (wp & 3)];
        d[0] = s.x; d[1] = s.y; d[2] = s.z; d[3] = s.w;
        __syncthreads();
        const int base = (int)(prod == 0 ? P_W2 : P_W3), n = tid & 15;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int k = (tid >> 4) + 16 * j;
            adam_one(a, base + (k0 + k) * H + n0 + n, sh[k][n] + sh[k][16 + n], lr, c1, c2, failed);
        }
    } else if (blockIdx.x + 1 < gridDim.x) {
        // parameter r of W1, b1, b2, b3, W4, b4, Ws, bs, Wq: its partial sums
        // lie `ld` apart, `cnt` of them, from `p` (none: the gradient is 0)
        const int r = (blockIdx.x - TU_TILES) * 32 + lane;
        const int L1 = KIN * H, L4 = H * NOUT;
        int i = -1;
        const float *p = nullptr;
        int64_t cnt = 0, ld = 0;
        auto small = [&](int prod, int c, int n) {
            p = w.part16 + (int64_t)prod * w.SS * (16 * H) + c * H + n;
            cnt = w.SS;
            ld = 16 * H;
        };
        auto skip = [&](int m, int c) {
            if (m >= 22 || c >= 6) return;
            p = w.skip + 6 * m + c;
            cnt = w.T;
            ld = SKIP_SUMS;
        };
        if (r < L1) {
            i = (int)P_W1 + r;
            if (r / H < 6) small(0, r / H, r % H);
        } else if (r < L1 + 3 * H) {
            const int l = (r - L1) / H, n = (r - L1) % H;
            i = (int)(l == 0 ? P_B1 : l == 1 ? P_B2 : P_B3) + n;
            p = w.bias + (int64_t)l * 2 * w.T * H + n;
            cnt = 2 * w.T;
            ld = H;
        } else if (r < L1 + 3 * H + L4) {
            const int e = r - L1 - 3 * H;
            i = (int)P_W4 + e;
            small(1, e % NOUT, e / NOUT);
        } else if (r < TU_REST) {
            const int e = r - L1 - 3 * H - L4, m = e / NOUT;    // b4, Ws (8), bs, Wq (16)
            i = (int)P_B4 + e;
            if (m == 0 || m == 9) skip(21, e % NOUT);
            else if (m < 9) { if (m - 1 < 6) skip(m - 1, e % NOUT); }
            else if (m - 10 < 15) skip(6 + m - 10, e % NOUT);
        }
        float s = 0.0f;
#pragma unroll 8
        for (int64_t z = wp; z < cnt; z += 8) s += __ldg(p + z * ld);
        sh[wp][lane] = s;
        __syncthreads();
        if (wp == 0 && i >= 0) {
            float g = 0.0f;
            for (int k = 0; k < 8; ++k) g += sh[k][lane];
            adam_one(a, i, g, lr, c1, c2, failed);
        }
    } else {
        for (int q = tid; q < 148; q += 256) {
            double s = 0.0;
            for (int64_t z = q; z < 2 * w.T; z += 148) s += w.loss[z];
            loss_part[q] = failed ? __longlong_as_double(0x7FF8000000000000ll) : s;
        }
    }
    // the last block to finish advances the schedule and clears the failure
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(w.ticket, 1) == (int)gridDim.x - 1) {
            if (failed) *w.failed = 0;
            else if (a.counter) *a.counter += 1;
        }
    }
}

// Places the scratch in the caller's work area; false if it does not fit
// (it always does: 8 * 256 + 24 floats a sample and SPLIT_WORK are more)
bool train_layout(TrainWork &w, float *work, int64_t B)
{
    w.T = (B + TS - 1) / TS;
    w.S = (int)((w.T + 1) / 2 < TG_SPLITS ? (w.T + 1) / 2 : TG_SPLITS);      // at least two tiles each
    w.SS = (int)(w.T < TG_SMALL_SPLITS ? w.T : TG_SMALL_SPLITS);
    unsigned char *p = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(work) + 127) & ~uintptr_t(127));
    auto take = [&](int64_t bytes) {
        unsigned char *q = p;
        p += (bytes + 127) & ~int64_t(127);
        return q;
    };
    w.failed = reinterpret_cast<unsigned long long *>(take(8));
    w.img = take(6 * w.T * TT_IMG);
    w.small = take(2 * w.T * TT_SMALL);
    w.wpk = take(16 * (int64_t)W_CHUNK_BYTES);
    w.part = reinterpret_cast<float *>(take(2 * (int64_t)w.S * H * H * 4));
    w.part16 = reinterpret_cast<float *>(take(2 * (int64_t)w.SS * 16 * H * 4));
    w.bias = reinterpret_cast<float *>(take(3 * 2 * w.T * H * 4));
    w.skip = reinterpret_cast<float *>(take(w.T * SKIP_SUMS * 4));
    w.loss = reinterpret_cast<double *>(take(2 * w.T * 8));
    w.ticket = reinterpret_cast<int32_t *>(take(4));
    const int64_t have = (8 * B * H + 24 * B + SPLIT_WORK) * 4;
    return p - reinterpret_cast<unsigned char *>(work) <= have;
}

bool g5_fits(int M, int N, int K) { return M >= G5_BM && N >= G5_BN && K >= G5_BK; }

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// one GEMM launch: the tcgen05 kernel for products of at least one full
// tile, gemm_tc for the narrow ones (N = 8 outputs, K = 8 inputs, M = 6)
cudaError_t launch_gemm(const float *A, int lda, int tA, const float *B, int ldb, int tB, float *C, int ldc, int M,
                        int N, int K, const float *bias, cudaStream_t s)
{
    if (g5_fits(M, N, K)) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_tc05, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G5_SMEM);
        if (e != cudaSuccess) return e;
        const dim3 grid((unsigned)((N + G5_BN - 1) / G5_BN), (unsigned)((M + G5_BM - 1) / G5_BM));
        const int vA = !tA && (lda & 3) == 0 && aligned16(A), vB = tB && (ldb & 3) == 0 && aligned16(B);
        gemm_tc05<<<grid, G5_THREADS, G5_SMEM, s>>>(A, lda, tA, B, ldb, tB, C, ldc, M, N, K, bias, vA, vB);
    } else {
        const dim3 grid((unsigned)((N + GT_N - 1) / GT_N), (unsigned)((M + GT_M - 1) / GT_M));
        gemm_tc<<<grid, 128, 0, s>>>(A, lda, tA, B, ldb, tB, C, ldc, M, N, K, bias);
    }
    return cudaGetLastError();
}

}  // namespace

// ------------------------------------------------------------------ C ABI


static_assert(PK_TOTAL == FFA_MLP_WPACK_BYTES, "inference weight pack size");
static_assert(TC_SMEM <= 232448, "inference kernel shared memory");


extern "C" int ffa_mlp_gemm(const float *A, int lda, int transA, const float *B, int ldb, int transB, float *C,
                            int ldc, int M, int N, int K, const float *bias, void *stream)
{
    if (!A || !B || !C || M <= 0 || N <= 0 || K <= 0) return FFA_ERR_INVALID;
    if ((M + GT_M - 1) / GT_M > 65535) return FFA_ERR_UNSUPPORTED;
    return launch_gemm(A, lda, transA ? 1 : 0, B, ldb, transB ? 1 : 0, C, ldc, M, N, K, bias,
                       (cudaStream_t)stream) == cudaSuccess ? FFA_OK : FFA_ERR_CUDA;
}

extern "C" int ffa_mlp_gemm_timeouts(int32_t *count)
{
    if (!count) return FFA_ERR_INVALID;
    int v = 0;
    FFA_CHECK_CUDA(cudaMemcpyFromSymbol(&v, g_gemm_timeouts, sizeof(int)));
    const int zero = 0;
    FFA_CHECK_CUDA(cudaMemcpyToSymbol(g_gemm_timeouts, &zero, sizeof(int)));
    *count = v;
    return FFA_OK;
}

extern "C" int ffa_mlp_train_step(const ffa_mlp_train_desc *d, void *stream)
{
    if (!d || !d->params || !d->grads || !d->adam_m || !d->adam_v || !d->x || !d->target || !d->work ||
        !d->loss_part || d->batch <= 0 || d->n_fit < 1 || d->n_fit > 6)
        return FFA_ERR_INVALID;
    const bool sched = d->lr_table != nullptr;
    if (sched != (d->counter != nullptr)) return FFA_ERR_INVALID;
    if (!sched && d->lr > 0.0f && d->step < 1) return FFA_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    const int64_t B = d->batch;
    if (B > 65535LL * GT_M || B * H > INT32_MAX) return FFA_ERR_UNSUPPORTED;
    TrainWork w;
    if (!train_layout(w, d->work, B)) return FFA_ERR_UNSUPPORTED;
    AdamArgs a{d->params, d->grads, d->adam_m, d->adam_v, d->mask, d->lr, d->beta1, d->beta2, d->eps, 1.0f, 1.0f,
               d->lr_table, d->counter, sched || d->lr > 0.0f};
    if (!sched && a.update) {
        a.c1 = 1.0f - powf(d->beta1, (float)d->step);
        a.c2 = 1.0f - powf(d->beta2, (float)d->step);
    }
    int dev = 0, sms = 0;
    FFA_CHECK_CUDA(cudaGetDevice(&dev));
    FFA_CHECK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const auto tile = d->n_fit <= 4 ? train_tile_kernel<4> : train_tile_kernel<6>;
    FFA_CHECK_CUDA(cudaFuncSetAttribute(tile, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TT_SMEM));
    FFA_CHECK_CUDA(cudaFuncSetAttribute(train_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TG_SMEM));
    train_pack_kernel<<<H * H / 4 / 256, 256, 0, s>>>(d->params, w);
    FFA_CHECK_CUDA(ffa::launch_chained(tile, (unsigned)(w.T < sms ? w.T : sms), TT_THREADS, TT_SMEM, s, d->params, d->x,
                                       d->target, w, B, d->n_fit));
    FFA_CHECK_CUDA(ffa::launch_chained(train_wgrad_kernel, 8 * w.S + 2 * w.SS, TG_THREADS, TG_SMEM, s, w));
    FFA_CHECK_CUDA(ffa::launch_chained(train_update_kernel, TU_BLOCKS, 256, 0, s, w, a, d->loss_part));
    return cudaGetLastError() == cudaSuccess ? FFA_OK : FFA_ERR_CUDA;
}


extern "C" int ffa_mlp_pack(const float *params, void *wpack, void *stream)
{
    if (!params || !wpack || (reinterpret_cast<uintptr_t>(wpack) & 15)) return FFA_ERR_INVALID;
    pack_weights_kernel<<<(H * H + 255) / 256, 256, 0, (cudaStream_t)stream>>>(
        params, reinterpret_cast<unsigned char *>(wpack));
    return cudaGetLastError() == cudaSuccess ? FFA_OK : FFA_ERR_CUDA;
}

extern "C" int ffa_mlp_infer(const ffa_mlp_infer_desc *d, void *stream)
{
    if (!d || !d->params || !d->wpack || !d->state || d->n < 0 || d->n_apply < 0 ||
        (reinterpret_cast<uintptr_t>(d->wpack) & 15) || (reinterpret_cast<uintptr_t>(d->state) & 15))
        return FFA_ERR_INVALID;
    if (d->n == 0 || d->n_apply == 0) {
        if (d->applied && d->n > 0) FFA_CHECK_CUDA(cudaMemsetAsync(d->applied, 0, sizeof(int32_t) * d->n, (cudaStream_t)stream));
        return FFA_OK;
    }
    int dev = 0, sms = 0;
    FFA_CHECK_CUDA(cudaGetDevice(&dev));
    FFA_CHECK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int64_t tiles = (d->n + TC_M - 1) / TC_M;
    const int grid = (int)(tiles < sms ? tiles : sms);
    if (tiles > sms) {
        // more tiles than SMs: two tiles in flight per SM
        FFA_CHECK_CUDA(cudaFuncSetAttribute(mlp_infer_tc2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)TC2_SMEM));
        mlp_infer_tc2_kernel<<<grid, TC_THREADS, TC2_SMEM, (cudaStream_t)stream>>>(
            d->params, reinterpret_cast<const unsigned char *>(d->wpack), d->state, d->applied, d->error, d->n,
            d->n_apply, d->radius2);
    } else {
        FFA_CHECK_CUDA(cudaFuncSetAttribute(mlp_infer_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)TC_SMEM));
        mlp_infer_tc_kernel<<<grid, TC_THREADS, TC_SMEM, (cudaStream_t)stream>>>(
            d->params, reinterpret_cast<const unsigned char *>(d->wpack), d->state, d->applied, d->error, d->n,
            d->n_apply, d->radius2);
    }
    return cudaGetLastError() == cudaSuccess ? FFA_OK : FFA_ERR_CUDA;
}
