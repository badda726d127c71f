// C[M,N] = A[M,K] . W[N,K]^T with fp32 FMA on the SIMT pipes, any sizes.
//
// This is the true 32-bit matrix product of the float32 path (no tensor cores, no TF32) and
// the fall-back of the bfloat16 path for shapes the tensor-core kernel refuses.  Activations A
// are float or bf16, weights W are float or bf16 independently (a weight stored in 32-bit
// stays so).  Accumulation is fp32 in an order that only K fixes, so a row's result does not
// depend on what else is in the batch:
//
//   * float x float with rows of whole 16-byte pieces (every product of the float32 path): K is
//     cut into KPARTS parts, a part's elements of even k and of odd k are summed apart with k
//     ascending, and the sums are added in order.  The parts are what lets a product of few tokens
//     keep the whole chip busy; three kernels share this order, one for few tokens (bound by the
//     weights' way in), one for many (bound by the FMA pipes) and one for many and few columns.
//   * anything else: k ascending over the whole row, the kernel for all sizes.
//
// Epilogues (the reference's are src/backend/cuda/k_gemm.cu:29-53):
//   0 store in the activation dtype      1 store fp32
//   2 add into an fp32 matrix (residual) 3 silu(c[2j]) * c[2j+1] over interleaved gate/up rows
//   6 relu(c[2j]) * c[2j+1] likewise     7 gelu(c[2j]) * c[2j+1], gelu in its tanh form
//   8 gelu(c) in its exact form (erf), stored in the activation dtype     9 max(c, 0)^2 likewise
// An optional fp32 bias[N] is added before the epilogue.
#include <type_traits>

#include "common.cuh"

EMBER_DEFINE_LAST_ERROR

namespace ember {

constexpr int BM = 64, BN = 64, BK = 16;

template <typename TA, typename TW, int EPI>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const TA* __restrict__ A, int lda, const TW* __restrict__ W, int ldw,
                 const float* __restrict__ bias, void* __restrict__ Cv, int ldc, int M, int N, int K) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    pdl_launch_dependents();
    pdl_wait();
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;  // tx -> columns, ty -> rows
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.0f;

    // loader mapping: 256 threads fetch 64 rows x 16 k: thread -> (row = id / 4, k = (id % 4) * 4 .. +3)
    const int lrow = threadIdx.x >> 2, lk = (threadIdx.x & 3) * 4;
    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int k = k0 + lk + j;
            const int am = m0 + lrow, wn = n0 + lrow;
            As[lk + j][lrow] = (am < M && k < K) ? to_float(A[(size_t)am * lda + k]) : 0.0f;
            Ws[lk + j][lrow] = (wn < N && k < K) ? to_float(W[(size_t)wn * ldw + k]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; k++) {
            float a[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = As[k][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; j++) w[j] = Ws[k][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }

#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int n = n0 + tx * 4 + j;
            if (n >= N) continue;
            float c = acc[i][j] + (bias ? bias[n] : 0.0f);
            if (EPI == 0 || EPI == 8 || EPI == 9) {
                if (EPI == 8) c = 0.5f * c * (1.0f + erff(c * 0.7071067811865476f));
                if (EPI == 9) { c = fmaxf(c, 0.0f); c *= c; }
                ((TA*)Cv)[(size_t)m * ldc + n] = from_float<TA>(c);
            } else if (EPI == 1) {
                ((float*)Cv)[(size_t)m * ldc + n] = c;
            } else if (EPI == 2) {
                float* p = (float*)Cv + (size_t)m * ldc + n;
                *p = *p + c;
            } else {
                if ((j & 1) == 0) {  // n even: gate; n + 1: up (same thread, N is even)
                    const float u = acc[i][j + 1] + (bias ? bias[n + 1] : 0.0f);
                    const float a = EPI == 6 ? fmaxf(c, 0.0f)
                                  : (EPI == 7 ? 0.5f * c * (1.0f + tanhf(0.7978845608028654f * fmaf(0.044715f * c * c, c, c))) : c / (1.0f + expf(-c)));
                    ((TA*)Cv)[(size_t)m * ldc + (n >> 1)] = from_float<TA>(a * u);
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------------------------
// float x float, 16-byte pieces.  Part p of K is [p * len, min(K, (p + 1) * len)), len a multiple of PART_UNIT.
constexpr int KPARTS = 8, PART_UNIT = 32;

__device__ __forceinline__ int part_length(int K) { return ((K + KPARTS - 1) / KPARTS + PART_UNIT - 1) / PART_UNIT * PART_UNIT; }

// 16 bytes from global to shared memory without a register; zeros when !valid (src is then not read).
__device__ __forceinline__ void copy16(float* dst, const float* src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Two fp32 multiply-adds in one instruction, on elements k and k + 1 of two rows as they lie in shared memory.
__device__ __forceinline__ unsigned long long fma_pair(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ float pair_sum(unsigned long long v) {
    return __uint_as_float((unsigned)v) + __uint_as_float((unsigned)(v >> 32));
}

// The sums of columns n and n + 1 (n even) of row m -> the output.
__device__ __forceinline__ void finish_pair(float c0, float c1, const float* __restrict__ bias, float* __restrict__ C, int ldc, int m,
                                            int n, int N, int epi) {
    const bool two = n + 1 < N;
    if (bias) {
        c0 += bias[n];
        if (two) c1 += bias[n + 1];
    }
    if (epi == 3 || epi == 6 || epi == 7) {                       // N is even
        const float a = epi == 6 ? fmaxf(c0, 0.0f)
                      : (epi == 7 ? 0.5f * c0 * (1.0f + tanhf(0.7978845608028654f * fmaf(0.044715f * c0 * c0, c0, c0))) : c0 / (1.0f + expf(-c0)));
        C[(size_t)m * ldc + (n >> 1)] = a * c1;
        return;
    }
    float* p = C + (size_t)m * ldc + n;
    if (epi == 8) {
        c0 = 0.5f * c0 * (1.0f + erff(c0 * 0.7071067811865476f));
        c1 = 0.5f * c1 * (1.0f + erff(c1 * 0.7071067811865476f));
    } else if (epi == 9) {
        c0 = fmaxf(c0, 0.0f); c0 *= c0;
        c1 = fmaxf(c1, 0.0f); c1 *= c1;
    } else if (epi == 2) {
        c0 += p[0];
        if (two) c1 += p[1];
    }
    p[0] = c0;
    if (two) p[1] = c1;
}

// Few tokens (MT of them per block): bound by the weights' way in.  A thread sums one part of K for one weight row
// and MT tokens; a warp holds NB weight rows x 32 / NB parts and feeds itself through a ring of cp.async stages of 32
// elements of k (a whole 128-byte line of each row), so nothing but the final addition of the parts needs a block
// barrier and 3 x 4.5 KB a warp are on their way.  Weights that no kernel still running writes (`settled`) are asked for
// before the wait for the kernel before.  Rows of 36 floats keep the 16-byte reads of a quarter warp in different banks.
// Four tokens at the 0.6B widths (hidden 1,024), in a step: o and down 9.0 and 13.8 us, q/k/v and gate/up 5, the head's
// 622 MB 100 us (6.2 TB/s); with the general kernel everywhere four requests of 75 tokens and four more steps took 143 ms,
// with this one and the next 23.
constexpr int FEW_K = 32, FEW_ROW = FEW_K + 4;

template <int MT, int NB>
constexpr size_t few_stage_floats() { return 32 * FEW_ROW + (32 / NB) * MT * FEW_K; }
template <int MT, int NB, int FEW_STAGES>
constexpr size_t few_smem() { return (NB * KPARTS / 32) * FEW_STAGES * few_stage_floats<MT, NB>() * sizeof(float); }

template <int MT, int NB, int FEW_STAGES>
__global__ void __launch_bounds__(NB * KPARTS)
gemm_f32_few_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, const float* __restrict__ bias,
                    float* __restrict__ C, int ldc, int M, int N, int K, int epi, int settled) {
    extern __shared__ __align__(16) float few_shared[];
    constexpr int WP = 32 / NB;                                   // parts of a warp
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n0 = blockIdx.x * NB, m0 = blockIdx.y * MT;
    const int len = part_length(K), steps = len / FEW_K;
    float* stages = few_shared + warp * FEW_STAGES * few_stage_floats<MT, NB>();
    const int piece = (lane & 7) * 4;                             // this lane's 16 bytes of a row of a stage

    auto fetch_w = [&](int step) {
        float* dst = stages + (step % FEW_STAGES) * few_stage_floats<MT, NB>();
#pragma unroll
        for (int r0 = 0; r0 < 32; r0 += 4) {
            const int r = r0 + (lane >> 3), part = warp * WP + r / NB, n = n0 + r % NB;
            const int k = part * len + step * FEW_K + piece;
            const bool ok = n < N && k < K;
            copy16(dst + r * FEW_ROW + piece, ok ? W + (size_t)n * ldw + k : W, ok);
        }
    };
    auto fetch_a = [&](int step) {
        float* dst = stages + (step % FEW_STAGES) * few_stage_floats<MT, NB>() + 32 * FEW_ROW;
#pragma unroll
        for (int r0 = 0; r0 < WP * MT; r0 += 4) {
            const int r = r0 + (lane >> 3), part = warp * WP + r / MT, m = m0 + r % MT;
            const int k = part * len + step * FEW_K + piece;
            const bool ok = m < M && k < K;
            if (r < WP * MT) copy16(dst + r * FEW_K + piece, ok ? A + (size_t)m * lda + k : A, ok);
        }
    };
    if (!settled) pdl_wait();
#pragma unroll
    for (int s = 0; s < FEW_STAGES - 1; s++)
        if (s < steps) fetch_w(s);
    pdl_wait();
#pragma unroll
    for (int s = 0; s < FEW_STAGES - 1; s++) {
        if (s < steps) fetch_a(s);
        copies_commit();
    }

    unsigned long long acc[MT];
#pragma unroll
    for (int m = 0; m < MT; m++) acc[m] = 0;
    for (int step = 0; step < steps; step++) {
        if (step + FEW_STAGES - 1 < steps) {
            fetch_w(step + FEW_STAGES - 1);
            fetch_a(step + FEW_STAGES - 1);
        }
        copies_commit();
        copies_wait<FEW_STAGES - 1>();
        __syncwarp();                                             // every lane's copies of this stage are there
        const float* ws = stages + (step % FEW_STAGES) * few_stage_floats<MT, NB>();
        const float* as = ws + 32 * FEW_ROW + (lane / NB) * MT * FEW_K;
        ws += lane * FEW_ROW;
#pragma unroll
        for (int k = 0; k < FEW_K; k += 4) {
            const ulonglong2 w = *(const ulonglong2*)(ws + k);
#pragma unroll
            for (int m = 0; m < MT; m++) {
                const ulonglong2 a = *(const ulonglong2*)(as + m * FEW_K + k);
                acc[m] = fma_pair(a.x, w.x, acc[m]);
                acc[m] = fma_pair(a.y, w.y, acc[m]);
            }
        }
        __syncwarp();                                             // the stage may be written again
    }

    copies_wait<0>();
    __syncthreads();
    float* parts = few_shared;                                    // [KPARTS][MT][NB]
    const int part = threadIdx.x / NB, nn = threadIdx.x % NB;
#pragma unroll
    for (int m = 0; m < MT; m++) parts[(part * MT + m) * NB + nn] = pair_sum(acc[m]);
    __syncthreads();
    for (int i = threadIdx.x; i < MT * NB / 2; i += NB * KPARTS) {
        const int m = i / (NB / 2), n = (i % (NB / 2)) * 2;
        if (m0 + m >= M || n0 + n >= N) continue;
        float c0 = parts[m * NB + n], c1 = parts[m * NB + n + 1];
#pragma unroll
        for (int q = 1; q < KPARTS; q++) {
            c0 += parts[(q * MT + m) * NB + n];
            c1 += parts[(q * MT + m) * NB + n + 1];
        }
        finish_pair(c0, c1, bias, C, ldc, m0 + m, n0 + n, N, epi);
    }
}

// Many tokens: bound by the FMA pipes.  A block makes a tile of 32 tokens x 64 columns, its eight warps one part of K
// each: a warp keeps the whole tile of its part in registers (8 x 8 pairs of sums a thread, sixteen 16-byte reads of
// shared memory per 128 paired multiply-adds) and feeds itself through two cp.async stages of 16 elements of k, so again
// only the addition of the parts needs block barriers.  Rows of 20 floats keep the eight rows that a warp reads at
// once in different banks.  Sums of one element of k at a time and tiles of 64 x 64 took 137 us for 300 tokens x 6,144
// columns x 1,024, this 132.
constexpr int MANY_M = 32, MANY_N = 64, MANY_K = 16, MANY_ROW = MANY_K + 4, MANY_OUT = MANY_N + 8;
constexpr int MANY_STAGE = (MANY_M + MANY_N) * MANY_ROW;          // floats
constexpr size_t MANY_SMEM = (size_t)KPARTS * 2 * MANY_STAGE * sizeof(float);
static_assert(MANY_SMEM >= (size_t)KPARTS * MANY_M * MANY_OUT * sizeof(float), "the parts' tiles take the stages' place");

__global__ void __launch_bounds__(KPARTS * 32, 1)
gemm_f32_many_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, const float* __restrict__ bias,
                     float* __restrict__ C, int ldc, int M, int N, int K, int epi, int settled) {
    extern __shared__ __align__(16) float many_shared[];
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tx = lane & 7, ty = lane >> 3;
    const int n0 = blockIdx.x * MANY_N, m0 = blockIdx.y * MANY_M;
    const int len = part_length(K), steps = len / MANY_K, k_first = warp * len;
    float* stages = many_shared + warp * 2 * MANY_STAGE;
    const int piece = (lane & 3) * 4;

    auto fetch_w = [&](int step) {
        float* dst = stages + (step & 1) * MANY_STAGE + MANY_M * MANY_ROW;
        const int k = k_first + step * MANY_K + piece;
#pragma unroll
        for (int r0 = 0; r0 < MANY_N; r0 += 8) {
            const int r = r0 + (lane >> 2);
            const bool ok = n0 + r < N && k < K;
            copy16(dst + r * MANY_ROW + piece, ok ? W + (size_t)(n0 + r) * ldw + k : W, ok);
        }
    };
    auto fetch_a = [&](int step) {
        float* dst = stages + (step & 1) * MANY_STAGE;
        const int k = k_first + step * MANY_K + piece;
#pragma unroll
        for (int r0 = 0; r0 < MANY_M; r0 += 8) {
            const int r = r0 + (lane >> 2);
            const bool ok = m0 + r < M && k < K;
            copy16(dst + r * MANY_ROW + piece, ok ? A + (size_t)(m0 + r) * lda + k : A, ok);
        }
    };
    if (!settled) pdl_wait();
    fetch_w(0);
    pdl_wait();
    fetch_a(0);
    copies_commit();

    unsigned long long acc[8][8];                                 // token i * 4 + ty, column j * 8 + tx
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = 0;
    for (int step = 0; step < steps; step++) {
        if (step + 1 < steps) {
            fetch_w(step + 1);
            fetch_a(step + 1);
        }
        copies_commit();
        copies_wait<1>();
        __syncwarp();
        const float* as = stages + (step & 1) * MANY_STAGE + ty * MANY_ROW;
        const float* ws = stages + (step & 1) * MANY_STAGE + (MANY_M + tx) * MANY_ROW;
#pragma unroll
        for (int k = 0; k < MANY_K; k += 4) {
            ulonglong2 a[8], w[8];
#pragma unroll
            for (int i = 0; i < 8; i++) a[i] = *(const ulonglong2*)(as + i * 4 * MANY_ROW + k);
#pragma unroll
            for (int j = 0; j < 8; j++) w[j] = *(const ulonglong2*)(ws + j * 8 * MANY_ROW + k);
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 8; j++) acc[i][j] = fma_pair(a[i].x, w[j].x, acc[i][j]);
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 8; j++) acc[i][j] = fma_pair(a[i].y, w[j].y, acc[i][j]);
        }
        __syncwarp();
    }

    copies_wait<0>();
    __syncthreads();
    float* parts = many_shared;                                   // [KPARTS][MANY_M][MANY_OUT]
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) parts[(warp * MANY_M + i * 4 + ty) * MANY_OUT + j * 8 + tx] = pair_sum(acc[i][j]);
    __syncthreads();
    for (int i = threadIdx.x; i < MANY_M * MANY_N / 2; i += KPARTS * 32) {
        const int m = i / (MANY_N / 2), n = (i % (MANY_N / 2)) * 2;
        if (m0 + m >= M || n0 + n >= N) continue;
        float2 c = *(const float2*)(parts + m * MANY_OUT + n);
#pragma unroll
        for (int q = 1; q < KPARTS; q++) {
            const float2 d = *(const float2*)(parts + (q * MANY_M + m) * MANY_OUT + n);
            c.x += d.x;
            c.y += d.y;
        }
        finish_pair(c.x, c.y, bias, C, ldc, m0 + m, n0 + n, N, epi);
    }
}

// Many tokens and few columns: with one block a tile the tiles above are one to three waves of blocks, the last of them mostly
// empty.  Here a cluster of four blocks makes a tile of 64 tokens x 64 columns, two to an SM: two parts of K a block, a warp
// for the even and one for the odd elements of k of each part.  A thread keeps 16 tokens x 8 columns of that sum, paired along
// the tokens; operands lie k-major, brought by 4-byte copies whose 8 k x 4 rows fall into 32 banks into a ring of three
// stages that the two warps of a part share.  The parts of a tile meet in distributed shared memory, every block finishes
// a quarter of its tokens.  The sums are those of the kernel above, in its order.
// Where it is ahead and where not: clusters_are_faster.  It reaches 39 TFLOP/s (2,048 tokens x 1,024 x 3,072), the kernel above 36:
// neither gets to the FMA pipes' 74.  The same sums by plain multiply-adds take 119 us where these take 88 (300 tokens x 4,096 x
// 1,024), and operands loaded 16 bytes at a time into registers and stored turned 104.
constexpr int NARROW_T = 64, NARROW_N = 64, NARROW_K = 16, NARROW_STAGES = 3, NARROW_CLUSTER = 4, NARROW_PARTS = KPARTS / NARROW_CLUSTER;
constexpr int NARROW_ROW = NARROW_N + 4;                          // floats of a k in a stage's operand, and of a row of sums
constexpr int NARROW_STAGE = 2 * NARROW_K * NARROW_ROW;           // floats
constexpr size_t NARROW_SMEM = (size_t)NARROW_PARTS * NARROW_STAGES * NARROW_STAGE * sizeof(float);
static_assert(NARROW_T == NARROW_N && NARROW_SMEM >= (size_t)NARROW_PARTS * NARROW_T * NARROW_ROW * sizeof(float), "the parts' tiles take the stages' place");

// 4 bytes from global to shared memory; zero when !valid.
__device__ __forceinline__ void copy4(float* dst, const float* src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(valid ? 4 : 0) : "memory");
}
__device__ __forceinline__ unsigned long long pack_pair(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(__float_as_uint(lo)), "r"(__float_as_uint(hi)));
    return r;
}

__global__ void __cluster_dims__(NARROW_CLUSTER, 1, 1) __launch_bounds__(NARROW_PARTS * 64, 2)
gemm_f32_narrow_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, const float* __restrict__ bias,
                       float* __restrict__ C, int ldc, int M, int N, int K, int epi, int settled) {
    extern __shared__ __align__(16) float narrow_shared[];
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tx = lane & 7, ty = lane >> 3;
    const int local = warp >> 1, odd = warp & 1, rank = blockIdx.x % NARROW_CLUSTER;
    const int n0 = (int)(blockIdx.x / NARROW_CLUSTER) * NARROW_N, m0 = blockIdx.y * NARROW_T;
    const int len = part_length(K), steps = len / NARROW_K, k_first = (rank * NARROW_PARTS + local) * len;
    float* stages = narrow_shared + local * NARROW_STAGES * NARROW_STAGE;
    const int ck = odd * 8 + tx;                                  // a warp copies 8 of a stage's 16 elements of k

    auto fetch = [&](float* dst, const float* X, int ldx, int first, int count, int step) {
        const int k = k_first + step * NARROW_K + ck;
        const float* src = X + (size_t)(first + ty) * ldx + k;
#pragma unroll
        for (int r = 0; r < 64; r += 4) {
            const bool ok = first + r + ty < count && k < K;
            copy4(dst + ck * NARROW_ROW + ty + r, ok ? src + (size_t)r * ldx : X, ok);
        }
    };
    auto fetch_w = [&](int step) { fetch(stages + (step % NARROW_STAGES) * NARROW_STAGE + NARROW_K * NARROW_ROW, W, ldw, n0, N, step); };
    auto fetch_a = [&](int step) { fetch(stages + (step % NARROW_STAGES) * NARROW_STAGE, A, lda, m0, M, step); };
    auto pair_sync = [&] { asm volatile("bar.sync %0, 64;" ::"r"(local + 1) : "memory"); };
    if (!settled) pdl_wait();
#pragma unroll
    for (int s = 0; s < NARROW_STAGES - 1; s++)
        if (s < steps) fetch_w(s);
    pdl_wait();
#pragma unroll
    for (int s = 0; s < NARROW_STAGES - 1; s++) {
        if (s < steps) fetch_a(s);
        copies_commit();
    }

    // tokens 16 g + 4 ty + 0..3 (pairs), columns 32 h + 4 tx + 0..3
    unsigned long long acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = 0;
    for (int step = 0; step < steps; step++) {
        copies_wait<NARROW_STAGES - 2>();
        pair_sync();                                              // both warps' copies of this stage are there, the one before is read
        if (step + NARROW_STAGES - 1 < steps) {
            fetch_w(step + NARROW_STAGES - 1);
            fetch_a(step + NARROW_STAGES - 1);
        }
        copies_commit();
        const float* as = stages + (step % NARROW_STAGES) * NARROW_STAGE + odd * NARROW_ROW + ty * 4;
        const float* ws = stages + (step % NARROW_STAGES) * NARROW_STAGE + (NARROW_K + odd) * NARROW_ROW + tx * 4;
#pragma unroll
        for (int k = 0; k < NARROW_K; k += 2) {
            ulonglong2 a[4];
            float4 w[2];
#pragma unroll
            for (int g = 0; g < 4; g++) a[g] = *(const ulonglong2*)(as + k * NARROW_ROW + g * 16);
#pragma unroll
            for (int h = 0; h < 2; h++) w[h] = *(const float4*)(ws + k * NARROW_ROW + h * 32);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const unsigned long long w2[4] = {pack_pair(w[h].x, w[h].x), pack_pair(w[h].y, w[h].y), pack_pair(w[h].z, w[h].z), pack_pair(w[h].w, w[h].w)};
#pragma unroll
                for (int j = 0; j < 4; j++)
#pragma unroll
                    for (int g = 0; g < 4; g++) {
                        acc[2 * g][h * 4 + j] = fma_pair(a[g].x, w2[j], acc[2 * g][h * 4 + j]);
                        acc[2 * g + 1][h * 4 + j] = fma_pair(a[g].y, w2[j], acc[2 * g + 1][h * 4 + j]);
                    }
            }
        }
    }
    copies_wait<0>();
    __syncthreads();

    // a part: the sums of even k, then those of odd k added
    float* part = narrow_shared + local * NARROW_T * NARROW_ROW;  // [tokens][NARROW_ROW]
#pragma unroll
    for (int who = 0; who < 2; who++) {
        if (odd == who) {
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int half = 0; half < 2; half++) {
                    const int m = (i >> 1) * 16 + ty * 4 + (i & 1) * 2 + half;
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        float* dst = part + m * NARROW_ROW + h * 32 + tx * 4;
                        float v[4];
#pragma unroll
                        for (int j = 0; j < 4; j++) v[j] = __uint_as_float((unsigned)(acc[i][h * 4 + j] >> (32 * half)));
                        if (who == 1) {
                            const float4 even = *(const float4*)dst;
                            v[0] = even.x + v[0]; v[1] = even.y + v[1]; v[2] = even.z + v[2]; v[3] = even.w + v[3];
                        }
                        *(float4*)dst = make_float4(v[0], v[1], v[2], v[3]);
                    }
                }
        }
        pair_sync();
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    // this block's quarter of the tokens, the parts in order
    uint32_t base[KPARTS];
#pragma unroll
    for (int q = 0; q < KPARTS; q++) {
        const uint32_t mine = (uint32_t)__cvta_generic_to_shared(narrow_shared + (q % NARROW_PARTS) * NARROW_T * NARROW_ROW);
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(base[q]) : "r"(mine), "r"(q / NARROW_PARTS));
    }
    constexpr int SHARE = NARROW_T / NARROW_CLUSTER;
    for (int i = threadIdx.x; i < SHARE * NARROW_N / 2; i += NARROW_PARTS * 64) {
        const int m = rank * SHARE + i / (NARROW_N / 2), n = (i % (NARROW_N / 2)) * 2;
        if (m0 + m >= M || n0 + n >= N) continue;
        float2 d[KPARTS];
#pragma unroll
        for (int q = 0; q < KPARTS; q++)
            asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(d[q].x), "=f"(d[q].y) : "r"(base[q] + (uint32_t)((m * NARROW_ROW + n) * 4)));
        float2 c = d[0];
#pragma unroll
        for (int q = 1; q < KPARTS; q++) { c.x += d[q].x; c.y += d[q].y; }
        finish_pair(c.x, c.y, bias, C, ldc, m0 + m, n0 + n, N, epi);
    }
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");      // (nobody leaves while its parts are read)
}

template <typename Kernel>
int launch_f32(Kernel kernel, dim3 grid, int threads, size_t smem, cudaStream_t st, const float* A, int lda, const float* W, int ldw,
               const float* bias, float* C, int ldc, int M, int N, int K, int epi, int settled) {
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return fail("gemm: shared memory %zu: %s", smem, cudaGetErrorString(e));
    }
    launch_kernel(kernel, grid, threads, smem, st, A, lda, W, ldw, bias, C, ldc, M, N, K, epi, settled);
    return check_launch("gemm_f32");
}

// Up to 16 tokens the kernel for few; 17 to 32, where two of its blocks read the same weights, while the tiles of 64 columns
// of the other one (of 32 tokens: one row of them) are fewer than half the SMs.  us at 17 and 32 tokens, few / many:
//   N x K   1,024 x 2,048  19 / 38  17 / 37     1,024 x 3,072  26 / 50  24 / 52     2,048 x 2,048  26 / 35  25 / 36
//           4,096 x 1,024  29 / 24  28 / 25     6,144 x 1,024  23 / 20  22 / 20    12,288 x 2,048  77 / 68  76 / 70
//         151,936 x 1,024  432 / 303  426 / 317
constexpr int FEW_TOKENS = 32, FEW_TOKENS_WIDE = 16, WIDE_COLUMNS = 4096;

// Whether the kernel for few looks eight stages ahead instead of three, with blocks of 8 weight rows.  Where an SM has no more than one
// block, its two warps are all that fetches there (the rings of 16 tokens also leave no room for a second one; three stages
// do, and a grid that does not fill the chip evenly gets some SMs two).  us, three / eight stages, K 2,048:
//   blocks          16            32            56            74            128           146           148           192
//   3, 4 tokens     5.7 / 4.7     6.1 / 4.9     6.5 / 5.6     6.1 / 4.9     9.0 / 5.9     9.1 / 6.1     6.3 / 5.4     9.3 / 6.8
//   5 to 8          7.5 / 7.8     7.8 / 7.7     9.0 / 7.9     7.8 / 7.9    12.8 / 8.2    12.4 / 8.1     7.9 / 8.1    12.5 / 14.5
//   9 to 16         9.8 / 11.1    9.9 / 10.9   12.5 / 11.2    9.7 / 11.2   16.8 / 11.5   16.7 / 11.6    9.8 / 11.6   17.0 / 20.4
// and alike at K 64 to 6,144.  Up to 8 tokens it does for 148 blocks and fewer (up to 5 % behind where blocks are few), beyond them not
// (3,072 rows of K 1,024, 4 tokens 6.3 / 7.6); 9 to 16 tokens from 52 blocks on (44 and 48: 10 % ahead to 10 % behind), but not
// where a grid of 74 or 148 blocks is even by itself.  One and two tokens are up to 36 % ahead from 96 blocks on and up to 12 %
// behind below; they have not been given it yet.
constexpr unsigned EVEN_BLOCKS = 148;          // a block an SM
static bool few_looks_far(int MT, unsigned blocks) {
    return MT >= 4 && blocks <= EVEN_BLOCKS && (MT < 16 || (blocks >= 52 && blocks != EVEN_BLOCKS / 2 && blocks != EVEN_BLOCKS));
}

template <int MT>
int launch_few(const float* A, int lda, const float* W, int ldw, const float* bias, float* C, int ldc, int M, int N, int K, int epi,
               int settled, cudaStream_t st) {
    const unsigned y = (unsigned)((M + MT - 1) / MT);
    auto run = [&](auto nb, auto depth) {
        constexpr int NB = decltype(nb)::value, ST = decltype(depth)::value;
        return launch_f32(gemm_f32_few_kernel<MT, NB, ST>, dim3((N + NB - 1) / NB, y), NB * KPARTS, few_smem<MT, NB, ST>(), st, A, lda, W, ldw, bias, C, ldc, M, N, K, epi, settled);
    };
    using std::integral_constant;
    // blocks of 16 weight rows once they fill the SMs twice, else of 8
    if (N >= 16 * 296) return run(integral_constant<int, 16>(), integral_constant<int, 3>());
    if (few_looks_far(MT, (unsigned)(N + 7) / 8 * y)) return run(integral_constant<int, 8>(), integral_constant<int, 8>());
    return run(integral_constant<int, 8>(), integral_constant<int, 3>());
}

// More than 32 tokens: whether clusters are the faster kernel.  The chip takes 148 tiles of the kernel for many at a time (32 tokens x 64
// columns) and 70 clusters (64 x 64; 71 and 72 are seen to leave some for a second turn), so they lose where the 64 tokens
// put them into one more turn than their halves.  us, many / clusters, K 1,024:
//   columns      512           1,024         1,280         1,536         2,048         2,304
//   65 tokens    20.0 / 18.9   19.9 / 19.4   19.9 / 19.7                 20.2 / 19.7   20.1 / 25.8
//   200          19.9 / 19.5   20.0 / 20.0   20.0 / 27.9   37.1 / 28.9   38.6 / 38.1   38.9 / 43.6
//   280          19.9 / 20.0   20.0 / 29.1   38.3 / 29.6   38.6 / 38.9   38.9 / 45.9
//   300          20.2 / 20.0   37.1 / 29.3   38.6 / 30.1                 55.8 / 46.2   56.9 / 53.7
//   520          20.0 / 27.2   39.0 / 43.7   56.8 / 52.5   57.5 / 60.7   75.9 / 78.2
//   1,024        39.1 / 39.7   76.2 / 70.9   94.5 / 87.4                 133 / 131     151 / 147
// (K 3,072: 53.9 / 48.3 for 1,024 columns and 200 tokens, 53.8 / 70.2 for 280.)  From 2,304 columns on they are ahead for 300 tokens and
// more (up to 17 %) and far behind for 65 to 200.  Over 592 products of 64 to 2,048 columns, K 1,024 to 3,072, the choice is
// within 0.1 % of the better kernel on average and at most 4.1 % off; clusters throughout were 2.5 % off, at most 47 %.
// Short K does not pay for the cluster's barriers: at K 64 to 256 they are 3 to 127 % slower (39 % on average), at 512 up to 72 %
// except for a few of them (8 clusters and fewer: 3 to 19 % faster).
constexpr int NARROW_COLUMNS = 2048, NARROW_AT_ONCE = 70;
static bool clusters_are_faster(int M, int N, int K) {
    if (N > NARROW_COLUMNS || K < 512) return false;
    const long long cols = (N + NARROW_N - 1) / NARROW_N, tiles = cols * ((M + MANY_M - 1) / MANY_M), clusters = cols * ((M + NARROW_T - 1) / NARROW_T);
    if (K < 1024) return clusters <= 8;
    return tiles > 3 * EVEN_BLOCKS || clusters <= NARROW_AT_ONCE * ((tiles + EVEN_BLOCKS - 1) / EVEN_BLOCKS);
}

int launch_pieces(const float* A, int lda, const float* W, int ldw, const float* bias, float* C, int ldc, int M, int N, int K, int epi,
                  int settled, cudaStream_t st) {
    if (M <= 1) return launch_few<1>(A, lda, W, ldw, bias, C, ldc, M, N, K, epi, settled, st);
    if (M <= 2) return launch_few<2>(A, lda, W, ldw, bias, C, ldc, M, N, K, epi, settled, st);
    if (M <= 4) return launch_few<4>(A, lda, W, ldw, bias, C, ldc, M, N, K, epi, settled, st);
    if (M <= 8) return launch_few<8>(A, lda, W, ldw, bias, C, ldc, M, N, K, epi, settled, st);
    if (M <= (N >= WIDE_COLUMNS ? FEW_TOKENS_WIDE : FEW_TOKENS)) return launch_few<16>(A, lda, W, ldw, bias, C, ldc, M, N, K, epi, settled, st);
    // a grid has at most 65,535 rows of blocks, half as many tokens here as the 64-row tiles of the general kernel take
    const bool narrow = clusters_are_faster(M, N, K);
    constexpr int ROWS = 65535 * MANY_M;
    for (long long m = 0; m < M; m += ROWS) {
        const int rows = M - m < ROWS ? (int)(M - m) : ROWS;
        const float* a = A + (size_t)m * lda;
        float* c = C + (size_t)m * ldc;
        const int rc = narrow ? launch_f32(gemm_f32_narrow_kernel, dim3((N + NARROW_N - 1) / NARROW_N * NARROW_CLUSTER, (rows + NARROW_T - 1) / NARROW_T), NARROW_PARTS * 64,
                                           NARROW_SMEM, st, a, lda, W, ldw, bias, c, ldc, rows, N, K, epi, settled)
                              : launch_f32(gemm_f32_many_kernel, dim3((N + MANY_N - 1) / MANY_N, (rows + MANY_M - 1) / MANY_M), KPARTS * 32, MANY_SMEM, st, a, lda, W, ldw,
                                           bias, c, ldc, rows, N, K, epi, settled);
        if (rc) return rc;
    }
    return 0;
}

template <typename TA, typename TW>
int launch(const void* A, int lda, const void* W, int ldw, const float* bias, void* C, int ldc, int M, int N, int K,
           int epi, cudaStream_t st) {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    const TA* a = (const TA*)A;
    const TW* w = (const TW*)W;
    switch (epi) {
        case 0: launch_kernel(gemm_simt_kernel<TA, TW, 0>, grid, 256, 0, st, a, lda, w, ldw, bias, C, ldc, M, N, K); break;
        case 1: launch_kernel(gemm_simt_kernel<TA, TW, 1>, grid, 256, 0, st, a, lda, w, ldw, bias, C, ldc, M, N, K); break;
        case 2: launch_kernel(gemm_simt_kernel<TA, TW, 2>, grid, 256, 0, st, a, lda, w, ldw, bias, C, ldc, M, N, K); break;
        case 3: launch_kernel(gemm_simt_kernel<TA, TW, 3>, grid, 256, 0, st, a, lda, w, ldw, bias, C, ldc, M, N, K); break;
        case 6: launch_kernel(gemm_simt_kernel<TA, TW, 6>, grid, 256, 0, st, a, lda, w, ldw, bias, C, ldc, M, N, K); break;
        case 7: launch_kernel(gemm_simt_kernel<TA, TW, 7>, grid, 256, 0, st, a, lda, w, ldw, bias, C, ldc, M, N, K); break;
        case 8: launch_kernel(gemm_simt_kernel<TA, TW, 8>, grid, 256, 0, st, a, lda, w, ldw, bias, C, ldc, M, N, K); break;
        case 9: launch_kernel(gemm_simt_kernel<TA, TW, 9>, grid, 256, 0, st, a, lda, w, ldw, bias, C, ldc, M, N, K); break;
        default: return fail("gemm: unknown epilogue %d", epi);
    }
    return check_launch("gemm_simt");
}

}  // namespace ember

using namespace ember;

// Whether a float32 product of few tokens, `mt` of them a block, looks eight stages ahead (host only).
EMBER_API int ember_gemm_f32_few_looks_far(int mt, int blocks) { return few_looks_far(mt, (unsigned)blocks) ? 1 : 0; }

// ... and whether one of more tokens goes to clusters.
EMBER_API int ember_gemm_f32_clusters(int M, int N, int K) { return clusters_are_faster(M, N, K) ? 1 : 0; }

EMBER_API int ember_gemm_simt(const void* A, int a_dtype, int lda, const void* W, int w_dtype, int ldw,
                              const float* bias, void* C, int ldc, int M, int N, int K, int epilogue, int settled, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return fail("gemm: K=%d", K);
    if (lda < K || ldw < K) return fail("gemm: row strides (%d, %d) smaller than K=%d", lda, ldw, K);
    const bool gated = epilogue == 3 || epilogue == 6 || epilogue == 7;
    if (gated && (N & 1)) return fail("gemm: the gated epilogue needs an even N, got %d", N);
    if (ldc < (gated ? N / 2 : N)) return fail("gemm: output stride %d too small for N=%d", ldc, N);
    if ((M + BM - 1) / BM > 65535) return fail("gemm: M=%d is too large for one launch", M);
    cudaStream_t st = (cudaStream_t)stream;
    const bool pieces = a_dtype == EMBER_F32 && w_dtype == EMBER_F32 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 &&
                        (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
    if (pieces) {
        if (epilogue != 0 && epilogue != 1 && epilogue != 2 && epilogue != 3 && !(epilogue >= 6 && epilogue <= 9))
            return fail("gemm: unknown epilogue %d", epilogue);
        return launch_pieces((const float*)A, lda, (const float*)W, ldw, bias, (float*)C, ldc, M, N, K, epilogue, settled, st);
    }
    if (a_dtype == EMBER_F32 && w_dtype == EMBER_F32)
        return launch<float, float>(A, lda, W, ldw, bias, C, ldc, M, N, K, epilogue, st);
    if (a_dtype == EMBER_F32 && w_dtype == EMBER_BF16)
        return launch<float, __nv_bfloat16>(A, lda, W, ldw, bias, C, ldc, M, N, K, epilogue, st);
    if (a_dtype == EMBER_BF16 && w_dtype == EMBER_F32)
        return launch<__nv_bfloat16, float>(A, lda, W, ldw, bias, C, ldc, M, N, K, epilogue, st);
    if (a_dtype == EMBER_BF16 && w_dtype == EMBER_BF16)
        return launch<__nv_bfloat16, __nv_bfloat16>(A, lda, W, ldw, bias, C, ldc, M, N, K, epilogue, st);
    return fail("gemm: unsupported dtypes %d/%d", a_dtype, w_dtype);
}
