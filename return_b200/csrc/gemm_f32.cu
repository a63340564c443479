// True float32 matrix product for the 32-bit path: C[M,N] = A[M,K] * W[N,K]^T.
//
// FFMA on the CUDA cores only: no tensor-core instruction, so no TF32 anywhere.  Every output
// element is accumulated over k = 0 .. K-1 in ascending order by one thread, so its value
// does not depend on M, on the row's place in the batch, on the launch shape, or on which of the
// kernels below computed it.
#include "common.cuh"

namespace {

__device__ __forceinline__ float4 ld4_guarded(const float* p, int left) {      // `left`: elements that exist from p on
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (left > 0) v.x = p[0];
    if (left > 1) v.y = p[1];
    if (left > 2) v.z = p[2];
    if (left > 3) v.w = p[3];
    return v;
}

__device__ __forceinline__ void cp16_zfill(float* smem, const float* gmem, int bytes) {       // bytes behind `bytes` become zero
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }

// ---------------------------------------------------------------- tiles: five rows and more
// A CTA computes BM x BN outputs, a thread TM x TN of them from registers, a warp (four lanes by eight) 4 TM x 8 TN.  Rows of
// both operands lie in shared memory as they do in memory, 32 values of k a stage, 36 floats apart: a thread takes four values
// of k of a row in one 16-byte read, the four (eight) rows that one such read of a warp touches fall on different banks, and
// the stages come by cp.async, STAGES - 1 in flight, without a register.  What bounds it is what shared memory hands to the
// registers, 32 floats a cycle and SM: TM TN / (TM + TN) FFMAs a float, which is the FFMA pipe's 128 a cycle for 8 x 8 outputs
// a thread and a third of it for 4 x 2.  Measured on a B200 (the FFMA pipe alone gives 64-70 TFLOP/s, one or two values an
// instruction alike): 2,048 x 24,576 x 4,096 45 TFLOP/s; 257 x (4,096 | 6,144) x 1,024 85 and 114 us, 257 x 1,024 x
// (2,048 | 3,072) 51 and 76 us, together 326 us where 64 x 64 tiles with one stage and 4-byte copies took 935.  Transposing
// into k-major stages through registers, with fragments read a group ahead, was no faster (8.7-9.3 ms, 86, 116, 55, 82 us).
constexpr int BK = 32, PITCH = BK + 4;

template <int BM, int BN, int TM, int TN, int STAGES>
__global__ void __launch_bounds__(BM * BN / (TM * TN))
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                int M, int N, int K, int lda, int ldw, int ldc, int vec) {
    constexpr int THREADS = BM * BN / (TM * TN);
    constexpr int COPIES = (BM + BN) * (BK / 4) / THREADS;
    constexpr int WARPS_N = BN / (8 * TN);
    static_assert(BM % (4 * TM) == 0 && BN % (8 * TN) == 0 && (BM + BN) * (BK / 4) % THREADS == 0, "whole warps and copies");
    extern __shared__ __align__(16) float tile_smem[];     // [stage][BM rows of A, then BN rows of W][PITCH]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int wm = (warp / WARPS_N) * (4 * TM) + (lane >> 3), wn = (warp % WARPS_N) * (8 * TN) + (lane & 7);
    const int steps = (K + BK - 1) / BK;
    pdl_wait();

    auto fetch = [&](int step) {
        float* stage = tile_smem + (step % STAGES) * (BM + BN) * PITCH;
#pragma unroll
        for (int i = 0; i < COPIES; ++i) {
            const int e = tid + i * THREADS, row = e / (BK / 4), k = step * BK + (e % (BK / 4)) * 4;
            const bool is_a = row < BM;
            const int r = is_a ? m0 + row : n0 + row - BM;
            const bool live = r < (is_a ? M : N) && k < K;
            const float* src = is_a ? A + (size_t)r * lda + k : W + (size_t)r * ldw + k;
            float* dst = stage + row * PITCH + (e % (BK / 4)) * 4;
            if (vec) cp16_zfill(dst, live ? src : W, live ? 16 : 0);
            else *reinterpret_cast<float4*>(dst) = live ? ld4_guarded(src, K - k) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < steps) fetch(s);
        cp_commit();
    }

    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2));
        __syncthreads();                                   // this stage is there, and the one before it has been used
        if (step + STAGES - 1 < steps) fetch(step + STAGES - 1);
        cp_commit();
        const float* a_s = tile_smem + (step % STAGES) * (BM + BN) * PITCH + wm * PITCH;
        const float* w_s = tile_smem + (step % STAGES) * (BM + BN) * PITCH + (BM + wn) * PITCH;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            float4 a[TM], b[TN];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4*>(w_s + 8 * j * PITCH + k);
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(a_s + 4 * i * PITCH + k);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
        }
    }
    pdl_trigger_late();
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + wm + 4 * i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + wn + 8 * j;
            if (n < N) C[(size_t)m * ldc + n] = acc[i][j];
        }
    }
}

template <int BM, int BN, int TM, int TN, int STAGES>
int launch_tiles(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int vec, cudaStream_t st) {
    const size_t smem = (size_t)STAGES * (BM + BN) * PITCH * sizeof(float);
    static PerDevice configured;
    const int rc = configured.once([&](int) {
        return cudaFuncSetAttribute(gemm_f32_kernel<BM, BN, TM, TN, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    });
    if (rc) return rc;
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    return rb_launch_pdl(gemm_f32_kernel<BM, BN, TM, TN, STAGES>, grid, dim3(BM * BN / (TM * TN)), smem, st, A, W, C, M, N, K, lda, ldw, ldc, vec);
}

// ---------------------------------------------------------------- up to four rows
// A lane owns one weight row (an output column), a warp half of the rows of A; every product's sum is a chain over k, so the
// chain's latency and the stream of weights bound it, not the arithmetic.  Stages of 32 weight rows by 128 k come by cp.async
// (four in flight); a lane reads its row 16 bytes at a time (rows 132 floats apart: conflict-free), the rows of A are broadcasts.
// 3 x 4,096 x 1,024: 16.9 us against 26.1 with 32 x 64 tiles; from five rows on the tiles are as fast (26 against 27 us for eight).
constexpr int THIN_ROWS = 4, THIN_BN = 32, THIN_BK = 128, THIN_STAGES = 4, THIN_THREADS = 64, THIN_PITCH = THIN_BK + 4;

template <int MR>
__global__ void __launch_bounds__(THIN_THREADS)
gemm_f32_thin_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                     int M, int N, int K, int lda, int ldw, int ldc, int vec) {
    constexpr int ROWS = 2 * MR;
    extern __shared__ __align__(16) float thin_smem[];     // [stage][32 weight rows, then ROWS rows of A][THIN_PITCH]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n0 = blockIdx.x * THIN_BN;
    auto fetch = [&](int step) {
        float* stage = thin_smem + (size_t)(step % THIN_STAGES) * (THIN_BN + ROWS) * THIN_PITCH;
        const int k0 = step * THIN_BK;
        for (int e = tid; e < (THIN_BN + ROWS) * (THIN_BK / 4); e += THIN_THREADS) {
            const int row = e / (THIN_BK / 4), k = k0 + (e % (THIN_BK / 4)) * 4;
            const bool is_w = row < THIN_BN;
            const int r = is_w ? n0 + row : row - THIN_BN;
            const bool live = r < (is_w ? N : M) && k < K;
            const float* src = is_w ? W + (size_t)r * ldw + k : A + (size_t)r * lda + k;
            float* dst = stage + row * THIN_PITCH + (k - k0);
            if (vec) cp16_zfill(dst, live ? src : W, live ? 16 : 0);
            else *reinterpret_cast<float4*>(dst) = live ? ld4_guarded(src, K - k) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    const int steps = (K + THIN_BK - 1) / THIN_BK;
    pdl_wait();
    for (int s = 0; s < THIN_STAGES - 1; ++s) {
        if (s < steps) fetch(s);
        cp_commit();
    }
    float acc[MR];
#pragma unroll
    for (int i = 0; i < MR; ++i) acc[i] = 0.f;
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(THIN_STAGES - 2));
        __syncthreads();                                   // this stage is there, and the one before it has been used
        if (step + THIN_STAGES - 1 < steps) fetch(step + THIN_STAGES - 1);
        cp_commit();
        const float* stage = thin_smem + (size_t)(step % THIN_STAGES) * (THIN_BN + ROWS) * THIN_PITCH;
        const float* w = stage + lane * THIN_PITCH;
        const float* a = stage + (THIN_BN + warp * MR) * THIN_PITCH;
        if (warp * MR < M) {
#pragma unroll 8
            for (int k = 0; k < THIN_BK; k += 4) {
                const float4 b = *reinterpret_cast<const float4*>(w + k);
#pragma unroll
                for (int i = 0; i < MR; ++i) {
                    const float4 v = *reinterpret_cast<const float4*>(a + i * THIN_PITCH + k);
                    acc[i] = fmaf(v.x, b.x, acc[i]);
                    acc[i] = fmaf(v.y, b.y, acc[i]);
                    acc[i] = fmaf(v.z, b.z, acc[i]);
                    acc[i] = fmaf(v.w, b.w, acc[i]);
                }
            }
        }
    }
    pdl_trigger_late();
    const int n = n0 + lane;
#pragma unroll
    for (int i = 0; i < MR; ++i) {
        const int m = warp * MR + i;
        if (m < M && n < N) C[(size_t)m * ldc + n] = acc[i];
    }
}

template <int MR>
int launch_thin(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int vec, cudaStream_t st) {
    const size_t smem = (size_t)THIN_STAGES * (THIN_BN + 2 * MR) * THIN_PITCH * sizeof(float);
    static PerDevice configured;
    const int rc = configured.once([&](int) {
        return cudaFuncSetAttribute(gemm_f32_thin_kernel<MR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    });
    if (rc) return rc;
    return rb_launch_pdl(gemm_f32_thin_kernel<MR>, dim3((N + THIN_BN - 1) / THIN_BN), dim3(THIN_THREADS), smem, st, A, W, C, M, N, K,
                         lda, ldw, ldc, vec);
}

// Which tiles: those with which the busiest SM is done first.  An SM's time is its tiles' outputs over what it gets through of
// that kind, measured in outputs a microsecond at K = 1,024 (one tile an SM / several): 128 x 128 146, 64 x 128 133, 64 x 64 92,
// 32 x 64 78 / 96.  So large tiles win where they fill the GPU (2,048 x 24,576 x 4,096: 9.2 ms against 13.1 with 32 x 64) and
// small ones where large ones would leave SMs idle (257 x 1,024 x 3,072: 76 us against 331).
struct TileKind { int bm, bn, alone, among; };
constexpr TileKind KINDS[4] = {{128, 128, 146, 146}, {64, 128, 133, 133}, {64, 64, 92, 92}, {32, 64, 78, 96}};

int pick(int M, int N, int sms) {
    int best = 0;
    double best_cost = 0.0;
    for (int i = 0; i < 4; ++i) {
        const TileKind& t = KINDS[i];
        const long long tiles = (long long)((M + t.bm - 1) / t.bm) * ((N + t.bn - 1) / t.bn), rounds = (tiles + sms - 1) / sms;
        const double cost = (double)rounds * t.bm * t.bn / (rounds > 1 ? t.among : t.alone);
        if (i == 0 || cost < best_cost) { best = i; best_cost = cost; }
    }
    return best;
}

}  // namespace

// kind: -1 the engine's choice; 0..3 a tile kind, 4 the kernel for few rows (measurements and tests; any choice gives the same bits)
RB_EXPORT int rb_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K,
                          int lda, int ldw, int ldc, int kind, cudaStream_t st) {
    if (M <= 0 || N <= 0) return 0;
    const int vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
    const int sms = rb_num_sms();
    if (sms <= 0) return (int)cudaErrorInvalidDevice;
    if (kind < 0) {
        kind = M <= THIN_ROWS ? 4 : pick(M, N, sms);
        // blockIdx.y ends at 65,535: more rows than that many tiles go to the tallest
        if (kind < 4 && (M + KINDS[kind].bm - 1) / KINDS[kind].bm > 65535) kind = 0;
    }
    switch (kind) {
        case 0: return launch_tiles<128, 128, 8, 8, 3>(A, W, C, M, N, K, lda, ldw, ldc, vec, st);
        case 1: return launch_tiles<64, 128, 8, 4, 4>(A, W, C, M, N, K, lda, ldw, ldc, vec, st);
        case 2: return launch_tiles<64, 64, 8, 4, 4>(A, W, C, M, N, K, lda, ldw, ldc, vec, st);
        case 3: return launch_tiles<32, 64, 4, 2, 5>(A, W, C, M, N, K, lda, ldw, ldc, vec, st);
        case 4: break;
        default: return (int)cudaErrorInvalidValue;
    }
    if (M > THIN_ROWS) return (int)cudaErrorInvalidValue;
    if (M <= 2) return launch_thin<1>(A, W, C, M, N, K, lda, ldw, ldc, vec, st);
    return launch_thin<2>(A, W, C, M, N, K, lda, ldw, ldc, vec, st);
}
