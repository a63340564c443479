// C[M,N] = A[M,K] * W[N,K]^T in float32 for sums of up to SHORT_K values: FFMA chains on the CUDA cores.
//
// The kernel of gemm_f32.cu pays some 7 us a round of tiles in front of and behind its products, which a short sum does not earn back (us, tensor cores /
// this): 2,048 x 4,096 x 64 52 / 33, x 96 65 / 45, 16 x 4,096 x 64 6.6 / 6.1.  Further on it depends on the number of rows (2,048 rows x 128
// 56 / 57, 257 x 128 10 / 14, 16 x 128 6.6 / 6.1), which must not choose: every element is accumulated over k = 0 .. K-1 in ascending
// order by one thread, so its value does not depend on M, on the row's place in the batch, or on which tile computed it.
//
// A CTA computes BM x BN outputs, a thread TM x TN of them from registers, a warp (four lanes by eight) 4 TM x 8 TN.  Rows of
// both operands lie in shared memory as they do in memory, 32 values of k a stage, 36 floats apart: a thread takes four values
// of k of a row in one 16-byte read, the four (eight) rows that one such read of a warp touches fall on different banks, and
// the stages come by cp.async, STAGES - 1 in flight, without a register.  What bounds it is what shared memory hands to the
// registers, 32 floats a cycle and SM: TM TN / (TM + TN) FFMAs a float, which is the FFMA pipe's 128 a cycle for 8 x 8 outputs
// a thread and a third of it for 4 x 2.
#include "common.cuh"

namespace {

constexpr int SHORT_K = 96, BK = 32, PITCH = BK + 4;

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

template <int BM, int BN, int TM, int TN, int STAGES>
__global__ void __launch_bounds__(BM * BN / (TM * TN))
gemm_f32_short_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
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
        return cudaFuncSetAttribute(gemm_f32_short_kernel<BM, BN, TM, TN, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    });
    if (rc) return rc;
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    return rb_launch_pdl(gemm_f32_short_kernel<BM, BN, TM, TN, STAGES>, grid, dim3(BM * BN / (TM * TN)), smem, st, A, W, C, M, N, K, lda, ldw, ldc, vec);
}

// Which tiles: those with which the busiest SM is done first.  An SM's time is its tiles' outputs over what it gets through of
// that kind, measured in outputs a microsecond at K = 1,024 (one tile an SM / several): 128 x 128 146, 64 x 128 133, 64 x 64 92, 32 x 64 78 / 96.
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

// Whether a product's sums are short; the choice looks at nothing that changes from step to step.
int rb_gemm_f32_short_takes(int K) { return K <= SHORT_K; }

// kind: -1 the engine's choice, otherwise its last two bits are a tile kind (any choice gives the same bits)
int rb_gemm_f32_short(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int kind, int sms, cudaStream_t st) {
    const int vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
    constexpr int MOST = 65535 * 32;                       // rows of a launch: its grid ends there with the lowest tiles
    for (long long m = 0; m < M; m += MOST) {
        const int rows = (int)(M - m < MOST ? M - m : MOST), k = kind < 0 ? pick(rows, N, sms) : kind & 3;
        const float* a = A + m * lda;
        float* c = C + m * ldc;
        const int rc = k == 0 ? launch_tiles<128, 128, 8, 8, 3>(a, W, c, rows, N, K, lda, ldw, ldc, vec, st)
                     : k == 1 ? launch_tiles<64, 128, 8, 4, 4>(a, W, c, rows, N, K, lda, ldw, ldc, vec, st)
                     : k == 2 ? launch_tiles<64, 64, 8, 4, 4>(a, W, c, rows, N, K, lda, ldw, ldc, vec, st)
                              : launch_tiles<32, 64, 4, 2, 5>(a, W, c, rows, N, K, lda, ldw, ldc, vec, st);
        if (rc) return rc;
    }
    return 0;
}
