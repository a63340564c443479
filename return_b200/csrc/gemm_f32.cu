// Matrix product of the 32-bit path: C[M,N] = A[M,K] * W[N,K]^T in float32's precision, on the fifth-generation tensor cores.
//
// Every operand is multiplied by 2^16 and split into three bfloat16 parts, 2^16 x = h + m + l, and six of the nine
// products are made (hh, hm, mh, hl, mm, lh; the other three are below 2^-24 of a product), each exactly, the largest in an
// accumulator of its own.  A tensor core's accumulator cuts off what it cannot hold instead of rounding, so it sums 128 values of k
// at most; from there on sums are made on the CUDA cores, which round to nearest.  An element's sum has one order: K is
// cut into four groups of whole blocks of 64, a group into runs of two blocks; runs are added up in their group and the four
// groups one behind the other.  So its value does not depend on M, on the row's place in the batch, on the launch shape, or on
// which of the shapes below computed it.  Error against 64 bits (2-norm over that of the result, normal operands): 1.3e-7 at K = 1,024,
// 1.4e-7 at 3,072, where a chain of FFMAs over k has 5.7e-7 and 9.9e-7.
//
// The factor is there for small operands: bfloat16 ends at 2^-133, where the last bits of a number below 2^-109 would lie; times 2^16
// the parts hold every bit of every float32.  (It takes the warps that split one more instruction a pair: 2,048 x 4,096 x 1,024 145 -> 153 us.)
// An infinity or a NaN has no parts, and neither has a number beyond 2^112, and sums end at 2^96: where a result is no finite
// number, it is made once more from the operands themselves, one FFMA behind the other over k.
#include <float.h>

#include "tc5.cuh"

namespace {

using namespace tc5;

// A CTA computes 128 columns of C (weight rows: the M side of the MMA, a TMEM lane each) by up to BN rows (the tokens: the N
// side), over all of K or, in a cluster of SPLIT CTAs, over its share of the groups.  Warps with fixed roles:
//   eight split  read float32 from memory (a block ahead, in registers) and write the parts as 128-byte-swizzled tiles;
//   eight read   the accumulators of a run and add them to the group's sums in registers (a lane a column of C);
//   one          thread issues the MMAs.
// The tokens' parts lie below each other, so that one MMA multiplies the weights' leading parts with all three of them (N = 3 BN),
// one the middle parts with two, one the last with one: three instructions for six products, which counts because an instruction
// takes 54 cycles at least.  Two stages of parts, two sets of accumulators.  A block of 64 takes a CTA 1.2 us at BN = 80 (2,048 x 4,096 x 1,024
// is six tiles one behind the other on an SM, 25.6 us each, 6.7 of them set-up and end), of which the tensor pipe works less than half (24 % of
// a launch of 257 x 4,096 x 1,024, ncu): bound by the warps that split, of which six more do not fit the registers.  The thread that issues the MMAs halves what its scheduler has left (measured with the warps' clocks), so no warp that splits shares it: 257 x 4,096 x
// 1,024 took 29.8 us with two of them there, and 37.8 with the path for ragged rows in the same loop, whose code then did not stay in
// the instruction cache.  Splitting by conversions, by integer rounding or by bfloat16-minus-float32 subtractions made no difference.
// Now 26.8 us (tiles of FFMAs: 86); 257 x 6,144 x 1,024 43 (128), 257 x 1,024 x 3,072 22 (77), 2,048 x 4,096 x 1,024 153 (397), 2,048 x 4,096 x
// 1,000, in pieces of four, 182 (409; one value at a time 311), x 3,001 673 (1,657),
// 3 x 8,192 x 1,024 11 (18), 16 x 1,024 x 3,072 13 (75).
constexpr int BK = 64;                     // values of k of a block: one 128-byte swizzle row of bfloat16
constexpr int BM = 128;                    // weight rows of a CTA
constexpr int RUN = 2;                     // blocks that one accumulator sums
constexpr int GROUPS = 4;                  // groups of blocks of one sum
constexpr int STAGES = 2;
constexpr float UP = 65536.f, DOWN = 1.f / (UP * UP);                      // what operands are multiplied by, and sums
constexpr unsigned long long UP2 = 0x4780000047800000ull;                 // UP twice
constexpr int CONV = 256, DRAIN = 256, W_DRAIN = 8, W_MMA = 16, THREADS = 19 * 32;

template <int BN> struct Shape {
    static constexpr unsigned A_BYTES = BM * BK * 2, B_BYTES = 3 * BN * BK * 2, STAGE_BYTES = 3 * A_BYTES + B_BYTES;
    static constexpr unsigned STASH_BYTES = BN * BM * 4, NEED_BYTES = STAGES * STAGE_BYTES + STASH_BYTES + 1024;
    // CTAs of a cluster wait for each other while they hold tensor memory, so they share an SM with no CTA of another stream's
    // kernel that might do the same: they ask for so much shared memory that none fits beside them.
    static constexpr unsigned ALONE_BYTES = 204 * 1024, CLUSTER_BYTES = NEED_BYTES > ALONE_BYTES ? NEED_BYTES : ALONE_BYTES;
    static constexpr int BUF = 3 * BN;                                     // columns of a set of accumulators
    static constexpr unsigned TMEM = 2 * BUF <= 128 ? 128 : 2 * BUF <= 256 ? 256 : 512;
    static constexpr int COLS = BN / 2;                                    // tokens of a warp that reads accumulators
    static constexpr int TASKS = BM * 8 / CONV + (BN * 8 + CONV - 1) / CONV;   // pieces of eight values a thread and block
    static_assert(BN % 16 == 0 && BUF <= 256 && GROUPS * (BN / 2) * BM * 4 <= STAGES * (int)STAGE_BYTES, "sizes of an MMA and of the exchange");
};

// What a row of both operands is: whole blocks of 64; whole pieces of four values, 16 bytes aligned like those; anything.
constexpr int ROW_WHOLE = 0, ROW_QUADS = 1, ROW_ANY = 2;

struct Args {
    const float* A; const float* W; float* C;
    int M, N, K, lda, ldw, ldc;
    int row;                               // ROW_WHOLE, ROW_QUADS or ROW_ANY
    int tile_m;                            // rows of C of a tile: at most BN
    int* status;
};

__device__ __forceinline__ void store_in_cluster(unsigned smem_addr, unsigned rank, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(map_to_cta(smem_addr, rank)), "f"(v) : "memory");
}
__device__ __forceinline__ void tmem_ld8(unsigned taddr, unsigned (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
// The middle parts come out negated: bfloat16 minus float32 is one instruction.
__device__ __forceinline__ void less(unsigned parts, float& x, float& y) {
    asm("{\n.reg .b16 lo, hi;\nmov.b32 {lo, hi}, %2;\nsub.rn.f32.bf16 %0, lo, %0;\nsub.rn.f32.bf16 %1, hi, %1;\n}" : "+f"(x), "+f"(y) : "r"(parts));
}
__device__ __forceinline__ void scaled_up(float& x, float& y) {          // times UP, both in one instruction
    asm("{\n.reg .b64 v;\nmov.b64 v, {%0, %1};\nmul.rn.f32x2 v, v, %2;\nmov.b64 {%0, %1}, v;\n}" : "+f"(x), "+f"(y) : "l"(UP2));
}
__device__ __forceinline__ unsigned upper(float x, float y) { return __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632); }
__device__ __forceinline__ void split(float x, float y, unsigned& h, unsigned& m, unsigned& l) {
    scaled_up(x, y);
    h = __byte_perm(__float_as_uint(x) + 0x8000u, __float_as_uint(y) + 0x8000u, 0x7632);
    less(h, x, y);
    m = upper(x, y);
    less(m, x, y);
    l = upper(x, y);
}

// A result that is no finite number, from the operands as they are.
__device__ __noinline__ float chain(const float* a, const float* w, int K) {
    float acc = 0.f;
    for (int k = 0; k < K; ++k) acc = fmaf(a[k], w[k], acc);
    return acc;
}

struct Piece { float4 lo, hi; };           // eight values of k of a row
__device__ __forceinline__ Piece whole_piece(const float* p) {
    return {*reinterpret_cast<const float4*>(p), *reinterpret_cast<const float4*>(p + 4)};
}
__device__ __forceinline__ Piece quads_of_piece(const float* p, int left) {      // `left`: values that exist from p on, a multiple of four
    const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
    return {left > 0 ? *reinterpret_cast<const float4*>(p) : none, left > 4 ? *reinterpret_cast<const float4*>(p + 4) : none};
}
__device__ __forceinline__ Piece part_of_piece(const float* p, int left) {
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = i < left ? p[i] : 0.f;
    return {make_float4(v[0], v[1], v[2], v[3]), make_float4(v[4], v[5], v[6], v[7])};
}

template <int BN, int SPLIT, int ROW>
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_kernel(const Args g) {
    using S = Shape<BN>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    float* stash = reinterpret_cast<float*>(base + STAGES * S::STAGE_BYTES);            // [token][weight row]: sums of the groups before
    __shared__ __align__(8) unsigned long long full[STAGES], empty[STAGES], acc_full[2], acc_empty[2];
    __shared__ unsigned tmem_slot;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = SPLIT > 1 ? (int)cluster_ctarank() : 0;
    const int n0 = ((int)blockIdx.x / SPLIT) * BM, m0 = (int)blockIdx.y * g.tile_m;
    const int rows = min(g.tile_m, g.M - m0);
    // this CTA's groups of blocks
    const int nb = (g.K + BK - 1) / BK, per = (nb + GROUPS - 1) / GROUPS;
    constexpr int MINE = GROUPS / SPLIT;
    const int g0 = rank * MINE;
    auto group_end = [&](int i) { return min(nb, (i + 1) * per); };
    const int b_begin = min(nb, g0 * per), b_end = group_end(g0 + MINE - 1);

    if (warp == W_MMA) tmem_alloc(smem_u32(&tmem_slot), S::TMEM);
    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < STAGES; ++i) { mbar_init(smem_u32(&full[i]), CONV / 32); mbar_init(smem_u32(&empty[i]), 1); }
#pragma unroll
        for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&acc_full[i]), 1); mbar_init(smem_u32(&acc_empty[i]), DRAIN / 32); }
        mbar_init_fence();
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const unsigned tmem = tmem_slot;
    bool ok = true;
    pdl_wait();

    constexpr int COLS = S::COLS;
    float sum[COLS];                                        // the readers' sums of the group at hand
    const int q = warp & 3, half = (warp - W_DRAIN) >> 2;
    const int wrow = q * 32 + lane;                         // a reader's weight row
    const bool reader = warp >= W_DRAIN && warp < W_MMA;
    if (!reader && warp != W_MMA) {                         // ---- split and store
        if (warp & 3) {                                     // (two warps of the MMA thread's scheduler stand idle)
        // A thread takes the same eight values of k of rows r0, r0 + 32, ...: first of the weights', then of the tokens'.  Rows that do not
        // exist stay zero: what comes of them is not stored.
        constexpr int ROWS = CONV / 8, W_TASKS = BM / ROWS;
        const int r0 = (warp < 4 ? warp - 1 : warp < 8 ? warp - 2 : warp - 11) * 4 + (lane >> 3), k0 = (lane & 7) * 8;
        const unsigned to0 = sw128_offset(r0, lane & 7);
        const float* w0 = g.W + (size_t)(n0 + r0) * g.ldw + k0;
        const float* a0 = g.A + (size_t)(m0 + r0) * g.lda + k0;
        const size_t w_step = (size_t)ROWS * g.ldw, a_step = (size_t)ROWS * g.lda;
        unsigned live = 0;                                  // a bit a row: it exists
#pragma unroll
        for (int u = 0; u < S::TASKS; ++u)
            live |= (u < W_TASKS ? n0 + r0 + ROWS * u < g.N : r0 + ROWS * (u - W_TASKS) < rows) ? 1u << u : 0u;
        Piece x[S::TASKS];
#pragma unroll
        for (int u = 0; u < S::TASKS; ++u) x[u] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
        auto fetch = [&](int u, int b) {
            const float* p = (u < W_TASKS ? w0 + u * w_step : a0 + (u - W_TASKS) * a_step) + b * BK;
            const int left = g.K - b * BK - k0;
            if (live >> u & 1) x[u] = ROW == ROW_WHOLE ? whole_piece(p) : ROW == ROW_QUADS ? quads_of_piece(p, left) : part_of_piece(p, left);
        };
        if (b_begin < b_end) {
#pragma unroll
            for (int u = 0; u < S::TASKS; ++u) fetch(u, b_begin);
        }
        for (int b = b_begin; b < b_end; ++b) {
            const int it = b - b_begin, s = it % STAGES;
            if (it >= STAGES) ok = ok && mbar_wait(smem_u32(&empty[s]), ((it / STAGES) - 1) & 1);
            unsigned char* stage = base + s * S::STAGE_BYTES + to0;
            const bool more = b + 1 < b_end;
#pragma unroll
            for (int u = 0; u < S::TASKS; ++u) {
                uint4 h, m, l;
                split(x[u].lo.x, x[u].lo.y, h.x, m.x, l.x);
                split(x[u].lo.z, x[u].lo.w, h.y, m.y, l.y);
                split(x[u].hi.x, x[u].hi.y, h.z, m.z, l.z);
                split(x[u].hi.z, x[u].hi.w, h.w, m.w, l.w);
                if (more) fetch(u, b + 1);
                const bool is_w = u < W_TASKS;
                if (is_w || BN % ROWS == 0 || r0 + ROWS * (u - W_TASKS) < BN) {
                    unsigned char* to = stage + (is_w ? ROWS * u * 128 : 3 * (int)S::A_BYTES + ROWS * (u - W_TASKS) * 128);
                    constexpr unsigned STEP_B = BN * BK * 2;
                    *reinterpret_cast<uint4*>(to) = h;
                    *reinterpret_cast<uint4*>(to + (is_w ? S::A_BYTES : STEP_B)) = m;
                    *reinterpret_cast<uint4*>(to + 2 * (is_w ? S::A_BYTES : STEP_B)) = l;
                }
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&full[s]));
        }
        }
    } else if (warp == W_MMA) {
        if (lane == 0) {                                    // ---- MMAs
            constexpr unsigned idesc3 = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(3 * BN >> 3) << 17) | ((unsigned)(BM >> 4) << 24);
            const unsigned idesc2 = instr_desc_bf16(BM, 2 * BN), idesc1 = instr_desc_bf16(BM, BN);
            int it = 0, run = 0;
            for (int i = g0; i < g0 + MINE; ++i) {
                for (int b = min(nb, i * per); b < group_end(i); b += RUN, ++run) {
                    const int buf = run & 1, last = min(b + RUN, group_end(i));
                    if (run >= 2) ok = ok && mbar_wait(smem_u32(&acc_empty[buf]), ((run >> 1) - 1) & 1);
                    fence_after_sync();
                    const unsigned d = tmem + buf * S::BUF;
                    for (int c = b; c < last; ++c, ++it) {
                        const int s = it % STAGES;
                        ok = ok && mbar_wait(smem_u32(&full[s]), (it / STAGES) & 1);
                        fence_after_sync();
                        const unsigned a = smem_u32(base + s * S::STAGE_BYTES), t = a + 3 * S::A_BYTES;
#pragma unroll
                        for (int k16 = 0; k16 < BK / 16; ++k16) {
                            const unsigned long long bd = smem_desc_sw128(t, k16 * 32);
                            mma_ss(d, smem_desc_sw128(a, k16 * 32), bd, idesc3, c > b || k16 > 0);
                            mma_ss(d + BN, smem_desc_sw128(a + S::A_BYTES, k16 * 32), bd, idesc2, true);
                            mma_ss(d + 2 * BN, smem_desc_sw128(a + 2 * S::A_BYTES, k16 * 32), bd, idesc1, true);
                        }
                        mma_commit(smem_u32(&empty[s]));
                    }
                    mma_commit(smem_u32(&acc_full[buf]));
                }
            }
        }
    } else {                                                // ---- read accumulators
        int run = 0;
        float* mine = stash + (size_t)half * COLS * BM + wrow;
        for (int i = g0; i < g0 + MINE; ++i) {
#pragma unroll
            for (int j = 0; j < COLS; ++j) sum[j] = 0.f;
            for (int b = min(nb, i * per); b < group_end(i); b += RUN, ++run) {
                const int buf = run & 1;
                ok = ok && mbar_wait(smem_u32(&acc_full[buf]), (run >> 1) & 1);
                fence_after_sync();
                const unsigned at = tmem + ((unsigned)(q * 32) << 16) + buf * S::BUF + half * COLS;
#pragma unroll
                for (int j = 0; j < COLS; j += 8) {
                    unsigned big[8], s1[8], s2[8];
                    tmem_ld8(at + j, big);
                    tmem_ld8(at + BN + j, s1);
                    tmem_ld8(at + 2 * BN + j, s2);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        sum[j + e] += __uint_as_float(big[e]) + (__uint_as_float(s2[e]) - __uint_as_float(s1[e]));
                }
                fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&acc_empty[buf]));
            }
            // the groups one behind the other; of a cluster's share the first of two waits beside the second
            if (SPLIT == 1) {
#pragma unroll
                for (int j = 0; j < COLS; ++j) mine[j * BM] = i > g0 ? mine[j * BM] + sum[j] : sum[j];
            } else if (i < g0 + MINE - 1) {
#pragma unroll
                for (int j = 0; j < COLS; ++j) mine[j * BM] = sum[j];
            }
        }
    }
    pdl_trigger_late();
    auto leave = [&](int t, int r, float v) {               // tile row t, weight row r of the tile
        const int n = n0 + r;
        if (t < rows && n < g.N) {
            v *= DOWN;
            if (!(fabsf(v) <= FLT_MAX)) v = chain(g.A + (size_t)(m0 + t) * g.lda, g.W + (size_t)n * g.ldw, g.K);
            g.C[(size_t)(m0 + t) * g.ldc + n] = v;
        }
    };
    if (SPLIT == 1) {
        __syncthreads();
#pragma unroll 1
        for (int e = tid; e < BN * BM; e += THREADS) leave(e / BM, e % BM, stash[e]);
    } else {
        // every CTA of the cluster adds the four groups up for its share of the tokens
        constexpr int SHARE = BN / SPLIT;
        float* inbox = reinterpret_cast<float*>(base);      // [group][token of the share][weight row], over the stages
        __syncwarp();
        cluster_sync_all();                                 // nobody's MMAs read them any more
        if (reader) {
#pragma unroll
            for (int j = 0; j < COLS; ++j) {
                const int t = half * COLS + j;
                const unsigned to = smem_u32(inbox + ((size_t)g0 * SHARE + t % SHARE) * BM + wrow);
                if (MINE == 2) {
                    store_in_cluster(to, t / SHARE, stash[(size_t)t * BM + wrow]);
                    store_in_cluster(to + SHARE * BM * 4, t / SHARE, sum[j]);
                } else {
                    store_in_cluster(to, t / SHARE, sum[j]);
                }
            }
        }
        __syncwarp();
        cluster_sync_all();
#pragma unroll 1
        for (int e = tid; e < SHARE * BM; e += THREADS) {
            float v = inbox[e];
#pragma unroll
            for (int i = 1; i < GROUPS; ++i) v += inbox[i * SHARE * BM + e];
            leave(rank * SHARE + e / BM, e % BM, v);
        }
    }
    if (!ok) atomicExch(g.status, 1);
    __syncwarp();
    fence_before_sync();
    __syncthreads();
    if (warp == W_MMA) tmem_dealloc(tmem, S::TMEM);
}

template <int BN, int SPLIT, int ROW>
int launch_as(const Args& g, cudaStream_t st) {
    constexpr unsigned smem = SPLIT > 1 ? Shape<BN>::CLUSTER_BYTES : Shape<BN>::NEED_BYTES;
    static PerDevice configured;
    const int rc = configured.once([&](int) {
        return cudaFuncSetAttribute(gemm_f32_kernel<BN, SPLIT, ROW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    });
    if (rc) return rc;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = SPLIT;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((g.N + BM - 1) / BM) * SPLIT, (unsigned)((g.M + g.tile_m - 1) / g.tile_m));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = RB_PDL_MODE == 3 ? 1 : 2;
    return (int)cudaLaunchKernelEx(&cfg, gemm_f32_kernel<BN, SPLIT, ROW>, g);
}

template <int BN, int SPLIT>
int launch(const Args& g, cudaStream_t st) {
    if (g.row == ROW_WHOLE) return launch_as<BN, SPLIT, ROW_WHOLE>(g, st);
    return g.row == ROW_QUADS ? launch_as<BN, SPLIT, ROW_QUADS>(g, st) : launch_as<BN, SPLIT, ROW_ANY>(g, st);
}

// Which shape: the one whose busiest SM is done first.  Measured, in units of 10 ns: what a CTA takes for a block of 64, for its set-up
// and end, and for the exchange of a cluster's sums.  One round of CTAs after the other: 240 of them take twice what 148 do
// (fewer than 148 where they come in clusters).
constexpr int WIDTHS[4] = {80, 64, 32, 16}, BLOCK_COST[4] = {108, 91, 74, 69}, FIXED_COST[4] = {670, 630, 450, 430}, SPLITS[3] = {1, 2, 4};
constexpr int EXCHANGE_COST = 120;

// CTAs that the device holds at once, by the place in SPLITS.
bool resident(int (&ctas)[3]) {
    static PerDevice asked;
    static int of_device[PerDevice::MAX_DEVICES][3] = {};
    const int rc = asked.once([&](int dev) {
        of_device[dev][0] = rb_num_sms();
        of_device[dev][1] = rb_cluster_ctas((const void*)gemm_f32_kernel<16, 2, ROW_WHOLE>, 2, THREADS, Shape<16>::CLUSTER_BYTES);
        of_device[dev][2] = rb_cluster_ctas((const void*)gemm_f32_kernel<16, 4, ROW_WHOLE>, 4, THREADS, Shape<16>::CLUSTER_BYTES);
        return of_device[dev][0] < 1 ? cudaErrorInvalidDevice : cudaSuccess;
    });
    int dev = 0;
    if (rc || cudaGetDevice(&dev) != cudaSuccess) return false;
    for (int l = 0; l < 3; ++l) ctas[l] = of_device[dev][l];
    return true;
}

int pick(int M, int N, int K, const int (&held)[3]) {
    int best = 0;
    long long best_cost = -1;
    const long long nb = (K + BK - 1) / BK, per = (nb + GROUPS - 1) / GROUPS;
    for (int kind = 0; kind < 12; ++kind) {
        if (held[kind % 3] < 1) continue;
        const int bn = WIDTHS[kind / 3], split = SPLITS[kind % 3];
        const long long tiles_m = (M + bn - 1) / bn, ctas = tiles_m * ((N + BM - 1) / BM) * split, rounds = (ctas + held[kind % 3] - 1) / held[kind % 3];
        const long long blocks = GROUPS / split * per < nb ? GROUPS / split * per : nb;
        const long long cost = rounds * (blocks * BLOCK_COST[kind / 3] + FIXED_COST[kind / 3] + (split > 1 ? EXCHANGE_COST : 0));
        if (best_cost < 0 || cost < best_cost) { best = kind; best_cost = cost; }
    }
    return best;
}

}  // namespace

// gemm_f32_short.cu: sums of few values
int rb_gemm_f32_short_takes(int K);
int rb_gemm_f32_short(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int kind, int sms, cudaStream_t st);

// kind: -1 the engine's choice; 0..11 a shape, 3 * (place in WIDTHS) + (place in SPLITS) (measurements and tests; any choice gives the same
// bits).  status: one int in device memory, set to 1 if a wait inside the kernel gave up.
RB_EXPORT int rb_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K,
                          int lda, int ldw, int ldc, int kind, int* status, cudaStream_t st) {
    if (M <= 0 || N <= 0) return 0;
    const bool quads = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
    const int row = !quads ? ROW_ANY : K % BK == 0 ? ROW_WHOLE : ROW_QUADS;
    const int sms = rb_num_sms();
    if (sms <= 0) return (int)cudaErrorInvalidDevice;
    if (kind >= 12) return (int)cudaErrorInvalidValue;
    if (rb_gemm_f32_short_takes(K)) return rb_gemm_f32_short(A, W, C, M, N, K, lda, ldw, ldc, kind, sms, st);
    constexpr int MOST = 65535 * 16;                        // rows of a launch: its grid ends there with the narrowest tiles
    for (long long m = MOST; m < M; m += MOST) {
        const int rc = rb_gemm_f32(A + m * lda, W, C + m * ldc, (int)(M - m < MOST ? M - m : MOST), N, K, lda, ldw, ldc, kind, status, st);
        if (rc) return rc;
    }
    if (M > MOST) M = MOST;
    if (kind < 0) {
        int held[3];
        if (!resident(held)) return (int)cudaErrorInvalidConfiguration;
        kind = pick(M, N, K, held);
    }
    const int bn = WIDTHS[kind / 3], tiles = (M + bn - 1) / bn;
    const Args g = {A, W, C, M, N, K, lda, ldw, ldc, row, (M + tiles - 1) / tiles, status};
    switch (kind) {
        case 0: return launch<80, 1>(g, st);
        case 1: return launch<80, 2>(g, st);
        case 2: return launch<80, 4>(g, st);
        case 3: return launch<64, 1>(g, st);
        case 4: return launch<64, 2>(g, st);
        case 5: return launch<64, 4>(g, st);
        case 6: return launch<32, 1>(g, st);
        case 7: return launch<32, 2>(g, st);
        case 8: return launch<32, 4>(g, st);
        case 9: return launch<16, 1>(g, st);
        case 10: return launch<16, 2>(g, st);
        default: return launch<16, 4>(g, st);
    }
}
