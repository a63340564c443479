// The experts' products of a step on the fifth-generation tensor cores: C[place, n] = sum_k A[place, k] W[e][n, k] over the
// (token, expert) pairs in the order of their experts (A holds their rows in that order), bfloat16 with float32 accumulation in
// tensor memory, operands by TMA.  Optionally the gated unit of the experts in the epilogue: W[e] then holds F gate rows and F up
// rows, and C[place, f] = g sigmoid(alpha g) (u + shift) of the two sums, capped (moe.cu, clamped_glu), so that the [places, 2F]
// intermediate is neither written nor read.
//
// The operands' roles are exchanged: an expert's weight rows are the M side of the MMA (256 a tile, by a pair of CTAs on
// neighbouring SMs with the two-SM form, cta_group::2: each CTA holds 128 of them, and their accumulators lie on its 128 TMEM
// lanes), the expert's places are the N side, of any multiple of 32 up to 256.  A run of n places is cut into as few tiles as
// possible, all of about the same width, so what a tile computes beside its places is at most 31 columns.  (With the places as M, a
// tile of 128 rows or a part of one: 25 % of the products of 32 experts and 8,192 pairs were of rows behind a run's end, and each CTA
// loaded 48 KB a k block where a pair loads 32 KB a CTA.)  Each CTA of a pair brings its weight rows and half of the places.
//
// Producer thread, MMA thread (of the even CTA, the leader), ring of stages, two accumulators: as in the pair kernel of
// gemm_tc5.cu.  The accumulators come out with a weight row a lane, so the epilogue turns blocks of 32 places by 32 rows round
// through shared memory before it stores them: neighbouring lanes then hold neighbouring columns of one place.  With the gated
// unit, gate rows lie on lanes 0-63 and their up rows on lanes 64-127: two warps exchange halves of each block and each does half
// of the units.  How many tiles there are follows from the router's choice, which only the device knows: every CTA works the
// list out from the offsets of the runs.
//
// Every mbarrier wait is bounded; a wait that gives up raises *status and the kernel still frees its tensor memory.
// Bound by the weights' and rows' way in: a pair's tile of 256 rows by 131 places loads half as many bytes an MMA again as one by 256,
// and the weights (402 + 201 MB below) come from HBM.  Measured (8,192 pairs on 32 experts, H = 2,048, F = 1,536): 131 us gated and 59-70 us
// down (the kernel with places as M, and a pass for the units: 199 and 22 us together).  With few and small tiles what counts is the set-up (the
// pair's barrier stands in front of the wait for the kernels before this one) and the last tile's epilogue, which nothing hides: 1,024 pairs on 16 experts
// of 1,024 x 768 take 57 us with everything around them, 61 before those two were looked at, 55 with places as M; 8,160 pairs 111, 118, 109.
// Boxes of 64 places instead of 32 took 8 % longer; asking the weights into L2 4 / 10 / 20 stages ahead, by TMA or by a warp of
// prefetches, 3 / 9 / 20 % and 2 / 6 / 28 % longer.
#include <cuda.h>

#include "tc5.cuh"
#include "tma.cuh"

namespace {

using namespace tc5;

constexpr int BK = 64;                    // bf16 elements: one 128-byte swizzle row
constexpr int BM = 128;                   // weight rows of a CTA
constexpr int MAX_BN = 256;               // places of a tile at most
constexpr int BOX = 64;                   // weight rows of a TMA box
constexpr int PBOX = 32;                  // places of a TMA box
constexpr int KPS = 2;                    // k blocks of 64 a stage
constexpr int STAGES = 3;
constexpr int SETS = 2;                   // sets of four epilogue warps: they take blocks of 32 places in turn
constexpr int THREADS = 64 + 128 * SETS;  // warp 0: TMA, warp 1: MMA, then the epilogue
constexpr int MAX_EXPERTS = 1024;
constexpr unsigned A_BYTES = BM * BK * 2, B_BYTES = (MAX_BN / 2) * BK * 2, BLOCK_BYTES = A_BYTES + B_BYTES, STAGE_BYTES = KPS * BLOCK_BYTES;
constexpr unsigned TURN_BYTES = 32 * 64;                  // a warp's block of 32 places by 32 rows of bf16 that is turned round, or what its partner handed it
constexpr unsigned SMEM_BYTES = STAGES * STAGE_BYTES + 4 * SETS * TURN_BYTES + 1024;

struct Unit { float limit, alpha, shift; const float* weight; const int* pair_at; };      // the gated unit, and what multiplies a place's sums first

struct Tile {
    int e;         // expert
    int m0;        // first place (row of A and of C)
    int rows;      // places of the tile
    int bn;        // the MMA's N: rows rounded up to 32
    int nt;        // tile of weight rows
};

// Places of a tile of a run of n places, but for the last.
__device__ __forceinline__ int run_width(int n) {
    const int k = (n + MAX_BN - 1) / MAX_BN;
    return k == 0 ? 32 : ((n + k - 1) / k + 31) & ~31;
}

// Tiles are numbered with the tiles of all experts' places fastest: the weights of a block of output columns are read once,
// and the places' rows stay in L2 across the blocks.
__device__ __forceinline__ Tile locate(const int* s_start, const int* s_off, int E, int total_m, int tile) {
    Tile t;
    t.nt = tile / total_m;
    const int r = tile - t.nt * total_m;
    int lo = 0, hi = E;                                     // the last expert whose first tile is not behind r
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (s_start[mid] <= r) lo = mid; else hi = mid;
    }
    const int width = run_width(s_off[lo + 1] - s_off[lo]);
    t.e = lo;
    t.m0 = s_off[lo] + (r - s_start[lo]) * width;
    t.rows = min(width, s_off[lo + 1] - t.m0);
    t.bn = (t.rows + 31) & ~31;
    return t;
}

__device__ __forceinline__ void mbar_arrive_in_cluster(unsigned cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void load_pair(unsigned smem_dst, const CUtensorMap* map, int x, int y, unsigned bar_in_cluster) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_dst), "l"(map), "r"(x), "r"(y), "r"(bar_in_cluster) : "memory");
}
__device__ __forceinline__ void mma_ss_pair(unsigned d_tmem, unsigned long long a_desc, unsigned long long b_desc, unsigned idesc, bool accumulate) {
    asm volatile(
        "{\n.reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"((unsigned)accumulate) : "memory");
}
__device__ __forceinline__ void mma_commit_pair(unsigned bar) {          // one arrival on this barrier in both CTAs
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((unsigned short)3) : "memory");
}

// 32 places (or 16) by 32 weight rows, place j of this lane's row in v[j]: written to `turn` [place][32] and stored with
// neighbouring lanes on neighbouring columns.  `first`: output of the first place and of this warp's first row.
template <int N>
__device__ __forceinline__ void turn_and_store(unsigned char* turn, const float (&v)[N], bf16* first, int ldo, int rows, int cols, bool vec, int lane) {
    bf16* t = reinterpret_cast<bf16*>(turn);
    __syncwarp();                                           // the block before this one has been taken
#pragma unroll
    for (int j = 0; j < N; ++j) t[j * 32 + lane] = __float2bfloat16_rn(v[j]);
    __syncwarp();
    if (vec && cols >= 32) {                                // four lanes a place, eight places an instruction
#pragma unroll
        for (int j = 0; j < N; j += 8) {
            const int p = j + (lane >> 2);
            if (p < rows) *reinterpret_cast<uint4*>(first + (size_t)p * ldo + (lane & 3) * 8) = *reinterpret_cast<const uint4*>(t + p * 32 + (lane & 3) * 8);
        }
    } else {
#pragma unroll
        for (int j = 0; j < N; ++j)
            if (j < rows && lane < cols) first[(size_t)j * ldo + lane] = t[j * 32 + lane];
    }
}

template <int ACT>
__device__ __forceinline__ void activate_all(float (&v)[32]) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = rb_activate(ACT, v[j], nullptr, 0, 0);
}

// g sigmoid(alpha g) (u + shift) of the capped sums.  The quotient by 1 + exp(-alpha g) is a product with its reciprocal, put right by what
// is left over (one step of Newton's method): off by no more than a rounding or two, for a fraction of a rounded division's instructions.
__device__ __forceinline__ float gated(float g, float u, const Unit& unit) {
    g = fminf(g, unit.limit);
    u = fminf(fmaxf(u, -unit.limit), unit.limit);
    const float den = 1.0f + expf(-unit.alpha * g);
    float rec;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rec) : "f"(den));
    const float q = g * rec;
    return (den < 1e36f ? fmaf(fmaf(-q, den, g), rec, q) : q) * (u + unit.shift);       // behind that the remainder is lost, or NaN
}

template <bool GATED>
__global__ void __launch_bounds__(THREADS)
moe_tc5_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
               const int* __restrict__ offsets, int E, bf16* __restrict__ out, int N, int K, int ldo,
               int* __restrict__ status, int act, int vec, Unit unit) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* turns = base + STAGES * STAGE_BYTES;
    __shared__ __align__(8) unsigned long long full_bar[STAGES], empty_bar[STAGES], acc_full[2], acc_empty[2];
    __shared__ unsigned tmem_slot;
    __shared__ int s_start[MAX_EXPERTS + 1], s_off[MAX_EXPERTS + 1];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned rank = cluster_ctarank();                // 0: the leader
    const int pair = (int)blockIdx.x >> 1, pairs = (int)gridDim.x >> 1;
    constexpr unsigned TMEM_COLS = 2 * MAX_BN;
    constexpr int TILE_N = GATED ? BM : 2 * BM;             // output columns of a pair's tile
    const int nkb = (K + BK * KPS - 1) / (BK * KPS);        // stages a tile; k blocks past K are zero-filled by the copy

    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        tma::prefetch_desc(&map_a);
        tma::prefetch_desc(&map_w);
#pragma unroll
        for (int s = 0; s < STAGES; ++s) { mbar_init(smem_u32(&full_bar[s]), 1); mbar_init(smem_u32(&empty_bar[s]), 1); }
#pragma unroll
        for (int b = 0; b < 2; ++b) { mbar_init(smem_u32(&acc_full[b]), 1); mbar_init(smem_u32(&acc_empty[b]), 2 * 4 * SETS); }
        mbar_init_fence();
    }
    fence_before_sync();
    cluster_sync_all();                                     // both CTAs' barriers exist before either is signalled
    fence_after_sync();
    pdl_wait();                                             // the offsets and the rows come from the kernels before
    for (int e = tid; e <= E; e += THREADS) s_off[e] = offsets[e];
    __syncthreads();
    if (warp == 0) {                                        // first tile of every expert: sums over 32 experts at a time
        int run = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int e = e0 + lane, n = e < E ? s_off[e + 1] - s_off[e] : 0;
            const int own = n > 0 ? (n + run_width(n) - 1) / run_width(n) : 0;
            int upto = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += v;
            }
            if (e < E) s_start[e] = run + upto - own;
            run += __shfl_sync(0xffffffffu, upto, 31);
        }
        if (lane == 0) s_start[E] = run;
    }
    __syncthreads();
    const int total_m = s_start[E];
    const int tiles = total_m * ((N + TILE_N - 1) / TILE_N);
    const unsigned tacc = tmem_slot;
    bool ok = true;

    // this CTA's two boxes of weight rows: gate and up rows of 64 outputs, or 128 rows in a run
    auto first_row = [&](const Tile& t) { return GATED ? t.e * 2 * N + t.nt * TILE_N + (int)rank * BOX : t.e * N + t.nt * TILE_N + (int)rank * BM; };
    const int second = GATED ? N : BOX;

    if (warp == 0) {
        if (lane == 0) {                                    // ---- producer (both CTAs)
            int it = 0;                                     // stages filled so far, over all tiles
            for (int tile = pair; tile < tiles; tile += pairs) {
                const Tile t = locate(s_start, s_off, E, total_m, tile);
                const int w0 = first_row(t), w1 = w0 + second;
                const int half = t.bn >> 1, m = t.m0 + (int)rank * half, boxes = (half + PBOX - 1) / PBOX;
                const unsigned bytes = A_BYTES + (unsigned)boxes * (PBOX * BK * 2);
                for (int kb = 0; kb < nkb; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (it >= STAGES) ok = mbar_wait(smem_u32(&empty_bar[s]), ((it / STAGES) - 1) & 1) && ok;
                    const unsigned full_local = smem_u32(&full_bar[s]);
                    if (rank == 0) mbar_arrive_expect_tx(full_local, 2 * KPS * bytes);
                    const unsigned full = map_to_cta(full_local, 0);
                    const unsigned dst = smem_u32(base + (size_t)s * STAGE_BYTES);
#pragma unroll
                    for (int j = 0; j < KPS; ++j) {
                        const unsigned d = dst + j * BLOCK_BYTES;
                        const int x = (kb * KPS + j) * BK;
                        load_pair(d, &map_w, x, w0, full);
                        load_pair(d + BOX * BK * 2, &map_w, x, w1, full);
                        for (int b = 0; b < boxes; ++b) load_pair(d + A_BYTES + b * (PBOX * BK * 2), &map_a, x, m + b * PBOX, full);
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {                       // ---- MMA issuer (the leader)
            int it = 0, local = 0;
            for (int tile = pair; tile < tiles; tile += pairs, ++local) {
                const Tile t = locate(s_start, s_off, E, total_m, tile);
                const unsigned idesc = instr_desc_bf16(2 * BM, t.bn);
                const int buf = local & 1;
                if (local >= 2) ok = mbar_wait(smem_u32(&acc_empty[buf]), ((local >> 1) - 1) & 1) && ok;
                fence_after_sync();
                const unsigned d = tacc + buf * MAX_BN;
                for (int kb = 0; kb < nkb; ++kb, ++it) {
                    const int s = it % STAGES;
                    ok = mbar_wait(smem_u32(&full_bar[s]), (it / STAGES) & 1) && ok;
                    fence_after_sync();
                    const unsigned a0 = smem_u32(base + (size_t)s * STAGE_BYTES);
#pragma unroll
                    for (int j = 0; j < KPS; ++j) {
                        const unsigned a = a0 + j * BLOCK_BYTES, b = a + A_BYTES;
#pragma unroll
                        for (int k16 = 0; k16 < BK / 16; ++k16)
                            mma_ss_pair(d, smem_desc_sw128(a, k16 * 32), smem_desc_sw128(b, k16 * 32), idesc, kb > 0 || j > 0 || k16 > 0);
                    }
                    mma_commit_pair(smem_u32(&empty_bar[s]));   // the stage is free in both CTAs once these MMAs have read it
                }
                mma_commit_pair(smem_u32(&acc_full[buf]));      // both halves of this tile's accumulator are complete
            }
        }
    } else {                                                // ---- epilogue (both CTAs): TMEM lanes by warp % 4
        const int q = warp & 3, set = (warp - 2) >> 2;
        unsigned char* turn = turns + (set * 4 + q) * TURN_BYTES;
        float* inbox = reinterpret_cast<float*>(turn);      // [16 places][32 rows]: the partner's sums of the places that this warp does
        float* outbox = reinterpret_cast<float*>(turns + (set * 4 + (q ^ 2)) * TURN_BYTES);
        const int meet = 1 + set * 2 + (q & 1);             // the named barrier of the two
        const unsigned acc_empty_leader0 = map_to_cta(smem_u32(&acc_empty[0]), 0), acc_empty_leader1 = map_to_cta(smem_u32(&acc_empty[1]), 0);
        int local = 0;
        for (int tile = pair; tile < tiles; tile += pairs, ++local) {
            const Tile t = locate(s_start, s_off, E, total_m, tile);
            const int buf = local & 1;
            ok = mbar_wait(smem_u32(&acc_full[buf]), (local >> 1) & 1) && ok;
            if (tile + pairs >= tiles) pdl_trigger_late();                 // the last tile of this CTA
            fence_after_sync();
            // this warp's first output column, and how many of its 32 exist
            const int n0 = t.nt * TILE_N + (GATED ? (int)rank * BOX + (q & 1) * 32 : (int)rank * BM + q * 32), cols = min(32, N - n0);
#pragma unroll 1
            for (int c0 = 32 * set; c0 < t.rows; c0 += 32 * SETS) {
                unsigned r[32];
                tmem_ld32(tacc + ((unsigned)(q * 32) << 16) + buf * MAX_BN + c0, r);
                tmem_ld_wait();
                const int left = t.rows - c0;
                bf16* to = out + (size_t)(t.m0 + c0) * ldo + n0;
                if (GATED) {
                    // warps q and q + 2 hold gate and up sums of the same 32 units: the first does places 0-15 of the block, the
                    // second 16-31; each hands the other its sums of the places that are not its own.
                    const bool up = q >= 2;
                    const int p0 = up ? 16 : 0;
                    if (unit.weight != nullptr) {           // lane j: what multiplies the sums of place j of the block
                        const int place = t.m0 + c0 + lane;
                        const float c = lane < left ? unit.weight[unit.pair_at ? unit.pair_at[place] : place] : 1.f;
#pragma unroll
                        for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__shfl_sync(0xffffffffu, c, j) * __uint_as_float(r[j]));
                    }
                    asm volatile("bar.sync %0, 64;" ::"r"(meet) : "memory");         // the partner is done with its inbox
#pragma unroll
                    for (int j = 0; j < 16; ++j) outbox[j * 32 + lane] = __uint_as_float(r[up ? j : 16 + j]);
                    asm volatile("bar.sync %0, 64;" ::"r"(meet) : "memory");
                    float v[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const float mine = __uint_as_float(r[up ? 16 + j : j]), other = inbox[j * 32 + lane];
                        v[j] = gated(up ? other : mine, up ? mine : other, unit);
                    }
                    if (cols > 0) turn_and_store<16>(turn, v, to + (size_t)p0 * ldo, ldo, left - p0, cols, vec, lane);
                } else {
                    float v[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
                    // one look at which activation it is: a look a sum put the code of all four between any two sums, and fetching it
                    // cost 0.7 us a block even where there was none
                    if (act == ACT_RELU2) activate_all<ACT_RELU2>(v);
                    else if (act == ACT_TANH) activate_all<ACT_TANH>(v);
                    else if (act == ACT_GELU_TANH) activate_all<ACT_GELU_TANH>(v);
                    else if (act == ACT_SILU) activate_all<ACT_SILU>(v);
                    if (cols > 0) turn_and_store<32>(turn, v, to, ldo, left, cols, vec, lane);
                }
            }
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive_in_cluster(buf ? acc_empty_leader1 : acc_empty_leader0);   // this warp has drained its quarter
        }
    }
    if (!ok) atomicExch(status, 1);
    __syncwarp();
    fence_before_sync();
    cluster_sync_all();                                     // neither CTA leaves, or gives its tensor memory back, while the other works
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tacc), "r"(TMEM_COLS) : "memory");
}

template <bool GATED>
int launch(const void* A, int lda, const void* W, const int* offsets, int E, void* out, int ldo, int places, int N, int K, int act, int* status,
           const Unit& unit, cudaStream_t st) {
    CUtensorMap ma, mw;
    if (!tma::make_map_bf16(&ma, A, places, K, lda, PBOX) || !tma::make_map_bf16(&mw, W, E * N * (GATED ? 2 : 1), K, K, BOX)) return (int)cudaErrorInvalidValue;
    // pairs that the device holds at once (an SM whose neighbour is switched off takes none)
    static PerDevice configured;
    static int pairs_of_device[PerDevice::MAX_DEVICES] = {0};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const int rc = configured.once([&](int dev) {
        cudaError_t e = cudaFuncSetAttribute(moe_tc5_kernel<GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES);
        if (e != cudaSuccess) return e;
        int clusters = 0;
        e = cudaOccupancyMaxActiveClusters(&clusters, moe_tc5_kernel<GATED>, &cfg);
        if (e != cudaSuccess) return e;
        if (clusters < 1) return cudaErrorInvalidConfiguration;
        pairs_of_device[dev] = clusters;
        return cudaSuccess;
    });
    if (rc != 0) return rc;
    int dev = 0;
    cudaGetDevice(&dev);
    const long long n_tiles = (N + (GATED ? BM : 2 * BM) - 1) / (GATED ? BM : 2 * BM);
    const long long worst = ((long long)places / MAX_BN + E) * n_tiles;      // a run of n places has ceil(n / MAX_BN) tiles at most, none if it is empty
    const int resident = pairs_of_device[dev];
    cfg.gridDim = dim3(2 * (unsigned)(worst < resident ? worst : resident));
    cfg.stream = st;
    cfg.numAttrs = RB_PDL_MODE == 3 ? 1 : 2;
    const int vec = ldo % 8 == 0 && N % 8 == 0 && ((uintptr_t)out & 15) == 0;
    return (int)cudaLaunchKernelEx(&cfg, moe_tc5_kernel<GATED>, ma, mw, offsets, E, (bf16*)out, N, K, ldo, status, act, vec, unit);
}

bool fits(const void* A, int lda, const void* W, int E, int rows, int K) {
    return E > 0 && E <= MAX_EXPERTS && K > 0 && K % 8 == 0 && lda % 8 == 0 && ((uintptr_t)A % 16) == 0 && ((uintptr_t)W % 16) == 0 &&
           (long long)E * rows <= 0x7fffffffLL;
}

}  // namespace

// A [places, K] (the pairs' rows in the order of their experts), W [E, N, K] contiguous, offsets int32 [E + 1] on the
// device, out [places, N] bfloat16; act: -1, or the number of an activation (rb_activate) on the float32 sums.  status: one int in
// device memory, set to 1 if a wait inside the kernel gave up.
RB_EXPORT int rb_moe_tc5_gemm(const void* A, int lda, const void* W, const int* offsets, int E, void* out, int ldo, int places,
                              int N, int K, int act, int* status, cudaStream_t st) {
    if (places <= 0 || N <= 0) return 0;
    if (act > ACT_SILU || !fits(A, lda, W, E, N, K)) return (int)cudaErrorInvalidValue;
    return launch<false>(A, lda, W, offsets, E, out, ldo, places, N, K, act, status, Unit{}, st);
}

// The same with the gated unit: W [E, 2F, K] (F gate rows, then F up rows), out [places, F].  limit, alpha, shift, weight, pair_at: as
// in rb_clamped_glu.
RB_EXPORT int rb_moe_tc5_gated(const void* A, int lda, const void* W, const int* offsets, int E, void* out, int ldo, int places, int F,
                               int K, float limit, float alpha, float shift, const float* weight, const int* pair_at, int* status,
                               cudaStream_t st) {
    if (places <= 0 || F <= 0) return 0;
    if (!fits(A, lda, W, E, 2 * F, K)) return (int)cudaErrorInvalidValue;
    return launch<true>(A, lda, W, offsets, E, out, ldo, places, F, K, -1, status, Unit{limit, alpha, shift, weight, pair_at}, st);
}
