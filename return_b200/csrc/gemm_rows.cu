// out[M, N] = x[M, K] * W[N, K]^T for the rows of an ordinary step (tens to a few hundred of them) in bfloat16, float32 accumulation:
// tcgen05 with the operand roles exchanged (weight rows are the MMA's M side, 128 TMEM lanes; the step's rows its N side), operands by
// TMA, and K cut over the CTAs of a cluster where the output has too few tiles to fill the GPU.  Optionally the gated unit over
// woven gate/up rows of W, or an activation, on the float32 sums.
//
// Such a product takes a few microseconds, so what counts beside its bytes is what stands in front of and behind them: the set-up
// overlaps the kernel before (programmatic dependent launch), a stage's two operands are one TMA instruction each (boxes of 128 values of k: an
// instruction takes the TMA unit some 85 ns whatever it brings), and the tile is as wide as its rows, rounded up to 16.
// A tile's sums go through shared memory once: a lane holds a weight row, a row of the output wants neighbouring columns in
// neighbouring lanes.  In a cluster the CTA of rank r adds the shares of K up (in their order) for the rows r, r + SPLIT, ...
//
// Every mbarrier wait is bounded; a wait that gives up raises *status and the kernel still frees its tensor memory.
#include <cuda.h>

#include "tc5.cuh"
#include "tma.cuh"

namespace {

using namespace tc5;

constexpr int BM = 128;                    // weight rows of a tile
constexpr int BK = 64;                     // one 128-byte swizzle row
constexpr int KPS = 2;                     // blocks of k of a stage
constexpr int MAX_BN = 256, MAX_STAGES = 8;
constexpr unsigned RING = 196 * 1024;      // bytes for stages
constexpr unsigned TWO_AN_SM = 80 * 1024;  // of so many bytes no third CTA fits an SM
constexpr int THREADS = 384;               // warp 0: TMA, 1: MMAs, 4 to 11: accumulators; all of them at the end

__host__ __device__ constexpr unsigned stage_bytes(int bn) { return KPS * (unsigned)(BM + bn) * BK * 2; }

struct Args {
    void* out;
    int M, N, K, ldo;
    int bn, tile_m, stages;                // width of a tile (a multiple of 16), rows of a tile, stages of the ring
    int blocks;                            // blocks of k of a box: KPS, or 1 where K is no multiple of 64
    int out_f32, gated, act, vec;          // gated: 0, or 1 + the gate; act: -1, or the activation; vec: output rows of whole 16-byte pieces
    int* status;
    // FUSED only
    const float* ssq_in; int ssq_count;    // shares of sum(v^2) of every row of x, or null: the sums are multiplied by 1 / sqrt(sum / norm_dim + eps)
    int norm_dim; float eps;
    float* stream;                         // [M, N], or null: v = stream + sums goes back there; out gets v (offset + norm_w), ssq_out a
    const void* norm_w; int norm_w_dtype;  // tile's share of sum(v^2) (out and norm_w null: neither)
    float offset;
    float* ssq_out;
    int ld_sums;
};

__device__ __forceinline__ void load_box(unsigned smem_dst, const CUtensorMap* map, int x, int row, int block, unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(smem_dst), "l"(map), "r"(x), "r"(row), "r"(block), "r"(bar) : "memory");
}

// LS: log2 of the CTAs that share a tile's K.
// FUSED: the norm before the product and the residual add behind it are folded in, as gemm_skinny.cu does for few rows: a layer is two launches
// shorter, which is what bounds such a step launch by launch: 512 tokens through six layers of 1,024 x 3,072 643 -> 563 us, 100 and 8 decoded
// ones 729 -> 645; captured, 16 decoded tokens 264 -> 248, 64 371 -> 355, 128 509 -> 492.  The rows' factors are worked out by two warps while
// the others wait for the operands, the first rows of the stream are asked for before that, and a half warp has a row's 128 columns.
template <int LS, bool FUSED>
__global__ void __launch_bounds__(THREADS, 1)
gemm_rows_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const Args g) {
    constexpr int SPLIT = 1 << LS;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) unsigned long long full[MAX_STAGES], empty[MAX_STAGES], done;
    __shared__ unsigned tmem_slot;
    __shared__ float rstd_s[FUSED ? MAX_BN : 1];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = LS > 0 ? (int)cluster_ctarank() : 0;
    const int n0 = ((int)blockIdx.x >> LS) * BM, m0 = (int)blockIdx.y * g.tile_m;
    const int bn = g.bn, stages = g.stages;
    const unsigned sbytes = stage_bytes(bn);
    const int all = (g.K + BK * KPS - 1) / (BK * KPS), per = (all + SPLIT - 1) >> LS;      // stages of the whole K and of a CTA
    const int s_begin = min(all, rank * per), s_end = min(all, s_begin + per);
    const unsigned tmem_cols = bn <= 32 ? 32 : bn <= 64 ? 64 : bn <= 128 ? 128 : 256;

    if (warp == 1) tmem_alloc(smem_u32(&tmem_slot), tmem_cols);
    if (tid == 0) {
        tma::prefetch_desc(&map_w);
        tma::prefetch_desc(&map_x);
        for (int i = 0; i < stages; ++i) { mbar_init(smem_u32(&full[i]), 1); mbar_init(smem_u32(&empty[i]), 1); }
        mbar_init(smem_u32(&done), 1);
        mbar_init_fence();
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const unsigned tmem = tmem_slot;
    bool ok = true;
    pdl_wait();
    const int share = bn >> LS;                             // rows of the tile that a CTA finishes: m0 + (slot << LS | rank)
    const int end = min(g.M, m0 + g.tile_m);
    // FUSED: this thread's eight columns (the same in all of its rows), their norm weights and the first row's part of the stream
    const int fused_col = n0 + 8 * (tid & 15);
    float w8[8], next8[8];
    auto ask = [&](int slot) {
        const int row = m0 + (slot << LS | rank);
        if (slot < share && row < end && fused_col < g.N) {
            const float4* f = reinterpret_cast<const float4*>(g.stream + (size_t)row * g.N + fused_col);
            const float4 lo = f[0], hi = f[1];
            next8[0] = lo.x; next8[1] = lo.y; next8[2] = lo.z; next8[3] = lo.w; next8[4] = hi.x; next8[5] = hi.y; next8[6] = hi.z; next8[7] = hi.w;
        }
    };
    if (FUSED && g.stream != nullptr) {
        ask(tid >> 4);
        if (g.norm_w != nullptr) {
#pragma unroll
            for (int i = 0; i < 8; ++i) w8[i] = fused_col < g.N ? g.offset + load_as_f32(g.norm_w, g.norm_w_dtype, fused_col + i) : 0.f;
        }
    }

    if (warp == 0) {
        if (lane == 0) {                                    // ---- operands
            for (int i = s_begin; i < s_end; ++i) {
                const int it = i - s_begin, s = it % stages;
                if (it >= stages) ok = ok && mbar_wait(smem_u32(&empty[s]), ((it / stages) - 1) & 1);
                const unsigned bar = smem_u32(&full[s]), a = smem_u32(base) + s * sbytes, b = a + KPS * BM * BK * 2;
                mbar_arrive_expect_tx(bar, sbytes);
                if (g.blocks == KPS) {
                    load_box(a, &map_w, 0, n0, i * KPS, bar);
                    load_box(b, &map_x, 0, m0, i * KPS, bar);
                } else {
                    for (int j = 0; j < KPS; ++j) {
                        load_box(a + j * BM * BK * 2, &map_w, (i * KPS + j) * BK, n0, 0, bar);
                        load_box(b + j * bn * BK * 2, &map_x, (i * KPS + j) * BK, m0, 0, bar);
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {                                    // ---- MMAs
            const unsigned idesc = instr_desc_bf16(BM, bn);
            for (int i = s_begin; i < s_end; ++i) {
                const int it = i - s_begin, s = it % stages;
                ok = ok && mbar_wait(smem_u32(&full[s]), (it / stages) & 1);
                fence_after_sync();
                const unsigned a = smem_u32(base) + s * sbytes, b = a + KPS * BM * BK * 2;
#pragma unroll
                for (int j = 0; j < KPS; ++j)
#pragma unroll
                    for (int k16 = 0; k16 < BK / 16; ++k16)
                        mma_ss(tmem, smem_desc_sw128(a + j * BM * BK * 2, k16 * 32), smem_desc_sw128(b + j * bn * BK * 2, k16 * 32), idesc,
                               it > 0 || j > 0 || k16 > 0);
                mma_commit(smem_u32(&empty[s]));
            }
            mma_commit(smem_u32(&done));
        }
    } else if (warp >= 4) {
        ok = mbar_wait(smem_u32(&done), 0);
        fence_after_sync();
    } else if (FUSED && g.ssq_in != nullptr) {              // ---- the rows' factors
        for (int slot = tid - 64; slot < share; slot += 64) {
            const int row = m0 + (slot << LS | rank);
            float sum = 0.f;
            if (row < end) {
                const float* f = g.ssq_in + (size_t)row * g.ld_sums;
                for (int i = 0; i < g.ssq_count; ++i) sum += f[i];
            }
            rstd_s[slot] = 1.0f / sqrtf(sum / (float)g.norm_dim + g.eps);
        }
    }
    pdl_trigger_late();
    // ---- the sums to shared memory, over the stages: [share of K][row of this CTA's][weight row]
    __syncwarp();
    if (LS > 0) cluster_sync_all();                         // nobody's MMAs read them any more
    if (warp >= 4) {
        const int q = warp & 3;
        unsigned to[SPLIT];
#pragma unroll
        for (int r = 0; r < SPLIT; ++r) {
            const unsigned own = smem_u32(base) + (unsigned)(rank * share * BM + q * 32 + lane) * 4;
            to[r] = LS > 0 ? map_to_cta(own, r) : own;
        }
        for (int c0 = 32 * ((warp - 4) >> 2); c0 < bn; c0 += 64) {
            unsigned r[32];
            if (s_begin < s_end) {
                tmem_ld32(tmem + ((unsigned)(q * 32) << 16) + c0, r);
                tmem_ld_wait();
            } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) r[j] = 0u;
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                if (j >= 16 && c0 + 16 >= bn) break;        // (a tile may end behind half a block)
                const unsigned at = to[j & (SPLIT - 1)] + (unsigned)((c0 + j) >> LS) * (BM * 4);
                if (LS > 0) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(at), "r"(r[j]) : "memory");
                else asm volatile("st.shared.u32 [%0], %1;" ::"r"(at), "r"(r[j]) : "memory");
            }
        }
    }
    __syncwarp();
    if (LS > 0) cluster_sync_all();
    else __syncthreads();
    const float* sums = reinterpret_cast<const float*>(base);
    auto eight = [&](int slot, int c, float (&v)[8]) {      // columns 8 c .. 8 c + 7 of a row, the shares of K added up
#pragma unroll
        for (int p = 0; p < SPLIT; ++p) {
            const float4* f = reinterpret_cast<const float4*>(sums + ((size_t)p * share + slot) * BM + 8 * c);
            const float4 lo = f[0], hi = f[1];
            if (p == 0) {
                v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w; v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
            } else {
                v[0] += lo.x; v[1] += lo.y; v[2] += lo.z; v[3] += lo.w; v[4] += hi.x; v[5] += hi.y; v[6] += hi.z; v[7] += hi.w;
            }
        }
    };
    const int width = g.gated ? g.N >> 1 : g.N;             // columns of the output
    auto store = [&](int row, int col, const float (&v)[8]) {
        const size_t at = (size_t)row * g.ldo + col;
        if (g.vec && col + 8 <= width) {
            if (g.out_f32) {
                float4* o = reinterpret_cast<float4*>((float*)g.out + at);
                o[0] = make_float4(v[0], v[1], v[2], v[3]);
                o[1] = make_float4(v[4], v[5], v[6], v[7]);
            } else {
                uint4 o;
                __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
                for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
                *reinterpret_cast<uint4*>((bf16*)g.out + at) = o;
            }
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (col + i < width) {
                    if (g.out_f32) ((float*)g.out)[at + i] = v[i];
                    else ((bf16*)g.out)[at + i] = __float2bfloat16_rn(v[i]);
                }
            }
        }
    };
    if (FUSED && g.stream != nullptr) {
        for (int slot = tid >> 4; slot < share; slot += THREADS / 16) {          // a half warp has the whole of a row's columns
            const int row = m0 + (slot << LS | rank);
            const bool live = row < end && fused_col < g.N;
            float v[8], had[8], ss = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) had[i] = next8[i];
            ask(slot + THREADS / 16);
            if (live) {
                eight(slot, tid & 15, v);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    v[i] = g.ssq_in ? had[i] + v[i] * rstd_s[slot] : had[i] + v[i];
                    ss += v[i] * v[i];
                }
                float4* f = reinterpret_cast<float4*>(g.stream + (size_t)row * g.N + fused_col);
                f[0] = make_float4(v[0], v[1], v[2], v[3]);
                f[1] = make_float4(v[4], v[5], v[6], v[7]);
                if (g.norm_w != nullptr) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[i] *= w8[i];
                    store(row, fused_col, v);
                }
            }
            if (g.ssq_out != nullptr) {
                const unsigned half = 0xffffu << (lane & 16);
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(half, ss, o);
                if ((lane & 15) == 0 && row < end) g.ssq_out[(size_t)row * g.ld_sums + ((int)blockIdx.x >> LS)] = ss;
            }
        }
    } else if (g.gated) {
        for (int e = tid; e < share * (BM / 16); e += THREADS) {
            const int slot = e / (BM / 16), c = e % (BM / 16), row = m0 + (slot << LS | rank), col = (n0 >> 1) + 8 * c;
            if (row >= end || col >= width) continue;
            float gate[8], up[8], v[8];
            eight(slot, 2 * c, gate);
            eight(slot, 2 * c + 1, up);
            if (FUSED && g.ssq_in != nullptr) {
#pragma unroll
                for (int i = 0; i < 8; ++i) { gate[i] *= rstd_s[slot]; up[i] *= rstd_s[slot]; }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = gate[i] / (1.0f + expf(-rb_gate_arg(g.gated - 1, gate[i]))) * up[i];
            store(row, col, v);
        }
    } else {
        for (int e = tid; e < share * (BM / 8); e += THREADS) {
            const int slot = e / (BM / 8), c = e % (BM / 8), row = m0 + (slot << LS | rank), col = n0 + 8 * c;
            if (row >= end || col >= width) continue;
            float v[8];
            eight(slot, c, v);
            if (FUSED && g.ssq_in != nullptr) {
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] *= rstd_s[slot];
            }
            if (g.act >= 0) {
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = rb_activate(g.act, v[i], nullptr, 0, 0);
            }
            store(row, col, v);
        }
    }
    if (!ok) atomicExch(g.status, 1);
    __syncwarp();
    fence_before_sync();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, tmem_cols);
}

// Rows of `k` values, `box_rows` of them a box.
bool make_map(CUtensorMap* map, const void* p, int rows, int K, long long ld, int box_rows) {
    tma::EncodeTiledFn encode = tma::encode_fn();
    if (encode == nullptr) return false;
    const bool whole = K % BK == 0;
    const cuuint64_t dims[3] = {(cuuint64_t)(whole ? BK : K), (cuuint64_t)rows, (cuuint64_t)(whole ? K / BK : 1)}, strides[2] = {(cuuint64_t)ld * 2, BK * 2};
    const cuuint32_t box[3] = {BK, (cuuint32_t)box_rows, whole ? KPS : 1u}, one[3] = {1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(p), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int LS, bool FUSED>
int launch(const CUtensorMap& mw, const CUtensorMap& mx, const Args& g, unsigned smem, cudaStream_t st) {
    static PerDevice configured;
    const int rc = configured.once([&](int) {
        return cudaFuncSetAttribute(gemm_rows_kernel<LS, FUSED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(RING + 1024));
    });
    if (rc) return rc;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1 << LS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((g.N + BM - 1) / BM) << LS, (unsigned)((g.M + g.tile_m - 1) / g.tile_m));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = RB_PDL_MODE == 3 ? 1 : 2;
    return (int)cudaLaunchKernelEx(&cfg, gemm_rows_kernel<LS, FUSED>, mw, mx, g);
}

// CTAs that the device holds at once, by log2 of their cluster's size: 148 SMs hold 148 in pairs and 132 in fours.
bool resident(int (&ctas)[3]) {
    static PerDevice asked;
    static int of_device[PerDevice::MAX_DEVICES][3] = {};
    const int rc = asked.once([&](int dev) {
        of_device[dev][0] = rb_num_sms();
        of_device[dev][1] = rb_cluster_ctas((const void*)gemm_rows_kernel<1, false>, 2, THREADS, RING + 1024);
        of_device[dev][2] = rb_cluster_ctas((const void*)gemm_rows_kernel<2, false>, 4, THREADS, RING + 1024);
        return of_device[dev][0] < 1 ? cudaErrorInvalidDevice : cudaSuccess;
    });
    int dev = 0;
    if (rc || cudaGetDevice(&dev) != cudaSuccess) return false;
    for (int l = 0; l < 3; ++l) ctas[l] = of_device[dev][l];
    return true;
}

// Rows of a tile and CTAs of a cluster: the choice whose busiest SM is done first.
void pick(int M, int N, int K, const int (&ctas)[3], int* tiles_m, int* ls) {
    long long best = -1;
    const long long all = (K + BK * KPS - 1) / (BK * KPS), tiles_n = (N + BM - 1) / BM;
    const int least = (M + MAX_BN - 1) / MAX_BN;
    for (int t = least; t <= least + 7; ++t) {
        const int rows = (M + t - 1) / t, bn = (rows + 15) & ~15;
        if (t > least && (M + t - 2) / (t - 1) <= 32) break;      // narrower still gains nothing
        for (int l = 0; l < 3; ++l) {
            if (all >> l < 2 && l > 0) break;
            if (ctas[l] < 1) continue;
            const long long rounds = (tiles_n * t * (1 << l) + ctas[l] - 1) / ctas[l];
            const long long mma = 8 * (bn > 108 ? bn / 2 : 54) + 300, load = (BM + bn) * 6;
            const long long cost = rounds * (((all + (1 << l) - 1) >> l) * (mma > load ? mma : load) + 5000 + bn * 16 + (l > 0 ? 1500 : 0));
            if (best < 0 || cost < best) { best = cost; *tiles_m = t; *ls = l; }
        }
    }
}

// What the two entries share: the shape's choice, the maps, the launch.
template <bool FUSED>
int run(Args& g, const void* x, const void* w, int ldx, int ldw, int tiles, int ls, cudaStream_t st) {
    const int M = g.M, N = g.N, K = g.K;
    if (K <= 0 || K % 8 || ldx % 8 || ldw % 8 || ((uintptr_t)x % 16) || ((uintptr_t)w % 16)) return (int)cudaErrorInvalidValue;
    if (tiles < 0) {
        int ctas[3];
        if (!resident(ctas)) return (int)cudaErrorInvalidConfiguration;
        pick(M, N, K, ctas, &tiles, &ls);
    }
    if (tiles < 1 || ls < 0 || ls > 2 || tiles > 65535 || (M + tiles - 1) / tiles > MAX_BN) return (int)cudaErrorInvalidValue;
    g.tile_m = (M + tiles - 1) / tiles;
    g.bn = (g.tile_m + 15) & ~15;
    g.blocks = K % BK == 0 ? KPS : 1;
    const int all = (K + BK * KPS - 1) / (BK * KPS), per = (all + (1 << ls) - 1) >> ls;
    g.stages = (int)(RING / stage_bytes(g.bn));
    g.stages = g.stages > MAX_STAGES ? MAX_STAGES : g.stages;
    g.stages = g.stages > per ? per : g.stages;
    g.vec = g.ldo % 8 == 0 && ((uintptr_t)g.out % 16) == 0;
    unsigned smem = g.stages * stage_bytes(g.bn);
    if (smem < (unsigned)g.bn * BM * 4) smem = (unsigned)g.bn * BM * 4;               // the sums lie over the stages
    // CTAs of a cluster wait for each other while they hold tensor memory, so an SM takes no more of them than it has columns for: two of 256,
    // four of 128 (52 KB each at least, so no fifth fits), and five, which is all that their threads leave room for, of fewer.
    if (ls > 0 && g.bn > 128 && smem < TWO_AN_SM) smem = TWO_AN_SM;
    CUtensorMap mw, mx;
    if (!make_map(&mw, w, N, K, ldw, BM) || !make_map(&mx, x, M, K, ldx, g.bn)) return (int)cudaErrorInvalidValue;
    if (ls == 0) return launch<0, FUSED>(mw, mx, g, smem + 1024, st);
    return ls == 1 ? launch<1, FUSED>(mw, mx, g, smem + 1024, st) : launch<2, FUSED>(mw, mx, g, smem + 1024, st);
}

}  // namespace

// out: bfloat16, or float32 with out_f32.  gated: 1 + the number of a gate (W's rows woven in eights, out [M, N / 2]), or 0; act: an activation's
// number (rb_activate, without a bias), or -1.  tiles, ls: how many tiles M falls into and log2 of the CTAs that share K, or -1: the engine's
// choice.  status: one int in device memory, set to 1 if a wait inside the kernel gave up.
RB_EXPORT int rb_gemm_rows(const void* x, const void* w, void* out, int out_f32, int gated, int act, int M, int N, int K, int ldx, int ldw, int ldo,
                           int tiles, int ls, int* status, cudaStream_t st) {
    if (M <= 0 || N <= 0) return 0;
    if (gated && (N % 16 || gated < 0 || gated - 1 > GATE_GELU_TANH || act >= 0)) return (int)cudaErrorInvalidValue;
    if (act > ACT_NEG_EXP_EXP) return (int)cudaErrorInvalidValue;
    Args g = {};
    g.out = out; g.M = M; g.N = N; g.K = K; g.ldo = ldo; g.out_f32 = out_f32; g.gated = gated; g.act = act; g.status = status;
    return run<false>(g, x, w, ldx, ldw, tiles, ls, st);
}

// The product with the norm before it and the residual add behind it folded in (as rb_gemm_skinny_fused, for more rows).
// ssq_in [M, ld_sums]: ssq_count shares of sum(v^2) a row, or null.  stream [M, N] float32, or null: with it out is null (no next norm) or gets
// v (offset + norm_w) for the next product, and ssq_out [M, ld_sums] (or null) one share a tile of 128 columns.
RB_EXPORT int rb_gemm_rows_fused(const void* x, const void* w, void* out, int gated, int M, int N, int K, int ldx, int ldw, int ldo,
                                 const float* ssq_in, int ssq_count, int norm_dim, float eps, float* stream, const void* norm_w,
                                 int norm_w_dtype, float offset, float* ssq_out, int ld_sums, int tiles, int ls, int* status, cudaStream_t st) {
    if (M <= 0 || N <= 0) return 0;
    if (gated && (N % 16 || gated < 0 || gated - 1 > GATE_GELU_TANH || stream != nullptr)) return (int)cudaErrorInvalidValue;
    if (ssq_in != nullptr && (ssq_count < 1 || ssq_count > ld_sums || norm_dim < 1)) return (int)cudaErrorInvalidValue;
    if (stream == nullptr && (out == nullptr || norm_w != nullptr || ssq_out != nullptr)) return (int)cudaErrorInvalidValue;
    if (stream != nullptr && (N % 8 || ((uintptr_t)stream % 16) || (out == nullptr) != (norm_w == nullptr))) return (int)cudaErrorInvalidValue;
    if (ssq_out != nullptr && (N + BM - 1) / BM > ld_sums) return (int)cudaErrorInvalidValue;
    Args g = {};
    g.out = out; g.M = M; g.N = N; g.K = K; g.ldo = ldo; g.gated = gated; g.act = -1; g.status = status;
    g.ssq_in = ssq_in; g.ssq_count = ssq_count; g.norm_dim = norm_dim; g.eps = eps;
    g.stream = stream; g.norm_w = norm_w; g.norm_w_dtype = norm_w_dtype; g.offset = offset; g.ssq_out = ssq_out; g.ld_sums = ld_sums;
    return run<true>(g, x, w, ldx, ldw, tiles, ls, st);
}

// The engine's choice for a product, on the current device: tiles that M falls into, log2 of the CTAs that share K, CTAs of the grid, and how many of them
// the device holds at once.
RB_EXPORT int rb_gemm_rows_plan(int M, int N, int K, int* out) {
    int ctas[3];
    if (M <= 0 || N <= 0 || K <= 0 || !resident(ctas)) return (int)cudaErrorInvalidValue;
    pick(M, N, K, ctas, &out[0], &out[1]);
    out[2] = (out[0] * ((N + BM - 1) / BM)) << out[1];
    out[3] = ctas[out[1]];
    return 0;
}
