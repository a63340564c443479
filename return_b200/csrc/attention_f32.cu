// Paged causal attention of the 32-bit path for head sizes 32, 64, 96 and 128: the scheme of attention_simt.cu (tiles of 32 keys aligned to
// absolute positions, an online softmax a row, CTAs of up to 32 rows of neighbouring tokens that share a key/value head), its two
// products on the matrix instructions in float32's precision.
//
// Operands are multiplied by 2^16 and split into three bfloat16 parts (which then hold every bit of every float32, small ones too:
// bfloat16 ends at 2^-133), six of nine products are made (the rest is below 2^-24 of a product), the largest in an accumulator of its own;
// a tile's 128 products of a score, or 32 of an output, are summed there, all else on the CUDA cores,
// which round to nearest.  A row of the products is worked out by itself and in one order, so the result for a token does not
// depend on how the prompt was cut into steps or on what else is in the batch: it is bit-identical.  An infinity, a NaN or a number beyond 2^112 has no
// parts: where a score or an output's sum over a tile is no finite number, it is made again from the operands, one FFMA behind the
// other over what the row sees, so a value reaches only the rows that see it.
//
// Eight warps.  Scores: a warp a 16 x 8 part of rows by keys, K's parts made as they are read.  Softmax: a warp four rows, a lane a key,
// the rows' reductions in step.  Outputs: a warp up to two blocks of eight columns for all rows, V's parts made once, accumulators in registers.
// Bound by what a tile of 32 keys waits for one behind the other: three parts and three barriers, 3 us a tile (one token behind 2,000 walks 63
// tiles in 188 us), at half of the issue slots and 6.5 % of the tensor pipe (ncu).  Measured (16 query and 8 key/value heads of 128), us,
// attention_simt.cu / this: 257 tokens of three requests 67 / 46, 219 64 / 35, 1,000 420 / 222, one token behind 2,000 281 / 188 (the factor's part
// of it 2 to 9 %).  P's parts made by the softmax's warps, and two sets of
// score accumulators: 2 to 10 % slower.
#include <float.h>

#include "common.cuh"

namespace {

constexpr int ROWS = 32, KEYS = 32, WARPS = 8, RW = 4;
constexpr int SP = KEYS + 8;              // floats of a row of scores: eight-byte reads of four rows by four lanes hit all banks

constexpr float UP = 65536.f, DOWN = 1.f / (UP * UP);                  // what operands are multiplied by, and sums
constexpr unsigned long long UP2 = 0x4780000047800000ull;             // UP twice

struct Parts { unsigned h, m, l; };       // of two neighbouring values, the first in the low half
__device__ __forceinline__ unsigned pack2(float lo, float hi) {
    unsigned r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ Parts split(float x, float y) {
    Parts p;
    p.h = pack2(x, y);
    x -= __uint_as_float(p.h << 16);
    y -= __uint_as_float(p.h & 0xffff0000u);
    p.m = pack2(x, y);
    x -= __uint_as_float(p.m << 16);
    y -= __uint_as_float(p.m & 0xffff0000u);
    p.l = pack2(x, y);
    return p;
}
__device__ __forceinline__ Parts split_up(float x, float y) {         // of both times UP, one instruction
    asm("{\n.reg .b64 v;\nmov.b64 v, {%0, %1};\nmul.rn.f32x2 v, v, %2;\nmov.b64 {%0, %1}, v;\n}" : "+f"(x), "+f"(y) : "l"(UP2));
    return split(x, y);
}
__device__ __forceinline__ void mma(float (&c)[4], const uint4& a, unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
struct First { uint4 h, m, l; };          // the parts of a first operand, 16 rows by 16 along the sum
struct Sums {                             // the product of the leading parts, the five others in three accumulators side by side
    float big[4], mm[4], hl[4], lh[4];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < 4; ++i) big[i] = mm[i] = hl[i] = lh[i] = 0.f;
    }
    __device__ __forceinline__ void add(const First& a, const Parts& p, const Parts& r) {
        mma(big, a.h, p.h, r.h);
        mma(mm, a.m, p.m, r.m);
        mma(hl, a.h, p.l, r.l);
        mma(lh, a.l, p.h, r.h);
        mma(mm, a.h, p.m, r.m);
        mma(hl, a.m, p.h, r.h);
    }
    __device__ __forceinline__ float get(int i) const { return (big[i] + ((mm[i] + hl[i]) + lh[i])) * DOWN; }
};
__device__ __forceinline__ bool finite(float x) { return fabsf(x) <= FLT_MAX; }

__device__ __forceinline__ void cp16(float* smem, const float* gmem, int bytes) {       // bytes behind `bytes` become zero
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem), "r"(bytes));
}

// Arguments as of attention_simt_kernel (attention_simt.cu).
struct Args {
    const float* q; int ld;
    const float* kpool; const float* vpool;
    const int* pos; const int* tok_seg; const int* block_table;
    int bt_stride, page_size;
    float* out;
    int T, Hq, Hkv;
    float scale;
    int window, chunk;
    float softcap;
    const float* slopes; const float* sink; const float* bias;
    int bias_n, keep, tb, heads;
};

template <int D> struct Smem {
    static constexpr int KT = D / 16, KP = D + 8, VP = D + 4;             // key and value rows lie so that a warp's reads hit all banks
    static constexpr int Q = 2 * KT * 384, TILE = KEYS * (KP + VP), S = ROWS * SP;
    static constexpr size_t BYTES = (size_t)(Q + 2 * TILE + 2 * S + 2 * ROWS) * 4;
};

// A score, and an output's sum over a tile, from the operands as they are.
__device__ __noinline__ float chain(const float* a, const float* b, int n) {
    float x = 0.f;
    for (int i = 0; i < n; ++i) x = fmaf(a[i], b[i], x);
    return x;
}
__device__ __noinline__ float chain_seen(const float* p, const float* v, int pitch, int from, int to, int kept, const int* page) {
    float x = 0.f;
    for (int j = 0; j < KEYS; ++j)
        if (page[j] >= 0 && j <= to && (j >= from || j < kept)) x = fmaf(p[j] * (1.f / UP), v[j * pitch], x);
    return x;
}

template <int D>
__global__ void __launch_bounds__(32 * WARPS, 2)
attention_f32_kernel(const Args a) {
    using M = Smem<D>;
    constexpr int KT = M::KT, KP = M::KP, VP = M::VP, NT = (D / 8 + WARPS - 1) / WARPS;      // NT: blocks of 8 columns of a warp: warp, warp + 8
    static_assert(D % 32 == 0, "whole rows by cp.async");
    // CTAs by heads, then by tokens, every tb-th of these first: most of those begin a block, and the others, which return at once, come
    // behind and beside them (in the tokens' order they held the last heads up by 15 us at 257 tokens)
    const int G = a.Hq / a.Hkv, splits = (G + a.heads - 1) / a.heads;
    const int by_head = blockIdx.x % (a.Hkv * splits), nth = blockIdx.x / (a.Hkv * splits), columns = (a.T + a.tb - 1) / a.tb;
    const int t0 = (nth % columns) * a.tb + nth / columns;
    if (t0 >= a.T) return;
    pdl_wait();                                                        // the tables may be the work of the kernel before this one
    const int seg = a.tok_seg[t0], p0 = a.pos[t0];
    if (t0 > 0 && a.tok_seg[t0 - 1] == seg && a.pos[t0 - 1] == p0 - 1 && p0 % a.tb != 0) return;   // an earlier token's CTA takes this one along
    const int until = a.tb - p0 % a.tb;
    int n = 1;
    while (n < until && t0 + n < a.T && a.tok_seg[t0 + n] == seg && a.pos[t0 + n] == p0 + n) ++n;
    const int kvh = by_head / splits, g0 = (by_head % splits) * a.heads, nh = min(a.heads, G - g0);
    const int rows = n * nh;                                           // row i: token t0 + i / nh, head kvh * G + g0 + i % nh

    extern __shared__ __align__(16) float f32_smem[];
    unsigned* qp = reinterpret_cast<unsigned*>(f32_smem);              // [block of rows][block of 16 dims][part][lane][4]
    float* tiles = f32_smem + M::Q;                                    // [2][keys, then values]
    float* Ss = tiles + 2 * M::TILE;
    float* Ps = Ss + M::S;
    float* alpha_s = Ps + M::S;
    float* inv_s = alpha_s + ROWS;
    __shared__ int page_of[2][KEYS], from_s[ROWS], to_s[ROWS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t2 = 2 * (lane & 3);
    const int* bt = a.block_table + (size_t)seg * a.bt_stride;
    const size_t head_stride = (size_t)a.page_size * D;
    auto q_row = [&](int row) { return a.q + (size_t)(t0 + row / nh) * a.ld + (size_t)(kvh * G + g0 + row % nh) * D; };

    // the tiles of kept positions come first, then those from the first row's lowest key on
    const int lo0 = a.window > 0 ? max(0, p0 - a.window + 1) : a.chunk > 0 ? (p0 / a.chunk) * a.chunk : 0;
    const int first0 = (lo0 / KEYS) * KEYS, p_last = p0 + n - 1;
    auto next = [&](int j0) { return j0 < first0 && j0 + KEYS >= a.keep ? first0 : j0 + KEYS; };
    // Pages are looked up a tile ahead of the copies that need them: a look waited for in front of every tile cost 0.8 us.
    int page_r[KEYS / WARPS];
    auto look = [&](int j0) {                                          // keys behind the last row are not there yet
#pragma unroll
        for (int i = 0; i < KEYS / WARPS; ++i) {
            const int j = j0 + warp + i * WARPS;
            page_r[i] = j <= p_last ? bt[j / a.page_size] : -2;
        }
    };
    auto fetch = [&](int j0, int buf) {                                // they, and pages that were given back, read as zero
        float* ks = tiles + buf * M::TILE;
#pragma unroll
        for (int i = 0; i < KEYS / WARPS; ++i) {
            const int jj = warp + i * WARPS, j = j0 + jj, page = page_r[i];
            if (lane == 0) page_of[buf][jj] = page;
            const size_t at = ((size_t)(page < 0 ? 0 : page) * a.Hkv + kvh) * head_stride + (size_t)(j % a.page_size) * D + 4 * lane;
            if (4 * lane < D) {
                cp16(ks + jj * KP + 4 * lane, a.kpool + at, page < 0 ? 0 : 16);
                cp16(ks + KEYS * KP + jj * VP + 4 * lane, a.vpool + at, page < 0 ? 0 : 16);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::);
        look(next(j0));
    };
    const int begin = a.keep > 0 ? 0 : first0;
    look(begin);
    fetch(begin, 0);

    for (int c = warp; c < 2 * KT; c += WARPS) {                       // the queries' parts
        const int ra = 16 * (c / KT) + g, d = 16 * (c % KT) + t2;
        float x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int row = ra + (i & 2 ? 8 : 0), at = d + (i & 1) + (i & 4 ? 8 : 0);
            x[i] = row < rows ? q_row(row)[at] : 0.f;
        }
        const Parts p0_ = split_up(x[0], x[1]), p1 = split_up(x[2], x[3]), p2 = split_up(x[4], x[5]), p3 = split_up(x[6], x[7]);
        uint4* to = reinterpret_cast<uint4*>(qp + c * 384) + lane;
        to[0] = make_uint4(p0_.h, p1.h, p2.h, p3.h);
        to[32] = make_uint4(p0_.m, p1.m, p2.m, p3.m);
        to[64] = make_uint4(p0_.l, p1.l, p2.l, p3.l);
    }
    // this warp's rows of the softmax
    const int r0 = warp * RW, nr = min(RW, rows - r0);
    int p[RW], lo[RW], hd[RW];
    float m[RW], l[RW];
#pragma unroll
    for (int i = 0; i < RW; ++i) {
        const int row = min(r0 + i, rows - 1);
        p[i] = p0 + row / nh;
        hd[i] = kvh * G + g0 + row % nh;
        lo[i] = a.window > 0 ? max(0, p[i] - a.window + 1) : a.chunk > 0 ? (p[i] / a.chunk) * a.chunk : 0;
        m[i] = -INFINITY;
        l[i] = 0.f;
    }
    const int mt = warp & 1, part = warp >> 1;                         // of the scores: block of 16 rows, block of 8 keys
    const bool there = 16 * mt < rows;
    const int blocks = rows > 16 ? 2 : 1;
    float o[2][NT][4];                                                 // block of 16 rows, of 8 columns
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) o[b][j][e] = 0.f;

    int buf = 0;
    for (int j0 = begin; j0 <= p_last; j0 = next(j0), buf ^= 1) {
        asm volatile("cp.async.wait_group 0;\n" ::);
        __syncthreads();                                               // this tile is there, and the one before it has been used
        if (next(j0) <= p_last) fetch(next(j0), buf ^ 1);
        const float* ks = tiles + buf * M::TILE;
        const float* vs = ks + KEYS * KP;
        if (there) {                                                   // ---- scores
            Sums s;
            s.clear();
            const float* kr = ks + (8 * part + g) * KP + t2;
            const uint4* qa = reinterpret_cast<const uint4*>(qp + mt * KT * 384) + lane;
#pragma unroll
            for (int k = 0; k < KT; ++k) {
                const First x = {qa[k * 96], qa[k * 96 + 32], qa[k * 96 + 64]};
                const float2 b0 = *reinterpret_cast<const float2*>(kr + 16 * k), b1 = *reinterpret_cast<const float2*>(kr + 16 * k + 8);
                s.add(x, split_up(b0.x, b0.y), split_up(b1.x, b1.y));
            }
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
                const int row = 16 * mt + g + 4 * e, key = 8 * part + t2;
                float2 v = make_float2(s.get(e), s.get(e + 1));
                if (row < rows && !(finite(v.x) && finite(v.y))) {
                    if (!finite(v.x)) v.x = chain(q_row(row), ks + key * KP, D);
                    if (!finite(v.y)) v.y = chain(q_row(row), ks + (key + 1) * KP, D);
                }
                *reinterpret_cast<float2*>(Ss + row * SP + key) = v;
            }
        }
        __syncthreads();
        if (nr > 0) {                                                  // ---- softmax, a lane a key
            const int j = j0 + lane, page = page_of[buf][lane];
            float sc[RW], mx[RW];
            bool on[RW], valid[RW];
#pragma unroll
            for (int i = 0; i < RW; ++i) {
                // a row takes the tiles from its own lowest key on, and those of kept positions
                on[i] = i < nr && j0 <= p[i] && (j0 >= (lo[i] / KEYS) * KEYS || j0 < a.keep);
                valid[i] = on[i] && (j >= lo[i] || j < a.keep) && j <= p[i];
                sc[i] = Ss[(r0 + i) * SP + lane] * a.scale;
            }
            if (a.softcap > 0.f) {
#pragma unroll
                for (int i = 0; i < RW; ++i) sc[i] = a.softcap * tanhf(sc[i] / a.softcap);
            }
            if (a.slopes) {
#pragma unroll
                for (int i = 0; i < RW; ++i) sc[i] -= a.slopes[hd[i]] * (float)(p[i] - j);
            }
            if (a.bias) {
#pragma unroll
                for (int i = 0; i < RW; ++i) sc[i] += a.bias[(size_t)hd[i] * a.bias_n + max(0, min(p[i] - j, a.bias_n - 1))];
            }
#pragma unroll
            for (int i = 0; i < RW; ++i) {                             // a page that was given back: show it as NaN
                sc[i] = !valid[i] ? -INFINITY : page < 0 ? __int_as_float(0x7fc00000) : sc[i];
                mx[i] = sc[i];
            }
#pragma unroll
            for (int w = 16; w > 0; w >>= 1)
#pragma unroll
                for (int i = 0; i < RW; ++i) mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], w));
            float pj[RW], sum[RW];
#pragma unroll
            for (int i = 0; i < RW; ++i) {
                mx[i] = fmaxf(m[i], mx[i]);
                const float e = expf(sc[i] - mx[i]);
                pj[i] = valid[i] ? e : 0.f;
                sum[i] = pj[i];
                Ps[(r0 + i) * SP + lane] = pj[i] * UP;
            }
#pragma unroll
            for (int w = 16; w > 0; w >>= 1)
#pragma unroll
                for (int i = 0; i < RW; ++i) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], w);
#pragma unroll
            for (int i = 0; i < RW; ++i) {
                const float old = expf(m[i] - mx[i]), alpha = on[i] ? old : 1.0f;        // m = -inf on the first tile gives 0
                l[i] = l[i] * alpha + sum[i];
                m[i] = mx[i];
                if (lane == 0) {
                    alpha_s[r0 + i] = alpha;
                    from_s[r0 + i] = lo[i] - j0;
                    to_s[r0 + i] = on[i] ? p[i] - j0 : -1;
                }
            }
        } else if (r0 < ((rows + 15) & ~15)) {                         // rows that fill up a block
#pragma unroll
            for (int i = 0; i < RW; ++i) {
                Ps[(r0 + i) * SP + lane] = 0.f;
                if (lane == 0) alpha_s[r0 + i] = 1.f;
            }
        }
        __syncthreads();
        // ---- outputs: a warp's columns for both blocks of rows, the values' parts made once
        if (8 * warp < D) {
            Sums u[2][NT];
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int j = 0; j < NT; ++j) u[b][j].clear();
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                Parts v0[NT], v1[NT];
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    const int col = 8 * (warp + WARPS * j) + g;
                    const float* vr = vs + (16 * k + t2) * VP + (col < D ? col : 0);
                    v0[j] = split_up(vr[0], vr[VP]);
                    v1[j] = split_up(vr[8 * VP], vr[9 * VP]);
                }
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    if (b >= blocks) break;
                    const float* pr = Ps + (16 * b + g) * SP + 16 * k + t2;
                    const float2 y0 = *reinterpret_cast<const float2*>(pr), y1 = *reinterpret_cast<const float2*>(pr + 8 * SP);
                    const float2 y2 = *reinterpret_cast<const float2*>(pr + 8), y3 = *reinterpret_cast<const float2*>(pr + 8 * SP + 8);
                    const Parts a0 = split(y0.x, y0.y), a1 = split(y1.x, y1.y), a2 = split(y2.x, y2.y), a3 = split(y3.x, y3.y);
                    const First x = {make_uint4(a0.h, a1.h, a2.h, a3.h), make_uint4(a0.m, a1.m, a2.m, a3.m), make_uint4(a0.l, a1.l, a2.l, a3.l)};
#pragma unroll
                    for (int j = 0; j < NT; ++j) u[b][j].add(x, v0[j], v1[j]);
                }
            }
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                if (b >= blocks) break;
                const float al[2] = {alpha_s[16 * b + g], alpha_s[16 * b + g + 8]};
                float x[NT][4];
                bool fine = true;
#pragma unroll
                for (int j = 0; j < NT; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        x[j][e] = u[b][j].get(e);
                        fine = fine && finite(x[j][e]);
                    }
                if (!fine) {
#pragma unroll 1
                    for (int i = 0; i < 4 * NT; ++i) {
                        const int e = i & 3, row = 16 * b + g + (e & 2 ? 8 : 0), col = 8 * (warp + WARPS * (i >> 2)) + t2 + (e & 1);
                        if (row >= rows || col >= D) continue;
                        const float y = chain_seen(Ps + row * SP, vs + col, VP, from_s[row], to_s[row], a.keep - j0, page_of[buf]);
#pragma unroll
                        for (int n = 0; n < 4 * NT; ++n)
                            if (n == i && !finite(x[n >> 2][n & 3])) x[n >> 2][n & 3] = y;
                    }
                }
#pragma unroll
                for (int j = 0; j < NT; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) o[b][j][e] = fmaf(o[b][j][e], al[e >> 1], x[j][e]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < RW; ++i) {
        if (i >= nr) continue;
        if (a.sink) l[i] += expf(a.sink[hd[i]] - m[i]);
        if (lane == 0) inv_s[r0 + i] = 1.0f / l[i];
    }
    pdl_trigger_late();
    __syncthreads();
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
            const int row = 16 * b + g + 4 * e;
            if (row >= rows) continue;
            const float inv = inv_s[row];
            float* to = a.out + ((size_t)(t0 + row / nh) * a.Hq + kvh * G + g0 + row % nh) * D + t2;
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const int col = 8 * (warp + WARPS * j);
                if (col >= D) continue;
                to[col] = o[b][j][e] * inv;
                to[col + 1] = o[b][j][e + 1] * inv;
            }
        }
}

template <int D>
int launch(const Args& a, int splits, cudaStream_t st) {
    static PerDevice configured;
    const int rc = configured.once([&](int) {
        return cudaFuncSetAttribute(attention_f32_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Smem<D>::BYTES);
    });
    if (rc) return rc;
    return rb_launch_pdl(attention_f32_kernel<D>, dim3((unsigned)((a.T + a.tb - 1) / a.tb * a.tb) * a.Hkv * splits), dim3(32 * WARPS), Smem<D>::BYTES, st, a);
}

}  // namespace

// Whether the kernel takes these sizes; the choice looks at nothing that changes from step to step, so a model's tokens all get one kernel's bits.
int rb_attention_f32_takes(int D, const void* kpool, const void* vpool) {
    return D % 32 == 0 && D >= 32 && D <= 128 && (((uintptr_t)kpool | (uintptr_t)vpool) & 15) == 0;
}

int rb_attention_f32(const float* q, int ld, const float* kpool, const float* vpool, const int* pos, const int* tok_seg, const int* block_table,
                     int bt_stride, int page_size, float* out, int T, int Hq, int Hkv, int D, float scale, int window, int chunk, float softcap,
                     const float* slopes, const float* sink, const float* bias, int bias_n, int keep, cudaStream_t st) {
    const int G = Hq / Hkv, heads = G < ROWS ? G : ROWS;
    int tb = 1;                                            // tokens of a CTA: a power of two whose rows fit
    while (2 * tb * heads <= ROWS && tb < 16) tb *= 2;
    const Args a = {q, ld, kpool, vpool, pos, tok_seg, block_table, bt_stride, page_size, out, T, Hq, Hkv, scale, window, chunk, softcap,
                    slopes, sink, bias, bias_n, keep, tb, heads};
    const int splits = (G + heads - 1) / heads;
    if (D == 128) return launch<128>(a, splits, st);
    if (D == 96) return launch<96>(a, splits, st);
    return D == 64 ? launch<64>(a, splits, st) : launch<32>(a, splits, st);
}
