// Paged causal attention on the CUDA cores, for any element type, head size, page size and
// segment shape: the kernel of the 32-bit path where attention_f32.cu does not take the head size, and the plain twin of the tensor-core kernels.
//
// A warp owns up to four (token, query head) rows.  Keys are taken in tiles of 32 that are aligned to
// absolute positions (0-31, 32-63, ...), lane j of a tile scores key j, and the online softmax
// (running maximum m, running sum l, float32 accumulators) advances tile by tile as in the
// reference's kernels (rollout/attention.py:125-139).  Because the tiles are fixed by position
// and a row never looks at another row, the result for a token does not depend on how the
// prompt was cut into steps or on what else is in the batch: it is bit-identical.
//
// A CTA of eight warps works on the rows of neighbouring tokens of one segment that share a key/value head, and brings a
// tile of keys and values to shared memory once for all of them, the next one on its way meanwhile (rows padded by four floats: a lane's 16-byte reads of its
// key are free of bank conflicts).  Which tokens: there is a CTA per token (and key/value head), and the one whose token
// starts a segment's portion or stands at a multiple of `tb` positions takes the tokens up to the next multiple; the
// others return at once.  So no table of blocks is needed, and decoded tokens get a CTA each.  The order of every sum is
// the row's own.  Bound by shared memory: a tile costs a warp four reads of keys and values for sixteen FFMAs.  Measured
// (257 tokens, 16 query and 8 key/value heads of 128, up to 219 keys): 68 us a layer; a warp per row that read its keys
// from global memory, a lane a key, took 326.
//
// q: rotated queries inside the QKV buffer, row stride ld.  K and V: one layer's pools
// [num_pages, Hkv, P, D].  A key at position j is visible to the query at position p iff
// lo <= j <= p with lo = max(0, p - window + 1) when window > 0, else 0.
//
// Options of the score, all off by default: `chunk` > 0 bounds the keys from below by the start of the query's own
// block of `chunk` positions (blocks counted from position 0) instead of a window; `softcap` > 0 turns a scaled score
// s into softcap * tanh(s / softcap); `slopes` [Hq] takes slopes[h] * (p - j) off the score of key j; `bias` [Hq, bias_n] adds
// bias[h, min(p - j, bias_n - 1)] to it; `keep` > 0 (with a window) leaves the first `keep` positions visible for every later query; `sink` [Hq] adds exp(sink[h]) to the softmax's denominator (a term with no key and
// no value).
#include "common.cuh"

#define SIMT_MAX_D 256
#define SIMT_WARPS 8
#define SIMT_RW 4                     // rows of a warp
#define SIMT_ROWS (SIMT_WARPS * SIMT_RW)
#define SIMT_KEYS 32                  // keys of a tile

__device__ __forceinline__ void simt_cp16(float* smem, const float* gmem, int bytes) {       // bytes behind `bytes` become zero
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem), "r"(bytes));
}

// NC: runs of 128 columns that a row's accumulators cover (a lane holds columns 4 lane + 128 c ..+ 3)
template <typename TA, int NC>
__global__ void __launch_bounds__(32 * SIMT_WARPS, NC == 1 ? 2 : 1)
attention_simt_kernel(const TA* __restrict__ q, int ld, const TA* __restrict__ kpool,
                      const TA* __restrict__ vpool, const int* __restrict__ pos,
                      const int* __restrict__ tok_seg, const int* __restrict__ block_table,
                      int bt_stride, int page_size, TA* __restrict__ out, int T, int Hq, int Hkv, int D,
                      float scale, int window, int chunk, float softcap, const float* __restrict__ slopes,
                      const float* __restrict__ sink, const float* __restrict__ bias, int bias_n, int keep,
                      int tb, int heads, int vec) {
    const int t0 = blockIdx.x;
    const int seg = tok_seg[t0], p0 = pos[t0];
    if (t0 > 0 && tok_seg[t0 - 1] == seg && pos[t0 - 1] == p0 - 1 && p0 % tb != 0) return;   // an earlier token's CTA takes this one along
    const int until = tb - p0 % tb;                                    // tokens up to the next multiple
    int n = 1;
    while (n < until && t0 + n < T && tok_seg[t0 + n] == seg && pos[t0 + n] == p0 + n) ++n;
    const int G = Hq / Hkv;
    const int splits = (G + heads - 1) / heads;                        // CTAs that share a key/value head's query heads
    const int kvh = blockIdx.y / splits, g0 = (blockIdx.y % splits) * heads;
    const int nh = min(heads, G - g0);                                 // query heads of this CTA
    const int rows = n * nh;                                           // row i: token t0 + i / nh, head kvh * G + g0 + i % nh

    const int D4 = (D + 3) & ~3, pitch = D4 + 4;
    extern __shared__ __align__(16) float simt_smem[];
    float* qs = simt_smem;                                             // [SIMT_ROWS][pitch]
    float* tiles = qs + SIMT_ROWS * pitch;                             // [2][keys, values][SIMT_KEYS][pitch]
    __shared__ int page_of[2][SIMT_KEYS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int* bt = block_table + (size_t)seg * bt_stride;
    const size_t head_stride = (size_t)page_size * D;                  // one kv head of one page

    const int r0 = warp * SIMT_RW, nr = min(SIMT_RW, rows - r0);       // this warp's rows (nr <= 0: none)
    int p[SIMT_RW], lo[SIMT_RW], hd[SIMT_RW];
    float m[SIMT_RW], l[SIMT_RW], acc[SIMT_RW][4 * NC];
#pragma unroll
    for (int i = 0; i < SIMT_RW; ++i) {
        const int row = min(r0 + i, rows - 1);
        p[i] = p0 + row / nh;
        hd[i] = kvh * G + g0 + row % nh;
        lo[i] = window > 0 ? max(0, p[i] - window + 1) : chunk > 0 ? (p[i] / chunk) * chunk : 0;
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < 4 * NC; ++c) acc[i][c] = 0.f;
    }
    for (int d = lane; d < D4; d += 32) {                              // a warp reads its own rows only; rows that do not exist are zero
        float x[SIMT_RW];
#pragma unroll
        for (int i = 0; i < SIMT_RW; ++i)
            x[i] = i < nr && d < D ? to_f32(q[(size_t)(t0 + p[i] - p0) * ld + (size_t)hd[i] * D + d]) : 0.f;
#pragma unroll
        for (int i = 0; i < SIMT_RW; ++i) qs[(r0 + i) * pitch + d] = x[i];
    }
    // the tiles of kept positions come first, then those from the first row's lowest key on
    const int lo0 = window > 0 ? max(0, p0 - window + 1) : chunk > 0 ? (p0 / chunk) * chunk : 0;
    const int first0 = (lo0 / 32) * 32, p_last = p0 + n - 1;
    auto next = [&](int j0) { return j0 < first0 && j0 + 32 >= keep ? first0 : j0 + 32; };
    // a tile on its way to shared memory: keys behind the last row are not there yet, pages that were given back read as zero
    const int per = D4 >> 2;
    auto fetch = [&](int j0, int buf) {
        float* ks = tiles + buf * 2 * SIMT_KEYS * pitch;
        int page_r[SIMT_KEYS / SIMT_WARPS];                            // looked up together, not one behind the other
#pragma unroll
        for (int i = 0; i < SIMT_KEYS / SIMT_WARPS; ++i) {
            const int j = j0 + warp + i * SIMT_WARPS;
            page_r[i] = j <= p_last ? bt[j / page_size] : -2;
        }
#pragma unroll
        for (int i = 0; i < SIMT_KEYS / SIMT_WARPS; ++i) {
            const int jj = warp + i * SIMT_WARPS, j = j0 + jj, page = page_r[i];
            if (lane == 0) page_of[buf][jj] = page;
            const size_t at = ((size_t)(page < 0 ? 0 : page) * Hkv + kvh) * head_stride + (size_t)(j % page_size) * D;
            float* kd = ks + jj * pitch;
            float* vd = kd + SIMT_KEYS * pitch;
            for (int c = lane; c < per; c += 32) {
                const int d = 4 * c;
                if (vec) {
                    simt_cp16(kd + d, reinterpret_cast<const float*>(kpool) + at + d, page < 0 ? 0 : 16);
                    simt_cp16(vd + d, reinterpret_cast<const float*>(vpool) + at + d, page < 0 ? 0 : 16);
                } else {
                    for (int i = d; i < d + 4; ++i) {
                        const bool there = page >= 0 && i < D;
                        kd[i] = there ? to_f32(kpool[at + i]) : 0.f;
                        vd[i] = there ? to_f32(vpool[at + i]) : 0.f;
                    }
                }
            }
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    int buf = 0;
    const int begin = keep > 0 ? 0 : first0;
    fetch(begin, 0);
    for (int j0 = begin; j0 <= p_last; j0 = next(j0), buf ^= 1) {
        asm volatile("cp.async.wait_group 0;\n" ::);
        __syncthreads();                                               // this tile is there, and the one before it has been used
        if (next(j0) <= p_last) fetch(next(j0), buf ^ 1);              // on its way while this one is worked on
        if (nr <= 0) continue;
        const float* ks = tiles + buf * 2 * SIMT_KEYS * pitch;
        const float* vs = ks + SIMT_KEYS * pitch;
        const int j = j0 + lane, page = page_of[buf][lane];
        float dot[SIMT_RW];
#pragma unroll
        for (int i = 0; i < SIMT_RW; ++i) dot[i] = 0.f;
        const float* kr = ks + lane * pitch;
        const float* qr = qs + r0 * pitch;
#pragma unroll 4
        for (int d = 0; d < D4; d += 4) {
            const float4 k4 = *reinterpret_cast<const float4*>(kr + d);
#pragma unroll
            for (int i = 0; i < SIMT_RW; ++i) {                        // rows that do not exist are zero
                const float4 q4 = *reinterpret_cast<const float4*>(qr + i * pitch + d);
                dot[i] = fmaf(q4.x, k4.x, dot[i]);
                dot[i] = fmaf(q4.y, k4.y, dot[i]);
                dot[i] = fmaf(q4.z, k4.z, dot[i]);
                dot[i] = fmaf(q4.w, k4.w, dot[i]);
            }
        }
        float pj[SIMT_RW];
        int from[SIMT_RW], to[SIMT_RW];                                // the keys of the tile that a row sees (besides kept ones)
#pragma unroll
        for (int i = 0; i < SIMT_RW; ++i) {
            // a row takes the tiles from its own lowest key on, and those of kept positions
            const bool on = i < nr && j0 <= p[i] && (j0 >= (lo[i] / 32) * 32 || j0 < keep);
            const bool valid = on && (j >= lo[i] || j < keep) && j <= p[i];
            from[i] = lo[i] - j0;
            to[i] = on ? p[i] - j0 : -1;
            float s = -INFINITY;
            if (valid) {
                if (page < 0) {
                    s = __int_as_float(0x7fc00000);                    // a page that was given back: show it as NaN
                } else {
                    s = dot[i] * scale;
                    if (softcap > 0.f) s = softcap * tanhf(s / softcap);
                    if (slopes) s -= slopes[hd[i]] * (float)(p[i] - j);
                    if (bias) s += bias[(size_t)hd[i] * bias_n + min(p[i] - j, bias_n - 1)];
                }
            }
            const float m_new = fmaxf(m[i], warp_max(s));
            pj[i] = valid ? expf(s - m_new) : 0.f;
            const float alpha = on ? expf(m[i] - m_new) : 1.0f;        // m = -inf on the first tile gives 0
            l[i] = l[i] * alpha + warp_sum(pj[i]);
#pragma unroll
            for (int c = 0; c < 4 * NC; ++c) acc[i][c] *= alpha;
            m[i] = m_new;
        }
        bool all = __all_sync(0xffffffffu, page >= 0);                 // every row sees every key of the tile
#pragma unroll
        for (int i = 0; i < SIMT_RW; ++i) all = all && (i >= nr || (from[i] <= 0 && to[i] >= SIMT_KEYS - 1));
        if (all) {
#pragma unroll 8
            for (int jj = 0; jj < SIMT_KEYS; ++jj) {
                float4 v4[NC];
#pragma unroll
                for (int c = 0; c < NC; ++c)
                    v4[c] = 4 * lane + 128 * c < D4 ? *reinterpret_cast<const float4*>(vs + jj * pitch + 4 * lane + 128 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int i = 0; i < SIMT_RW; ++i) {
                    const float pjj = __shfl_sync(0xffffffffu, pj[i], jj);
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        acc[i][4 * c] = fmaf(pjj, v4[c].x, acc[i][4 * c]);
                        acc[i][4 * c + 1] = fmaf(pjj, v4[c].y, acc[i][4 * c + 1]);
                        acc[i][4 * c + 2] = fmaf(pjj, v4[c].z, acc[i][4 * c + 2]);
                        acc[i][4 * c + 3] = fmaf(pjj, v4[c].w, acc[i][4 * c + 3]);
                    }
                }
            }
            continue;
        }
        const int jend = min(SIMT_KEYS, p_last - j0 + 1);
#pragma unroll 4
        for (int jj = 0; jj < jend; ++jj) {
            if (page_of[buf][jj] < 0) continue;
            const bool kept = j0 + jj < keep;
            float4 v4[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c)
                v4[c] = 4 * lane + 128 * c < D4 ? *reinterpret_cast<const float4*>(vs + jj * pitch + 4 * lane + 128 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < SIMT_RW; ++i) {
                const float pjj = __shfl_sync(0xffffffffu, pj[i], jj);
                if (jj <= to[i] && (jj >= from[i] || kept)) {          // uniform over the warp; a key the row does not see may hold anything
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        acc[i][4 * c] = fmaf(pjj, v4[c].x, acc[i][4 * c]);
                        acc[i][4 * c + 1] = fmaf(pjj, v4[c].y, acc[i][4 * c + 1]);
                        acc[i][4 * c + 2] = fmaf(pjj, v4[c].z, acc[i][4 * c + 2]);
                        acc[i][4 * c + 3] = fmaf(pjj, v4[c].w, acc[i][4 * c + 3]);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < SIMT_RW; ++i) {
        if (i >= nr) continue;
        if (sink) l[i] += expf(sink[hd[i]] - m[i]);
        const float inv = 1.0f / l[i];
        TA* orow = out + ((size_t)(t0 + (r0 + i) / nh) * Hq + hd[i]) * D;
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int d = 4 * lane + 128 * c + k;
                if (d < D) orow[d] = from_f32<TA>(acc[i][4 * c + k] * inv);
            }
    }
}

template <typename TA, int NC>
static int launch_simt(const void* q, int ld, const void* kpool, const void* vpool, const int* pos, const int* tok_seg,
                       const int* block_table, int bt_stride, int page_size, void* out, int T, int Hq, int Hkv, int D, float scale,
                       int window, int chunk, float softcap, const float* slopes, const float* sink, const float* bias, int bias_n,
                       int keep, cudaStream_t st) {
    const int G = Hq / Hkv, heads = G < SIMT_ROWS ? G : SIMT_ROWS;
    int tb = 1;                                            // tokens of a CTA: a power of two whose rows fit
    while (2 * tb * heads <= SIMT_ROWS && tb < 16) tb *= 2;
    const size_t smem = (size_t)(SIMT_ROWS + 4 * SIMT_KEYS) * (((D + 3) & ~3) + 4) * sizeof(float);
    static PerDevice configured;
    const int rc = configured.once([&](int) {
        return cudaFuncSetAttribute(attention_simt_kernel<TA, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)((SIMT_ROWS + 4 * SIMT_KEYS) * (128 * NC + 4) * sizeof(float)));
    });
    if (rc) return rc;
    const int vec = sizeof(TA) == 4 && D % 4 == 0 && (((uintptr_t)kpool | (uintptr_t)vpool) & 15) == 0;
    dim3 grid(T, Hkv * ((G + heads - 1) / heads));
    attention_simt_kernel<TA, NC><<<grid, 32 * SIMT_WARPS, smem, st>>>(
        (const TA*)q, ld, (const TA*)kpool, (const TA*)vpool, pos, tok_seg, block_table, bt_stride, page_size, (TA*)out, T, Hq, Hkv, D,
        scale, window, chunk, softcap, slopes, sink, bias, bias_n, keep, tb, heads, vec);
    return rb_launch_status();
}

// attention_f32.cu: the 32-bit path's kernel where it takes the head size and the pools lie on 16-byte boundaries (257 tokens as above: 46 us).
int rb_attention_f32_takes(int D, const void* kpool, const void* vpool);
int rb_attention_f32(const float* q, int ld, const float* kpool, const float* vpool, const int* pos, const int* tok_seg, const int* block_table,
                     int bt_stride, int page_size, float* out, int T, int Hq, int Hkv, int D, float scale, int window, int chunk, float softcap,
                     const float* slopes, const float* sink, const float* bias, int bias_n, int keep, cudaStream_t st);

RB_EXPORT int rb_attention_simt_mod(const void* q, int ld, const void* kpool, const void* vpool,
                                const int* pos, const int* tok_seg, const int* block_table,
                                int bt_stride, int page_size, void* out, int act_dtype, int T,
                                int Hq, int Hkv, int D, float scale, int window, int chunk, float softcap,
                                const float* slopes, const float* sink, const float* bias, int bias_n, int keep, cudaStream_t st) {
    if (T <= 0) return 0;
    if (bias != nullptr && bias_n < 1) return (int)cudaErrorInvalidValue;
    if ((window > 0 && chunk > 0) || keep < 0 || (keep > 0 && window <= 0)) return (int)cudaErrorInvalidValue;
    if (D > SIMT_MAX_D || D <= 0 || Hkv <= 0 || Hq % Hkv) return (int)cudaErrorInvalidValue;
    if (act_dtype == RB_F32 && rb_attention_f32_takes(D, kpool, vpool))
        return rb_attention_f32((const float*)q, ld, (const float*)kpool, (const float*)vpool, pos, tok_seg, block_table, bt_stride, page_size,
                                (float*)out, T, Hq, Hkv, D, scale, window, chunk, softcap, slopes, sink, bias, bias_n, keep, st);
    auto launch = act_dtype == RB_F32 ? (D <= 128 ? launch_simt<float, 1> : launch_simt<float, 2>)
                                      : (D <= 128 ? launch_simt<bf16, 1> : launch_simt<bf16, 2>);
    return launch(q, ld, kpool, vpool, pos, tok_seg, block_table, bt_stride, page_size, out, T, Hq, Hkv, D, scale, window, chunk,
                  softcap, slopes, sink, bias, bias_n, keep, st);
}

RB_EXPORT int rb_attention_simt(const void* q, int ld, const void* kpool, const void* vpool,
                                const int* pos, const int* tok_seg, const int* block_table,
                                int bt_stride, int page_size, void* out, int act_dtype, int T,
                                int Hq, int Hkv, int D, float scale, int window, cudaStream_t st) {
    return rb_attention_simt_mod(q, ld, kpool, vpool, pos, tok_seg, block_table, bt_stride, page_size, out, act_dtype, T,
                                 Hq, Hkv, D, scale, window, 0, 0.f, nullptr, nullptr, nullptr, 0, 0, st);
}
