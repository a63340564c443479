// The recurrences of recurrent.cu over the long segments of a step, 32 tokens at a time instead of one.
//
// With decays g_t (a vector over the key rows, or one number), P_t their product from the chunk's start through token t, and S0
// the state before the chunk, every mode but the matrix memory has the form
//     U = T (v - (k * P) S0)  (delta rules; otherwise U = v, times the step in the state-space scan)
//     o = (q * P) S0 + M U,      S = diag(P_32) S0 + (k * P_32 / P_t)^T U
// with two lower triangular 32 x 32 matrices: M[t, s] = q_t . (P_t / P_s * k_s), and for the delta rules T = (I + diag(beta) A)^-1
// diag(beta), A[t, s] = k_t . (P_t / P_s * k_s) for s < t.  No quotient is ever formed: a ratio P_t / P_s is a product of the
// decays between s and t, so decays as small as they come cost no accuracy (they underflow to zero where the true value does).
//
// `chunk_prep_kernel` works out k * P, q * P, k * P_32 / P_t, T, M and P_32 for all chunks and heads side by side and leaves them in the
// order in which the second kernel's matrix instructions want them.  `chunk_serial_kernel` walks the chunks of a segment in order,
// a CTA per 16 value columns of a head, for the long segments only: a CTA takes an SM's shared memory, so one that finds nothing to do
// still holds up those behind it.  The state stays in registers and S0 goes through matrix instructions.
//
// All arithmetic keeps float32's precision.  The products run as bfloat16 matrix instructions on operands split into three
// bfloat16 parts (x = h + m + l, 24 bits down to 2^-109, below which bfloat16 ends before they do), six of the nine products (hh, hm, mh, hl, lh, mm; the rest is below 2^-24), the five small
// ones in an accumulator of their own.  Per flop that is as fast as three TF32 products, which would keep 22 bits, and 1.3 times
// the CUDA cores' peak, of which register blocks this small reach a third.
#include "tc5.cuh"

#define CHUNK_DECAY 0            // the modes of recurrent.cu
#define CHUNK_DELTA 2
#define CHUNK_BONUS 3
#define CHUNK_SSM 4
#define CHUNK_DELTA_HEAD 5

namespace {

constexpr int CT = 32;                   // tokens of a chunk
constexpr int THREADS = 256;
constexpr int COLS = 16;                 // value columns of a CTA of the second kernel

struct ChunkArgs {
    const void* q; const void* k; const void* v;        // (t, head, i) at base + t * ld + head * dim + i
    int q_ld, k_ld, v_ld;
    int q_f32, k_f32, v_f32;                            // 1: float32, 0: bfloat16
    const float* gate_a; const float* gate_b; const float* extra;       // as in ScanArgs (recurrent.cu)
    float q_scale;
    float* state; long long state_stride; int s_off;
    const int* cu_q; const int* seg_slot;
    float* scratch;                                     // [chunk of the window][head][per_head floats]
    float* out;                                         // [T, H * V]
    int* status;                                        // set to 1 if a wait gave up
    int H, G, D, V, segments;
    int min_tokens;                                     // segments of fewer tokens are none of these kernels' business
    int longs;                                          // how many segments are long (at most)
    int first, count;                                   // the window: these chunks of all segments' chunks, counted in order
};

// What a chunk leaves per head, in floats: q * P, k * P_32 / P_t, M, P_32, eight marks (one a warp: whether anything is not an
// ordinary number; 32 places, so that chunks lie on 128-byte boundaries), then (delta rules) k * P, T.  Matrices lie in the order of
// m16n8k16's second operand: [block of 16 along the sum][block of 8 along the other side][lane][4], lane l holding column l / 4
// and rows 2 (l % 4) + {0, 1, 8, 9}.
template <int DP> struct Layout {
    static constexpr int X = CT * DP;
    static constexpr int Q = 0, KS = X, M = 2 * X, G = 2 * X + CT * CT, MARKS = G + DP, KP = MARKS + 32, T = KP + X, DELTA = T + CT * CT, PLAIN = KP;
};

template <int MODE> constexpr bool is_delta() { return MODE == CHUNK_DELTA || MODE == CHUNK_DELTA_HEAD; }

__device__ __forceinline__ float ld_elem(const void* p, int f32, size_t i) {
    return f32 ? ((const float*)p)[i] : __bfloat162float(((const bf16*)p)[i]);
}

// Chunks of segments base + 32 u + lane (0: a segment that is none of these kernels' business), and where these begin and end, all
// looked up together.
struct Found { int own[4], begin[4], end[4]; };
__device__ __forceinline__ Found own_chunks(const ChunkArgs& a, int base, int lane) {
    Found f;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int s = base + 32 * u + lane;
        f.begin[u] = s < a.segments ? a.cu_q[s] : 0;
        f.end[u] = s < a.segments ? a.cu_q[s + 1] : 0;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int len = f.end[u] - f.begin[u];
        f.own[u] = len >= a.min_tokens ? (len + CT - 1) / CT : 0;
    }
    return f;
}
struct Place { int seg, chunk, begin, end; };            // a segment (-1: none), a chunk or a number of chunks, the segment's tokens

// The `which`-th long segment and how many chunks lie in front of it, by one warp.
__device__ __forceinline__ Place find_segment(const ChunkArgs& a, int which, int lane) {
    Place p = {-1, 0, 0, 0};
    for (int base = 0; base < a.segments && p.seg < 0; base += 128) {
        const Found f = own_chunks(a, base, lane);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const unsigned there = __ballot_sync(0xffffffffu, f.own[u] > 0);
            const bool here = p.seg < 0 && which < __popc(there);
            const bool it = here && f.own[u] > 0 && __popc(there & ((1u << lane) - 1u)) == which;
            const int at = here ? __ffs(__ballot_sync(0xffffffffu, it)) - 1 : 0;
            if (p.seg < 0) p.chunk += __reduce_add_sync(0xffffffffu, !here || lane < at ? f.own[u] : 0);
            if (here) {
                p.seg = base + 32 * u + at;
                p.begin = __shfl_sync(0xffffffffu, f.begin[u], at);
                p.end = __shfl_sync(0xffffffffu, f.end[u], at);
            }
            which -= __popc(there);
        }
    }
    return p;
}

// The segment that chunk `c` belongs to and the chunk's number in it, by one warp.
__device__ __forceinline__ Place find_chunk(const ChunkArgs& a, int c, int lane) {
    for (int base = 0; base < a.segments; base += 128) {
        const Found f = own_chunks(a, base, lane);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int all = __reduce_add_sync(0xffffffffu, f.own[u]);
            if (c < all) {
                int upto = f.own[u];                     // inclusive sums over the lanes
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, upto, o);
                    if (lane >= o) upto += v;
                }
                const int at = __ffs(__ballot_sync(0xffffffffu, c < upto)) - 1;
                return {base + 32 * u + at, c - __shfl_sync(0xffffffffu, upto - f.own[u], at), __shfl_sync(0xffffffffu, f.begin[u], at),
                        __shfl_sync(0xffffffffu, f.end[u], at)};
            }
            c -= all;
        }
    }
    return {-1, 0, 0, 0};
}

// ---------------------------------------------------------------- float32 products by three bfloat16 parts
// Beyond this the leading part would be an infinity.  An infinity or a NaN has no parts, and multiplied with the zeros above a
// triangle's diagonal it would reach the tokens before its own: chunks in which one turns up make a segment take the slow way (walk_tokens).
constexpr float LARGEST = 3.38e38f;
__device__ __forceinline__ bool ordinary(float x) { return fabsf(x) <= LARGEST; }
__device__ __forceinline__ bool ordinary(const float4& x) { return ordinary(x.x) && ordinary(x.y) && ordinary(x.z) && ordinary(x.w); }

struct Parts { unsigned h, m, l; };      // of two neighbouring elements: the first in the low half

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
__device__ __forceinline__ void mma(float (&c)[4], const uint4& a, unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
struct First { uint4 h, m, l; };         // the parts of a first operand
__device__ __forceinline__ First first_of(const unsigned* planes, int lane) {
    const uint4* p = reinterpret_cast<const uint4*>(planes) + lane;
    return {p[0], p[32], p[64]};
}
// big[j] += the product of the leading parts with b[j], small[j] += the five others; one kind of product after the other over
// all j, so that no instruction waits for the one before it
template <int N>
__device__ __forceinline__ void mma6(float (&big)[N][4], float (&small)[N][4], const First& a, const float4 (&b)[N]) {
    Parts p[N], r[N];
#pragma unroll
    for (int j = 0; j < N; ++j) { p[j] = split(b[j].x, b[j].y); r[j] = split(b[j].z, b[j].w); }
#pragma unroll
    for (int j = 0; j < N; ++j) mma(big[j], a.h, p[j].h, r[j].h);
#pragma unroll
    for (int j = 0; j < N; ++j) mma(small[j], a.m, p[j].m, r[j].m);
#pragma unroll
    for (int j = 0; j < N; ++j) mma(small[j], a.h, p[j].l, r[j].l);
#pragma unroll
    for (int j = 0; j < N; ++j) mma(small[j], a.l, p[j].h, r[j].h);
#pragma unroll
    for (int j = 0; j < N; ++j) mma(small[j], a.h, p[j].m, r[j].m);
#pragma unroll
    for (int j = 0; j < N; ++j) mma(small[j], a.m, p[j].h, r[j].h);
}
// Two blocks along the sum of one block of a second operand, `stride` floats apart.
__device__ __forceinline__ void two_blocks(float4 (&x)[2], const float* b, int stride, int lane) {
#pragma unroll
    for (int k = 0; k < 2; ++k) x[k] = *reinterpret_cast<const float4*>(b + k * stride + lane * 4);
}
// sum of up to two products, for a tile that stands alone: the small products run in three accumulators side by side
__device__ __forceinline__ void mma6_alone(float (&out)[4], const unsigned* planes, const float4 (&b)[2], int blocks, int lane) {
    float acc[2][4][4];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[k][j][i] = 0.f;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        if (k < blocks) {
            const First a = first_of(planes + k * 384, lane);
            const Parts p = split(b[k].x, b[k].y), r = split(b[k].z, b[k].w);
            mma(acc[k][0], a.h, p.h, r.h);
            mma(acc[k][1], a.m, p.m, r.m);
            mma(acc[k][2], a.h, p.l, r.l);
            mma(acc[k][3], a.l, p.h, r.h);
            mma(acc[k][1], a.h, p.m, r.m);
            mma(acc[k][2], a.m, p.h, r.h);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        out[i] = (acc[0][0][i] + acc[1][0][i]) + ((acc[0][1][i] + acc[1][1][i]) + (acc[0][2][i] + acc[1][2][i]) + (acc[0][3][i] + acc[1][3][i]));
}

// ---------------------------------------------------------------- first kernel: everything that does not need the state
// Tokens stand in four blocks of eight.  Pairs within a block: a warp per block and matrix, lanes over the key rows, a running
// product of decays from the later token down to the earlier, and one exchange that sums 32 pairs over the 32 lanes (31
// shuffles instead of 160).  Pairs of two blocks a > b: P_t / P_s is (decays of a up to t) (whole blocks between) (decays of b
// behind s), three factors of at most one, so the pairs are a product of 16 x DP (k and q rows of a) by DP x 8 on the matrix
// instructions.  T follows by forward substitution, a lane a column, while the other warps write.
constexpr int PAD = 8;                   // floats between rows in shared memory: 8-byte reads of 4 rows x 4 lanes hit all banks

// Sums 32 values over the lanes; lane l gets the sum of value l.
__device__ __forceinline__ float exchange_sums(float (&v)[32], int lane) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            if (j < o) {
                const float send = up ? v[j] : v[j + o], keep = up ? v[j + o] : v[j];
                v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
    }
    return v[0];
}

// 32 rows of D elements of a matrix into shared memory, all of a thread's loads in flight together; what does not exist is `none`.
template <int DP>
__device__ __forceinline__ void load_rows(float* to, const void* p, int f32, int t0, int n, int ld, int off, int D, float scale, float none) {
    constexpr int PITCH = DP + PAD, N = CT * DP / 4 / THREADS;
    const int tid = threadIdx.x;
    const bool vec = D % 4 == 0 && ld % 4 == 0 && off % 4 == 0 && (reinterpret_cast<uintptr_t>(p) & (f32 ? 15 : 7)) == 0;
    uint4 x[N];
    if (vec) {
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const int e = tid + u * THREADS, t = e / (DP / 4), i = (e % (DP / 4)) * 4;
            const size_t at = (size_t)(t0 + t) * ld + off + i;
            const bool live = t < n && i < D;
            if (f32) {
                x[u] = live ? *reinterpret_cast<const uint4*>((const float*)p + at) : make_uint4(0u, 0u, 0u, 0u);
            } else {
                const uint2 b = live ? *reinterpret_cast<const uint2*>((const bf16*)p + at) : make_uint2(0u, 0u);
                x[u] = make_uint4(b.x << 16, b.x & 0xffff0000u, b.y << 16, b.y & 0xffff0000u);
            }
        }
    }
#pragma unroll
    for (int u = 0; u < N; ++u) {
        const int e = tid + u * THREADS, t = e / (DP / 4), i = (e % (DP / 4)) * 4;
        float v[4];
        if (vec) {
            v[0] = __uint_as_float(x[u].x); v[1] = __uint_as_float(x[u].y); v[2] = __uint_as_float(x[u].z); v[3] = __uint_as_float(x[u].w);
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) v[c] = t < n && i + c < D ? ld_elem(p, f32, (size_t)(t0 + t) * ld + off + i + c) : 0.f;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) to[t * PITCH + i + c] = t < n && i + c < D ? v[c] * scale : none;
    }
}

template <int MODE, int DP>
__global__ void __launch_bounds__(THREADS, 3)
chunk_prep_kernel(const ChunkArgs a) {
    using L = Layout<DP>;
    constexpr bool DELTA = is_delta<MODE>();
    constexpr bool ROWS = MODE == CHUNK_DELTA || MODE == CHUNK_BONUS;    // a decay per key row
    constexpr int PITCH = DP + PAD, VEC = DP / 32;
    extern __shared__ __align__(16) float prep_smem[];
    float* Ks = prep_smem;                               // k, then k times the decays of its block up to it
    float* Qs = Ks + CT * PITCH;                         // q likewise
    float* Gs = Qs + CT * PITCH;                         // decays, then k times the decays of its block behind it
    __shared__ double bd[4][DP];                         // decays of the whole blocks: products are rounded once, where they are used
    __shared__ __align__(16) float Am[CT][CT + 4], Mm[CT][CT + 4], Tm[CT][CT + 4];
    __shared__ float beta[CT];
    __shared__ Place which;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int h = blockIdx.y;
    pdl_wait();
    if (warp == 0) {
        const Place w = find_chunk(a, a.first + blockIdx.x, lane);
        if (lane == 0) which = w;
    }
    for (int e = tid; e < CT * CT; e += THREADS) Am[e / CT][e % CT] = Mm[e / CT][e % CT] = 0.f;
    __syncthreads();
    if (which.seg < 0) return;
    const int t0 = which.begin + which.chunk * CT, n = min(CT, which.end - t0);
    const int H = a.H, D = a.D, kvh = h / (H / a.G);
    load_rows<DP>(Ks, a.k, a.k_f32, t0, n, a.k_ld, kvh * D, D, 1.f, 0.f);
    load_rows<DP>(Qs, a.q, a.q_f32, t0, n, a.q_ld, kvh * D, D, a.q_scale, 0.f);
    if (ROWS) {
        load_rows<DP>(Gs, a.gate_a, 1, t0, n, H * D, h * D, D, 1.f, 1.f);
    } else {
        const float g = MODE == CHUNK_DECAY ? a.gate_a[h] : lane < n ? a.gate_a[(size_t)(t0 + lane) * H + h] : 1.f;    // lane: token
#pragma unroll
        for (int t = warp; t < CT; t += THREADS / 32) {
            const float gt = t < n ? __shfl_sync(0xffffffffu, g, t) : 1.f;
#pragma unroll
            for (int i = lane; i < DP; i += 32) Gs[t * PITCH + i] = gt;
        }
    }
    if (DELTA && tid < CT) beta[tid] = tid < n ? a.gate_b[(size_t)(t0 + tid) * H + h] : 0.f;
    __syncthreads();

    // ---- pairs within a block: even warps A, odd warps M
    if (DELTA || (warp & 1)) {
        const int b = warp >> 1;
        const bool is_m = warp & 1;
        const float* X = is_m ? Qs : Ks;
        float k[8][VEC], g[8][VEC], v[32];
#pragma unroll
        for (int t = 0; t < 8; ++t)
#pragma unroll
            for (int c = 0; c < VEC; ++c) {
                k[t][c] = Ks[(8 * b + t) * PITCH + VEC * lane + c];
                g[t][c] = Gs[(8 * b + t) * PITCH + VEC * lane + c];
            }
        float diag[4];                                   // of tokens 4 to 7 (those of 0 to 3 ride along with the pairs)
#pragma unroll
        for (int j = 0; j < 4; ++j) { v[28 + j] = 0.f; diag[j] = 0.f; }
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            float y[VEC];
#pragma unroll
            for (int c = 0; c < VEC; ++c) y[c] = X[(8 * b + t) * PITCH + VEC * lane + c];
            if (is_m) {
                float d = 0.f;
#pragma unroll
                for (int c = 0; c < VEC; ++c) {
                    const int i = VEC * lane + c;
                    const float own = MODE == CHUNK_BONUS ? (i < D ? a.extra[(size_t)h * D + i] : 0.f) : 1.f;
                    d = fmaf(y[c] * own, k[t][c], d);
                }
                if (t < 4) v[28 + t] = d; else diag[t - 4] = d;
            }
            if (MODE != CHUNK_BONUS || !is_m) {          // the bonus rule reads the state before the token's own decay
#pragma unroll
                for (int c = 0; c < VEC; ++c) y[c] *= g[t][c];
            }
#pragma unroll
            for (int s = 7; s >= 0; --s) {
                if (s >= t) continue;
                float d = 0.f;
#pragma unroll
                for (int c = 0; c < VEC; ++c) {
                    d = fmaf(y[c], k[s][c], d);
                    y[c] *= g[s][c];
                }
                v[t * (t - 1) / 2 + s] = d;
            }
        }
        const float sum = exchange_sums(v, lane);
        float (*to)[CT + 4] = is_m ? Mm : Am;
        if (lane < 28) {
            int t = 1;
            while ((t + 1) * t / 2 <= lane) ++t;
            to[8 * b + t][8 * b + lane - t * (t - 1) / 2] = sum;
        } else if (is_m) {
            to[8 * b + lane - 28][8 * b + lane - 28] = sum;
        }
        if (is_m) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float d = warp_sum(diag[j]);
                if (lane == 0) to[8 * b + 4 + j][8 * b + 4 + j] = d;
            }
        }
    }
    __syncthreads();
    // ---- decays within the blocks
    for (int e = tid; e < 4 * DP; e += THREADS) {
        const int b = e / DP, i = e % DP;
        float* k = Ks + 8 * b * PITCH + i;
        float* q = Qs + 8 * b * PITCH + i;
        float* gk = Gs + 8 * b * PITCH + i;
        float g[8], ks[8];
        double p = 1.0;
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            g[t] = gk[t * PITCH];
            ks[t] = k[t * PITCH];
            if (MODE == CHUNK_BONUS) q[t * PITCH] *= (float)p;
            p *= (double)g[t];
            if (MODE != CHUNK_BONUS) q[t * PITCH] *= (float)p;
            if (DELTA) k[t * PITCH] = ks[t] * (float)p;
        }
        bd[b][i] = p;
        p = 1.0;
#pragma unroll
        for (int t = 7; t >= 0; --t) {
            gk[t * PITCH] = ks[t] * (float)p;
            p *= (double)g[t];
        }
    }
    __syncthreads();
    // ---- pairs of two blocks: six of them, a warp each
    if (warp < 6) {
        const int hi = warp < 1 ? 1 : warp < 3 ? 2 : 3, lo = warp - hi * (hi - 1) / 2;
        const int r = lane >> 2, c2 = 2 * (lane & 3);
        float big[1][4] = {{0.f, 0.f, 0.f, 0.f}}, small[1][4] = {{0.f, 0.f, 0.f, 0.f}};
        const float* kx = Ks + (8 * hi + r) * PITCH + c2;
        const float* qx = Qs + (8 * hi + r) * PITCH + c2;
        const float* sx = Gs + (8 * lo + r) * PITCH + c2;
#pragma unroll 2
        for (int kt = 0; kt < DP / 16; ++kt) {
            const int i = 16 * kt;
            float2 b0 = *(const float2*)(sx + i), b1 = *(const float2*)(sx + i + 8);
            for (int mid = lo + 1; mid < hi; ++mid) {
                const double* w = bd[mid] + i + c2;
                b0.x *= (float)w[0]; b0.y *= (float)w[1]; b1.x *= (float)w[8]; b1.y *= (float)w[9];
            }
            const float2 q0 = *(const float2*)(qx + i), q1 = *(const float2*)(qx + i + 8);
            const Parts p1 = split(q0.x, q0.y), p3 = split(q1.x, q1.y);
            Parts p0 = {0u, 0u, 0u}, p2 = {0u, 0u, 0u};
            if (DELTA) {
                const float2 k0 = *(const float2*)(kx + i), k1 = *(const float2*)(kx + i + 8);
                p0 = split(k0.x, k0.y);
                p2 = split(k1.x, k1.y);
            }
            const First x = {make_uint4(p0.h, p1.h, p2.h, p3.h), make_uint4(p0.m, p1.m, p2.m, p3.m), make_uint4(p0.l, p1.l, p2.l, p3.l)};
            const float4 y[1] = {make_float4(b0.x, b0.y, b1.x, b1.y)};
            mma6<1>(big, small, x, y);
        }
        const int t = 8 * hi + r, s = 8 * lo + c2;
        if (DELTA) { Am[t][s] = big[0][0] + small[0][0]; Am[t][s + 1] = big[0][1] + small[0][1]; }
        Mm[t][s] = big[0][2] + small[0][2];
        Mm[t][s + 1] = big[0][3] + small[0][3];
    }
    __syncthreads();
    float* to = a.scratch + ((size_t)blockIdx.x * H + h) * (DELTA ? L::DELTA : L::PLAIN);
    bool fine = true;
    auto leave = [&](int at, const float4& x) {
        *(float4*)(to + at) = x;
        fine = fine && ordinary(x);
    };
    // ---- T by forward substitution (warp 0; a lane a column), the writes by the others
    if (DELTA && warp == 0) {
        float T[CT];
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            float s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int s = 0; s < t; s += 4) {
                const float4 a4 = *(const float4*)&Am[t][s];             // zero on and above the diagonal
                s4[0] = fmaf(a4.x, T[s], s4[0]);
                if (s + 1 < t) s4[1] = fmaf(a4.y, T[s + 1], s4[1]);
                if (s + 2 < t) s4[2] = fmaf(a4.z, T[s + 2], s4[2]);
                if (s + 3 < t) s4[3] = fmaf(a4.w, T[s + 3], s4[3]);
            }
            T[t] = beta[t] * ((t == lane ? 1.f : 0.f) - ((s4[0] + s4[1]) + (s4[2] + s4[3])));
            Tm[t][lane] = T[t];
        }
    } else {
        const int w0 = DELTA ? warp - 1 : warp, ws = DELTA ? 7 : 8;
        const int r = lane >> 2, c2 = 2 * (lane & 3);
        // second operands whose sum runs over the key rows: q * P and k * P
        for (int e = w0; e < (DP / 16) * (CT / 8); e += ws) {
            const int kt = e / (CT / 8), nt = e % (CT / 8), i = 16 * kt + c2;
            double d[4] = {1.0, 1.0, 1.0, 1.0};
            for (int b = 0; b < nt; ++b) { d[0] *= bd[b][i]; d[1] *= bd[b][i + 1]; d[2] *= bd[b][i + 8]; d[3] *= bd[b][i + 9]; }
            const float p[4] = {(float)d[0], (float)d[1], (float)d[2], (float)d[3]};
            const float* q = Qs + (8 * nt + r) * PITCH + i;
            leave(L::Q + e * 128 + lane * 4, make_float4(q[0] * p[0], q[1] * p[1], q[8] * p[2], q[9] * p[3]));
            if (DELTA) {
                const float* k = Ks + (8 * nt + r) * PITCH + i;
                leave(L::KP + e * 128 + lane * 4, make_float4(k[0] * p[0], k[1] * p[1], k[8] * p[2], k[9] * p[3]));
            }
        }
        // ... over the tokens: k * P_32 / P_t
        for (int e = w0; e < (CT / 16) * (DP / 8); e += ws) {
            const int kt = e / (DP / 8), i = 8 * (e % (DP / 8)) + r, t = 16 * kt + c2;
            double d = 1.0;                              // decays of the blocks behind the second eight tokens, then the first
            for (int b = 2 * kt + 2; b < 4; ++b) d *= bd[b][i];
            const float p1 = (float)d, p0 = (float)(d * bd[2 * kt + 1][i]);
            const float* k = Gs + t * PITCH + i;
            leave(L::KS + e * 128 + lane * 4, make_float4(k[0] * p0, k[PITCH] * p0, k[8 * PITCH] * p1, k[9 * PITCH] * p1));
        }
        if (w0 == 0) {
            for (int i = lane; i < DP; i += 32) {
                const float g = (float)(bd[0][i] * bd[1][i] * bd[2][i] * bd[3][i]);
                to[L::G + i] = g;
                fine = fine && ordinary(g);
            }
        }
        for (int e = w0; e < (CT / 16) * (CT / 8); e += ws) {
            const int kt = e / (CT / 8), t = 8 * (e % (CT / 8)) + r, s = 16 * kt + c2;
            leave(L::M + e * 128 + lane * 4, make_float4(Mm[t][s], Mm[t][s + 1], Mm[t][s + 8], Mm[t][s + 9]));
        }
    }
    if (DELTA) {
        __syncthreads();
        const int kt = warp / (CT / 8), t = 8 * (warp % (CT / 8)) + (lane >> 2), s = 16 * kt + 2 * (lane & 3);
        leave(L::T + warp * 128 + lane * 4, make_float4(Tm[t][s], Tm[t][s + 1], Tm[t][s + 8], Tm[t][s + 9]));
    }
    const bool marked = __any_sync(0xffffffffu, !fine);
    if (lane == 0) to[L::MARKS + warp] = marked ? 1.f : 0.f;
    pdl_trigger_late();
}

// ---------------------------------------------------------------- second kernel: the chunks of a segment in order
// Everything is transposed: value columns are the 16 rows of the matrix instructions' first operand, so that their results
// (state, v - (k * P) S0, U) are already laid out as the next product's first operand, lane by lane.  Of the 16 warps (8 for keys
// up to 64) one half works on k * P, the other on q * P, each warp on 16 of the key rows over which those products sum; the parts
// meet in shared memory.  U = T (v - ...) is made by the first four warps, the outputs by the last four (while the next chunk's U is
// made), and every warp updates eight of the state's rows, which it keeps in float32 registers, and leaves their three parts for
// the next chunk.  Chunks come by bulk copies, two ahead; every wait for one is bounded (status word).  Bound by the latency of
// a chunk's steps one behind the other: 2.3 us a chunk of the delta rule with keys of 128 (64 chunks of 16 heads of 128 x 128: 149 us;
// the matrix instructions alone would be 0.75 us a chunk), 1.6 us of the others (100 us).  With cp.async by all threads in the place of the
// bulk copies and the outputs finished in their own chunk: 187 and 128 us; with eight warps instead of sixteen and the values'
// conversion behind their load: 167 and 184; with the outputs' sums and the checks of U and of the state on the chain: 157 and 107.
// The first kernel takes 54 and 38 us there (62 and 45 with two CTAs an SM instead of three); token by token it was 893 and 508.
// Whether everything was an ordinary number is asked of the outputs only and answered once, behind the last chunk.
constexpr int STAGES = 3;

__device__ __forceinline__ void bulk_copy(unsigned smem, const float* gmem, unsigned bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem), "l"(gmem), "r"(bytes), "r"(bar) : "memory");
}

template <int DP> constexpr int serial_warps() { return DP / 8; }

template <int DP, bool DELTA> constexpr size_t serial_smem() {
    return (size_t)STAGES * (DELTA ? Layout<DP>::DELTA : Layout<DP>::PLAIN) * 4      // chunks
           + (size_t)(DELTA ? 2 : 1) * (DP / 16) * 512 * 4                           // parts of the sums over the key rows
           + (size_t)(DP / 16 + 2 + 4) * 384 * 4;                                    // the state, v - (k * P) S0 and U (of two chunks) in three parts
}

// Tokens t0 .. t0 + n - 1 one by one, by the CTA that keeps the state S (two rows of two columns a thread, laid out as in
// chunk_serial_kernel): a segment in which an infinity or a NaN turned up, once more from the state that it began with, so that it reaches
// the tokens and columns that it reaches in recurrent.cu, and no others.  `sums`: 48 floats a warp.
template <int MODE, int DP>
__device__ __noinline__ float4 walk_tokens(const ChunkArgs& a, int t0, int n, int h, int col, float4 S4, float* sums) {
    constexpr bool DELTA = is_delta<MODE>(), ROWS = MODE == CHUNK_DELTA || MODE == CHUNK_BONUS;
    constexpr int WARPS = serial_warps<DP>();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c8 = lane >> 2, i0 = 8 * warp + 2 * (lane & 3);
    const int H = a.H, D = a.D, V = a.V, kvh = h / (H / a.G);
    float S[4] = {S4.x, S4.y, S4.z, S4.w};
    const bool ok[2] = {col < V, col + 8 < V}, row[2] = {i0 < D, i0 + 1 < D};
    auto quad = [](float x) {
        x += __shfl_xor_sync(0xffffffffu, x, 1);
        return x + __shfl_xor_sync(0xffffffffu, x, 2);
    };
    // the sums over a column's rows: this warp's, left in shared memory; then (behind a barrier) all warps'
    auto put_sums = [&](float* to, float x, float y) {
        x = quad(x);
        y = quad(y);
        if ((lane & 3) == 0) { to[warp * 16 + c8] = x; to[warp * 16 + 8 + c8] = y; }
    };
    auto all_of = [&](const float* from, int c) {
        float x = 0.f;
        for (int w = 0; w < WARPS; ++w) x += from[w * 16 + 8 * c + c8];
        return x;
    };
    __syncthreads();                                     // nobody reads what lay here before
    for (int i = 0; i < n; ++i) {
        const size_t t = (size_t)(t0 + i);
        float k[2], q[2], g[2], w[2], v[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            k[r] = row[r] ? ld_elem(a.k, a.k_f32, t * a.k_ld + (size_t)kvh * D + i0 + r) : 0.f;
            q[r] = row[r] ? ld_elem(a.q, a.q_f32, t * a.q_ld + (size_t)kvh * D + i0 + r) * a.q_scale : 0.f;
            g[r] = !row[r] ? 1.f : MODE == CHUNK_DECAY ? a.gate_a[h] : ROWS ? a.gate_a[(t * H + h) * D + i0 + r] : a.gate_a[t * H + h];
            w[r] = MODE == CHUNK_BONUS && row[r] ? a.extra[(size_t)h * D + i0 + r] : 0.f;
            v[r] = ok[r] ? ld_elem(a.v, a.v_f32, t * a.v_ld + (size_t)h * V + col + 8 * r) : 0.f;
        }
        float u[2] = {v[0], v[1]}, o[2] = {0.f, 0.f};
        if (DELTA) {
            float p[2] = {0.f, 0.f};
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    S[2 * c + r] *= g[r];
                    if (row[r]) p[c] = fmaf(S[2 * c + r], k[r], p[c]);
                }
            put_sums(sums, p[0], p[1]);
            __syncthreads();
            const float beta = a.gate_b[t * H + h];
#pragma unroll
            for (int c = 0; c < 2; ++c) u[c] = beta * (v[c] - all_of(sums, c));
        } else if (MODE == CHUNK_SSM) {
            const float step = a.gate_b[t * H + h];
            u[0] *= step;
            u[1] *= step;
        }
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                if (!row[r]) continue;
                float& s = S[2 * c + r];
                if (MODE == CHUNK_BONUS) o[c] = fmaf(fmaf(w[r], k[r] * u[c], s), q[r], o[c]);
                s = DELTA ? fmaf(k[r], u[c], s) : fmaf(g[r], s, k[r] * u[c]);
                if (MODE != CHUNK_BONUS) o[c] = fmaf(s, q[r], o[c]);
            }
        float* mine = sums + (1 + (i & 1)) * 16 * WARPS;
        put_sums(mine, o[0], o[1]);
        __syncthreads();
        if (warp == 0 && (lane & 3) == 0) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                float x = all_of(mine, c);
                if (MODE == CHUNK_SSM) x = fmaf(a.extra[h], v[c], x);
                if (ok[c]) a.out[(t * H + h) * V + col + 8 * c] = x;
            }
        }
    }
    __syncthreads();
    return make_float4(S[0], S[1], S[2], S[3]);
}

template <int MODE, int DP>
__global__ void __launch_bounds__(32 * serial_warps<DP>(), 1)
chunk_serial_kernel(const ChunkArgs a) {
    using L = Layout<DP>;
    constexpr bool DELTA = is_delta<MODE>();
    constexpr int PER = DELTA ? L::DELTA : L::PLAIN;
    constexpr int WARPS = serial_warps<DP>(), KT = DP / 16, TB = DELTA ? 4 : 2;      // KT: blocks of 16 key rows; TB: blocks of 8 tokens of a warp
    constexpr bool PAIRED = WARPS == 16;                 // two warps share a block of tokens of v - (k * P) S0, a column of a lane each
    extern __shared__ __align__(128) float serial_smem_base[];
    float* stages = serial_smem_base;
    float* part = stages + STAGES * PER;                 // [k * P, q * P][KT][4 blocks of tokens][lane][4]
    unsigned* Sp = reinterpret_cast<unsigned*>(part + (DELTA ? 2 : 1) * KT * 512);   // [KT][3][lane][4]
    unsigned* Rp = Sp + KT * 384;                        // [2][3][lane][4]
    unsigned* Up = Rp + 2 * 384;                         // [chunk % 2][2][3][lane][4]
    __shared__ __align__(8) unsigned long long full[STAGES];
    __shared__ Place which;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int h = blockIdx.y, j0 = blockIdx.x * COLS;
    pdl_wait();
    if (warp == 0) {
        const Place w = find_segment(a, blockIdx.z, lane);
        if (lane == 0) {
            which = w;
#pragma unroll
            for (int i = 0; i < STAGES; ++i) tc5::mbar_init(tc5::smem_u32(&full[i]), 1);
            tc5::mbar_init_fence();
        }
    }
    __syncthreads();
    const int seg = which.seg, before = which.chunk, t_first = which.begin, t_end = which.end;
    if (seg < 0) return;
    // this segment's chunks that lie in the window
    const int c_begin = max(0, a.first - before);
    const int c_end = min((t_end - t_first + CT - 1) / CT, a.first + a.count - before);
    if (c_begin >= c_end) return;
    const int H = a.H, D = a.D, V = a.V, nrd = (D + 7) >> 3;
    const float* src = a.scratch + ((size_t)(before + c_begin - a.first) * H + h) * PER;
    const int chunks = c_end - c_begin;
    auto fetch = [&](int c) {                            // by one thread; every copy is waited for in its turn
        if (tid == 0 && c < chunks) {
            const unsigned bar = tc5::smem_u32(&full[c % STAGES]);
            tc5::mbar_arrive_expect_tx(bar, PER * 4);
            bulk_copy(tc5::smem_u32(stages + (c % STAGES) * PER), src + (size_t)c * H * PER, PER * 4, bar);
        }
    };
    fetch(0);
    fetch(1);

    const int col = j0 + (lane >> 2);                    // and col + 8
    const bool ok0 = col < V, ok1 = col + 8 < V;
    const bool in0 = warp < nrd && ok0, in1 = warp < nrd && ok1;
    // rows 8 warp + 2 (lane % 4) + {0, 1} of col and of col + 8; a slot's row may begin on any float
    float* home = a.state + (long long)a.seg_slot[seg] * a.state_stride + a.s_off + (size_t)h * nrd * 8 * V + ((size_t)warp * V + col) * 8 + 2 * (lane & 3);
    float S[4] = {in0 ? home[0] : 0.f, in0 ? home[1] : 0.f, in1 ? home[64] : 0.f, in1 ? home[65] : 0.f};
    // A first operand of 16 along the sum: registers 0, 1 are the first block of 8 (columns col and col + 8), 2, 3 the second.
    auto put = [&](unsigned* planes, int block, const float (&x)[4]) {
        const Parts lo = split(x[0], x[1]), hi = split(x[2], x[3]);
        unsigned* at = planes + (block >> 1) * 384 + lane * 4 + (block & 1) * 2;
        *(uint2*)at = make_uint2(lo.h, hi.h);
        *(uint2*)(at + 128) = make_uint2(lo.m, hi.m);
        *(uint2*)(at + 256) = make_uint2(lo.l, hi.l);
    };
    auto put_half = [&](unsigned* planes, int block, int which, float x0, float x1) {        // one of the two columns
        const Parts p = split(x0, x1);
        unsigned* at = planes + (block >> 1) * 384 + lane * 4 + (block & 1) * 2 + which;
        at[0] = p.h; at[128] = p.m; at[256] = p.l;
    };
    put(Sp, warp, S);
    const float skip = MODE == CHUNK_SSM ? a.extra[h] : 0.f;
    // who takes v - (k * P) S0 or v (block rb of 8 tokens; with PAIRED column rc of the two), and who the outputs (block ob)
    const bool right = warp < WARPS / 2, output = warp >= WARPS - 4;
    const int rb = PAIRED ? warp >> 1 : warp, rc = PAIRED ? warp & 1 : 0, ob = warp - (WARPS - 4);
    // Values of a chunk, asked for a chunk ahead: tokens ta, ta + 1 of col, then of col + 8, by the warps that need them (what is not
    // there stays zero).  The loaded bits stay as they are until they are used: a conversion right behind a load would make the warp
    // wait for it there.
    unsigned v_next[4] = {0u, 0u, 0u, 0u};
    float step_next[2] = {0.f, 0.f};
    const bool has_values = right || (MODE == CHUNK_SSM && output);
    const bool c0 = ok0 && !(PAIRED && right && rc), c1 = ok1 && !(PAIRED && right && !rc);
    int t_next = t_first + c_begin * CT + 8 * (right ? rb : ob) + 2 * (lane & 3);
    const int t_stop = min(t_end, t_first + c_end * CT);
    const char* v_at = (const char*)a.v + ((size_t)t_next * a.v_ld + (size_t)h * V + col) * (a.v_f32 ? 4 : 2);
    const size_t v_row = (size_t)a.v_ld * (a.v_f32 ? 4 : 2);
    auto values = [&]() {
        if (!has_values) return;
        const bool l0 = t_next < t_stop, l1 = t_next + 1 < t_stop;
        if (a.v_f32) {
            const unsigned* p = (const unsigned*)v_at;
            const unsigned* n = (const unsigned*)(v_at + v_row);
            v_next[0] = l0 && c0 ? p[0] : 0u;
            v_next[1] = l1 && c0 ? n[0] : 0u;
            v_next[2] = l0 && c1 ? p[8] : 0u;
            v_next[3] = l1 && c1 ? n[8] : 0u;
        } else {
            const unsigned short* p = (const unsigned short*)v_at;
            const unsigned short* n = (const unsigned short*)(v_at + v_row);
            v_next[0] = l0 && c0 ? p[0] : 0u;
            v_next[1] = l1 && c0 ? n[0] : 0u;
            v_next[2] = l0 && c1 ? p[8] : 0u;
            v_next[3] = l1 && c1 ? n[8] : 0u;
        }
        if (MODE == CHUNK_SSM && right) {
            step_next[0] = l0 ? a.gate_b[(size_t)t_next * H + h] : 0.f;
            step_next[1] = l1 ? a.gate_b[(size_t)(t_next + 1) * H + h] : 0.f;
        }
        t_next += CT;
        v_at += CT * v_row;
    };
    values();
    // A chunk's outputs are finished while the next one's U is made, by warps that have nothing to do with that: they keep
    // (q * P) S0, their rows of M and (for the skip) the values.  An infinity or a NaN anywhere (in the state, in U, in a value) is in some
    // output of its column, times a zero or not, so they alone are looked at, and the marks of what the first kernel left.
    float o_sum[4], o_skip[4] = {0.f, 0.f, 0.f, 0.f};
    float4 o_m[2];
    bool ok = true, odd = false;                         // odd: something was no ordinary number
    auto finish = [&](int c) {
        float own[4];
        mma6_alone(own, Up + (c & 1) * 768, o_m, (ob >> 1) + 1, lane);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            own[i] += o_sum[i];
            if (MODE == CHUNK_SSM) own[i] = fmaf(skip, o_skip[i], own[i]);
            odd = odd || !ordinary(own[i]);
        }
        const int ta = t_first + (c_begin + c) * CT + 8 * ob + 2 * (lane & 3);
        float* o = a.out + ((size_t)ta * H + h) * V + col;
        if (ta < t_end) {
            if (ok0) o[0] = own[0];
            if (ok1) o[8] = own[2];
        }
        if (ta + 1 < t_end) {
            if (ok0) o[(size_t)H * V] = own[1];
            if (ok1) o[(size_t)H * V + 8] = own[3];
        }
    };

    for (int c = 0; c < chunks; ++c) {
        ok = tc5::mbar_wait(tc5::smem_u32(&full[c % STAGES]), (c / STAGES) & 1) && ok;
        __syncthreads();                                 // the state's parts are there; nobody is in chunk c - 1
        fetch(c + 2);
        const float* X = stages + (c % STAGES) * PER;
        if (warp == WARPS / 2 && lane < 8) odd = odd || X[L::MARKS + lane] != 0.f;
        float v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[i] = __uint_as_float(a.v_f32 ? v_next[i] : v_next[i] << 16);
            if (MODE == CHUNK_SSM && right) v[i] *= step_next[i & 1];
        }
        values();
        // ---- products with the state, over 16 of the key rows
        {
            const int half = warp / KT, kt = warp % KT, nt0 = DELTA ? 0 : 2 * half;
            const float* B = X + (DELTA && half == 0 ? L::KP : L::Q) + (kt * 4 + nt0) * 128 + lane * 4;
            float big[TB][4], small[TB][4];
            float4 b[TB];
#pragma unroll
            for (int nt = 0; nt < TB; ++nt) {
                b[nt] = *reinterpret_cast<const float4*>(B + nt * 128);
#pragma unroll
                for (int i = 0; i < 4; ++i) big[nt][i] = small[nt][i] = 0.f;
            }
            mma6<TB>(big, small, first_of(Sp + kt * 384, lane), b);
            float* to = part + ((DELTA ? half * KT : 0) + kt) * 512 + nt0 * 128 + lane * 4;
#pragma unroll
            for (int nt = 0; nt < TB; ++nt)
                *(float4*)(to + nt * 128) = make_float4(big[nt][0] + small[nt][0], big[nt][1] + small[nt][1], big[nt][2] + small[nt][2],
                                                        big[nt][3] + small[nt][3]);
        }
        if (!DELTA && output && c > 0) finish(c - 1);
        if (!DELTA && right) {
            if (PAIRED) put_half(Up + (c & 1) * 768, rb, rc, rc ? v[2] : v[0], rc ? v[3] : v[1]);
            else put(Up + (c & 1) * 768, rb, v);
        }
        __syncthreads();
        float o_new[4] = {0.f, 0.f, 0.f, 0.f};
        if (output) {
            const float* from = part + (DELTA ? KT * 512 : 0) + ob * 128 + lane * 4;
#pragma unroll
            for (int w = 0; w < KT; ++w) {
                const float4 x = *(const float4*)(from + w * 512);
                o_new[0] += x.x; o_new[1] += x.y; o_new[2] += x.z; o_new[3] += x.w;
            }
        }
        if (DELTA) {
            if (right) {
                const float* from = part + rb * 128 + lane * 4;
                if (PAIRED) {
                    float x0 = rc ? v[2] : v[0], x1 = rc ? v[3] : v[1], s0 = 0.f, s1 = 0.f;
#pragma unroll
                    for (int w = 0; w < KT; ++w) {
                        const float2 x = *(const float2*)(from + w * 512 + 2 * rc);
                        s0 += x.x; s1 += x.y;
                    }
                    put_half(Rp, rb, rc, x0 - s0, x1 - s1);
                } else {
                    float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int w = 0; w < KT; ++w) {
                        const float4 x = *(const float4*)(from + w * 512);
                        sum[0] += x.x; sum[1] += x.y; sum[2] += x.z; sum[3] += x.w;
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[i] -= sum[i];
                    put(Rp, rb, v);
                }
            }
            __syncthreads();
            if (warp < 4) {
                float u[4];
                float4 x[2];
                two_blocks(x, X + L::T + warp * 128, 512, lane);
                mma6_alone(u, Rp, x, (warp >> 1) + 1, lane);
                put(Up + (c & 1) * 768, warp, u);
            } else if (output && c > 0) {
                finish(c - 1);
            }
            __syncthreads();
        }
        if (output) {
#pragma unroll
            for (int i = 0; i < 4; ++i) { o_sum[i] = o_new[i]; o_skip[i] = v[i]; }
            two_blocks(o_m, X + L::M + ob * 128, 512, lane);
        }
        // ---- the state behind the chunk, eight rows; it is added to on the CUDA cores, which round to nearest
        {
            const float2 g = *(const float2*)(X + L::G + 8 * warp + 2 * (lane & 3));
            float upd[4];
            float4 x[2];
            two_blocks(x, X + L::KS + warp * 128, (DP / 8) * 128, lane);
            mma6_alone(upd, Up + (c & 1) * 768, x, 2, lane);
            S[0] = fmaf(S[0], g.x, upd[0]); S[1] = fmaf(S[1], g.y, upd[1]);
            S[2] = fmaf(S[2], g.x, upd[2]); S[3] = fmaf(S[3], g.y, upd[3]);
            put(Sp, warp, S);
        }
    }
    if (output) finish(chunks - 1);
    // Looked at once, behind the last chunk: the slot still holds the state before the first, and every output is written again.
    if (__syncthreads_or(odd)) {
        const int t0 = t_first + c_begin * CT;
        const float4 s4 = walk_tokens<MODE, DP>(a, t0, min(t_end, t_first + c_end * CT) - t0, h, col,
                                                make_float4(in0 ? home[0] : 0.f, in0 ? home[1] : 0.f, in1 ? home[64] : 0.f, in1 ? home[65] : 0.f), part);
        S[0] = s4.x; S[1] = s4.y; S[2] = s4.z; S[3] = s4.w;
    }
    if (!ok) atomicExch(a.status, 1);
    pdl_trigger_late();
    if (in0) { home[0] = S[0]; home[1] = S[1]; }
    if (in1) { home[64] = S[2]; home[65] = S[3]; }
}

template <int MODE, int DP>
int launch_chunks(const ChunkArgs& a, cudaStream_t st) {
    constexpr size_t prep_bytes = (size_t)3 * CT * (DP + PAD) * 4, serial_bytes = serial_smem<DP, is_delta<MODE>()>();
    static PerDevice configured;
    int rc = configured.once([&](int) {
        const cudaError_t e = cudaFuncSetAttribute(chunk_prep_kernel<MODE, DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prep_bytes);
        return e != cudaSuccess ? e : cudaFuncSetAttribute(chunk_serial_kernel<MODE, DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)serial_bytes);
    });
    if (rc) return rc;
    rc = rb_launch_pdl(chunk_prep_kernel<MODE, DP>, dim3(a.count, a.H), dim3(THREADS), prep_bytes, st, a);
    if (rc) return rc;
    return rb_launch_pdl(chunk_serial_kernel<MODE, DP>, dim3((a.V + COLS - 1) / COLS, a.H, a.longs), dim3(32 * serial_warps<DP>()), serial_bytes, st, a);
}

template <int MODE>
int launch_mode(const ChunkArgs& a, cudaStream_t st) {
    return a.D <= 64 ? launch_chunks<MODE, 64>(a, st) : launch_chunks<MODE, 128>(a, st);
}

}  // namespace

// Floats of scratch for one chunk of all heads (0: a mode or size that these kernels do not take).
RB_EXPORT long long rb_chunked_scan_floats(int mode, int H, int D) {
    if (D <= 0 || D > 128 || H <= 0) return 0;
    const bool delta = mode == CHUNK_DELTA || mode == CHUNK_DELTA_HEAD;
    if (!delta && mode != CHUNK_DECAY && mode != CHUNK_BONUS && mode != CHUNK_SSM) return 0;
    if (D <= 64) return (long long)H * (delta ? Layout<64>::DELTA : Layout<64>::PLAIN);
    return (long long)H * (delta ? Layout<128>::DELTA : Layout<128>::PLAIN);
}

// The segments of at least `min_tokens` tokens, of which there are `longs` at most; `first` and `count`: which of their chunks, counted over all such segments in
// order.  A caller with less scratch than all chunks need goes through them window by window, in order.
RB_EXPORT int rb_chunked_scan(int mode, const void* q, const void* k, const void* v, int q_ld, int k_ld, int v_ld, int q_f32, int k_f32,
                              int v_f32, const float* gate_a, const float* gate_b, const float* extra, float q_scale, float* state,
                              long long state_stride, int s_off, const int* cu_q, const int* seg_slot, float* scratch, float* out, int H,
                              int G, int D, int V, int segments, int min_tokens, int longs, int first, int count, int* status, cudaStream_t st) {
    if (segments <= 0 || count <= 0) return 0;
    if (rb_chunked_scan_floats(mode, H, D) == 0 || V <= 0 || G <= 0 || H % G || min_tokens < 1 || first < 0) return (int)cudaErrorInvalidValue;
    if (((uintptr_t)scratch & 15) || longs < 1 || longs > 65535) return (int)cudaErrorInvalidValue;
    ChunkArgs a;
    a.q = q; a.k = k; a.v = v; a.q_ld = q_ld; a.k_ld = k_ld; a.v_ld = v_ld;
    a.q_f32 = q_f32; a.k_f32 = k_f32; a.v_f32 = v_f32;
    a.gate_a = gate_a; a.gate_b = gate_b; a.extra = extra; a.q_scale = q_scale;
    a.state = state; a.state_stride = state_stride; a.s_off = s_off; a.cu_q = cu_q; a.seg_slot = seg_slot;
    a.scratch = scratch; a.out = out; a.status = status; a.H = H; a.G = G; a.D = D; a.V = V; a.segments = segments;
    a.min_tokens = min_tokens; a.longs = longs; a.first = first; a.count = count;
    if (mode == CHUNK_DECAY) return launch_mode<CHUNK_DECAY>(a, st);
    if (mode == CHUNK_DELTA) return gate_b ? launch_mode<CHUNK_DELTA>(a, st) : (int)cudaErrorInvalidValue;
    if (mode == CHUNK_DELTA_HEAD) return gate_b ? launch_mode<CHUNK_DELTA_HEAD>(a, st) : (int)cudaErrorInvalidValue;
    if (mode == CHUNK_BONUS) return extra ? launch_mode<CHUNK_BONUS>(a, st) : (int)cudaErrorInvalidValue;
    return extra && gate_b ? launch_mode<CHUNK_SSM>(a, st) : (int)cudaErrorInvalidValue;
}
