// Causal grouped-query attention of the FP32 path over the paged cache, heads of 64 and 128: FP32 multiply-adds throughout,
// and a token's result bit for bit the same whether it comes in a portion or alone, whatever else is in the step.
//
// attention_generic.cu reads every key once per query head and walks the keys one by one; here a block keeps the rows of one
// kv head that read the same keys (tokens x heads of the group) and multiplies tiles.  To keep a token's result independent
// of the cut, the order of every operation on it follows from absolute key positions alone and is the same in both kernels:
//     keys in blocks of 64 [64 b, 64 b + 63], blocks in segments of 8 [512 s, 512 s + 511];
//     score: for every 32 dimensions two chains of multiply-adds, over the even and the odd ones, added; these sums one after the
//            other; times the scale (a masked key: -inf);
//     block: m' = max(m, its scores), p = exp(s - m'), l = l exp(m - m') + sum p, acc = acc exp(m - m') then + p v key by key;
//            the sum of p: keys j, j + 16, j + 32, j + 48 as (+) + (+), then a binary tree over j from its lowest bit up;
//     segment: from (-inf, 0, 0), merged into the running (m, l, acc) when it ends; the sink is where the running sums start.
// A block or segment of which a token sees nothing changes none of its bits, so tokens of one tile may differ in what they see.
// Formula, windows, chunks and sinks as in attention_generic.cu.
//
// Portions (attention_f32_tile): 64 rows (32 at heads of 128) x 64 keys per step, 128 threads of 8 x 4 scores and 8 x 4
// outputs, packed multiply-adds, keys and values through two buffers of asynchronous copies.  Bound by shared memory (12
// loads of 16 bytes for 128 multiply-adds) and by the blocks that an SM holds: two at heads of 64 (255 registers), one at heads of
// 128 (161 KB of shared memory).  Single tokens (attention_f32_rows): a
// block per (token, kv head, segment), partial results merged by a second launch - or per (token, kv head) where the segments
// would not fill the GPU any better.  1,087 tokens in three portions, 32 heads of 64: 188 us against 2,054 us of
// attention_generic.cu; two single tokens over 130 keys: 8.6 against 134 us.  2,048 tokens of 24/8 heads of 128: 1,423 us (1,673 with
// chains over the whole head and empty rows that made every key block an edge).
#include "common.cuh"

#define AF_KB 64                    // keys of a block
#define AF_SEG 512                  // keys of a segment
#define AF_CHAIN 32                 // dimensions of a score's chains
#define AF_THREADS 128
#define AF_MAX_GROUP 16

struct AfParams {
    const float *q, *k, *v;
    float* out;
    const int *block_table, *positions, *seq_of_token;
    const float* sinks;
    int bt_stride, n_q, n_kv, group, page, page_shift, window, chunk;      // page_shift: -1 where the page size is no power of two
    float scale;
};

__device__ __forceinline__ void af_copy16(float* dst_smem, const float* src, bool live) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
    const int n = live ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void af_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void af_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void af_fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long af_pair(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 af_split(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
// exp(a - b) where a <= b, and 1 where they are the same (both may be -inf).
__device__ __forceinline__ float af_factor(float a, float b) { return a == b ? 1.f : expf(a - b); }
__device__ __forceinline__ float af_scale(float a, float f) { return __fmul_rn(a, f); }
// A score's next two chains added to what came before them: rounded, never contracted into what follows.
__device__ __forceinline__ float af_score(float before, unsigned long long chains) {
    const float2 c = af_split(chains);
    return __fadd_rn(before, __fadd_rn(c.x, c.y));
}
// First key that the token at position pos sees.
__device__ __forceinline__ int af_first(const AfParams& p, int pos) {
    int lo = (p.window > 0 && pos - p.window + 1 > 0) ? pos - p.window + 1 : 0;
    if (p.chunk > 0 && pos - pos % p.chunk > lo) lo = pos - pos % p.chunk;
    return lo;
}

// Keys [64 b, 64 b + 64) of one request and kv head into shared memory, zeros outside [from, to].
template <int HD>
__device__ __forceinline__ void af_fetch(const AfParams& p, const int* table, int kvh, int b, int from, int to, float* ks, float* vs) {
    constexpr int G16 = HD / 4, PITCH = HD + 4;
    for (int i = threadIdx.x; i < AF_KB * G16; i += AF_THREADS) {
        const int row = i / G16, c = 4 * (i % G16), key = b * AF_KB + row;
        const bool live = key >= from && key <= to;
        size_t at = 0;
        if (live) {
            const int page = p.page_shift >= 0 ? key >> p.page_shift : key / p.page;
            at = (((size_t)table[page] * p.n_kv + kvh) * p.page + (key - page * p.page)) * HD + c;
        }
        af_copy16(ks + row * PITCH + c, p.k + at, live);
        af_copy16(vs + row * PITCH + c, p.v + at, live);
    }
}

// ---- portions --------------------------------------------------------------------------------------------------------
// Tile t of the plan covers tile_tokens query tokens of one request from tile_row0 on; a block takes one slice of it that
// fills its rows with (token, head of the group) pairs, and one kv head.
template <int HD, int RM>
__global__ void __launch_bounds__(AF_THREADS)
attention_f32_tile_kernel(AfParams p, const int* __restrict__ tile_seq, const int* __restrict__ tile_row0, int tile_tokens,
                          const int* __restrict__ cu_q, const int* __restrict__ kv_len, int slices) {
    constexpr int ROWS = 8 * RM, PITCH = HD + 4, PP = AF_KB + 4, DV = HD / 64;       // DV: groups of four output columns per thread
    extern __shared__ __align__(16) float af_smem[];
    ni_launch_dependents();                                // the output projection asks for its weights meanwhile
    float* qs = af_smem;                                   // [ROWS][PITCH]
    float* ks = qs + ROWS * PITCH;                         // [2][64][PITCH]
    float* vs = ks + 2 * AF_KB * PITCH;                    // [2][64][PITCH]
    float* ps = vs + 2 * AF_KB * PITCH;                    // [ROWS][PP]
    const int tile = blockIdx.x / slices, slice = blockIdx.x % slices, kvh = blockIdx.y;
    const int seq = tile_seq[tile], q_len = cu_q[seq + 1] - cu_q[seq], start = kv_len[seq] - q_len;
    const int per = ROWS / p.group;                        // tokens of a block
    const int tok0 = tile_row0[tile] + slice * per;        // in the portion
    int tok1 = tok0 + per;
    if (tok1 > tile_row0[tile] + tile_tokens) tok1 = tile_row0[tile] + tile_tokens;
    if (tok1 > q_len) tok1 = q_len;
    if (tok0 >= tok1) return;
    const int rows = (tok1 - tok0) * p.group;
    const int* table = p.block_table + (size_t)seq * p.bt_stride;
    const size_t q_row0 = (size_t)(cu_q[seq] + tok0);
    for (int i = threadIdx.x; i < ROWS * (HD / 4); i += AF_THREADS) {
        const int r = i / (HD / 4), c = 4 * (i % (HD / 4));
        const bool live = r < rows;
        const size_t at = live ? ((q_row0 + r / p.group) * p.n_q + kvh * p.group + r % p.group) * HD + c : 0;
        af_copy16(qs + r * PITCH + c, p.q + at, live);
    }
    const int pos_first = start + tok0, pos_last = start + tok1 - 1;
    const int from = af_first(p, pos_first), b_first = from / AF_KB, b_last = pos_last / AF_KB;      // af_first grows with pos
    af_fetch<HD>(p, table, kvh, b_first, from, pos_last, ks, vs);
    af_commit();

    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4, r0 = ty * RM;
    int pos[RM], lo[RM];
    float m_run[RM], l_run[RM], m[RM], l[RM];
    unsigned long long run[RM][2 * DV], acc[RM][2 * DV];
#pragma unroll
    for (int i = 0; i < RM; ++i) {
        const int r = r0 + i;
        pos[i] = r < rows ? start + tok0 + r / p.group : -1;               // a row that is not there sees nothing
        lo[i] = r < rows ? af_first(p, pos[i]) : 0;
        m_run[i] = p.sinks && r < rows ? p.sinks[kvh * p.group + r % p.group] : -INFINITY;
        l_run[i] = p.sinks && r < rows ? 1.f : 0.f;
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int d = 0; d < 2 * DV; ++d) run[i][d] = acc[i][d] = 0ull;
    }
    for (int b = b_first; b <= b_last; ++b) {
        const int buf = (b - b_first) & 1;
        if (b < b_last) af_fetch<HD>(p, table, kvh, b + 1, from, pos_last, ks + (buf ^ 1) * AF_KB * PITCH, vs + (buf ^ 1) * AF_KB * PITCH);
        af_commit();
        af_wait<1>();
        __syncthreads();
        const float* kb = ks + buf * AF_KB * PITCH + tx * PITCH;
        const float* qb = qs + r0 * PITCH;
        float s[RM][4];
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 1
        for (int d0 = 0; d0 < HD; d0 += AF_CHAIN) {
            unsigned long long s2[RM][4];
#pragma unroll
            for (int i = 0; i < RM; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s2[i][j] = 0ull;
#pragma unroll 4
            for (int d = d0; d < d0 + AF_CHAIN; d += 4) {
                ulonglong2 kk[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) kk[j] = *reinterpret_cast<const ulonglong2*>(kb + 16 * j * PITCH + d);
#pragma unroll
                for (int i = 0; i < RM; ++i) {
                    const ulonglong2 qq = *reinterpret_cast<const ulonglong2*>(qb + i * PITCH + d);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        af_fma2(s2[i][j], qq.x, kk[j].x);
                        af_fma2(s2[i][j], qq.y, kk[j].y);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < RM; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[i][j] = af_score(s[i][j], s2[i][j]);
        }
        const int key = b * AF_KB + tx;
        // (a row that is not there counts as one that sees everything: it is never stored)
        const bool edge = b * AF_KB + AF_KB - 1 > pos_first || b * AF_KB < af_first(p, pos_last);
        // (the rows side by side in every step: a row's four exchanges and its exponentials are a chain of their own)
        float top[RM];
#pragma unroll
        for (int i = 0; i < RM; ++i) {
            top[i] = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const bool seen = !edge || (key + 16 * j <= pos[i] && key + 16 * j >= lo[i]);
                s[i][j] = seen ? af_scale(s[i][j], p.scale) : -INFINITY;
                top[i] = fmaxf(top[i], s[i][j]);
            }
        }
#pragma unroll
        for (int o = 1; o < 16; o <<= 1)
#pragma unroll
            for (int i = 0; i < RM; ++i) top[i] = fmaxf(top[i], __shfl_xor_sync(0xffffffffu, top[i], o));
        float sum[RM];
#pragma unroll
        for (int i = 0; i < RM; ++i) {
            const float m_new = fmaxf(m[i], top[i]), corr = af_factor(m[i], m_new);
            float w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const bool seen = !edge || (key + 16 * j <= pos[i] && key + 16 * j >= lo[i]);
                w[j] = seen ? expf(s[i][j] - m_new) : 0.f;
                ps[(r0 + i) * PP + tx + 16 * j] = w[j];
            }
            sum[i] = __fadd_rn(__fadd_rn(w[0], w[1]), __fadd_rn(w[2], w[3]));
            m[i] = m_new;
            top[i] = corr;
#pragma unroll
            for (int d = 0; d < 2 * DV; ++d) {
                const float2 a = af_split(acc[i][d]);
                acc[i][d] = af_pair(af_scale(a.x, corr), af_scale(a.y, corr));
            }
        }
#pragma unroll
        for (int o = 1; o < 16; o <<= 1)
#pragma unroll
            for (int i = 0; i < RM; ++i) sum[i] = __fadd_rn(sum[i], __shfl_xor_sync(0xffffffffu, sum[i], o));
#pragma unroll
        for (int i = 0; i < RM; ++i) l[i] = fmaf(l[i], top[i], sum[i]);
        __syncwarp();                                      // a half warp reads only the rows it has written itself
        const float* vb = vs + buf * AF_KB * PITCH + 4 * tx;
        const float* pb = ps + r0 * PP;
        // a key that a row does not see has the weight 0 there, which leaves the row alone unless its value is not a number or
        // infinite: then (never, in a sound model) the row must not touch it at all
        bool plain = true;
        if (edge) {
            bool odd = false;
            for (int i = threadIdx.x; i < AF_KB * (HD / 4); i += AF_THREADS) {
                const float4 v = *reinterpret_cast<const float4*>(vs + buf * AF_KB * PITCH + (i / (HD / 4)) * PITCH + 4 * (i % (HD / 4)));
                odd |= !(isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w));
            }
            plain = !__syncthreads_or(odd);
        }
        if (plain) {
#pragma unroll 2
            for (int j = 0; j < AF_KB; j += 4) {
                float4 w[RM];
#pragma unroll
                for (int i = 0; i < RM; ++i) w[i] = *reinterpret_cast<const float4*>(pb + i * PP + j);
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int g = 0; g < DV; ++g) {
                        const ulonglong2 vv = *reinterpret_cast<const ulonglong2*>(vb + (j + u) * PITCH + 64 * g);
#pragma unroll
                        for (int i = 0; i < RM; ++i) {
                            const float x = u == 0 ? w[i].x : u == 1 ? w[i].y : u == 2 ? w[i].z : w[i].w;
                            const unsigned long long xx = af_pair(x, x);
                            af_fma2(acc[i][2 * g], xx, vv.x);
                            af_fma2(acc[i][2 * g + 1], xx, vv.y);
                        }
                    }
            }
        } else {
            for (int j = 0; j < AF_KB; ++j) {
                const int at = b * AF_KB + j;
#pragma unroll
                for (int i = 0; i < RM; ++i) {
                    if (at > pos[i] || at < lo[i]) continue;
                    const float x = pb[i * PP + j];
                    const unsigned long long xx = af_pair(x, x);
#pragma unroll
                    for (int g = 0; g < DV; ++g) {
                        const ulonglong2 vv = *reinterpret_cast<const ulonglong2*>(vb + j * PITCH + 64 * g);
                        af_fma2(acc[i][2 * g], xx, vv.x);
                        af_fma2(acc[i][2 * g + 1], xx, vv.y);
                    }
                }
            }
        }
        if (b == b_last || (b + 1) * AF_KB % AF_SEG == 0) {
#pragma unroll
            for (int i = 0; i < RM; ++i) {
                const float m_new = fmaxf(m_run[i], m[i]), fr = af_factor(m_run[i], m_new), fs = af_factor(m[i], m_new);
                l_run[i] = fmaf(l[i], fs, af_scale(l_run[i], fr));
                m_run[i] = m_new;
#pragma unroll
                for (int d = 0; d < 2 * DV; ++d) {
                    const float2 a = af_split(run[i][d]), c = af_split(acc[i][d]);
                    run[i][d] = af_pair(fmaf(c.x, fs, af_scale(a.x, fr)), fmaf(c.y, fs, af_scale(a.y, fr)));
                    acc[i][d] = 0ull;
                }
                m[i] = -INFINITY;
                l[i] = 0.f;
            }
        }
        __syncthreads();                                   // everybody has left this buffer before it is filled again
    }
#pragma unroll
    for (int i = 0; i < RM; ++i) {
        const int r = r0 + i;
        if (r >= rows) continue;
        const float inv = 1.0f / l_run[i];
        float* o = p.out + ((q_row0 + r / p.group) * p.n_q + kvh * p.group + r % p.group) * HD + 4 * tx;
#pragma unroll
        for (int g = 0; g < DV; ++g) {
            const float2 a = af_split(run[i][2 * g]), c = af_split(run[i][2 * g + 1]);
            *reinterpret_cast<float4*>(o + 64 * g) = make_float4(a.x * inv, a.y * inv, c.x * inv, c.y * inv);
        }
    }
}

// ---- single tokens ---------------------------------------------------------------------------------------------------
// A block per (token, kv head) and, with partials given, per segment (blockIdx.y).  partials: [item][segment][group][HD + 2]
// (acc, m, l of that segment alone), item = (index in the launch) * n_kv + kv head.
template <int HD, int GM>
__global__ void __launch_bounds__(AF_THREADS)
attention_f32_rows_kernel(AfParams p, const int* __restrict__ token_list, float* __restrict__ partials) {
    constexpr int PITCH = HD + 4, PP = AF_KB + 4, STEP = AF_THREADS / HD, OUTS = (GM + STEP - 1) / STEP;
    constexpr int QR = GM / 2 > 0 ? (GM + 1) / 2 : 1;      // rows of scores per thread (64 keys x 2)
    extern __shared__ __align__(16) float af_smem[];
    ni_launch_dependents();
    float* qs = af_smem;                                   // [GM][PITCH]
    float* ks = qs + GM * PITCH;
    float* vs = ks + 2 * AF_KB * PITCH;
    float* ps = vs + 2 * AF_KB * PITCH;                    // [GM][PP]
    float* corr_s = ps + GM * PP;                          // [GM]
    float* m_s = corr_s + GM;                              // [GM] of the segment, then l
    float* l_s = m_s + GM;
    const int item = blockIdx.x, kvh = item % p.n_kv, ti = item / p.n_kv;
    const int t = token_list ? token_list[ti] : ti;
    const int pos = p.positions[t], lo = af_first(p, pos);
    const int* table = p.block_table + (size_t)p.seq_of_token[t] * p.bt_stride;
    int b_first = lo / AF_KB, b_last = pos / AF_KB;
    if (partials) {
        const int s = blockIdx.y, s0 = s * (AF_SEG / AF_KB), s1 = s0 + AF_SEG / AF_KB - 1;
        if (s0 > b_last || s1 < b_first) return;           // nothing of this segment is seen
        if (s0 > b_first) b_first = s0;
        if (s1 < b_last) b_last = s1;
    }
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, G = p.group;
    for (int i = tid; i < G * (HD / 4); i += AF_THREADS) {
        const int r = i / (HD / 4), c = 4 * (i % (HD / 4));
        af_copy16(qs + r * PITCH + c, p.q + ((size_t)t * p.n_q + kvh * G + r) * HD + c, true);
    }
    af_fetch<HD>(p, table, kvh, b_first, lo, pos, ks, vs);
    af_commit();
    if (tid < G) { m_s[tid] = -INFINITY; l_s[tid] = 0.f; }
    const int d = tid % HD, rb = tid / HD;                 // outputs (rb + i STEP, d)
    float acc[OUTS], run[OUTS], m_run[OUTS], l_run[OUTS];
#pragma unroll
    for (int i = 0; i < OUTS; ++i) {
        const int r = rb + i * STEP;
        acc[i] = run[i] = 0.f;
        m_run[i] = p.sinks && r < G ? p.sinks[kvh * G + r] : -INFINITY;
        l_run[i] = p.sinks && r < G ? 1.f : 0.f;
    }
    for (int b = b_first; b <= b_last; ++b) {
        const int buf = (b - b_first) & 1;
        if (b < b_last) af_fetch<HD>(p, table, kvh, b + 1, lo, pos, ks + (buf ^ 1) * AF_KB * PITCH, vs + (buf ^ 1) * AF_KB * PITCH);
        af_commit();
        af_wait<1>();
        __syncthreads();
        const int kj = tid & 63, q0 = tid >> 6;
        const float* kb = ks + buf * AF_KB * PITCH + kj * PITCH;
        float s1[QR];
#pragma unroll
        for (int i = 0; i < QR; ++i) s1[i] = 0.f;
#pragma unroll 1
        for (int c0 = 0; c0 < HD; c0 += AF_CHAIN) {
            unsigned long long s2[QR];
#pragma unroll
            for (int i = 0; i < QR; ++i) s2[i] = 0ull;
#pragma unroll 4
            for (int c = c0; c < c0 + AF_CHAIN; c += 4) {
                const ulonglong2 kk = *reinterpret_cast<const ulonglong2*>(kb + c);
#pragma unroll
                for (int i = 0; i < QR; ++i)
                    if (q0 + 2 * i < G) {
                        const ulonglong2 qq = *reinterpret_cast<const ulonglong2*>(qs + (q0 + 2 * i) * PITCH + c);
                        af_fma2(s2[i], qq.x, kk.x);
                        af_fma2(s2[i], qq.y, kk.y);
                    }
            }
#pragma unroll
            for (int i = 0; i < QR; ++i) s1[i] = af_score(s1[i], s2[i]);
        }
        const int key = b * AF_KB + kj;
        const bool seen = key <= pos && key >= lo;
#pragma unroll
        for (int i = 0; i < QR; ++i)
            if (q0 + 2 * i < G) ps[(q0 + 2 * i) * PP + kj] = seen ? af_scale(s1[i], p.scale) : -INFINITY;
        __syncthreads();
        for (int r = warp; r < G; r += AF_THREADS / 32) {  // a warp per row; its halves do the same
            const int j0 = lane & 15, k0 = b * AF_KB + j0;
            float s[4], top = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                s[j] = ps[r * PP + j0 + 16 * j];
                top = fmaxf(top, s[j]);
            }
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            const float m_old = m_s[r], m_new = fmaxf(m_old, top), corr = af_factor(m_old, m_new);
            float w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = k0 + 16 * j <= pos && k0 + 16 * j >= lo ? expf(s[j] - m_new) : 0.f;
            float sum = __fadd_rn(__fadd_rn(w[0], w[1]), __fadd_rn(w[2], w[3]));
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, o));
            __syncwarp();
            if (lane < 16) {
#pragma unroll
                for (int j = 0; j < 4; ++j) ps[r * PP + j0 + 16 * j] = w[j];
            }
            if (lane == 0) {
                corr_s[r] = corr;
                l_s[r] = fmaf(l_s[r], corr, sum);
                m_s[r] = m_new;
            }
            __syncwarp();
        }
        __syncthreads();
        const float* vb = vs + buf * AF_KB * PITCH + d;
#pragma unroll
        for (int i = 0; i < OUTS; ++i)
            if (rb + i * STEP < G) acc[i] = af_scale(acc[i], corr_s[rb + i * STEP]);
        const int j_lo = lo > b * AF_KB ? lo - b * AF_KB : 0, j_hi = pos - b * AF_KB < AF_KB - 1 ? pos - b * AF_KB : AF_KB - 1;
        // unseen keys carry the weight 0 and a value of zeros; only whole groups of them are left out
#pragma unroll 4
        for (int j = j_lo & ~3; j <= j_hi; j += 4) {
            const float v0 = vb[j * PITCH], v1 = vb[(j + 1) * PITCH], v2 = vb[(j + 2) * PITCH], v3 = vb[(j + 3) * PITCH];
#pragma unroll
            for (int i = 0; i < OUTS; ++i)
                if (rb + i * STEP < G) {
                    const float4 w = *reinterpret_cast<const float4*>(ps + (rb + i * STEP) * PP + j);
                    acc[i] = fmaf(w.x, v0, acc[i]);
                    acc[i] = fmaf(w.y, v1, acc[i]);
                    acc[i] = fmaf(w.z, v2, acc[i]);
                    acc[i] = fmaf(w.w, v3, acc[i]);
                }
        }
        if (!partials && (b == b_last || (b + 1) * AF_KB % AF_SEG == 0)) {
#pragma unroll
            for (int i = 0; i < OUTS; ++i) {
                const int r = rb + i * STEP;
                if (r >= G) continue;
                const float m_new = fmaxf(m_run[i], m_s[r]), fr = af_factor(m_run[i], m_new), fs = af_factor(m_s[r], m_new);
                l_run[i] = fmaf(l_s[r], fs, af_scale(l_run[i], fr));
                m_run[i] = m_new;
                run[i] = fmaf(acc[i], fs, af_scale(run[i], fr));
                acc[i] = 0.f;
            }
            __syncthreads();
            if (tid < G) { m_s[tid] = -INFINITY; l_s[tid] = 0.f; }
        }
        __syncthreads();
    }
    if (partials) {
        float* at = partials + ((size_t)item * gridDim.y + blockIdx.y) * G * (HD + 2);
#pragma unroll
        for (int i = 0; i < OUTS; ++i)
            if (rb + i * STEP < G) at[(rb + i * STEP) * (HD + 2) + d] = acc[i];
        if (tid < G) {
            at[tid * (HD + 2) + HD] = m_s[tid];
            at[tid * (HD + 2) + HD + 1] = l_s[tid];
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < OUTS; ++i) {
        const int r = rb + i * STEP;
        if (r < G) p.out[((size_t)t * p.n_q + kvh * G + r) * HD + d] = run[i] * (1.0f / l_run[i]);
    }
}

// The segments of a token merged in order: a block of HD threads per (token, query head).
template <int HD>
__global__ void __launch_bounds__(HD)
attention_f32_merge_kernel(AfParams p, const int* __restrict__ token_list, const float* __restrict__ partials, int segments) {
    ni_launch_dependents();
    const int ti = blockIdx.x / p.n_q, head = blockIdx.x % p.n_q, kvh = head / p.group, r = head % p.group, d = threadIdx.x;
    const int t = token_list ? token_list[ti] : ti;
    const int pos = p.positions[t], s0 = af_first(p, pos) / AF_SEG, s1 = pos / AF_SEG;
    const float* at = partials + ((size_t)(ti * p.n_kv + kvh) * segments) * p.group * (HD + 2) + r * (HD + 2);
    float m = p.sinks ? p.sinks[head] : -INFINITY, l = p.sinks ? 1.f : 0.f, acc = 0.f;
    for (int s = s0; s <= s1; ++s) {
        const float* one = at + (size_t)s * p.group * (HD + 2);
        const float ms = one[HD], m_new = fmaxf(m, ms), fr = af_factor(m, m_new), fs = af_factor(ms, m_new);
        l = fmaf(one[HD + 1], fs, af_scale(l, fr));
        acc = fmaf(one[d], fs, af_scale(acc, fr));
        m = m_new;
    }
    p.out[((size_t)t * p.n_q + head) * HD + d] = acc * (1.0f / l);
}

static int af_params(AfParams& p, const float* q, const float* k, const float* v, float* out, const int* block_table, int bt_stride,
                     const int* positions, const int* seq_of_token, int n_q, int n_kv, int head_dim, int page, int window,
                     int chunk, const float* sinks, float scale) {
    if (n_q <= 0 || n_kv <= 0 || n_q % n_kv || page <= 0 || chunk < 0) return NI_ERR_BAD_ARGUMENT;
    if ((head_dim != 64 && head_dim != 128) || n_q / n_kv > AF_MAX_GROUP || n_kv > 65535) return NI_ERR_UNSUPPORTED_SIZE;
    if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)out) % 16) return NI_ERR_BAD_ARGUMENT;
    const int shift = (page & (page - 1)) == 0 ? __builtin_ctz((unsigned)page) : -1;
    p = AfParams{q, k, v, out, block_table, positions, seq_of_token, sinks, bt_stride, n_q, n_kv, n_q / n_kv, page, shift, window, chunk, scale};
    return NI_OK;
}

// Portions: n_tiles tiles of up to tile_tokens query tokens (request tile_seq[i], first row tile_row0[i] of its portion).
NI_EXPORT int ni_attention_f32_tiles(const float* q, const float* k, const float* v, float* out, const int* tile_seq,
                                     const int* tile_row0, int n_tiles, int tile_tokens, const int* cu_q, const int* kv_len,
                                     const int* block_table, int bt_stride, int n_q, int n_kv, int head_dim, int page,
                                     int window, int chunk, const float* sinks, float scale, cudaStream_t stream) {
    if (n_tiles <= 0) return NI_OK;
    AfParams p;
    if (int rc = af_params(p, q, k, v, out, block_table, bt_stride, nullptr, nullptr, n_q, n_kv, head_dim, page, window, chunk, sinks, scale)) return rc;
    if (tile_tokens <= 0) return NI_ERR_BAD_ARGUMENT;
#define LAUNCH(HD, RM)                                                                                                     \
    do {                                                                                                                   \
        constexpr int SMEM = (8 * RM * (HD + 4) + 4 * AF_KB * (HD + 4) + 8 * RM * (AF_KB + 4)) * (int)sizeof(float);        \
        auto kernel = attention_f32_tile_kernel<HD, RM>;                                                                   \
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);             \
        if (e != cudaSuccess) return (int)e;                                                                               \
        const int per = 8 * RM / p.group, slices = (tile_tokens + per - 1) / per;                                          \
        if ((long long)n_tiles * slices > 2147483647LL) return NI_ERR_UNSUPPORTED_SIZE;                                    \
        kernel<<<dim3(n_tiles * slices, n_kv), AF_THREADS, SMEM, stream>>>(p, tile_seq, tile_row0, tile_tokens, cu_q, kv_len, slices); \
    } while (0)
    if (head_dim == 64) LAUNCH(64, 8);
    else LAUNCH(128, 4);
#undef LAUNCH
    NI_RETURN_LAUNCH_STATUS();
}

// Into how many segments a launch over n_tokens tokens with up to max_kv keys is split: 1, or one block per segment of 512
// keys (a launch of few tokens leaves the GPU idle otherwise), and the floats of partial results that this takes.
NI_EXPORT int ni_attention_f32_segments(int n_tokens, int n_q, int n_kv, int head_dim, long long max_kv) {
    const long long segments = (max_kv + AF_SEG - 1) / AF_SEG;
    if (segments <= 1 || (long long)n_tokens * n_kv >= 4LL * ni_sm_count() || segments > 65535) return 1;
    return (long long)n_tokens * n_q * segments * (head_dim + 2) <= (16LL << 20) ? (int)segments : 1;      // 64 MB
}

// Single tokens (or any tokens, one by one): n_tokens entries of token_list, or tokens 0 .. n_tokens - 1.  segments as
// ni_attention_f32_segments says, partials [n_tokens * n_q * segments * (head_dim + 2)] floats if that is above 1.
NI_EXPORT int ni_attention_f32_rows(const float* q, const float* k, const float* v, float* out, const int* token_list, int n_tokens,
                                    const int* positions, const int* seq_of_token, const int* block_table, int bt_stride,
                                    int n_q, int n_kv, int head_dim, int page, int window, int chunk, const float* sinks,
                                    float scale, int segments, float* partials, cudaStream_t stream) {
    if (n_tokens <= 0) return NI_OK;
    AfParams p;
    if (int rc = af_params(p, q, k, v, out, block_table, bt_stride, positions, seq_of_token, n_q, n_kv, head_dim, page, window, chunk, sinks, scale)) return rc;
    if (segments < 1 || (segments > 1 && (!partials || (long long)segments * AF_SEG < (long long)bt_stride * page))) return NI_ERR_BAD_ARGUMENT;
    if (segments > 65535 || (long long)n_tokens * n_q > 2147483647LL) return NI_ERR_UNSUPPORTED_SIZE;
    if (segments == 1) partials = nullptr;
#define LAUNCH(HD, GM)                                                                                                     \
    do {                                                                                                                   \
        constexpr int SMEM = (GM * (HD + 4) + 4 * AF_KB * (HD + 4) + GM * (AF_KB + 4) + 3 * GM) * (int)sizeof(float);      \
        auto kernel = attention_f32_rows_kernel<HD, GM>;                                                                   \
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);             \
        if (e != cudaSuccess) return (int)e;                                                                               \
        kernel<<<dim3(n_tokens * n_kv, segments), AF_THREADS, SMEM, stream>>>(p, token_list, partials);                    \
        if (partials) attention_f32_merge_kernel<HD><<<n_tokens * n_q, HD, 0, stream>>>(p, token_list, partials, segments); \
    } while (0)
    if (head_dim == 64) {
        if (p.group <= 4) LAUNCH(64, 4);
        else LAUNCH(64, 16);
    } else {
        if (p.group <= 4) LAUNCH(128, 4);
        else LAUNCH(128, 16);
    }
#undef LAUNCH
    NI_RETURN_LAUNCH_STATUS();
}
