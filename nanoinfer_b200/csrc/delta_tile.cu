// The gated delta rule with one decay per head over prompt portions, sixteen tokens at a time, for key heads of 128 (formula and
// layouts of delta_rule.cu; delta_block.cu has the other sizes, four tokens at a time).
//
// With S the state before a tile, P(t, s) the product of the decays of tokens s + 1 .. t of the tile and c_t that of tokens 0 .. t:
//     R = K S,   X_t = beta_t v_t - beta_t c_t R_t,   U = T X,   T = (1 + L)^-1,   L_ts = beta_t P(t, s) (k_t . k_s)  (s < t)
//     O_t = c_t (Q S)_t + sum_{s<=t} A_ts U_s,   A_ts = P(t, s) (q_t . k_s)
//     S  <- c_15 S + sum_s P(15, s) k_s U_s^T
// T, A and the vectors are made for all tiles at once; what is left of the chain is five small products, on the tensor cores
// (mma.sync, bfloat16 operands, FP32 sums): every FP32 number is the exact sum of three bfloat16 numbers, and six of the nine
// products of parts are taken (2^-24 of a product is left out).  The sums of the largest parts leave the tensor core, which cuts, after
// one instruction and are added with rounding; the diagonals of T and A are left to FP32, and the state itself is never an accumulator.  Only products of decays over stretches of
// a tile appear, never quotients; they are formed in 64 bits, since their error is common to all of the state and would not average
// out along a portion.  Tokens that a last tile lacks have beta 0, decay 1 and zeros for k, q and v, which leaves S alone.
//
// The state lies transposed in the warps' accumulator layout, 16 columns of v by 64 of the 128 rows: read as the first operand of the
// next product it needs no exchange.  k, q, T and A are cut by the preparation, once, and lie as the second operands are read: a
// lane's numbers of a 16 x 8 piece side by side.  Two warps share 16 columns; they add their halves of R and Q S through shared
// memory, one barrier per tile.  What bounds a portion is the chain of its tiles, about 2,850 clocks each: 1,010 instructions of a
// lone warp per scheduler, which issues nothing else for 8 clocks while one of its 162 MMAs enters the tensor core.  (Four warps per 16
// columns: 148 us instead of 129 at the time, since their products come in the same phases; FP32 multiply-adds in the same tiles: 183 us.)
//
// Portions of 1,201 and 847 tokens, 16 heads of 128: 170 us with the preparation (51), against 245 us in blocks of four; 2,048 tokens 247
// (337), 8 x 512 260 (328), 512 69 (89); 2,048 tokens of 4 heads 213 (314), of 64 511 (669).  Error against 64 bits of the whole rule, read-outs / states, means over eight inputs of up to
// 1,100 tokens: decays of a few tokens 1.2e-7 / 1.1e-7 (blocks of four 1.3e-7 / 1.2e-7), of some tens 1.1e-7 / 1.2e-7 (1.4e-7 / 1.5e-7),
// of some hundreds 1.3e-7 / 1.5e-7 (3.0e-7 / 4.5e-7), decays near one 1.6e-7 / 1.8e-7 (1.7e-6 / 2.7e-6).  Decays and beta in 64 bits and
// the keys' norms with one step of Newton's method are worth more than what the cuts cost (in FP32: states 1.07 times the error of
// blocks of four where a decay lasts a few tokens); they take 2 us.
#include <type_traits>

#include "common.cuh"

#define DT_TOK 16
#define DT_D 128
// A piece of 16 x 8 of a second operand: per lane four numbers (rows 2 t, 2 t + 1, 2 t + 8, 2 t + 9 of column lane / 4, t = lane % 4) as
// three parts: 16 bytes with the first two for every lane, then 8 bytes with the third.
#define DT_PIECE 768
#define DT_KEYS (3 * 16 * DT_PIECE)         // of a tile and q/k head: k for R (8 pieces of rows x 2 of tokens), q likewise, k for S (16)
// of a tile and head: T, A less their diagonals (2 pieces each), then floats beta, beta c, c, P(15, .), A_tt and room to a multiple of 128
// bytes (without it, reads of every other tile start in the middle of a row of banks: 136 us instead of 131)
#define DT_COEF (4 * DT_PIECE + 96 * 4)

struct DtDims {
    int G, H, V, taps, ld, b_off, a_off;
    __host__ __device__ int C() const { return 2 * G * DT_D + H * V; }
    __host__ __device__ size_t hist_off() const { return (size_t)H * DT_D * V; }
};

__device__ __forceinline__ float dt_silu(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ double dt_softplus(double z) { return z > 20.0 ? z : log1p(exp(z)); }
// 1 / sqrt(s): the error of the division and the root (a factor of all of a row's numbers) is put right by one step of Newton's method
// whose residual is exact.
__device__ __forceinline__ float dt_rsqrt(float s) {
    const float r = 1.0f / sqrtf(s), h = s * r, left = fmaf(-h, r, 1.0f) - fmaf(s, r, -h) * r;
    return fmaf(0.5f * r, left, r);
}

// Tiles before request `seq` (all of a warp's lanes get it).
__device__ __forceinline__ int dt_tiles_before(const int* __restrict__ cu_q, int seq) {
    int n = 0;
    for (int i = threadIdx.x & 31; i < seq; i += 32) n += (cu_q[i + 1] - cu_q[i] + DT_TOK - 1) / DT_TOK;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    return n;
}
// The request that tile number b belongs to and its number there (false: there is no such tile).  One warp.
__device__ __forceinline__ bool dt_find(const int* __restrict__ cu_q, int n_seqs, int b, int& seq, int& in_seq) {
    const int lane = threadIdx.x & 31;
    int before = 0;
    for (int s0 = 0; s0 < n_seqs; s0 += 32) {
        const int s = s0 + lane;
        const int mine = s < n_seqs ? (cu_q[s + 1] - cu_q[s] + DT_TOK - 1) / DT_TOK : 0;
        int upto = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += x;
        }
        const unsigned past = __ballot_sync(0xffffffffu, before + upto > b);
        if (past) {
            const int src = __ffs(past) - 1;
            seq = s0 + src;
            in_seq = b - (before + __shfl_sync(0xffffffffu, upto - mine, src));
            return true;
        }
        before += __shfl_sync(0xffffffffu, upto, 31);
    }
    return false;
}

// Four channels of an input row; `at` counts from the portion's first token (a negative number reads the history).
template <typename T>
__device__ __forceinline__ float4 dt_row(const T* __restrict__ proj, const float* __restrict__ hist, const DtDims& dm, int first,
                                         int at, int c) {
    if (at >= 0) {
        const T* p = proj + (size_t)(first + at) * dm.ld + c;
        if (sizeof(T) == 4) return *reinterpret_cast<const float4*>(p);
        return make_float4(ni_to_float(p[0]), ni_to_float(p[1]), ni_to_float(p[2]), ni_to_float(p[3]));
    }
    return *reinterpret_cast<const float4*>(hist + (size_t)(dm.taps - 1 + at) * dm.C() + c);
}

// Convolution and silu of channels c .. c + 3 at four tokens from `at` on (zeros where a token does not exist).  TAPS 4: rows and
// the channels' weights in registers; 0: any number of taps, weights read where they are used.
template <typename T, int TAPS>
__device__ __forceinline__ void dt_conv(const T* __restrict__ proj, const float* __restrict__ conv_w, const float* __restrict__ hist,
                                        const DtDims& dm, int first, int at, int live, int c, float4 y[4]) {
    float4 acc[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) acc[t] = make_float4(0.f, 0.f, 0.f, 0.f);
    const float* w = conv_w + (size_t)c * dm.taps;
    if (live > 0) {
        if (TAPS == 4) {
            float4 x[7];                                       // inputs of tokens at - 3 .. at + 3
#pragma unroll
            for (int r = 0; r < 7; ++r) x[r] = r - 3 < live ? dt_row(proj, hist, dm, first, at - 3 + r, c) : make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 w0 = *reinterpret_cast<const float4*>(w), w1 = *reinterpret_cast<const float4*>(w + 4);
            const float4 w2 = *reinterpret_cast<const float4*>(w + 8), w3 = *reinterpret_cast<const float4*>(w + 12);
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                acc[t].x = fmaf(w0.w, x[t + 3].x, fmaf(w0.z, x[t + 2].x, fmaf(w0.y, x[t + 1].x, w0.x * x[t].x)));
                acc[t].y = fmaf(w1.w, x[t + 3].y, fmaf(w1.z, x[t + 2].y, fmaf(w1.y, x[t + 1].y, w1.x * x[t].y)));
                acc[t].z = fmaf(w2.w, x[t + 3].z, fmaf(w2.z, x[t + 2].z, fmaf(w2.y, x[t + 1].z, w2.x * x[t].z)));
                acc[t].w = fmaf(w3.w, x[t + 3].w, fmaf(w3.z, x[t + 2].w, fmaf(w3.y, x[t + 1].w, w3.x * x[t].w)));
            }
        } else {
            for (int r = 0; r < 4 + dm.taps - 1; ++r) {        // row r holds the inputs of token at - (taps - 1) + r
                if (r - (dm.taps - 1) >= live) break;
                const float4 x = dt_row(proj, hist, dm, first, at - (dm.taps - 1) + r, c);
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const int j = r - t;                       // this row is tap j of token t
                    if (j >= 0 && j < dm.taps) {
                        acc[t].x = fmaf(w[j], x.x, acc[t].x);
                        acc[t].y = fmaf(w[dm.taps + j], x.y, acc[t].y);
                        acc[t].z = fmaf(w[2 * dm.taps + j], x.z, acc[t].z);
                        acc[t].w = fmaf(w[3 * dm.taps + j], x.w, acc[t].w);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int t = 0; t < 4; ++t)
        y[t] = t < live ? make_float4(dt_silu(acc[t].x), dt_silu(acc[t].y), dt_silu(acc[t].z), dt_silu(acc[t].w))
                        : make_float4(0.f, 0.f, 0.f, 0.f);
}

__device__ __forceinline__ float dt_dot4(const float4& a, const float4& b, float acc) {
    return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, acc))));
}
// The three parts of two numbers, each a pair of bfloat16 (rounded: the parts' mean is zero).
__device__ __forceinline__ void dt_parts(float x, float y, uint32_t p[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
        p[i] = *reinterpret_cast<const uint32_t*>(&h);
        x -= __bfloat162float(h.x);
        y -= __bfloat162float(h.y);
    }
}
__device__ __forceinline__ void dt_put(uint8_t* pieces, int n_pieces, int piece, int lane, float a, float b, float c, float d) {
    uint32_t lo[3], hi[3];
    dt_parts(a, b, lo);
    dt_parts(c, d, hi);
    *reinterpret_cast<uint4*>(pieces + piece * 512 + lane * 16) = make_uint4(lo[0], hi[0], lo[1], hi[1]);
    *reinterpret_cast<uint2*>(pieces + n_pieces * 512 + piece * 256 + lane * 8) = make_uint2(lo[2], hi[2]);
}

// A block of 4 warps per (tile, q/k head), four tokens per warp: convolution, silu and unit norms, then all products k . k and q . k of
// the tile from shared memory, then T and A of each of the head's value heads; or per (tile, 128 channels of v): convolution and silu.
#define DT_PITCH 132
template <typename T, int TAPS>
__global__ void __launch_bounds__(128)
delta_tile_prepare_kernel(const T* __restrict__ proj, const float* __restrict__ conv_w, const float* __restrict__ a_log,
                          const float* __restrict__ dt_bias, const float* __restrict__ state, long long state_stride,
                          const int* __restrict__ cu_q, const int* __restrict__ slots, int n_seqs, DtDims dm,
                          float* __restrict__ values, uint8_t* __restrict__ keys, uint8_t* __restrict__ coef) {
    __shared__ __align__(16) float qs[DT_TOK][DT_PITCH];
    __shared__ __align__(16) float ks[DT_TOK][DT_PITCH];
    __shared__ float kk[DT_TOK][DT_TOK + 1], qk[DT_TOK][DT_TOK + 1];
    __shared__ float low[4][DT_TOK][DT_TOK], ts[4][DT_TOK][DT_TOK + 1], as[4][DT_TOK][DT_TOK + 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int seq, in_seq;
    if (!dt_find(cu_q, n_seqs, blockIdx.x, seq, in_seq)) return;
    const int C = dm.C(), first = cu_q[seq], tile0 = in_seq * DT_TOK, left = cu_q[seq + 1] - first - tile0;
    const int at = tile0 + 4 * warp, mine = left - 4 * warp, live = mine < 0 ? 0 : mine < 4 ? mine : 4;
    const float* hist = state + (size_t)slots[seq] * state_stride + dm.hist_off();
    float4 y[4];
    if ((int)blockIdx.y >= dm.G) {                             // values
        const int c = 2 * dm.G * DT_D + (blockIdx.y - dm.G) * 128 + 4 * lane;
        if (c >= C) return;
        dt_conv<T, TAPS>(proj, conv_w, hist, dm, first, at, live, c, y);
#pragma unroll
        for (int t = 0; t < 4; ++t)
            if (t < live) *reinterpret_cast<float4*>(values + (size_t)(first + at + t) * dm.H * dm.V + (c - 2 * dm.G * DT_D)) = y[t];
        return;
    }
    const int g = blockIdx.y;
#pragma unroll
    for (int which = 0; which < 2; ++which) {                  // q, then k
        const int c = (which * dm.G + g) * DT_D + 4 * lane;
        dt_conv<T, TAPS>(proj, conv_w, hist, dm, first, at, live, c, y);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const float r = dt_rsqrt((ni_warp_sum(dt_dot4(y[t], y[t], 0.f)) + 1e-6f) * (which ? 1.0f : (float)DT_D));
            y[t].x *= r; y[t].y *= r; y[t].z *= r; y[t].w *= r;
            *reinterpret_cast<float4*>(which ? &ks[4 * warp + t][4 * lane] : &qs[4 * warp + t][4 * lane]) = y[t];
        }
    }
    __syncthreads();
    {
        uint8_t* o = keys + ((size_t)blockIdx.x * dm.G + g) * DT_KEYS;
        const int t = 2 * (lane & 3), r = lane >> 2;
        for (int i = warp; i < 16; i += 4) {                   // pieces of k and q: rows 16 (i / 2) .., tokens 8 (i % 2) ..
            const int d = 16 * (i >> 1) + t, tok = 8 * (i & 1) + r;
            dt_put(o, 16, i, lane, ks[tok][d], ks[tok][d + 1], ks[tok][d + 8], ks[tok][d + 9]);
            dt_put(o + 16 * DT_PIECE, 16, i, lane, qs[tok][d], qs[tok][d + 1], qs[tok][d + 8], qs[tok][d + 9]);
            const int row = 8 * i + r;                         // of k as it enters S: tokens by rows 8 i ..
            dt_put(o + 32 * DT_PIECE, 16, i, lane, ks[t][row], ks[t + 1][row], ks[t + 8][row], ks[t + 9][row]);
        }
    }
    {                                                          // thread 8 t + s: products of token t with tokens s and s + 8
        const int t = threadIdx.x >> 3, s = threadIdx.x & 7;
        const auto add = [](float4& acc, const float4& x, const float4& y) {
            acc.x = fmaf(x.x, y.x, acc.x); acc.y = fmaf(x.y, y.y, acc.y); acc.z = fmaf(x.z, y.z, acc.z); acc.w = fmaf(x.w, y.w, acc.w);
        };
        const auto all = [](const float4& acc) { return (double)((acc.x + acc.y) + (acc.z + acc.w)); };
        double sum[4] = {0.0, 0.0, 0.0, 0.0};                  // sums of 16 channels, FP32, are added in 64 bits
#pragma unroll 2
        for (int d0 = 0; d0 < DT_D; d0 += 16) {
            float4 a0 = make_float4(0.f, 0.f, 0.f, 0.f), a1 = a0, b0 = a0, b1 = a0;
#pragma unroll
            for (int d = d0; d < d0 + 16; d += 4) {
                const float4 kt = *reinterpret_cast<const float4*>(&ks[t][d]), qt = *reinterpret_cast<const float4*>(&qs[t][d]);
                const float4 k0 = *reinterpret_cast<const float4*>(&ks[s][d]);
                add(a0, kt, k0);
                add(b0, qt, k0);
                if (warp >= 2) {                               // tokens from 8 on meet tokens from 8 on
                    const float4 k1 = *reinterpret_cast<const float4*>(&ks[s + 8][d]);
                    add(a1, kt, k1);
                    add(b1, qt, k1);
                }
            }
            sum[0] += all(a0); sum[1] += all(b0);
            if (warp >= 2) { sum[2] += all(a1); sum[3] += all(b1); }
        }
        kk[t][s] = (float)sum[0]; kk[t][s + 8] = (float)sum[2];
        qk[t][s] = (float)sum[1]; qk[t][s + 8] = (float)sum[3];
    }
    __syncthreads();
    const int per = dm.H / dm.G, j = lane & 15;
    for (int h = g * per + warp; h < (g + 1) * per; h += 4) {
        // lane t < 16: token t's decay and beta, in 64 bits: their errors are factors of all of the state
        double decay = 1.0, beta = 0.0;
        if (lane < DT_TOK && lane < left) {
            const T* row = proj + (size_t)(first + tile0 + lane) * dm.ld;
            decay = exp(-exp((double)a_log[h]) * dt_softplus((double)ni_to_float(row[dm.a_off + h]) + (double)dt_bias[h]));
            beta = 1.0 / (1.0 + exp(-(double)ni_to_float(row[dm.b_off + h])));
        }
        uint8_t* o = coef + ((size_t)blockIdx.x * dm.H + h) * DT_COEF;
        float* vec = reinterpret_cast<float*>(o + 4 * DT_PIECE);
        // lane j (and j + 16): column j of A and L, running down the tokens; c and P(15, .) on the way.  Products of decays stay in
        // 64 bits, since their error would not average out along a portion.
        double p = 1.0, c = 1.0, ct = 1.0;
#pragma unroll
        for (int t = 0; t < DT_TOK; ++t) {
            const double dt = __shfl_sync(0xffffffffu, decay, t), bt = __shfl_sync(0xffffffffu, beta, t);
            c *= dt;
            if (t == j) ct = c;
            p = t > j ? p * dt : 1.0;
            if (lane < DT_TOK) {
                as[warp][t][j] = t > j ? (float)p * qk[t][j] : 0.f;
                low[warp][t][j] = t > j ? (float)(bt * p) * kk[t][j] : 0.f;
            }
        }
        __syncwarp();
        if (lane < DT_TOK) {
            float x[DT_TOK];                                   // column j of T
#pragma unroll
            for (int t = 0; t < DT_TOK; ++t) {
                float a = 0.f;
#pragma unroll
                for (int s = 0; s < t; ++s) a = fmaf(low[warp][t][s], x[s], a);
                x[t] = t == j ? 1.f : t > j ? -a : 0.f;
                ts[warp][t][j] = t > j ? x[t] : 0.f;
            }
            vec[j] = (float)beta;
            vec[16 + j] = (float)(beta * ct);
            vec[32 + j] = (float)ct;
            vec[48 + j] = (float)p;                            // P(15, j)
            vec[64 + j] = qk[j][j];
        }
        __syncwarp();
        const int t = 2 * (lane & 3), r = lane >> 2;
#pragma unroll
        for (int m = 0; m < 2; ++m) {                          // rows 8 m .. of T and A as columns of a second operand
            dt_put(o, 2, m, lane, ts[warp][8 * m + r][t], ts[warp][8 * m + r][t + 1], ts[warp][8 * m + r][t + 8], ts[warp][8 * m + r][t + 9]);
            dt_put(o + 2 * DT_PIECE, 2, m, lane, as[warp][8 * m + r][t], as[warp][8 * m + r][t + 1], as[warp][8 * m + r][t + 8], as[warp][8 * m + r][t + 9]);
        }
        __syncwarp();
    }
}

__device__ __forceinline__ void dt_copy16(void* dst_smem, const void* src, bool live) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
    const int n = live ? 16 : 0;                               // 0: sixteen bytes of zeros, nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
// d += a b, sum += a b: 16 x 16 by 16 x 8
__device__ __forceinline__ void dt_mma(float d[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void dt_mma_zero(float d[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// The three parts of two accumulators of 16 x 8 (columns 0 .. 7 and 8 .. 15) as a first operand of 16 x 16: upper halves of the
// numbers, of what is left, and of what is left then.
struct DtOperand { uint32_t p[3][4]; };
__device__ __forceinline__ void dt_operand(const float c[4], const float d[4], DtOperand& o) {
    const float x[8] = {c[0], c[1], c[2], c[3], d[0], d[1], d[2], d[3]};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float a = x[2 * i], b = x[2 * i + 1];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const uint32_t h = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
            o.p[k][i] = h;
            a -= __uint_as_float(h << 16);
            b -= __uint_as_float(h & 0xffff0000u);
        }
    }
}
// One piece of a second operand, and its six products: the largest parts apart.
struct DtPiece { uint4 ab; uint2 c; };
__device__ __forceinline__ DtPiece dt_piece(const uint8_t* pieces, int n_pieces, int piece, int lane) {
    DtPiece b;
    b.ab = *reinterpret_cast<const uint4*>(pieces + piece * 512 + lane * 16);
    b.c = *reinterpret_cast<const uint2*>(pieces + n_pieces * 512 + piece * 256 + lane * 8);
    return b;
}
// Coefficient (t, s) of two pieces that hold T or A: the sum of its parts.
__device__ __forceinline__ float dt_coefficient(const uint8_t* pieces, int t, int s) {
    const DtPiece b = dt_piece(pieces, 2, t >> 3, 4 * (t & 7) + ((s & 7) >> 1));
    const uint32_t p[3] = {s >> 3 ? b.ab.y : b.ab.x, s >> 3 ? b.ab.w : b.ab.z, s >> 3 ? b.c.y : b.c.x};
    float sum = 0.f;
#pragma unroll
    for (int k = 2; k >= 0; --k) sum += __uint_as_float((s & 1) ? p[k] & 0xffff0000u : p[k] << 16);
    return sum;
}
// sum_{s<t} C_ts x_s without the tokens from t on, for the tokens and columns of this lane's numbers: what the tensor core makes of
// infinities and NaN (its zeros times a later token's) is taken back this way.
__device__ __noinline__ void dt_masked(const uint8_t* pieces, const float x[8], float y[8]) {
    const int lane = threadIdx.x & 31, q4 = lane & 3;
    float acc[8] = {};
#pragma unroll
    for (int s = 0; s < DT_TOK; ++s) {
        const int src = (lane & ~3) + ((s & 7) >> 1);
        const float a = __shfl_sync(0xffffffffu, x[4 * (s >> 3) + (s & 1)], src), b = __shfl_sync(0xffffffffu, x[4 * (s >> 3) + (s & 1) + 2], src);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = 8 * (i >> 1) + 2 * q4 + (i & 1), at = 4 * (i >> 1) + (i & 1);
            if (s < t) {
                const float c = dt_coefficient(pieces, t, s);
                acc[at] = fmaf(c, a, acc[at]);
                acc[at + 2] = fmaf(c, b, acc[at + 2]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) y[i] = acc[i];
}
#define DT_STAGES 2
#define DT_VP 36               // row pitch of the values in shared memory
#define DT_STAGE (DT_KEYS + DT_COEF + DT_TOK * DT_VP * 4)
#define DT_SMEM (DT_STAGES * DT_STAGE + 2 * 6 * 32 * 16)

// A block per (request, head, 32 columns): warps 2 w and 2 w + 1 have 16 of the columns, rows 0 .. 63 and 64 .. 127 of the state.
__global__ void __launch_bounds__(128)
delta_tile_recurrence_kernel(const float* __restrict__ values, const uint8_t* __restrict__ keys, const uint8_t* __restrict__ coef,
                             float* __restrict__ state, long long state_stride, const int* __restrict__ cu_q,
                             const int* __restrict__ slots, DtDims dm, float* __restrict__ out) {
    extern __shared__ __align__(16) uint8_t dt_smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q4 = lane & 3, row = lane >> 2;
    const int team = warp >> 1, half = warp & 1;
    const int h = blockIdx.y, seq = blockIdx.z, g = h / (dm.H / dm.G), V = dm.V;
    const int col0 = blockIdx.x * 32, col = col0 + 16 * team + row;            // this lane's columns: col and col + 8
    const int first = cu_q[seq], n = cu_q[seq + 1] - first;
    if (n <= 0) return;
    const int tiles = (n + DT_TOK - 1) / DT_TOK, tile0 = dt_tiles_before(cu_q, seq);
    const uint8_t* key_src = keys + ((size_t)tile0 * dm.G + g) * DT_KEYS;
    const uint8_t* coef_src = coef + ((size_t)tile0 * dm.H + h) * DT_COEF;
    float4* exch = reinterpret_cast<float4*>(dt_smem + DT_STAGES * DT_STAGE) + team * 6 * 32;   // [2 halves][R of 8 tokens, of 8 more, Q S][lane]

    auto fetch = [&](int tile) {
        if (tile < tiles) {
            uint8_t* st = dt_smem + (tile % DT_STAGES) * DT_STAGE;
            const uint8_t* k = key_src + (size_t)tile * dm.G * DT_KEYS;
#pragma unroll
            for (int i = 0; i < DT_KEYS / 2048; ++i) dt_copy16(st + (i * 128 + tid) * 16, k + (i * 128 + tid) * 16, true);
            const uint8_t* c = coef_src + (size_t)tile * dm.H * DT_COEF;
            for (int i = tid; i < DT_COEF / 16; i += 128) dt_copy16(st + DT_KEYS + i * 16, c + i * 16, true);
            const int t = tid >> 3, d = 4 * (tid & 7), tok = tile * DT_TOK + t;
            const bool live = tok < n && col0 + d < V;
            dt_copy16(st + DT_KEYS + DT_COEF + (t * DT_VP + d) * 4, live ? values + (size_t)(first + tok) * dm.H * V + h * V + col0 + d : values, live);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");   // one group per tile, empty or not
    };
    static_assert(DT_KEYS % 2048 == 0 && DT_COEF % 16 == 0, "whole pieces for every thread");

    // state: accumulator i holds columns col, col + 8 by rows 64 half + 8 i + 2 q4, + 1
    const bool there = col0 + 16 * team < V;                   // V is a multiple of 16: all of a team's columns or none
    float* S = state + (size_t)slots[seq] * state_stride + ((size_t)h * DT_D + 64 * half + 2 * q4) * V + col;
    float s[8][4];
    const auto walk = [&](auto masked) {
        constexpr bool MASKED = decltype(masked)::value;
        fetch(0);
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[i][e] = there ? S[(size_t)(8 * i + (e & 1)) * V + 8 * (e >> 1)] : 0.f;
        for (int tile = 0; tile < tiles; ++tile) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();                                       // the tile is there; every warp has left the one before
            fetch(tile + 1);
            const uint8_t* st = dt_smem + (tile % DT_STAGES) * DT_STAGE;
            const uint8_t* Tm = st + DT_KEYS;
            const uint8_t* Am = Tm + 2 * DT_PIECE;
            const float* vec = reinterpret_cast<const float*>(Tm + 4 * DT_PIECE);
            const float* vs = reinterpret_cast<const float*>(st + DT_KEYS + DT_COEF) + 16 * team + row;

            // R^T and (Q S)^T, this half of the rows: [16 columns] x [tokens 8 j .. 8 j + 7]; j: k, k, q, q
            float sum[4][4], small[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                DtOperand a;
                dt_operand(s[2 * i], s[2 * i + 1], a);
                DtPiece b[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) b[j] = dt_piece(st + (j >> 1) * 16 * DT_PIECE, 16, 2 * (4 * half + i) + (j & 1), lane);
                float big[4][4];
#pragma unroll
                for (int j = 0; j < 4; ++j) dt_mma_zero(big[j], a.p[0], b[j].ab.x, b[j].ab.y);
                if (i == 0) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) dt_mma_zero(small[j], a.p[0], b[j].c.x, b[j].c.y);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) dt_mma(small[j], a.p[0], b[j].c.x, b[j].c.y);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) dt_mma(small[j], a.p[2], b[j].ab.x, b[j].ab.y);
#pragma unroll
                for (int j = 0; j < 4; ++j) dt_mma(small[j], a.p[1], b[j].ab.z, b[j].ab.w);
#pragma unroll
                for (int j = 0; j < 4; ++j) dt_mma(small[j], a.p[0], b[j].ab.z, b[j].ab.w);
#pragma unroll
                for (int j = 0; j < 4; ++j) dt_mma(small[j], a.p[1], b[j].ab.x, b[j].ab.y);
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) sum[j][e] = i == 0 ? big[j][e] : sum[j][e] + big[j][e];
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) sum[j][e] += small[j][e];
            exch[(3 * half) * 32 + lane] = make_float4(sum[0][0], sum[0][1], sum[0][2], sum[0][3]);
            exch[(3 * half + 1) * 32 + lane] = make_float4(sum[1][0], sum[1][1], sum[1][2], sum[1][3]);
            // the other warp writes the read-outs of tokens 8 (1 - half) ..
            exch[(3 * half + 2) * 32 + lane] = half ? make_float4(sum[2][0], sum[2][1], sum[2][2], sum[2][3])
                                                    : make_float4(sum[3][0], sum[3][1], sum[3][2], sum[3][3]);
            asm volatile("bar.sync %0, 64;" ::"r"(1 + team) : "memory");
            float o[4], x[2][4];
            {
                const float4 y[3] = {exch[(3 * (1 - half)) * 32 + lane], exch[(3 * (1 - half) + 1) * 32 + lane], exch[(3 * (1 - half) + 2) * 32 + lane]};
#pragma unroll
                for (int j = 0; j < 2; ++j) {                      // X: tokens 8 j + 2 q4, + 1 of columns col, col + 8
                    const int t = 8 * j + 2 * q4;
                    const float2 be = *reinterpret_cast<const float2*>(vec + t), bc = *reinterpret_cast<const float2*>(vec + 16 + t);
                    x[j][0] = fmaf(-bc.x, sum[j][0] + y[j].x, be.x * vs[t * DT_VP]);
                    x[j][1] = fmaf(-bc.y, sum[j][1] + y[j].y, be.y * vs[(t + 1) * DT_VP]);
                    x[j][2] = fmaf(-bc.x, sum[j][2] + y[j].z, be.x * vs[t * DT_VP + 8]);
                    x[j][3] = fmaf(-bc.y, sum[j][3] + y[j].w, be.y * vs[(t + 1) * DT_VP + 8]);
                }
                o[0] = (half ? sum[3][0] : sum[2][0]) + y[2].x; o[1] = (half ? sum[3][1] : sum[2][1]) + y[2].y;
                o[2] = (half ? sum[3][2] : sum[2][2]) + y[2].z; o[3] = (half ? sum[3][3] : sum[2][3]) + y[2].w;
            }
            // U^T = X^T + X^T (T - 1)^T, in both warps
            float u[2][4];
            {
                DtOperand a;
                dt_operand(x[0], x[1], a);
                float d[2][4];
                DtPiece b[2];
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    b[m] = dt_piece(Tm, 2, m, lane);
                    dt_mma_zero(u[m], a.p[0], b[m].ab.x, b[m].ab.y);
                    dt_mma_zero(d[m], a.p[0], b[m].c.x, b[m].c.y);
                }
#pragma unroll
                for (int m = 0; m < 2; ++m) dt_mma(d[m], a.p[2], b[m].ab.x, b[m].ab.y);
#pragma unroll
                for (int m = 0; m < 2; ++m) dt_mma(d[m], a.p[1], b[m].ab.z, b[m].ab.w);
#pragma unroll
                for (int m = 0; m < 2; ++m) dt_mma(d[m], a.p[0], b[m].ab.z, b[m].ab.w);
#pragma unroll
                for (int m = 0; m < 2; ++m) dt_mma(d[m], a.p[1], b[m].ab.x, b[m].ab.y);
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int e = 0; e < 4; ++e) u[m][e] = x[m][e] + (u[m][e] + d[m][e]);
            }
            float later[4] = {0.f, 0.f, 0.f, 0.f};                 // what A U is without the tensor core
            if (MASKED) {
                float in[8], sums[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) in[i] = x[i >> 2][i & 3];
                dt_masked(Tm, in, sums);
#pragma unroll
                for (int i = 0; i < 8; ++i) in[i] = u[i >> 2][i & 3] = x[i >> 2][i & 3] + sums[i];
                dt_masked(Am, in, sums);
#pragma unroll
                for (int e = 0; e < 4; ++e) later[e] = half ? sums[4 + e] : sums[e];
            }
            // read-outs of tokens 8 half ..: c (Q S) + A U, what FP32 adds to them first
            {
                const float2 c = *reinterpret_cast<const float2*>(vec + 32 + 8 * half + 2 * q4), own = *reinterpret_cast<const float2*>(vec + 64 + 8 * half + 2 * q4);
                o[0] = fmaf(c.x, o[0], own.x * (half ? u[1][0] : u[0][0])); o[1] = fmaf(c.y, o[1], own.y * (half ? u[1][1] : u[0][1]));
                o[2] = fmaf(c.x, o[2], own.x * (half ? u[1][2] : u[0][2])); o[3] = fmaf(c.y, o[3], own.y * (half ? u[1][3] : u[0][3]));
            }
            // S^T <- c_15 S^T + (U P(15, .))^T K
            {
                float w[2][4];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float2 tail = *reinterpret_cast<const float2*>(vec + 48 + 8 * j + 2 * q4);
                    w[j][0] = u[j][0] * tail.x; w[j][1] = u[j][1] * tail.y; w[j][2] = u[j][2] * tail.x; w[j][3] = u[j][3] * tail.y;
                }
                DtOperand a;
                dt_operand(w[0], w[1], a);
                const float all = vec[32 + 15];
#pragma unroll
                for (int i0 = 0; i0 < 8; i0 += 4) {
                    DtPiece b[4];
                    float big[4][4], d[4][4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        b[i] = dt_piece(st + 32 * DT_PIECE, 16, 8 * half + i0 + i, lane);
                        dt_mma_zero(big[i], a.p[0], b[i].ab.x, b[i].ab.y);
                        dt_mma_zero(d[i], a.p[0], b[i].c.x, b[i].c.y);
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) dt_mma(d[i], a.p[2], b[i].ab.x, b[i].ab.y);
#pragma unroll
                    for (int i = 0; i < 4; ++i) dt_mma(d[i], a.p[1], b[i].ab.z, b[i].ab.w);
#pragma unroll
                    for (int i = 0; i < 4; ++i) dt_mma(d[i], a.p[0], b[i].ab.z, b[i].ab.w);
#pragma unroll
                    for (int i = 0; i < 4; ++i) dt_mma(d[i], a.p[1], b[i].ab.x, b[i].ab.y);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int e = 0; e < 4; ++e) s[i0 + i][e] = fmaf(all, s[i0 + i][e], big[i][e] + d[i][e]);
                }
            }
            // ... and A U
            {
                DtOperand a;
                dt_operand(u[0], u[1], a);
                const DtPiece b = dt_piece(Am, 2, half, lane);
                float big[4], d[4];
                dt_mma_zero(big, a.p[0], b.ab.x, b.ab.y);
                dt_mma_zero(d, a.p[0], b.c.x, b.c.y);
                dt_mma(d, a.p[2], b.ab.x, b.ab.y);
                dt_mma(d, a.p[1], b.ab.z, b.ab.w);
                dt_mma(d, a.p[0], b.ab.z, b.ab.w);
                dt_mma(d, a.p[1], b.ab.x, b.ab.y);
#pragma unroll
                for (int e = 0; e < 4; ++e) o[e] += MASKED ? later[e] : big[e] + d[e];
                const int t = 8 * half + 2 * q4, tok = tile * DT_TOK + t;
                float* dst = out + (size_t)(first + tok) * dm.H * V + (size_t)h * V + col;
                if (there && tok < n) {
                    dst[0] = o[0];
                    dst[8] = o[2];
                }
                if (there && tok + 1 < n) {
                    dst[(size_t)dm.H * V] = o[1];
                    dst[(size_t)dm.H * V + 8] = o[3];
                }
            }
        }
    };
    walk(std::false_type{});
    // An infinity or a NaN in U: the tensor core has given it (0 times it) to the tokens before its own in its tile, too.  It has reached
    // the state's column as well, and stays there: then once more, T and A times nothing but earlier tokens.  (Looked for in every tile:
    // 3 to 7 us of 131.)
    float zero = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) zero += s[i][e] - s[i][e];
    if (__syncthreads_or(zero != 0.f)) walk(std::true_type{});
    if (there) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) S[(size_t)(8 * i + (e & 1)) * V + 8 * (e >> 1)] = s[i][e];
    }
}

// Bytes of scratch for n_tokens tokens of n_seqs requests: values (float), keys, coefficients.
NI_EXPORT long long ni_delta_tile_values(int n_tokens, int H, int V) { return 4LL * n_tokens * H * V; }
NI_EXPORT long long ni_delta_tile_keys(int n_tokens, int n_seqs, int G) { return ((long long)n_tokens / DT_TOK + n_seqs) * G * DT_KEYS; }
NI_EXPORT long long ni_delta_tile_coefs(int n_tokens, int n_seqs, int H) { return ((long long)n_tokens / DT_TOK + n_seqs) * H * DT_COEF; }

// The whole rule but its gated norm (and the new history, which ni_delta_gated_norm writes): proj [T, ld] from q's first
// column on (b_off, a_off: columns of b and a), values, keys and coef are scratch, out [T, H V].
NI_EXPORT int ni_delta_tile(const void* proj, int proj_dtype, const float* conv_w, const float* a_log, const float* dt_bias,
                            float* state, long long state_stride, const int* cu_q, const int* slots, int n_tokens, int n_seqs,
                            int G, int H, int V, int taps, int ld, int b_off, int a_off, float* values, uint8_t* keys, uint8_t* coef,
                            float* out, cudaStream_t stream) {
    if (n_tokens <= 0 || n_seqs <= 0) return NI_OK;
    if (G <= 0 || H <= 0 || H % G || V <= 0 || V % 16 || taps <= 0 || taps > 64) return NI_ERR_UNSUPPORTED_SIZE;
    DtDims dm{G, H, V, taps, ld, b_off, a_off};
    const auto aligned = [](const void* q) { return (reinterpret_cast<size_t>(q) & 15) == 0; };
    if (b_off < 0 || a_off < 0 || ld < dm.C() || ld < b_off + H || ld < a_off + H) return NI_ERR_BAD_ARGUMENT;
    if (state_stride % 4 || !aligned(state) || !aligned(values) || !aligned(keys) || !aligned(coef)) return NI_ERR_BAD_ARGUMENT;
    if (proj_dtype == NI_DTYPE_F32 && (ld % 4 || !aligned(proj))) return NI_ERR_BAD_ARGUMENT;      // (bfloat16 rows are read number by number)
    if (proj_dtype != NI_DTYPE_F32 && proj_dtype != NI_DTYPE_BF16) return NI_ERR_BAD_ARGUMENT;
    const dim3 pgrid(n_tokens / DT_TOK + n_seqs, G + (H * V + 127) / 128);
    if (H > 65535 || n_seqs > 65535 || pgrid.y > 65535) return NI_ERR_UNSUPPORTED_SIZE;
    const bool four = taps == 4 && aligned(conv_w);
#define PREPARE(T, TAPS)                                                                                                       \
    delta_tile_prepare_kernel<T, TAPS><<<pgrid, 128, 0, stream>>>((const T*)proj, conv_w, a_log, dt_bias, state, state_stride, cu_q, \
                                                                  slots, n_seqs, dm, values, keys, coef)
    if (proj_dtype == NI_DTYPE_F32) { if (four) PREPARE(float, 4); else PREPARE(float, 0); }
    else { if (four) PREPARE(__nv_bfloat16, 4); else PREPARE(__nv_bfloat16, 0); }
#undef PREPARE
    if (cudaError_t e = cudaGetLastError()) return (int)e;
    const cudaError_t e = cudaFuncSetAttribute(delta_tile_recurrence_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DT_SMEM);
    if (e != cudaSuccess) return (int)e;
    delta_tile_recurrence_kernel<<<dim3((V + 31) / 32, H, n_seqs), 128, DT_SMEM, stream>>>(values, keys, coef, state, state_stride, cu_q, slots,
                                                                                           dm, out);
    NI_RETURN_LAUNCH_STATUS();
}
