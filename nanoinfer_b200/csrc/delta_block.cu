// The gated delta rule with one decay per head over prompt portions, four tokens at a time, FP32 throughout (formula and
// layouts of delta_rule.cu, which walks the tokens one by one; longer portions of key heads of 128 go sixteen tokens at a time,
// delta_tile.cu).
//
// A request's tokens are taken in blocks of four from its portion's start on.  With S the state before a block, P(t, s) the
// product of the decays of tokens s + 1 .. t of the block and c_t that of tokens 0 .. t:
//     u_t = beta_t (v_t - c_t S^T k_t - sum_{s<t} P(t, s) (k_t . k_s) u_s)
//     o_t = c_t S^T q_t + sum_{s<=t} P(t, s) (q_t . k_s) u_s
//     S  <- c_3 S + sum_s P(3, s) k_s u_s^T
// so a block's eight products with S do not wait for one another, and one exchange between lanes serves four tokens: what
// bounds a portion is the chain of its blocks (0.64 us each, measured from 512 to 2,048 tokens of one request with 128 thread blocks of
// 4 warps: 1,270 clocks at 1,965 MHz), no longer the chain of its tokens (0.35 us each).  2,048 tokens, 16 heads of 128: 337 us with
// the preparation against 715; portions of 1,201 and 847 tokens 245 against 502 us; 8 portions of 512 tokens 329 against 536 us.
// Only products of decays over stretches of a block appear, never quotients.  Tokens that a last block lacks have beta 0,
// decay 1 and zeros for k, q and v, which leaves S alone.
//
// Two launches:
//   delta_block_prepare     a warp per (block, q/k head): convolution, silu and unit norms of four tokens from seven rows held
//                           in registers, the block's products k . k and q . k, and the coefficients above for each of its
//                           value heads; a warp per (block, 128 channels of v): convolution and silu.  Before, a warp per token
//                           read every row once per tap: 83 us for 2,048 tokens of 16 heads of 128
//   delta_block_recurrence  a block of 4 warps per (request, head, 8 COLS columns): a lane keeps ROWS = D / 16 rows of COLS
//                           columns of S in registers, 16 lanes share a column and add up by halving exchanges (a lane ends
//                           with whole sums of its own).  A lane that reads a k or q uses it for COLS columns, since shared
//                           memory hands out 128 bytes per clock however many lanes share them.
#include "common.cuh"

struct DbDims {
    int G, H, D, V, taps, ld, b_off, a_off;
    __host__ __device__ int C() const { return 2 * G * D + H * V; }
    __host__ __device__ size_t hist_off() const { return (size_t)H * D * V; }
};

// Coefficients of a block and head: 0 beta c | 4 beta | 8 c | 12 P(3, .) | 16 a 4 x 4 matrix: on and below its diagonal
// P(t, s) q_t . k_s at [t][s], above it beta_t P(t, s) k_t . k_s at [s][t].
#define DB_COEF 32
#define DB_T 4

__device__ __forceinline__ float db_silu(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float db_softplus(float z) { return z > 20.0f ? z : log1pf(expf(z)); }

// Blocks of four tokens before request `seq` (all of a warp's lanes get it).
__device__ __forceinline__ int db_blocks_before(const int* __restrict__ cu_q, int seq) {
    int n = 0;
    for (int i = threadIdx.x & 31; i < seq; i += 32) n += (cu_q[i + 1] - cu_q[i] + DB_T - 1) / DB_T;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    return n;
}
// The request that block number b belongs to and its number there (false: there is no such block).  One warp.
__device__ __forceinline__ bool db_find(const int* __restrict__ cu_q, int n_seqs, int b, int& seq, int& in_seq) {
    const int lane = threadIdx.x & 31;
    int before = 0;
    for (int s0 = 0; s0 < n_seqs; s0 += 32) {
        const int s = s0 + lane;
        const int mine = s < n_seqs ? (cu_q[s + 1] - cu_q[s] + DB_T - 1) / DB_T : 0;
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

// Four channels of an input row `back` tokens before the portion's token `at` (a negative index reads the history).
template <typename T>
__device__ __forceinline__ float4 db_row(const T* __restrict__ proj, const float* __restrict__ hist, const DbDims& dm, int first,
                                         int at, int c) {
    if (at >= 0) {
        const T* p = proj + (size_t)(first + at) * dm.ld + c;
        if (sizeof(T) == 4) return *reinterpret_cast<const float4*>(p);
        float4 v;
        v.x = ni_to_float(p[0]); v.y = ni_to_float(p[1]); v.z = ni_to_float(p[2]); v.w = ni_to_float(p[3]);
        return v;
    }
    return *reinterpret_cast<const float4*>(hist + (size_t)(dm.taps - 1 + at) * dm.C() + c);
}

// Convolution and silu of channels c .. c + 3 at the block's four tokens (zeros where a token does not exist).  TAPS 4: the
// four channels' weights are four 16-byte loads; 0: any number of taps, weights read where they are used.
template <typename T, int TAPS>
__device__ __forceinline__ void db_conv(const T* __restrict__ proj, const float* __restrict__ conv_w, const float* __restrict__ hist,
                                        const DbDims& dm, int first, int at, int live, int c, float4 y[DB_T]) {
    float4 acc[DB_T];
#pragma unroll
    for (int t = 0; t < DB_T; ++t) acc[t] = make_float4(0.f, 0.f, 0.f, 0.f);
    const float* w = conv_w + (size_t)c * dm.taps;
    if (TAPS == 4) {
        float4 x[DB_T + 3];                                        // inputs of tokens at - 3 .. at + 3
#pragma unroll
        for (int r = 0; r < DB_T + 3; ++r) x[r] = r - 3 < live ? db_row(proj, hist, dm, first, at - 3 + r, c) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 w0 = *reinterpret_cast<const float4*>(w), w1 = *reinterpret_cast<const float4*>(w + 4);
        const float4 w2 = *reinterpret_cast<const float4*>(w + 8), w3 = *reinterpret_cast<const float4*>(w + 12);
#pragma unroll
        for (int t = 0; t < DB_T; ++t) {
            acc[t].x = fmaf(w0.w, x[t + 3].x, fmaf(w0.z, x[t + 2].x, fmaf(w0.y, x[t + 1].x, w0.x * x[t].x)));
            acc[t].y = fmaf(w1.w, x[t + 3].y, fmaf(w1.z, x[t + 2].y, fmaf(w1.y, x[t + 1].y, w1.x * x[t].y)));
            acc[t].z = fmaf(w2.w, x[t + 3].z, fmaf(w2.z, x[t + 2].z, fmaf(w2.y, x[t + 1].z, w2.x * x[t].z)));
            acc[t].w = fmaf(w3.w, x[t + 3].w, fmaf(w3.z, x[t + 2].w, fmaf(w3.y, x[t + 1].w, w3.x * x[t].w)));
        }
    } else {
        for (int r = 0; r < DB_T + dm.taps - 1; ++r) {             // row r holds the inputs of token at - (taps - 1) + r
            if (r - (dm.taps - 1) >= live) break;                  // inputs of tokens that do not exist
            const float4 x = db_row(proj, hist, dm, first, at - (dm.taps - 1) + r, c);
#pragma unroll
            for (int t = 0; t < DB_T; ++t) {
                const int j = r - t;                               // this row is tap j of token t
                if (j >= 0 && j < dm.taps) {
                    acc[t].x = fmaf(w[j], x.x, acc[t].x);
                    acc[t].y = fmaf(w[dm.taps + j], x.y, acc[t].y);
                    acc[t].z = fmaf(w[2 * dm.taps + j], x.z, acc[t].z);
                    acc[t].w = fmaf(w[3 * dm.taps + j], x.w, acc[t].w);
                }
            }
        }
    }
#pragma unroll
    for (int t = 0; t < DB_T; ++t)
        y[t] = t < live ? make_float4(db_silu(acc[t].x), db_silu(acc[t].y), db_silu(acc[t].z), db_silu(acc[t].w))
                        : make_float4(0.f, 0.f, 0.f, 0.f);
}

__device__ __forceinline__ float db_dot4(const float4& a, const float4& b, float acc) {
    return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, acc))));
}

#define DB_WARPS 4
template <typename T, int NC, int TAPS>       // NC: channels of a q or k head per lane / 4 (D <= 128 NC)
__global__ void __launch_bounds__(DB_WARPS * 32)
delta_block_prepare_kernel(const T* __restrict__ proj, const float* __restrict__ conv_w, const float* __restrict__ a_log,
                           const float* __restrict__ dt_bias, const float* __restrict__ state, long long state_stride,
                           const int* __restrict__ cu_q, const int* __restrict__ slots, int n_seqs, DbDims dm,
                           float* __restrict__ qkv, float* __restrict__ coef) {
    const int lane = threadIdx.x & 31;
    int unit = blockIdx.y * DB_WARPS + (threadIdx.x >> 5);
    const int C = dm.C(), HV = dm.H * dm.V;
    if (unit >= dm.G + (HV + 127) / 128) return;
    int seq, in_seq;
    if (!db_find(cu_q, n_seqs, blockIdx.x, seq, in_seq)) return;
    const int first = cu_q[seq], at = in_seq * DB_T, left = cu_q[seq + 1] - first - at, live = left < DB_T ? left : DB_T;
    const float* hist = state + (size_t)slots[seq] * state_stride + dm.hist_off();
    float* out = qkv + (size_t)(first + at) * C;
    float4 y[DB_T];
    if (unit >= dm.G) {                       // values
        const int c = 2 * dm.G * dm.D + (unit - dm.G) * 128 + 4 * lane;
        if (c >= C) return;
        db_conv<T, TAPS>(proj, conv_w, hist, dm, first, at, live, c, y);
#pragma unroll
        for (int t = 0; t < DB_T; ++t)
            if (t < live) *reinterpret_cast<float4*>(out + (size_t)t * C + c) = y[t];
        return;
    }
    const int g = unit, D = dm.D;
    float4 q[NC][DB_T], k[NC][DB_T];
#pragma unroll
    for (int n = 0; n < NC; ++n) {
        const int d = 128 * n + 4 * lane;
        if (d < D) {
            db_conv<T, TAPS>(proj, conv_w, hist, dm, first, at, live, g * D + d, q[n]);
            db_conv<T, TAPS>(proj, conv_w, hist, dm, first, at, live, (dm.G + g) * D + d, k[n]);
        } else {
#pragma unroll
            for (int t = 0; t < DB_T; ++t) q[n][t] = k[n][t] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    float rq[DB_T], rk[DB_T];                 // the factors that make unit vectors (q also times D^-1/2)
#pragma unroll
    for (int t = 0; t < DB_T; ++t) {
        float a = 0.f, b = 0.f;
#pragma unroll
        for (int n = 0; n < NC; ++n) {
            a = db_dot4(q[n][t], q[n][t], a);
            b = db_dot4(k[n][t], k[n][t], b);
        }
        rq[t] = (1.0f / sqrtf(ni_warp_sum(a) + 1e-6f)) * (1.0f / sqrtf((float)D));
        rk[t] = 1.0f / sqrtf(ni_warp_sum(b) + 1e-6f);
    }
#pragma unroll
    for (int n = 0; n < NC; ++n) {
        const int d = 128 * n + 4 * lane;
#pragma unroll
        for (int t = 0; t < DB_T; ++t) {
            q[n][t].x *= rq[t]; q[n][t].y *= rq[t]; q[n][t].z *= rq[t]; q[n][t].w *= rq[t];
            k[n][t].x *= rk[t]; k[n][t].y *= rk[t]; k[n][t].z *= rk[t]; k[n][t].w *= rk[t];
            if (d < D && t < live) {
                *reinterpret_cast<float4*>(out + (size_t)t * C + g * D + d) = q[n][t];
                *reinterpret_cast<float4*>(out + (size_t)t * C + (dm.G + g) * D + d) = k[n][t];
            }
        }
    }
    // lane 4 t + s, s <= t: q_t . k_s; s > t: k_s . k_t
    float pair = 0.f;
#pragma unroll
    for (int t = 0; t < DB_T; ++t)
#pragma unroll
        for (int s = 0; s < DB_T; ++s) {
            float a = 0.f;
#pragma unroll
            for (int n = 0; n < NC; ++n) a = db_dot4(s <= t ? q[n][t] : k[n][t], k[n][s], a);
            a = ni_warp_sum(a);
            if (lane == 16 + 4 * t + s) pair = a;
        }
    const int per = dm.H / dm.G;
    for (int h = g * per; h < (g + 1) * per; ++h) {
        float decay = 1.f, beta = 0.f;        // lane t < 4: token t's
        if (lane < live) {
            const T* row = proj + (size_t)(first + at + lane) * dm.ld;
            decay = expf(-expf(a_log[h]) * db_softplus(ni_to_float(row[dm.a_off + h]) + dt_bias[h]));
            beta = 1.0f / (1.0f + expf(-ni_to_float(row[dm.b_off + h])));
        }
        float d[DB_T], b[DB_T];
#pragma unroll
        for (int t = 0; t < DB_T; ++t) {
            d[t] = __shfl_sync(0xffffffffu, decay, t);
            b[t] = __shfl_sync(0xffffffffu, beta, t);
        }
        // this lane's coefficient: decays of tokens lo .. hi, times what belongs to it
        const int t = (lane >> 2) & 3, s = lane & 3;
        int lo, hi;
        float f;
        if (lane < 4) { lo = 0; hi = s; f = b[s == 0 ? 0 : s == 1 ? 1 : s == 2 ? 2 : 3]; }
        else if (lane < 8) { lo = 1; hi = 0; f = b[s == 0 ? 0 : s == 1 ? 1 : s == 2 ? 2 : 3]; }
        else if (lane < 12) { lo = 0; hi = s; f = 1.f; }
        else if (lane < 16) { lo = s + 1; hi = 3; f = 1.f; }
        else if (s <= t) { lo = s + 1; hi = t; f = pair; }
        else { lo = t + 1; hi = s; f = pair * (s == 1 ? b[1] : s == 2 ? b[2] : b[3]); }      // the later token's beta
#pragma unroll
        for (int i = 0; i < DB_T; ++i)
            if (i >= lo && i <= hi) f *= d[i];
        coef[((size_t)blockIdx.x * dm.H + h) * DB_COEF + lane] = f;
    }
}

__device__ __forceinline__ void db_copy16(float* dst_smem, const float* src, bool live) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
    const int n = live ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void db_fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long db_mul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long db_pair(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 db_split(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

// A lane's COLS (2 or 4) neighbouring columns of a row of S: one access.  (V is a multiple of 4 and a lane's first column one of
// COLS, so they lie on 4 COLS bytes.)
template <int COLS> __device__ __forceinline__ void db_load(const float* p, float* v) {
    if (COLS == 4) {
        const float4 x = *reinterpret_cast<const float4*>(p);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    } else {
        const float2 x = *reinterpret_cast<const float2*>(p);
        v[0] = x.x; v[1] = x.y;
    }
}
template <int COLS> __device__ __forceinline__ void db_store(float* p, const float* v) {
    if (COLS == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
}

#define DB_STAGES 4
// ROWS rows of COLS columns per lane: row quads 64 j + 4 (lane % 16) .. + 3, columns of half warp lane / 16.
template <int ROWS, int COLS>
__global__ void __launch_bounds__(DB_WARPS * 32)
delta_block_recurrence_kernel(const float* __restrict__ qkv, const float* __restrict__ coef, float* __restrict__ state,
                              long long state_stride, const int* __restrict__ cu_q, const int* __restrict__ slots, DbDims dm,
                              float* __restrict__ out) {
    constexpr int D = 16 * ROWS, QUADS = ROWS / 4, BCOLS = DB_WARPS * 2 * COLS;
    constexpr int STAGE = 2 * DB_T * D + DB_T * BCOLS + DB_COEF, VALS = 2 * DB_T * COLS;       // VALS sums per half warp
    extern __shared__ __align__(16) float db_smem[];
    float* exch = db_smem + DB_STAGES * STAGE + (threadIdx.x >> 4) * VALS;                     // this half warp's
    const int tid = threadIdx.x, lane = tid & 31, rg = lane & 15, half_warp = tid >> 4;
    const int h = blockIdx.y, seq = blockIdx.z, g = h / (dm.H / dm.G), C = dm.C();
    const int col0 = blockIdx.x * BCOLS, col = col0 + half_warp * COLS;
    const int first = cu_q[seq], n = cu_q[seq + 1] - first;
    if (n <= 0) return;
    const int blocks = (n + DB_T - 1) / DB_T;
    const float* cf = coef + ((size_t)db_blocks_before(cu_q, seq) * dm.H + h) * DB_COEF;
    // Each thread's share of a block: chunks of 16 bytes of the four tokens' k, then q (PER of them), and one chunk of the
    // values or of the coefficients for some; the sources move on by four tokens per block.
    constexpr int PER = 2 * DB_T * D / 4 / (DB_WARPS * 32);
    const float* kq_src[PER];
    int kq_tok[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int i = tid + j * DB_WARPS * 32, t = i / (D / 4), d = 4 * (i % (D / 4));
        kq_tok[j] = t & 3;
        kq_src[j] = qkv + (size_t)(first + (t & 3)) * C + (t < DB_T ? dm.G + g : g) * D + d;
    }
    constexpr int VCH = DB_T * BCOLS / 4;
    static_assert(VCH + DB_COEF / 4 <= DB_WARPS * 32, "one chunk of values or coefficients per thread");
    const int v_tok = tid / (BCOLS / 4), v_col = 4 * (tid % (BCOLS / 4));
    const bool v_mine = tid < VCH, v_there = col0 + v_col < dm.V, c_mine = !v_mine && tid < VCH + DB_COEF / 4;
    const float* x_src = v_mine ? qkv + (size_t)(first + v_tok) * C + 2 * dm.G * D + h * dm.V + col0 + (v_there ? v_col : 0)
                                : cf + 4 * (tid - VCH);
    const size_t step = (size_t)DB_T * C;
    int fetched = 0;
    float* stage_in = db_smem;
    auto fetch = [&]() {
        if (fetched < blocks) {
            const int tok = fetched * DB_T;
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                const bool live = tok + kq_tok[j] < n;
                db_copy16(stage_in + 4 * (tid + j * DB_WARPS * 32), live ? kq_src[j] : qkv, live);
                kq_src[j] += step;
            }
            if (v_mine) {
                const bool live = v_there && tok + v_tok < n;
                db_copy16(stage_in + 2 * DB_T * D + 4 * tid, live ? x_src : qkv, live);
                x_src += step;
            } else if (c_mine) {
                db_copy16(stage_in + 2 * DB_T * D + 4 * tid, x_src, true);
                x_src += (size_t)dm.H * DB_COEF;
            }
        }
        ++fetched;
        stage_in = stage_in == db_smem + (DB_STAGES - 1) * STAGE ? db_smem : stage_in + STAGE;
        asm volatile("cp.async.commit_group;" ::: "memory");       // one group per block of tokens, empty or not
    };
    for (int p = 0; p < DB_STAGES - 1; ++p) fetch();
    const bool there = col < dm.V;                                  // V is a multiple of COLS: all of a half warp's columns or none
    float* S = state + (size_t)slots[seq] * state_stride + ((size_t)h * D + 4 * rg) * dm.V + col;
    unsigned long long s2[ROWS / 2][COLS];
#pragma unroll
    for (int r = 0; r < ROWS / 2; ++r) {
        const size_t row = 64 * (r / 2) + 2 * (r & 1);
        float a[COLS], b[COLS];
#pragma unroll
        for (int c = 0; c < COLS; ++c) a[c] = b[c] = 0.f;
        if (there) {
            db_load<COLS>(S + row * dm.V, a);
            db_load<COLS>(S + (row + 1) * dm.V, b);
        }
#pragma unroll
        for (int c = 0; c < COLS; ++c) s2[r][c] = db_pair(a[c], b[c]);
    }
    const float* stage = db_smem;
    for (int b = 0; b < blocks; ++b) {
        asm volatile("cp.async.wait_group %0;" ::"n"(DB_STAGES - 2) : "memory");
        __syncthreads();                                            // block b is there; every warp has left block b - 1
        fetch();
        const float* ks = stage + 4 * rg;
        const float* qs = ks + DB_T * D;
        const float* vs = stage + 2 * DB_T * D + half_warp * COLS;
        const float* cs = stage + 2 * DB_T * D + DB_T * BCOLS;
        stage = stage == db_smem + (DB_STAGES - 1) * STAGE ? db_smem : stage + STAGE;
        ulonglong2 k[DB_T][QUADS];
        float sum[VALS];
#pragma unroll
        for (int t = 0; t < DB_T; ++t) {
            unsigned long long a[COLS], o[COLS];
#pragma unroll
            for (int c = 0; c < COLS; ++c) a[c] = o[c] = 0ull;
#pragma unroll
            for (int j = 0; j < QUADS; ++j) {
                k[t][j] = *reinterpret_cast<const ulonglong2*>(ks + t * D + 64 * j);
                const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(qs + t * D + 64 * j);
#pragma unroll
                for (int c = 0; c < COLS; ++c) {
                    db_fma2(a[c], k[t][j].x, s2[2 * j][c]);
                    db_fma2(o[c], q.x, s2[2 * j][c]);
                    db_fma2(a[c], k[t][j].y, s2[2 * j + 1][c]);
                    db_fma2(o[c], q.y, s2[2 * j + 1][c]);
                }
            }
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                const float2 x = db_split(a[c]), y = db_split(o[c]);
                sum[t * COLS + c] = x.x + x.y;
                sum[DB_T * COLS + t * COLS + c] = y.x + y.y;
            }
        }
        // halving exchanges over the 16 lanes of a column group: lane rg ends with sums rg VALS / 16 .. of the VALS ones
        int width = VALS / 2;
#pragma unroll
        for (int off = 8; off > 0; off >>= 1, width >>= 1) {
            const bool upper = rg & off;
#pragma unroll
            for (int i = 0; i < VALS / 2; ++i)
                if (i < width) {
                    const float give = upper ? sum[i] : sum[i + width], keep = upper ? sum[i + width] : sum[i];
                    sum[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
                }
        }
#pragma unroll
        for (int i = 0; i < VALS / 16; ++i) exch[rg * (VALS / 16) + i] = sum[i];
        __syncwarp();
        float u[DB_T][COLS];
        {
            const float4 bc = *reinterpret_cast<const float4*>(cs), be = *reinterpret_cast<const float4*>(cs + 4);
            const float4 m0 = *reinterpret_cast<const float4*>(cs + 16), m1 = *reinterpret_cast<const float4*>(cs + 20),
                         m2 = *reinterpret_cast<const float4*>(cs + 24);
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                const float r0 = be.x * vs[c] - bc.x * exch[c], r1 = be.y * vs[BCOLS + c] - bc.y * exch[COLS + c];
                const float r2 = be.z * vs[2 * BCOLS + c] - bc.z * exch[2 * COLS + c];
                const float r3 = be.w * vs[3 * BCOLS + c] - bc.w * exch[3 * COLS + c];
                u[0][c] = r0;
                u[1][c] = fmaf(-m0.y, u[0][c], r1);
                u[2][c] = fmaf(-m1.z, u[1][c], fmaf(-m0.z, u[0][c], r2));
                u[3][c] = fmaf(-m2.w, u[2][c], fmaf(-m1.w, u[1][c], fmaf(-m0.w, u[0][c], r3)));
            }
        }
        // read-outs: lanes t COLS + c of the half warp, one number each
        if (rg < DB_T * COLS) {
            const int t = rg / COLS, c = rg % COLS, tok = b * DB_T + t;
            const float4 m = *reinterpret_cast<const float4*>(cs + 16 + 4 * t);
            float uc[DB_T];
#pragma unroll
            for (int i = 0; i < DB_T; ++i) {
                uc[i] = u[i][0];
#pragma unroll
                for (int j = 1; j < COLS; ++j) uc[i] = c == j ? u[i][j] : uc[i];
            }
            float y = cs[8 + t] * exch[DB_T * COLS + rg];
            y = fmaf(m.x, uc[0], y);
            if (t > 0) y = fmaf(m.y, uc[1], y);
            if (t > 1) y = fmaf(m.z, uc[2], y);
            if (t > 2) y = fmaf(m.w, uc[3], y);
            if (there && tok < n) out[(size_t)(first + tok) * dm.H * dm.V + h * dm.V + col + c] = y;
        }
        const float4 tail = *reinterpret_cast<const float4*>(cs + 12);
        const float c3 = cs[11];
        const unsigned long long all = db_pair(c3, c3);
#pragma unroll
        for (int c = 0; c < COLS; ++c) {
            const float w0 = tail.x * u[0][c], w1 = tail.y * u[1][c], w2 = tail.z * u[2][c], w3 = tail.w * u[3][c];
            const unsigned long long p0 = db_pair(w0, w0), p1 = db_pair(w1, w1), p2 = db_pair(w2, w2), p3 = db_pair(w3, w3);
#pragma unroll
            for (int j = 0; j < QUADS; ++j) {
                unsigned long long x = db_mul2(s2[2 * j][c], all), y = db_mul2(s2[2 * j + 1][c], all);
                db_fma2(x, k[0][j].x, p0); db_fma2(y, k[0][j].y, p0);
                db_fma2(x, k[1][j].x, p1); db_fma2(y, k[1][j].y, p1);
                db_fma2(x, k[2][j].x, p2); db_fma2(y, k[2][j].y, p2);
                db_fma2(x, k[3][j].x, p3); db_fma2(y, k[3][j].y, p3);
                s2[2 * j][c] = x;
                s2[2 * j + 1][c] = y;
            }
        }
        __syncwarp();                                               // exch has been read before the next block writes it
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (there) {
#pragma unroll
        for (int r = 0; r < ROWS / 2; ++r) {
            const size_t row = 64 * (r / 2) + 2 * (r & 1);
            float a[COLS], b[COLS];
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                const float2 x = db_split(s2[r][c]);
                a[c] = x.x;
                b[c] = x.y;
            }
            db_store<COLS>(S + row * dm.V, a);
            db_store<COLS>(S + (row + 1) * dm.V, b);
        }
    }
}

// Whether these sizes are taken: key heads of 64, 128 or 256, whole 16-byte groups everywhere.
static int db_supports(int G, int H, int D, int V, int taps) {
    return G > 0 && H > 0 && H % G == 0 && (D == 64 || D == 128 || D == 256) && V > 0 && V % 4 == 0 && taps > 0 && taps <= 64;
}
// Floats of the coefficients of n_tokens tokens of n_seqs requests.
NI_EXPORT long long ni_delta_block_coefs(int n_tokens, int n_seqs, int H) {
    return ((long long)n_tokens / DB_T + n_seqs) * H * DB_COEF;
}

// The whole rule but its gated norm (and the new history, which ni_delta_gated_norm writes): proj [T, ld] from q's first
// column on (b_off, a_off: columns of b and a), qkv [T, C] and coef are scratch, out [T, H V].
NI_EXPORT int ni_delta_block(const void* proj, int proj_dtype, const float* conv_w, const float* a_log, const float* dt_bias,
                             float* state, long long state_stride, const int* cu_q, const int* slots, int n_tokens, int n_seqs,
                             int G, int H, int D, int V, int taps, int ld, int b_off, int a_off, float* qkv, float* coef,
                             float* out, cudaStream_t stream) {
    if (n_tokens <= 0 || n_seqs <= 0) return NI_OK;
    if (!db_supports(G, H, D, V, taps)) return NI_ERR_UNSUPPORTED_SIZE;
    DbDims dm{G, H, D, V, taps, ld, b_off, a_off};
    const auto aligned = [](const void* q) { return (reinterpret_cast<size_t>(q) & 15) == 0; };
    if (b_off < 0 || a_off < 0 || ld < dm.C() || ld < b_off + H || ld < a_off + H) return NI_ERR_BAD_ARGUMENT;
    if (state_stride % 4 || !aligned(state) || !aligned(qkv) || !aligned(coef)) return NI_ERR_BAD_ARGUMENT;
    if (proj_dtype == NI_DTYPE_F32 && (ld % 4 || !aligned(proj))) return NI_ERR_BAD_ARGUMENT;      // (bfloat16 rows are read number by number)
    if (H > 65535 || n_seqs > 65535) return NI_ERR_UNSUPPORTED_SIZE;
    const int units = G + (H * V + 127) / 128;
    const dim3 pgrid(n_tokens / DB_T + n_seqs, (units + DB_WARPS - 1) / DB_WARPS);
    if (pgrid.y > 65535) return NI_ERR_UNSUPPORTED_SIZE;
#define PREPARE(T, NC)                                                                                                   \
    if (taps == 4 && aligned(conv_w)) PREPARE_T(T, NC, 4); else PREPARE_T(T, NC, 0)
#define PREPARE_T(T, NC, TAPS)                                                                                           \
    delta_block_prepare_kernel<T, NC, TAPS><<<pgrid, DB_WARPS * 32, 0, stream>>>((const T*)proj, conv_w, a_log, dt_bias, state, \
                                                                          state_stride, cu_q, slots, n_seqs, dm, qkv, coef)
    if (proj_dtype == NI_DTYPE_F32) {
        if (D <= 128) { PREPARE(float, 1); } else { PREPARE(float, 2); }
    } else if (proj_dtype == NI_DTYPE_BF16) {
        if (D <= 128) { PREPARE(__nv_bfloat16, 1); } else { PREPARE(__nv_bfloat16, 2); }
    } else {
        return NI_ERR_BAD_ARGUMENT;
    }
#undef PREPARE
#undef PREPARE_T
    if (cudaError_t e = cudaGetLastError()) return (int)e;
    // Four columns per lane read a k and q from shared memory for twice as many columns; two halve what a lane does for a block
    // of tokens, which is faster as long as twice the blocks still have an SM each.  Heads of 128, us with four / two columns: 64
    // blocks of four columns (one portion of 512, 16 heads) 102.9 / 89.5, 96 (3 x 256 tokens, 8 heads) 56.8 / 63.6, 128 (2 x 256,
    // 16 heads) 58.5 / 65.2, 256 89.8 / 105.4; heads of 64: 64 blocks 47.9 / 46.7, 96 49.7 / 56.6.
    const bool few = 2LL * ((V + 31) / 32) * H * n_seqs <= ni_sm_count();
#define LAUNCH(ROWS, COLS)                                                                                                \
    do {                                                                                                                  \
        constexpr int B = DB_WARPS * 2 * (COLS);                                                                          \
        constexpr int SMEM = (DB_STAGES * (2 * DB_T * 16 * (ROWS) + DB_T * B + DB_COEF) + 8 * 2 * DB_T * (COLS)) * (int)sizeof(float); \
        auto kernel = delta_block_recurrence_kernel<ROWS, COLS>;                                                          \
        if (SMEM > 48 * 1024) {                                                                                           \
            const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);        \
            if (e != cudaSuccess) return (int)e;                                                                          \
        }                                                                                                                 \
        kernel<<<dim3((V + B - 1) / B, H, n_seqs), DB_WARPS * 32, SMEM, stream>>>(qkv, coef, state, state_stride, cu_q, slots, dm, out); \
    } while (0)
    if (D == 64) { if (few) LAUNCH(4, 2); else LAUNCH(4, 4); }
    else if (D == 128) { if (few) LAUNCH(8, 2); else LAUNCH(8, 4); }
    else LAUNCH(16, 2);
#undef LAUNCH
    NI_RETURN_LAUNCH_STATUS();
}
