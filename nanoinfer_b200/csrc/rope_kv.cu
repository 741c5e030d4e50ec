// Rotary position encoding of queries and keys, fused with the write of keys and values
// into their cache pages.
//
// The reference does this in three launches over FP32 tensors: rotation in place from a
// precomputed sin/cos table (src/op/kernels/cuda/rope_kernel.cu:32-84, table built at
// :95-132), then a paged write for decode (paged_kv_writed_kernel.cu:33-75) or for a
// prefill chunk (prefill_attention_kernel.cu:219-248).  Here one launch reads the fused
// QKV projection once: queries go rotated to a dense buffer, keys go rotated and values
// go unchanged straight to their page slots.  The angle is the FP32 product
// float(position) * inv_freq, as in the reference's table (rope_kernel.cu:127), and sin/cos
// are evaluated in FP32 per element instead of being read from a table of
// max_position rows.
//
// Page layout: [num_pages, num_kv_heads, page_size, head_dim]; the page of token t is
// block_table[seq_of_token[t] * bt_stride + position / page_size].
#include "common.cuh"

template <typename T>
__global__ void rope_kv_write_kernel(const T* __restrict__ qkv, T* __restrict__ q_out,
                                     T* __restrict__ k_pages, T* __restrict__ v_pages,
                                     const int* __restrict__ positions,
                                     const int* __restrict__ seq_of_token,
                                     const int* __restrict__ block_table, int bt_stride,
                                     const float* __restrict__ inv_freq, int n_q_heads,
                                     int n_kv_heads, int head_dim, int rotary_dim,
                                     int interleaved, int page_size, int write_cache) {
    const int t = blockIdx.x;
    const int pos = positions[t];
    const int half = head_dim / 2;
    const int rot_half = rotary_dim / 2;
    const int row_width = (n_q_heads + 2 * n_kv_heads) * head_dim;
    const T* row = qkv + (size_t)t * row_width;
    size_t kv_base = 0;
    if (write_cache) {
        const int page = block_table[(size_t)seq_of_token[t] * bt_stride + pos / page_size];
        kv_base = ((size_t)page * n_kv_heads * page_size + (pos % page_size)) * head_dim;
    }
    const int n_pairs = (n_q_heads + 2 * n_kv_heads) * half;
    for (int p = threadIdx.x; p < n_pairs; p += blockDim.x) {
        const int head = p / half;
        const int i = p - head * half;
        int ia, ib;
        bool rotate = false;
        if (i < rot_half && head < n_q_heads + n_kv_heads) {
            rotate = true;
            if (interleaved) { ia = 2 * i; ib = 2 * i + 1; }
            else { ia = i; ib = i + rot_half; }
        } else if (head < n_q_heads + n_kv_heads) {
            // dimensions beyond rotary_dim pass through unchanged
            ia = rotary_dim + 2 * (i - rot_half); ib = ia + 1;
        } else {
            ia = 2 * i; ib = 2 * i + 1;
        }
        float a = ni_to_float(row[head * head_dim + ia]);
        float b = ni_to_float(row[head * head_dim + ib]);
        if (rotate) {
            float s, c;
            sincosf((float)pos * inv_freq[i], &s, &c);
            const float ra = a * c - b * s;
            const float rb = a * s + b * c;
            a = ra; b = rb;
        }
        T* dst;
        if (head < n_q_heads) {
            dst = q_out + ((size_t)t * n_q_heads + head) * head_dim;
        } else if (!write_cache) {
            continue;
        } else if (head < n_q_heads + n_kv_heads) {
            dst = k_pages + kv_base + (size_t)(head - n_q_heads) * page_size * head_dim;
        } else {
            dst = v_pages + kv_base + (size_t)(head - n_q_heads - n_kv_heads) * page_size * head_dim;
        }
        dst[ia] = ni_from_float<T>(a);
        dst[ib] = ni_from_float<T>(b);
    }
}

// Adjacent-pair rotation with 16-byte accesses: one thread takes 8 consecutive elements (4
// rotary pairs) of one head of one token.  head_dim a multiple of 8.
template <typename T> struct Chunk8;
template <> struct Chunk8<__nv_bfloat16> {
    static __device__ __forceinline__ void load(const __nv_bfloat16* p, float v[8]) {
        const uint4 r = *reinterpret_cast<const uint4*>(p);
        const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&w[i]);
            v[2 * i] = __bfloat162float(b.x);
            v[2 * i + 1] = __bfloat162float(b.y);
        }
    }
    static __device__ __forceinline__ void store(__nv_bfloat16* p, const float v[8]) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            w[i] = *reinterpret_cast<uint32_t*>(&b);
        }
        *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
    }
};
template <> struct Chunk8<float> {
    static __device__ __forceinline__ void load(const float* p, float v[8]) {
        const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
    static __device__ __forceinline__ void store(float* p, const float v[8]) {
        *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
    }
};

// Adjacent-pair rotation with 16-byte accesses.  A block takes one token at a time: the token's
// rotary_dim / 2 (cos, sin) pairs are computed once into shared memory (they are the same for all
// of its heads) and its page is looked up once; then every thread rotates 8-element chunks.
template <typename T>
__global__ void rope_kv_write_vec_kernel(const T* __restrict__ qkv, T* __restrict__ q_out,
                                         T* __restrict__ k_pages, T* __restrict__ v_pages,
                                         const int* __restrict__ positions,
                                         const int* __restrict__ seq_of_token,
                                         const int* __restrict__ block_table, int bt_stride,
                                         const float* __restrict__ inv_freq, int n_tokens, int n_q_heads,
                                         int n_kv_heads, int head_dim, int rotary_dim, int page_size,
                                         int write_cache) {
    extern __shared__ float rope_cs[];                 // [rotary_dim / 2][cos, sin]
    const int chunks_per_head = head_dim >> 3;
    const int heads = n_q_heads + 2 * n_kv_heads;
    const int items = heads * chunks_per_head;
    for (int t = blockIdx.x; t < n_tokens; t += gridDim.x) {
        const int pos = positions[t];
        __syncthreads();                               // the table of the token before is no longer read
        for (int i = threadIdx.x; i < (rotary_dim >> 1); i += blockDim.x) {
            float s, cs;
            sincosf((float)pos * inv_freq[i], &s, &cs);
            rope_cs[2 * i] = cs;
            rope_cs[2 * i + 1] = s;
        }
        __syncthreads();
        const int page = write_cache ? block_table[(size_t)seq_of_token[t] * bt_stride + pos / page_size] : 0;
        const int slot = pos % page_size;
        // four chunks per thread and pass: all loads are issued before the first store, since what
        // bounds this kernel is the number of bytes in flight
        for (int item0 = threadIdx.x; item0 < items; item0 += 4 * blockDim.x) {
            float v[4][8];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int item = item0 + u * blockDim.x;
                if (item < items) {
                    const int head = item / chunks_per_head, c = item - head * chunks_per_head;
                    Chunk8<T>::load(qkv + ((size_t)t * heads + head) * head_dim + 8 * c, v[u]);
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int item = item0 + u * blockDim.x;
                if (item >= items) continue;
                const int head = item / chunks_per_head, c = item - head * chunks_per_head;
                if (head < n_q_heads + n_kv_heads) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int d = 8 * c + 2 * i;
                        if (d < rotary_dim) {
                            const float cs = rope_cs[d], sn = rope_cs[d + 1];
                            const float a = v[u][2 * i], b = v[u][2 * i + 1];
                            v[u][2 * i] = a * cs - b * sn;
                            v[u][2 * i + 1] = a * sn + b * cs;
                        }
                    }
                }
                T* dst;
                if (head < n_q_heads) {
                    dst = q_out + ((size_t)t * n_q_heads + head) * head_dim + 8 * c;
                } else {
                    if (!write_cache) continue;
                    const bool is_k = head < n_q_heads + n_kv_heads;
                    const int kvh = is_k ? head - n_q_heads : head - n_q_heads - n_kv_heads;
                    dst = (is_k ? k_pages : v_pages) + (((size_t)page * n_kv_heads + kvh) * page_size + slot) * head_dim + 8 * c;
                }
                Chunk8<T>::store(dst, v[u]);
            }
        }
    }
}

// The same for heads whose 8-element chunks divide a warp (head sizes 16, 32, 64, 128, 256): a lane keeps one chunk column of
// every head it visits, so its four cosines and sines are computed once and stay in registers - no table in shared memory, no
// barrier -, and the loads of all its heads (which need no position) are on their way before the token's position, angles and
// page are known.  A block is a token; a warp visits 32 / chunks heads at a time, ITEMS times at most before it stores.
// Bound by the chain position -> angles -> page -> stores of a token (one wave of blocks), not yet by its bytes: 2,048 tokens
// of 48 heads of 64 (25 MB) 8.1 -> 7.4 us, 1,914 tokens of 48 heads of 128 (47 MB) 17.0 -> 10.9 us against the table (replayed
// launches, the cache warm).
template <typename T, int ITEMS>
__global__ void __launch_bounds__(256)
rope_kv_write_lanes_kernel(const T* __restrict__ qkv, T* __restrict__ q_out, T* __restrict__ k_pages, T* __restrict__ v_pages,
                           const int* __restrict__ positions, const int* __restrict__ seq_of_token,
                           const int* __restrict__ block_table, int bt_stride, const float* __restrict__ inv_freq,
                           int n_q_heads, int n_kv_heads, int head_dim, int log_chunks, int rotary_dim, int page_size,
                           int write_cache) {
    const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int c = lane & ((1 << log_chunks) - 1), at_once = 32 >> log_chunks;
    const int heads = n_q_heads + 2 * n_kv_heads, used = write_cache ? heads : n_q_heads;
    const T* row = qkv + (size_t)t * heads * head_dim + 8 * c;
    float cs[4], sn[4];
    size_t kv_base = 0;
    bool first = true;
    for (int h0 = warp * at_once + (lane >> log_chunks); h0 - (lane >> log_chunks) < used; h0 += ITEMS * warps * at_once) {
        float v[ITEMS][8];
#pragma unroll
        for (int u = 0; u < ITEMS; ++u) {
            const int head = h0 + u * warps * at_once;
            if (head < used) Chunk8<T>::load(row + (size_t)head * head_dim, v[u]);
        }
        if (first) {
            first = false;
            const int pos = positions[t];
            if (write_cache) {
                const int page = block_table[(size_t)seq_of_token[t] * bt_stride + pos / page_size];
                kv_base = ((size_t)page * n_kv_heads * page_size + pos % page_size) * head_dim + 8 * c;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                cs[i] = 1.f;
                sn[i] = 0.f;
                if (8 * c + 2 * i < rotary_dim) sincosf((float)pos * inv_freq[4 * c + i], &sn[i], &cs[i]);
            }
        }
#pragma unroll
        for (int u = 0; u < ITEMS; ++u) {
            const int head = h0 + u * warps * at_once;
            if (head >= used) continue;
            T* dst;
            if (head < n_q_heads) dst = q_out + ((size_t)t * n_q_heads + head) * head_dim + 8 * c;
            else if (head < n_q_heads + n_kv_heads) dst = k_pages + kv_base + (size_t)(head - n_q_heads) * page_size * head_dim;
            else dst = v_pages + kv_base + (size_t)(head - n_q_heads - n_kv_heads) * page_size * head_dim;
            if (head < n_q_heads + n_kv_heads) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (8 * c + 2 * i < rotary_dim) {
                        const float a = v[u][2 * i], b = v[u][2 * i + 1];
                        v[u][2 * i] = a * cs[i] - b * sn[i];
                        v[u][2 * i + 1] = a * sn[i] + b * cs[i];
                    }
            }
            Chunk8<T>::store(dst, v[u]);
        }
    }
}

NI_EXPORT int ni_rope_kv_write(const void* qkv, int dtype, void* q_out, void* k_pages,
                               void* v_pages, const int* positions, const int* seq_of_token,
                               const int* block_table, int bt_stride, const float* inv_freq,
                               int n_tokens, int n_q_heads, int n_kv_heads, int head_dim,
                               int rotary_dim, int interleaved, int page_size, int write_cache,
                               cudaStream_t stream) {
    if (n_tokens <= 0) return NI_OK;
    if (head_dim <= 0 || head_dim % 2 || rotary_dim < 0 || rotary_dim % 2 || rotary_dim > head_dim ||
        n_q_heads <= 0 || n_kv_heads <= 0 || page_size <= 0)
        return NI_ERR_BAD_ARGUMENT;
    const int chunks = head_dim / 8;
    if (interleaved && head_dim % 8 == 0 && chunks >= 2 && chunks <= 32 && (chunks & (chunks - 1)) == 0) {
        // Groups of heads (a warp's worth of chunks each) per warp: two, over up to eight warps.  Four, where up to four warps then
        // hold them all and the launch has tokens enough to keep the SMs busy with fewer warps, half of which compute the angles:
        // 12 groups x 2,048 tokens 7.7 us with two, 7.4 with four, x 1,024 (heads of 128) 5.5 / 4.8, 8 groups x 2,048 5.8 / 5.4; but 12
        // groups x 512 3.6 / 4.2, x 8 3.0 / 3.8, 3 groups x 2,048 3.8 / 4.3, and 24 groups x 1,914 10.2 / 14.6.  In bfloat16 alone: the
        // two are separate compilations of the rotation, and a float32 token's bits must not depend on the step's size.
        int log_chunks = 0;
        while ((1 << log_chunks) < chunks) ++log_chunks;
        const int groups = ((n_q_heads + 2 * n_kv_heads) * chunks + 31) / 32, halves = (groups + 1) / 2;
        const bool four = dtype == NI_DTYPE_BF16 && groups <= 16 && (long long)n_tokens * halves >= 32LL * ni_sm_count();
        const int warps = four ? (groups + 3) / 4 : halves <= 8 ? halves : 8;
#define LAUNCHL(T, ITEMS)                                                                              \
    rope_kv_write_lanes_kernel<T, ITEMS><<<n_tokens, 32 * warps, 0, stream>>>(                         \
        (const T*)qkv, (T*)q_out, (T*)k_pages, (T*)v_pages, positions, seq_of_token, block_table,      \
        bt_stride, inv_freq, n_q_heads, n_kv_heads, head_dim, log_chunks, rotary_dim, page_size, write_cache)
        if (dtype == NI_DTYPE_F32) LAUNCHL(float, 2);
        else if (dtype == NI_DTYPE_BF16 && four) LAUNCHL(__nv_bfloat16, 4);
        else if (dtype == NI_DTYPE_BF16) LAUNCHL(__nv_bfloat16, 2);
        else return NI_ERR_BAD_ARGUMENT;
#undef LAUNCHL
        NI_RETURN_LAUNCH_STATUS();
    }
    if (interleaved && head_dim % 8 == 0) {
        const int items = (n_q_heads + 2 * n_kv_heads) * (head_dim / 8);
        const int threads = items >= 512 ? 256 : (items >= 256 ? 128 : 64);      // about four chunks per thread
        const int blocks = n_tokens < ni_sm_count() * 16 ? n_tokens : ni_sm_count() * 16;
#define LAUNCHV(T)                                                                                     \
    rope_kv_write_vec_kernel<T><<<blocks, threads, rotary_dim * sizeof(float), stream>>>(               \
        (const T*)qkv, (T*)q_out, (T*)k_pages, (T*)v_pages, positions, seq_of_token, block_table,     \
        bt_stride, inv_freq, n_tokens, n_q_heads, n_kv_heads, head_dim, rotary_dim, page_size, write_cache)
        if (dtype == NI_DTYPE_F32) LAUNCHV(float);
        else if (dtype == NI_DTYPE_BF16) LAUNCHV(__nv_bfloat16);
        else return NI_ERR_BAD_ARGUMENT;
#undef LAUNCHV
        NI_RETURN_LAUNCH_STATUS();
    }
    const int n_pairs = (n_q_heads + 2 * n_kv_heads) * head_dim / 2;
    const int threads = n_pairs >= 1024 ? 256 : 128;
#define LAUNCH(T)                                                                                  \
    rope_kv_write_kernel<T><<<n_tokens, threads, 0, stream>>>(                                     \
        (const T*)qkv, (T*)q_out, (T*)k_pages, (T*)v_pages, positions, seq_of_token, block_table, \
        bt_stride, inv_freq, n_q_heads, n_kv_heads, head_dim, rotary_dim, interleaved, page_size, \
        write_cache)
    if (dtype == NI_DTYPE_F32) LAUNCH(float);
    else if (dtype == NI_DTYPE_BF16) LAUNCH(__nv_bfloat16);
    else return NI_ERR_BAD_ARGUMENT;
#undef LAUNCH
    NI_RETURN_LAUNCH_STATUS();
}
