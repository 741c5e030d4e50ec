// out[M, N] = x[M, K] . w[N, K]^T in true FP32: FFMA on CUDA cores, no tensor-core mode.  The 32-bit path's products over rows of
// fewer than 1,024 columns; longer rows go to gemm_f32_tc.cu.
//
// The reference calls cublasSgemm with the default math mode for every projection
// (src/op/kernels/cuda/matmul_kernel.cu:48-89).  These kernels keep the FP32 path free of
// any library's choice of algorithm: each output element is one chain of fused
// multiply-adds over k = 0 .. K-1 in ascending order, whatever M is and whichever kernel or tile
// takes it, so a token's result does not depend on its batch.  K is therefore never split; what the
// kernels differ in is how many chains a block runs side by side and how the operands reach them.
#include "common.cuh"

__device__ __forceinline__ void gf_copy16(float* dst_smem, const float* src, bool live) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
    const int n = live ? 16 : 0;                                // 0: sixteen bytes of zeros, nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

// ---- many rows: tiles ------------------------------------------------------------------------------------------------
// A block's tile of BM x BN outputs, TM x TN per thread, k in steps of 16 through two buffers in shared memory; the next
// step's operands wait in registers while the current one is multiplied.  Both operands lie k by k, so that a thread reads
// neighbouring rows and columns as 16 bytes; neighbouring columns are the two halves of a packed multiply-add (two independent
// IEEE chains per instruction - the plain one, with three different registers, runs at two thirds of its rate).  Shared
// memory hands out 128 bytes per clock whatever the lanes share, so the thread's tile decides: 8 x 8 reads 16 numbers for 64
// multiply-adds (16 clocks of loads beside 16 of arithmetic per warp and k); 8 x 16 in blocks of 128 x 128 was no faster
// (2,780 against 2,620 us at 2,048 x 16,384 x 2,048: two blocks per SM instead of three).
#define GF_BK 16

template <int BM, int BN, int TM, int TN, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_f32_tile_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ out,
                     int M, int N, int K, int ldx, int ldo) {
    constexpr int THREADS = (BM / TM) * (BN / TN), TX = BN / TN;
    constexpr int PX = BM + 4, PW = BN + 4;                     // row pitches: 16-byte rows, few conflicts between k
    constexpr int QX = BM * GF_BK / 4, QW = BN * GF_BK / 4;     // groups of four k of a step
    constexpr int NX = QX / THREADS, NW = QW / THREADS;
    static_assert(TM % 4 == 0 && TN % 4 == 0 && TX % 8 == 0, "a thread's rows and columns come in fours, a warp is 4 x 8 threads");
    static_assert(QX % THREADS == 0 && QW % THREADS == 0, "every thread fetches the same number of groups");
    __shared__ __align__(16) float xs[2][GF_BK][PX];
    __shared__ __align__(16) float ws[2][GF_BK][PW];
    // one product per blockIdx.z (a head): its activations are columns [z K, (z+1) K) of x, its
    // matrix is w[z], its results are columns [z N, (z+1) N) of out
    x += (size_t)blockIdx.z * K;
    w += (size_t)blockIdx.z * N * K;
    out += (size_t)blockIdx.z * N;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = (warp % (TX / 8)) * 8 + (lane & 7), ty = (warp / (TX / 8)) * 4 + (lane >> 3);
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float4 xr[NX], wr[NW];

    auto fetch4 = [&](const float* row, bool live, int k) -> float4 {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (VEC) {
            if (live && k < K) v = *reinterpret_cast<const float4*>(row + k);
        } else if (live) {
            if (k < K) v.x = row[k];
            if (k + 1 < K) v.y = row[k + 1];
            if (k + 2 < K) v.z = row[k + 2];
            if (k + 3 < K) v.w = row[k + 3];
        }
        return v;
    };
    auto fetch = [&](int k0) {
#pragma unroll
        for (int e = 0; e < NX; ++e) {
            const int q = tid + e * THREADS, r = q >> 2;
            xr[e] = fetch4(x + (size_t)(m0 + r) * ldx, m0 + r < M, k0 + 4 * (q & 3));
        }
#pragma unroll
        for (int e = 0; e < NW; ++e) {
            const int q = tid + e * THREADS, r = q >> 2;
            wr[e] = fetch4(w + (size_t)(n0 + r) * K, n0 + r < N, k0 + 4 * (q & 3));
        }
    };
    auto keep = [&](int buf) {
#pragma unroll
        for (int e = 0; e < NX; ++e) {
            const int q = tid + e * THREADS, r = q >> 2, k = 4 * (q & 3);
            xs[buf][k][r] = xr[e].x; xs[buf][k + 1][r] = xr[e].y; xs[buf][k + 2][r] = xr[e].z; xs[buf][k + 3][r] = xr[e].w;
        }
#pragma unroll
        for (int e = 0; e < NW; ++e) {
            const int q = tid + e * THREADS, r = q >> 2, k = 4 * (q & 3);
            ws[buf][k][r] = wr[e].x; ws[buf][k + 1][r] = wr[e].y; ws[buf][k + 2][r] = wr[e].z; ws[buf][k + 3][r] = wr[e].w;
        }
    };

    unsigned long long acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;      // two zeros

    fetch(0);
    keep(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += GF_BK) {
        const bool more = k0 + GF_BK < K;
        if (more) fetch(k0 + GF_BK);
#pragma unroll
        for (int kk = 0; kk < GF_BK; ++kk) {
            float a[TM];
            unsigned long long b[TN / 2];
#pragma unroll
            for (int g = 0; g < TM / 4; ++g) {
                const float4 u = *reinterpret_cast<const float4*>(&xs[buf][kk][4 * ty + g * (BM / (TM / 4))]);
                a[4 * g] = u.x; a[4 * g + 1] = u.y; a[4 * g + 2] = u.z; a[4 * g + 3] = u.w;
            }
#pragma unroll
            for (int g = 0; g < TN / 4; ++g) {
                const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(&ws[buf][kk][4 * tx + g * (BN / (TN / 4))]);
                b[2 * g] = u.x; b[2 * g + 1] = u.y;
            }
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                unsigned long long aa;
                asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "f"(a[i]));
#pragma unroll
                for (int j = 0; j < TN / 2; ++j)
                    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(aa), "l"(b[j]));
            }
        }
        if (more) {
            keep(buf ^ 1);                                      // its readers passed the barrier of the step before
            __syncthreads();
            buf ^= 1;
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + 4 * ty + (i & 3) + (i >> 2) * (BM / (TM / 4));
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) {
            const int n = n0 + 4 * tx + 2 * (j & 1) + (j >> 1) * (BN / (TN / 4));
            const float2 v = *reinterpret_cast<const float2*>(&acc[i][j]);
            if (n < N) out[(size_t)m * ldo + n] = v.x;
            if (n + 1 < N) out[(size_t)m * ldo + n + 1] = v.y;
        }
    }
}

// ---- few rows: a warp per tile, fed by a second one ------------------------------------------------------------------
// A block of two warps: one fetches rows of w and x, KC columns at a time, through a ring of STAGES stages (asynchronous
// copies), the other multiplies, LN x (32 / LN) lanes with TN x TM outputs each.  Few rows mean few chains, so what bounds
// the block is the latency of its own chain (4 clocks per k) or, with many weight rows, memory: the multiplying warp must do
// nothing else, and several such blocks share an SM so that 60 KB or more of weights are on their way.  2 rows: [2048, 8192]
// 25 us (the chain alone: 17), [16384, 2048] 32 us (memory alone: 20.5); one warp doing both: 40 and 33 us.  The hand-overs are
// the block's named barriers (stage s: "full" 1 + s, "empty" 1 + STAGES + s), which wait in hardware.
__device__ __forceinline__ void gr_sync(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void gr_arrive(int id) { asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory"); }

template <int LN, int TN, int TM, int KC, int STAGES, int U>
__global__ void __launch_bounds__(64)
gemm_f32_ring_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ out,
                     int M, int N, int K, int ldx, int ldo) {
    constexpr int LM = 32 / LN, BN = LN * TN, BM = LM * TM, ROWS = BN + BM;
    constexpr int PITCH = KC + 4, STAGE = ROWS * PITCH;         // 16-byte rows; eight rows side by side lie in different bank groups
    constexpr int GROUPS = KC / 4, STEP = 32 / GROUPS;          // 16-byte groups of a row; rows that a warp copies at once
    static_assert(2 * STAGES + 1 <= 16 && GROUPS <= 32 && BN % STEP == 0 && BM % STEP == 0 && KC % (8 * U) == 0, "ring");
    extern __shared__ __align__(16) float gf_smem[];
    x += (size_t)blockIdx.z * K;
    w += (size_t)blockIdx.z * N * K;
    out += (size_t)blockIdx.z * N;
    const int lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
    const int chunks = (K + KC - 1) / KC;
    // Blocks of two warps fill an SM's warp slots, and with them its four schedulers, as 0 1, 2 3, 0 1, 2 3.  A block in slots 4
    // to 7 (8 to 11 as 0 to 3, and so on) lets its other warp multiply, so that four blocks multiply on four schedulers instead
    // of two: 177 rows x [2048, 8192] 346 -> 263 us, 16 rows x [16384, 2048] 67 -> 54 us.  (Which warp it is changes no result;
    // the slot is only read to spread the work.)
    __shared__ unsigned gr_slot;
    if (threadIdx.x == 0) asm volatile("mov.u32 %0, %%warpid;" : "=r"(gr_slot));
    __syncthreads();
    const int multiplier = (gr_slot >> 2) & 1;
    if ((int)(threadIdx.x >> 5) != multiplier) {                // the fetching warp
        const int row = lane / GROUPS, col = 4 * (lane % GROUPS);
        const bool whole = n0 + BN <= N && m0 + BM <= M;        // every row of the tile exists
        const float* wp = w + (size_t)(n0 + row) * K + col;
        const float* xp = x + (size_t)(m0 + row) * ldx + col;
        for (int c = 0; c < chunks + STAGES - 1; ++c, wp += KC, xp += KC) {
            // what has arrived is handed over before this warp waits for a stage to be left: the other one goes on meanwhile
            if (c >= STAGES - 1) {
                asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
                gr_arrive(1 + (c - (STAGES - 1)) % STAGES);     // chunk c - (STAGES - 1) is there
            }
            if (c < chunks) {
                const int s = c % STAGES;
                if (c >= STAGES) gr_sync(1 + STAGES + s);       // the stage has been read
                float* st = gf_smem + s * STAGE + row * PITCH + col;
                if (whole && (c + 1) * KC <= K) {
#pragma unroll
                    for (int i = 0; i < BN; i += STEP) gf_copy16(st + i * PITCH, wp + (size_t)i * K, true);
#pragma unroll
                    for (int i = 0; i < BM; i += STEP) gf_copy16(st + (BN + i) * PITCH, xp + (size_t)i * ldx, true);
                } else {
                    const bool in_k = c * KC + col < K;
                    for (int i = 0; i < BN; i += STEP) {
                        const bool live = in_k && n0 + row + i < N;
                        gf_copy16(st + i * PITCH, live ? wp + (size_t)i * K : w, live);
                    }
                    for (int i = 0; i < BM; i += STEP) {
                        const bool live = in_k && m0 + row + i < M;
                        gf_copy16(st + (BN + i) * PITCH, live ? xp + (size_t)i * ldx : x, live);
                    }
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");            // one group per turn, empty or not
        }
        return;
    }
    const int ln = lane % LN, lm = lane / LN;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
    for (int c = 0; c < chunks; ++c) {
        const int s = c % STAGES;
        gr_sync(1 + s);
        const float* wr = gf_smem + s * STAGE + ln * PITCH;
        const float* xr = gf_smem + s * STAGE + (BN + lm) * PITCH;
        // the numbers of the next U groups of four k are asked for before the current ones are multiplied: a chain must not
        // wait for shared memory
        float4 b[2][U][TN], a[2][U][TM];
        auto load = [&](int half, int k) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
#pragma unroll
                for (int j = 0; j < TN; ++j) b[half][u][j] = *reinterpret_cast<const float4*>(wr + j * LN * PITCH + k + 4 * u);
#pragma unroll
                for (int i = 0; i < TM; ++i) a[half][u][i] = *reinterpret_cast<const float4*>(xr + i * LM * PITCH + k + 4 * u);
            }
        };
        auto multiply = [&](int half) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[half][u][i].x, b[half][u][j].x, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[half][u][i].y, b[half][u][j].y, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[half][u][i].z, b[half][u][j].z, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[half][u][i].w, b[half][u][j].w, acc[i][j]);
            }
        };
        load(0, 0);
#pragma unroll
        for (int k = 0; k < KC; k += 8 * U) {
            load(1, k + 4 * U);
            multiply(0);
            if (k + 8 * U < KC) load(0, k + 8 * U);
            multiply(1);
        }
        if (c + STAGES < chunks) gr_arrive(1 + STAGES + s);     // as many arrivals as the fetching warp waits for
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + lm + i * LM;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + ln + j * LN;
            if (m < M && n < N) out[(size_t)m * ldo + n] = acc[i][j];
        }
    }
}

// ---- choice and launch -----------------------------------------------------------------------------------------------
enum { GF_AUTO = 0, GF_RING_2 = 1, GF_RING_4 = 2, GF_RING_8 = 3, GF_RING_16 = 4, GF_RING_32x16 = 5, GF_TILE = 6, GF_VARIANTS = 7 };

template <int BM, int BN, int TM, int TN>
static int gf_launch_tile(const float* x, const float* w, float* out, int M, int N, int K, int ldx, int ldo, int H, bool vec,
                          cudaStream_t stream) {
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, H);
    if (grid.y > 65535 || H > 65535) return NI_ERR_UNSUPPORTED_SIZE;
    auto kernel = vec ? gemm_f32_tile_kernel<BM, BN, TM, TN, true> : gemm_f32_tile_kernel<BM, BN, TM, TN, false>;
    kernel<<<grid, (BM / TM) * (BN / TN), 0, stream>>>(x, w, out, M, N, K, ldx, ldo);
    NI_RETURN_LAUNCH_STATUS();
}

template <int LN, int TN, int TM, int KC, int STAGES, int U>
static int gf_launch_ring(const float* x, const float* w, float* out, int M, int N, int K, int ldx, int ldo, int H,
                          cudaStream_t stream) {
    constexpr int BN = LN * TN, BM = 32 / LN * TM, SMEM = STAGES * (BN + BM) * (KC + 4) * (int)sizeof(float);
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, H);
    if (grid.y > 65535 || H > 65535) return NI_ERR_UNSUPPORTED_SIZE;
    auto kernel = gemm_f32_ring_kernel<LN, TN, TM, KC, STAGES, U>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return (int)e;
    kernel<<<grid, 64, SMEM, stream>>>(x, w, out, M, N, K, ldx, ldo);
    NI_RETURN_LAUNCH_STATUS();
}

// Up to 16 rows the narrowest ring that holds them all: weights are read once.  Beyond, the ring's 32 x 16 tiles (three
// blocks per SM) or the 64 x 128 tiles, whichever is done first by what they measured at K = 2,048 (both go with K, which
// is below 1,024 in the 32-bit path itself):
// a ring tile takes 34 us alone and 0.077 us each once the SMs are full, a 64 x 128 tile 128 us and 0.64 us.  [2048, K]
// weights: 64 rows 37 / 130 us, 177 rows 74 / 130 us, 256 rows 99 / 130 us, 512 rows 200 / 130 us; [16384, K]: 17 rows
// 103 / 130 us, 64 rows 170 / 132 us.  Before (64 x 64 tiles of 4 x 4 outputs per thread, one k-step of 16 at a time): 190 us and
// up for any few rows, [16384, K] at 2,048 rows 5,863 us against 2,620 us (0.70 of the FMA rate).
static int gf_choose(int M, int N, int H, bool vec) {
    if (!vec) return GF_TILE;
    if (M <= 16) return M <= 2 ? GF_RING_2 : M <= 4 ? GF_RING_4 : M <= 8 ? GF_RING_8 : GF_RING_16;
    const double fill = 148.0 / ni_sm_count();
    const double ring = (double)((N + 31) / 32) * ((M + 15) / 16) * H * fill, tile = (double)((N + 127) / 128) * ((M + 63) / 64) * H * fill;
    const double ring_us = 14.0 + 0.077 * ring, tile_us = 50.0 + 0.64 * tile;
    if ((M + 15) / 16 > 65535) return GF_TILE;                  // more row tiles of 16 than a grid has room for
    return (ring_us > 34.0 ? ring_us : 34.0) <= (tile_us > 128.0 ? tile_us : 128.0) ? GF_RING_32x16 : GF_TILE;
}

static int gf_run(int variant, const float* x, const float* w, float* out, int M, int N, int K, int ldx, int ldo, int H,
                  cudaStream_t stream) {
    // 16-byte loads of both operands: whole groups of four k, rows on 16 bytes
    const bool vec = K % 4 == 0 && ldx % 4 == 0 && ((uintptr_t)x | (uintptr_t)w) % 16 == 0;
    if (variant == GF_AUTO) variant = gf_choose(M, N, H, vec);
    if (!vec && variant != GF_TILE) return NI_ERR_BAD_ARGUMENT;
    switch (variant) {
        case GF_RING_2: return gf_launch_ring<16, 1, 1, 128, 6, 4>(x, w, out, M, N, K, ldx, ldo, H, stream);
        case GF_RING_4: return gf_launch_ring<16, 1, 2, 128, 5, 4>(x, w, out, M, N, K, ldx, ldo, H, stream);
        case GF_RING_8: return gf_launch_ring<8, 2, 2, 128, 5, 2>(x, w, out, M, N, K, ldx, ldo, H, stream);
        case GF_RING_16: return gf_launch_ring<8, 2, 4, 64, 6, 2>(x, w, out, M, N, K, ldx, ldo, H, stream);
        case GF_RING_32x16: return gf_launch_ring<8, 4, 4, 64, 5, 1>(x, w, out, M, N, K, ldx, ldo, H, stream);
        case GF_TILE: return gf_launch_tile<64, 128, 8, 8>(x, w, out, M, N, K, ldx, ldo, H, vec, stream);
    }
    return NI_ERR_BAD_ARGUMENT;
}

NI_EXPORT int ni_gemm_f32(const float* x, const float* w, float* out, int M, int N, int K,
                          cudaStream_t stream) {
    if (M <= 0 || N <= 0) return NI_OK;
    if (K <= 0) return NI_ERR_BAD_ARGUMENT;
    return gf_run(GF_AUTO, x, w, out, M, N, K, K, N, 1, stream);
}

// The same product by a named kernel (one of the numbers above): all of them give the same bits.
NI_EXPORT int ni_gemm_f32_variant(int variant, const float* x, const float* w, float* out, int M, int N, int K,
                                  cudaStream_t stream) {
    if (M <= 0 || N <= 0) return NI_OK;
    if (K <= 0 || variant < 0 || variant >= GF_VARIANTS) return NI_ERR_BAD_ARGUMENT;
    return gf_run(variant, x, w, out, M, N, K, K, N, 1, stream);
}

// One product per head: out[m, h, :] = x[m, h, :] . w[h]^T with x [M, H, K] (rows ldx floats apart: it may
// be some columns of a wider matrix), w [H, N, K], out [M, H, N], each output element the same ascending
// chain of fused multiply-adds as above.
NI_EXPORT int ni_gemm_f32_heads(const float* x, int ldx, const float* w, float* out, int M, int N, int K, int H,
                                cudaStream_t stream) {
    if (M <= 0 || N <= 0 || H <= 0) return NI_OK;
    if (K <= 0) return NI_ERR_BAD_ARGUMENT;
    if (ldx < H * K) return NI_ERR_BAD_ARGUMENT;
    return gf_run(GF_AUTO, x, w, out, M, N, K, ldx, H * N, H, stream);
}
