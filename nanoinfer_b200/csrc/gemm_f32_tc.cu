// out[M, N] = x[M, K] . w[N, K]^T of FP32 matrices with long rows on the fifth-generation tensor cores, with errors smaller than
// those of a chain of FP32 multiply-adds.  Every FP32 number is cut in two: its upper 11 bits of mantissa (what the tensor core's
// tf32 keeps of an operand) and what is left (13 bits, of which it keeps 11 again):
//
//     x w = xh wh + (xh wl + xl wh)  [+ xl wl, 2^-22 of x w and left out; xh is rounded, wh cut, so its mean is zero]
//
// The tensor core adds into its FP32 accumulator by cutting, a bias that grows with the number of additions (-1.3e-7 after 32
// columns, -2.9e-7 after 64).  So the accumulator of the large products (xh wh) is emptied every 64 columns into registers, where it
// is added with rounding to nearest, and the small ones, 2^-11 of the large, have an accumulator of their own that is emptied every
// 256:
//     slice s of 256:  sum_s = (((hh_0 + hh_1) + hh_2) + hh_3) + small          result = (sum_0 + sum_1) + ...
// This order is the same for every tile size, number of rows and split of K, so an element's bits depend on its two rows alone.
// Relative error against 64 bits, normal (positive) numbers: 3.0e-7 (3.7e-7) at 1,024 columns where the chain has 5.7e-7 (4.9e-7),
// 3.1e-7 (3.6e-7) at 8,192 where it has 1.6e-6 (1.3e-6).
//
// What bounds it: at many rows the cutting and the MMAs' reads of shared memory (2,048 x 16,384 weights and 1,087 rows: 418 us, 175
// TFLOP/s; chains on CUDA cores 1,417); at few the weights, [128256, 2048] 174 us (6.0 TB/s; the ring of chains 177, at 8 rows 239),
// and for small matrices the way of one block: 6 us of start, first load and last sum, 0.65 us for 64 columns ([2048, 2048] 12.4 us
// alone, less behind a kernel that lets it start early).
//
// The 128 lanes of the tcgen05 tile are weight rows, its columns BT rows of x (16 .. 128): few rows read the weights once, at
// many rows 128 x 128 tiles.  Blocks are persistent; a block's warps:
//   0 - ..  cut: GROUPS groups take turns at the stages of 32 columns that TMA has filled: the numbers stay where they are (the
//           tensor core ignores the bits that it does not keep), what is left goes beside them.  Those of x lie so that xh and
//           xl, or xl and xh, are 2 BT rows of one operand
//   then    empty the accumulators, 4 or 8 warps
//   last    two: the MMAs, and TMA
// A product with few weight rows cuts the slices of K over the blocks of a cluster; their sums go to the block that owns the row
// of x (through its shared memory, once all MMAs are done) and are added there in the order of the slices.
//
// An element that is not finite is computed once more as one chain of fused multiply-adds: inf - inf among the parts of an
// infinite operand, or an overflow that only the order of these sums has, does not show.
#include <cuda.h>

#include <mutex>

#include "common.cuh"

#define GT_ROWS 128            // weight rows of a tile
#define GT_HALF 32             // columns of a box in shared memory: 128 bytes
#define GT_BK 64               // k-block: what the accumulator of large products adds up
#define GT_SLICE 4             // k-blocks of a slice
#define GT_ERR_LOAD 51
#define GT_ERR_CUT 52
#define GT_ERR_MMA 53
#define GT_ERR_SUMS 54

// RAW stages of SUB boxes of 32 columns as they are loaded, STAGES of cut ones (PLACE: the same stages, the rests beside the numbers);
// GROUPS of GROUP cutting warps; ACC warps that empty accumulators; COLS of tensor memory (3 BT for the accumulators, the rest for
// sums of slices)
template <int BT> struct GtCfg;
template <> struct GtCfg<16> { static constexpr int RAW = 4, STAGES = 2, SUB = 2, GROUPS = 2, GROUP = 8, ACC = 4, COLS = 256; static constexpr bool PLACE = false; };
template <> struct GtCfg<32> { static constexpr int RAW = 3, STAGES = 2, SUB = 2, GROUPS = 2, GROUP = 8, ACC = 4, COLS = 512; static constexpr bool PLACE = false; };
template <> struct GtCfg<64> { static constexpr int RAW = 4, STAGES = 4, SUB = 1, GROUPS = 4, GROUP = 2, ACC = 8, COLS = 512; static constexpr bool PLACE = true; };
template <> struct GtCfg<128> { static constexpr int RAW = 3, STAGES = 3, SUB = 1, GROUPS = 3, GROUP = 4, ACC = 16, COLS = 512; static constexpr bool PLACE = true; };
template <int BT> struct GtSizes {
    using C = GtCfg<BT>;
    static constexpr int A = GT_ROWS * 128, B = BT * 128;                            // bytes of a box of weights and of x
    // A loaded stage: weights, x.  A cut one: rests of the weights, per box of x numbers and rests.  In place: weights, their rests,
    // per box of x room for both.
    static constexpr int RAW_STAGE = C::SUB * (C::PLACE ? 2 * A + 2 * B : A + B), STAGE = C::SUB * (C::PLACE ? 2 * A + 2 * B : A + 2 * B);
    static constexpr int RAW_X = C::SUB * (C::PLACE ? 2 * A : A), REST_A = C::PLACE ? C::SUB * A : 0, CUT_X = C::SUB * (C::PLACE ? 2 * A : A);
    static constexpr int CUT_RING = C::PLACE ? 0 : C::RAW * RAW_STAGE;               // where the stages of cut numbers begin
    static constexpr int RING = C::RAW * RAW_STAGE + (C::PLACE ? 0 : C::STAGES * STAGE), SMEM = 1024 + RING + 256;
    static constexpr int REGIONS = C::COLS / BT - 3;                                 // sums of slices that a block can keep
    static constexpr int CUT = C::GROUPS * C::GROUP, THREADS = (CUT + C::ACC + 2) * 32;
    static_assert(C::GROUPS <= C::STAGES && C::RAW >= C::STAGES && (!C::PLACE || C::RAW == C::STAGES), "see the cutting warps' waits");
    static_assert(SMEM <= 232448, "shared memory");
};

__device__ __forceinline__ uint32_t gt_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void gt_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(gt_smem(bar)), "r"(count));
}
__device__ __forceinline__ void gt_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(gt_smem(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void gt_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(gt_smem(bar)) : "memory");
}
// How long a wait may last, in clock ticks (about a second), and a switch for the tests: with it the emptying warps wait once
// more at the end for a phase that nothing completes.  Set by ni_gemm_f32_tc_set_wait.
__constant__ long long gt_wait_limit = 2000000000LL;
__constant__ int gt_extra_wait = 0;

__device__ __forceinline__ bool gt_wait(uint64_t* bar, uint32_t parity, int* error, int code) {
    const uint32_t addr = gt_smem(bar);
    long long start = 0;
    for (int iter = 0;; ++iter) {
        uint32_t done;
        asm volatile(
            "{\n.reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.b32 %0, 1, 0, p;\n}\n"
            : "=r"(done) : "r"(addr), "r"(parity) : "memory");
        if (done) return true;
        if ((iter & 1023) == 1023) {
            const long long now = clock64();
            if (start == 0) start = now;
            if (now - start > gt_wait_limit) {
                atomicExch(error, code);
                return false;
            }
        }
    }
}
// Whether three phases have ended, asked for at once (the answers take about 100 clocks each).
__device__ __forceinline__ bool gt_ended(uint64_t* a, uint32_t pa, uint64_t* b, uint32_t pb, uint64_t* c, uint32_t pc) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p, q, r;\n"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "mbarrier.test_wait.parity.shared::cta.b64 q, [%3], %4;\n"
        "mbarrier.test_wait.parity.shared::cta.b64 r, [%5], %6;\n"
        "and.pred p, p, q;\n"
        "and.pred p, p, r;\n"
        "selp.b32 %0, 1, 0, p;\n}\n"
        : "=r"(done) : "r"(gt_smem(a)), "r"(pa), "r"(gt_smem(b)), "r"(pb), "r"(gt_smem(c)), "r"(pc) : "memory");
    return done != 0;
}
__device__ __forceinline__ void gt_tma_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n"
        ::"r"(gt_smem(dst)), "l"(map), "r"(gt_smem(bar)), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void gt_tma_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n"
        ::"r"(gt_smem(dst)), "l"(map), "r"(gt_smem(bar)), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void gt_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void gt_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ uint64_t gt_desc(const void* tile) {   // K-major, 128-byte swizzle, 8-row groups 1024 bytes apart
    const uint32_t addr = gt_smem(tile);
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
__host__ __device__ constexpr uint32_t gt_idesc(int n) {          // TF32 x TF32 -> FP32, M = 128, N = n
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(GT_ROWS >> 4) << 24);
}
__device__ __forceinline__ void gt_mma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void gt_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
                 ::"r"(gt_smem(bar)) : "memory");
}
__device__ __forceinline__ void gt_ld16(uint32_t taddr, uint32_t r[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void gt_st16(uint32_t taddr, const float* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};\n"
        ::"f"(r[0]), "f"(r[1]), "f"(r[2]), "f"(r[3]), "f"(r[4]), "f"(r[5]), "f"(r[6]), "f"(r[7]),
          "f"(r[8]), "f"(r[9]), "f"(r[10]), "f"(r[11]), "f"(r[12]), "f"(r[13]), "f"(r[14]), "f"(r[15]), "r"(taddr) : "memory");
}
__device__ __forceinline__ void gt_pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void gt_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void gt_st_cluster(const float* mine, uint32_t rank, float v) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(gt_smem(mine)), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;\n" ::"r"(remote), "f"(v) : "memory");
}

// Pairs of numbers, for packed arithmetic.
typedef unsigned long long GtPair;
__device__ __forceinline__ GtPair gt_pair(float a, float b) {
    GtPair r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ GtPair gt_fma(GtPair a, GtPair b, GtPair c) {
    GtPair r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ GtPair gt_sub(GtPair a, GtPair b) { return gt_fma(b, gt_pair(-1.f, -1.f), a); }
// Rounded to 11 bits of mantissa by Veltkamp's splitting (the larger part of v's two): t = (2^13 + 1) v, t - (t - v).  What is not
// finite, or overflows in t, ends as NaN.
__device__ __forceinline__ GtPair gt_rounded(GtPair v) {
    const GtPair t = gt_fma(v, gt_pair(8192.f, 8192.f), v);
    return gt_sub(t, gt_sub(t, v));
}
// What the tensor core does not keep of two numbers, where it cuts them.
__device__ __forceinline__ GtPair gt_rest_of_cut(float a, float b) {
    const float ca = __uint_as_float(__float_as_uint(a) & 0xffffe000u), cb = __uint_as_float(__float_as_uint(b) & 0xffffe000u);
    return gt_sub(gt_pair(a, b), gt_pair(ca, cb));
}
// Four columns of a row in global memory, one by one (zeros beyond K): rows that TMA does not take.
__device__ __forceinline__ float4 gt_load4(const float* __restrict__ p, int k, int K, bool live) {
    float4 v;
    v.x = live && k < K ? p[k] : 0.f;
    v.y = live && k + 1 < K ? p[k + 1] : 0.f;
    v.z = live && k + 2 < K ? p[k + 2] : 0.f;
    v.w = live && k + 3 < K ? p[k + 3] : 0.f;
    return v;
}

// A sum that is not finite, as one chain (NaN stays NaN, so the chain may end there).
__device__ __forceinline__ float gt_chain(const float* __restrict__ x, const float* __restrict__ w, int K) {
    float a = 0.f;
    for (int k = 0; k < K && a == a; ++k) a = fmaf(x[k], w[k], a);
    return a;
}
__device__ __forceinline__ bool gt_finite(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }

struct GtParams {
    const float* x;
    const float* w;
    float* out;
    int M, N, K, H, ldx, ldo, splits;
    int* error;
};

// A unit of work: 128 weight rows and BT rows of x of one head (rows of x vary fastest: the blocks at work read few weights at a
// time), or a block's slices of it.
template <int BT> struct GtUnit {
    int n0, m0, head;
    __device__ __forceinline__ GtUnit(const GtParams& p, int unit) {
        const int m_tiles = (p.M + BT - 1) / BT, n_tiles = (p.N + GT_ROWS - 1) / GT_ROWS, nz = unit / m_tiles;
        m0 = (unit - nz * m_tiles) * BT;
        head = nz / n_tiles;
        n0 = (nz - head * n_tiles) * GT_ROWS;
    }
};

// TMA: rows on 16 bytes, whole groups of four columns; otherwise the cutting warps read global memory number by number.
template <int BT, bool TMA>
__global__ void __launch_bounds__(GtSizes<BT>::THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const GtParams p) {
    using S = GtSizes<BT>;
    constexpr int RAW = GtCfg<BT>::RAW, STAGES = GtCfg<BT>::STAGES, GROUPS = GtCfg<BT>::GROUPS, ACC = GtCfg<BT>::ACC;
    constexpr int SUB = GtCfg<BT>::SUB, P = GT_BK / GT_HALF / SUB;                           // stages of a k-block
    constexpr int CPT = BT * 4 / ACC;                                                        // columns of an emptying thread
    extern __shared__ uint8_t gt_smem_raw[];
    uint8_t* ring = reinterpret_cast<uint8_t*>(((uintptr_t)gt_smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* loaded = reinterpret_cast<uint64_t*>(ring + S::RING);
    uint64_t* full = loaded + RAW;
    uint64_t* empty = full + STAGES;
    uint64_t* raw_empty = GtCfg<BT>::PLACE ? empty : empty + STAGES;
    uint64_t* hh_full = raw_empty + RAW;
    uint64_t* hh_empty = hh_full + 2;
    uint64_t* small_empty = hh_empty + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(small_empty + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int splits = p.splits, K = p.K, rank = blockIdx.x % splits;
    const int k_blocks = (K + GT_BK - 1) / GT_BK, slices = (k_blocks + GT_SLICE - 1) / GT_SLICE;
    const int s0 = slices * rank / splits, s1 = slices * (rank + 1) / splits;                // this block's slices
    const int b0 = s0 * GT_SLICE, b1 = s1 * GT_SLICE < k_blocks ? s1 * GT_SLICE : k_blocks;  // and their k-blocks
    const int n_units = ((p.M + BT - 1) / BT) * ((p.N + GT_ROWS - 1) / GT_ROWS) * p.H;
    const int unit0 = blockIdx.x / splits, step = gridDim.x / splits;                        // (split: one unit per cluster)

    const int steps = (b1 - b0) * P;                                                         // stages of a unit
    auto tma_load = [&](int i, int n0, int m0, int head, int k, bool weights, bool x) {
        const int rs = i % RAW, buf = i / P & 1;
        uint8_t* a = ring + rs * S::RAW_STAGE;
        uint8_t* b = a + S::RAW_X + (GtCfg<BT>::PLACE && buf ? S::B : 0);
        if (weights) gt_expect_tx(&loaded[rs], SUB * (S::A + S::B));
#pragma unroll
        for (int h = 0; h < SUB; ++h) {                             // (a box beyond K is zeros)
            if (weights) gt_tma_2d(a + h * S::A, &map_w, k + h * GT_HALF, head * p.N + n0, &loaded[rs]);
            if (x) gt_tma_3d(b + (GtCfg<BT>::PLACE ? 2 : 1) * h * S::B, &map_x, k + h * GT_HALF, head, m0, &loaded[rs]);
        }
    };
    const int ahead = !TMA || unit0 >= n_units ? 0 : steps < RAW ? steps : RAW;              // stages asked for at once
    if (threadIdx.x == (S::CUT + ACC + 1) * 32) {
        for (int s = 0; s < STAGES; ++s) { gt_init(&full[s], GtCfg<BT>::GROUP); gt_init(&empty[s], 1); }
        for (int s = 0; s < RAW; ++s) { gt_init(&loaded[s], 1); if (!GtCfg<BT>::PLACE) gt_init(&raw_empty[s], 1); }
        for (int a = 0; a < 2; ++a) { gt_init(&hh_full[a], 1); gt_init(&hh_empty[a], ACC); }
        gt_init(small_empty, ACC);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        // The first weights are asked for before the kernel in front has ended, and before the block is set up: they depend on
        // nothing.
        const GtUnit<BT> u(p, unit0);
        for (int j = 0; j < ahead; ++j) tma_load(j, u.n0, u.m0, u.head, b0 * GT_BK + j * SUB * GT_HALF, true, false);
    }
    if (warp == S::CUT + ACC) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n"
                     ::"r"(gt_smem(tmem_slot)), "r"(GtCfg<BT>::COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    gt_fence_before();
    __syncthreads();
    gt_fence_after();
    const uint32_t tmem = *tmem_slot;
    gt_pdl_wait();                                                  // x is there, and nobody reads what out was

    if (warp < S::CUT) {
        // ---- cut: stage number i of this block is group i % GROUPS's.  A thread takes 16 bytes wherever they lie in the swizzle;
        // only numbers from global memory need their row and columns ----
        constexpr int T = 32 * GtCfg<BT>::GROUP, AU = S::A / 16 / T, BU = (S::B / 16 + T - 1) / T;
        constexpr int AB = AU < 8 ? AU : 8, BB = BU < 8 ? BU : 8;                   // 16-byte pieces read before the first is written
        static_assert(AU % AB == 0 && BU % BB == 0, "whole batches");
        static_assert(S::B / 16 < T || S::B / 16 % T == 0, "a thread has the same pieces of x as the others, or one or none");
        const int group = warp / GtCfg<BT>::GROUP, t = threadIdx.x % T;
        int first = 0;                                             // number of the unit's first stage
        bool ok = true;
        for (int unit = unit0; unit < n_units && ok; unit += step, first += steps) {
            const GtUnit<BT> u(p, unit);
            for (int i = first + (group + GROUPS - first % GROUPS) % GROUPS; i < first + steps; i += GROUPS) {
                const int rs = i % RAW, stage = i % STAGES, buf = i / P & 1;
                // (In this order: MMAs end in order, so every stage up to i - STAGES has been cut, and the loaded stage cannot be
                // waiting for number i - RAW still, whose phase has the other parity.)
                ok = gt_wait(&empty[stage], ((i / STAGES) & 1) ^ 1, p.error, GT_ERR_CUT);
                ok = ok && gt_wait(TMA ? &loaded[rs] : &raw_empty[rs], (i / RAW & 1) ^ (TMA ? 0 : 1), p.error, GT_ERR_CUT);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
#pragma unroll
                for (int h = 0; h < SUB; ++h) {
                    uint8_t* a = ring + rs * S::RAW_STAGE + h * S::A + 16 * t;
                    uint8_t* a_rest = ring + S::CUT_RING + stage * S::STAGE + S::REST_A + h * S::A + 16 * t;
                    const uint8_t* x = ring + rs * S::RAW_STAGE + S::RAW_X + (GtCfg<BT>::PLACE ? 2 * h * S::B + (buf ? S::B : 0) : h * S::B) + 16 * t;
                    uint8_t* b = ring + S::CUT_RING + stage * S::STAGE + S::CUT_X + 2 * h * S::B + 16 * t;
                    uint8_t* b_rest = b + (buf ? 0 : S::B);
                    b += buf ? S::B : 0;                           // (x before its rests, or behind them)
                    auto load = [&](const float* base, int ld, int rows, int at) -> float4 {
                        const int row = at >> 3, k = b0 * GT_BK + ((i - first) * SUB + h) * GT_HALF + 4 * ((at & 7) ^ (row & 7));
                        return gt_load4(base + (size_t)row * ld, k, K, row < rows);
                    };
#pragma unroll
                    for (int j0 = 0; j0 < AU; j0 += AB) {
                        float4 v[AB];
#pragma unroll
                        for (int j = 0; j < AB; ++j)
                            if (TMA) v[j] = *reinterpret_cast<const float4*>(a + (j0 + j) * 16 * T);
                            else v[j] = load(p.w + ((size_t)u.head * p.N + u.n0) * K, K, p.N - u.n0, t + (j0 + j) * T);
#pragma unroll
                        for (int j = 0; j < AB; ++j) {
                            if (!TMA) *reinterpret_cast<float4*>(a + (j0 + j) * 16 * T) = v[j];
                            *reinterpret_cast<ulonglong2*>(a_rest + (j0 + j) * 16 * T) =
                                make_ulonglong2(gt_rest_of_cut(v[j].x, v[j].y), gt_rest_of_cut(v[j].z, v[j].w));
                        }
                    }
                    if (S::B / 16 >= T || t < S::B / 16) {
#pragma unroll
                        for (int j0 = 0; j0 < BU; j0 += BB) {
                            float4 v[BB];
#pragma unroll
                            for (int j = 0; j < BB; ++j)
                                if (TMA) v[j] = *reinterpret_cast<const float4*>(x + (j0 + j) * 16 * T);
                                else v[j] = load(p.x + (size_t)u.head * K + (size_t)u.m0 * p.ldx, p.ldx, p.M - u.m0, t + (j0 + j) * T);
#pragma unroll
                            for (int j = 0; j < BB; ++j) {
                                const GtPair v0 = gt_pair(v[j].x, v[j].y), v1 = gt_pair(v[j].z, v[j].w);
                                const GtPair h0 = gt_rounded(v0), h1 = gt_rounded(v1);
                                *reinterpret_cast<ulonglong2*>(b + (j0 + j) * 16 * T) = make_ulonglong2(h0, h1);
                                *reinterpret_cast<ulonglong2*>(b_rest + (j0 + j) * 16 * T) =
                                    make_ulonglong2(gt_sub(v0, h0), gt_sub(v1, h1));
                            }
                        }
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");     // the MMAs read through the other proxy
                __syncwarp();
                if (lane == 0) gt_arrive(&full[stage]);
            }
        }
        __syncwarp();
    } else if (warp == S::CUT + ACC + 1) {
        // ---- TMA ----
        if (TMA && lane == 0) {
            int i = 0;
            bool ok = true;
            if (ahead) {
                const GtUnit<BT> u(p, unit0);
                for (int j = 0; j < ahead; ++j) tma_load(j, u.n0, u.m0, u.head, b0 * GT_BK + j * SUB * GT_HALF, false, true);
            }
            for (int unit = unit0; unit < n_units && ok; unit += step) {
                const GtUnit<BT> u(p, unit);
                for (int j = 0; j < steps; ++j, ++i) {
                    if (i < ahead) continue;
                    if (!gt_wait(&raw_empty[i % RAW], ((i / RAW) & 1) ^ 1, p.error, GT_ERR_LOAD)) { ok = false; break; }
                    tma_load(i, u.n0, u.m0, u.head, b0 * GT_BK + j * SUB * GT_HALF, true, true);
                }
            }
        }
        __syncwarp();
    } else if (warp == S::CUT + ACC) {
        // ---- MMAs: warp-uniform loop, one elected lane issues ----
        constexpr uint32_t one = gt_idesc(BT), two = gt_idesc(2 * BT);
        constexpr uint64_t BL = S::B >> 4;
        uint32_t elected;
        asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.b32 %0, 1, 0, p;\n}\n" : "=r"(elected));
        const bool leader = elected != 0;
        const uint64_t da0 = gt_desc(ring), dr0 = gt_desc(ring + S::CUT_RING + S::REST_A), db0 = gt_desc(ring + S::CUT_RING + S::CUT_X);
        int rs = 0, stage = 0, buf = 0;
        uint32_t phase = 0, small_phase = 1, hh_phase = 1;         // (the accumulators alternate: one phase for a pair of them)
        bool ok = true;
        for (int unit = unit0; unit < n_units && ok; unit += step) {
            for (int i = 0; i < steps; ++i) {
                const bool begins = P == 1 || i % P == 0, ends = P == 1 || i % P == P - 1, first = i % (P * GT_SLICE) == 0;
                // (A k-block in the middle asks for one barrier twice rather than for two.)
                ok = gt_ended(&full[stage], phase, begins ? &hh_empty[buf] : &full[stage], begins ? hh_phase : phase,
                              first ? small_empty : &full[stage], first ? small_phase : phase);
                if (!__all_sync(0xffffffffu, ok)) {
                    ok = !begins || gt_wait(&hh_empty[buf], hh_phase, p.error, GT_ERR_MMA);
                    ok = ok && (!first || gt_wait(small_empty, small_phase, p.error, GT_ERR_MMA));
                    ok = __all_sync(0xffffffffu, ok && gt_wait(&full[stage], phase, p.error, GT_ERR_MMA));
                }
                if (first) small_phase ^= 1;
                if (!ok) break;
                gt_fence_after();
                if (leader) {
                    const uint64_t da = da0 + (uint64_t)((rs * S::RAW_STAGE) >> 4);
                    const uint64_t dr = dr0 + (uint64_t)((stage * S::STAGE) >> 4), db = db0 + (uint64_t)((stage * S::STAGE) >> 4);
                    const uint32_t d_hh = tmem + (buf ? 2 * BT : 0), d_small = tmem + BT, d_both = tmem + (buf ? BT : 0);
#pragma unroll
                    for (int k = 0; k < SUB * GT_HALF / 8; ++k) {
                        const int h = k / (GT_HALF / 8);
                        const uint64_t o = (uint64_t)((k * 32 % 128) >> 4);
                        const uint64_t a = da + h * (S::A >> 4) + o, b = db + 2 * h * BL + o, bh = b + (buf ? BL : 0), bl = b + (buf ? 0 : BL);
                        if (k == 0 && begins && !first) {           // the large ones begin anew, the small ones go on
                            gt_mma(d_hh, a, bh, one, 0u);
                            gt_mma(d_small, a, bl, one, 1u);
                        } else {
                            gt_mma(d_both, a, b, two, k == 0 && first ? 0u : 1u);
                        }
                        gt_mma(d_small, dr + h * (S::A >> 4) + o, bh, one, 1u);
                    }
                    gt_commit(&empty[stage]);
                    if (!GtCfg<BT>::PLACE) gt_commit(&raw_empty[rs]);
                    if (ends) gt_commit(&hh_full[buf]);
                }
                __syncwarp();
                if (ends) { hh_phase ^= buf; buf ^= 1; }
                if (++rs == RAW) rs = 0;
                if (++stage == STAGES) { stage = 0; phase ^= 1; }
            }
        }
        __syncwarp();
    } else {
        // ---- empty the accumulators: a warp reads the lanes of its quarter (warp & 3), CPT of the columns ----
        const int quarter = warp & 3, c0 = (warp - S::CUT) / 4 * CPT;
        const uint32_t t = tmem + ((uint32_t)(quarter * 32) << 16) + c0;
        int i = 0;
        bool ok = true;
        for (int unit = unit0; unit < n_units && ok; unit += step) {
            const GtUnit<BT> u(p, unit);
            float s[CPT];
            for (int kb = b0; kb < b1; ++kb, ++i) {
                const int buf = i & 1, slice = kb / GT_SLICE;
                const bool first = kb % GT_SLICE == 0, end = kb == b1 - 1, last = end || kb % GT_SLICE == GT_SLICE - 1;
                ok = __all_sync(0xffffffffu, gt_wait(&hh_full[buf], (i >> 1) & 1, p.error, GT_ERR_SUMS));
                if (!ok) break;
                gt_fence_after();
                uint32_t v[16];
                if (first) {
#pragma unroll
                    for (int c = 0; c < CPT; ++c) s[c] = 0.f;
                }
#pragma unroll
                for (int c = 0; c < CPT; c += 16) {
                    gt_ld16(t + (buf ? 2 * BT : 0) + c, v);
#pragma unroll
                    for (int j = 0; j < 16; ++j) s[c + j] += __uint_as_float(v[j]);
                }
                if (last) {
#pragma unroll
                    for (int c = 0; c < CPT; c += 16) {
                        gt_ld16(t + BT + c, v);
#pragma unroll
                        for (int j = 0; j < 16; ++j) s[c + j] += __uint_as_float(v[j]);
                    }
                }
                gt_fence_before();
                __syncwarp();
                if (lane == 0) {
                    gt_arrive(&hh_empty[buf]);
                    if (last) gt_arrive(small_empty);
                }
                if (!last) continue;
                if (splits > 1) {                                   // kept until the cluster's MMAs are all done
#pragma unroll
                    for (int c = 0; c < CPT; c += 16) gt_st16(t + (3 + slice - s0) * BT + c, s + c);
                    asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                    continue;
                }
                // the sum so far lies in tensor memory
                if (slice > 0) {
#pragma unroll
                    for (int c = 0; c < CPT; c += 16) {
                        gt_ld16(t + 3 * BT + c, v);
#pragma unroll
                        for (int j = 0; j < 16; ++j) s[c + j] = __uint_as_float(v[j]) + s[c + j];
                    }
                }
                if (!end) {
#pragma unroll
                    for (int c = 0; c < CPT; c += 16) gt_st16(t + 3 * BT + c, s + c);
                    asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                }
            }
            const int n = u.n0 + quarter * 32 + lane;
            if (splits == 1 && ok && n < p.N) {
                const float* x = p.x + (size_t)u.head * K;
                const float* w = p.w + ((size_t)u.head * p.N + n) * K;
                float* out = p.out + (size_t)u.head * p.N + n;
                bool finite = true;
#pragma unroll
                for (int c = 0; c < CPT; ++c) {
                    const int m = u.m0 + c0 + c;
                    if (m < p.M) {
                        out[(size_t)m * p.ldo] = s[c];
                        finite = finite && gt_finite(s[c]);
                    }
                }
                if (!finite) {
#pragma unroll 1
                    for (int m = u.m0 + c0; m < u.m0 + c0 + CPT && m < p.M; ++m)
                        if (!gt_finite(out[(size_t)m * p.ldo])) out[(size_t)m * p.ldo] = gt_chain(x + (size_t)m * p.ldx, w, K);
                }
            }
        }
        if (gt_extra_wait) gt_wait(&hh_full[i & 1], (i >> 1) & 1, p.error, GT_ERR_SUMS);       // tests: a wait that runs out
        __syncwarp();
    }
    if (splits > 1) {
        const GtUnit<BT> u(p, unit0);
        const int rows = p.M - u.m0 < BT ? p.M - u.m0 : BT, per = (rows + splits - 1) / splits;
        float* slots = reinterpret_cast<float*>(ring);              // [slices][per][128]
        gt_cluster_sync();                                          // every block's loads have arrived and its MMAs are done
        if (warp >= S::CUT && warp < S::CUT + ACC) {
            const int quarter = warp & 3, c0 = (warp - S::CUT) / 4 * CPT;
            const uint32_t t = tmem + ((uint32_t)(quarter * 32) << 16) + c0;
#pragma unroll 1
            for (int s = s0; s < s1; ++s) {
                int owner = c0 / per, local = c0 - owner * per;
#pragma unroll 1
                for (int c = 0; c < CPT && c0 + c < rows; c += 16) {
                    uint32_t v[16];
                    gt_ld16(t + (3 + s - s0) * BT + c, v);
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        if (c0 + c + j < rows)
                            gt_st_cluster(slots + ((size_t)s * per + local) * GT_ROWS + quarter * 32 + lane, (uint32_t)owner, __uint_as_float(v[j]));
                        if (++local == per) { local = 0; ++owner; }
                    }
                }
            }
        }
        gt_cluster_sync();                                          // all sums have arrived
        if (warp >= S::CUT && warp < S::CUT + ACC) {
            const int quarter = warp & 3, row = quarter * 32 + lane, n = u.n0 + row;
            const float* mine = slots + row;
#pragma unroll 1
            for (int l = (warp - S::CUT) / 4; l < per && rank * per + l < rows; l += ACC / 4) {
                float v = mine[(size_t)l * GT_ROWS];
                for (int s = 1; s < slices; ++s) v += mine[((size_t)s * per + l) * GT_ROWS];
                const int m = u.m0 + rank * per + l;
                if (n < p.N) {
                    if (!gt_finite(v))
                        v = gt_chain(p.x + (size_t)u.head * K + (size_t)m * p.ldx, p.w + ((size_t)u.head * p.N + n) * K, K);
                    p.out[(size_t)u.head * p.N + n + (size_t)m * p.ldo] = v;
                }
            }
        }
    }
    gt_fence_before();
    __syncthreads();
    if (warp == S::CUT + ACC) {
        gt_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(GtCfg<BT>::COLS) : "memory");
    }
}

// ---- choice and launch -----------------------------------------------------------------------------------------------
// ticks: how long a wait inside the kernel may last, in clock ticks (<= 0: the default of about a second); extra_wait != 0: the
// emptying warps wait once more for a phase that never completes.  Holds for the current device until set again.
NI_EXPORT int ni_gemm_f32_tc_set_wait(long long ticks, int extra_wait) {
    if (ticks <= 0) ticks = 2000000000LL;
    cudaError_t e = cudaMemcpyToSymbol(gt_wait_limit, &ticks, sizeof(ticks));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(gt_extra_wait, &extra_wait, sizeof(extra_wait));
    return e == cudaSuccess ? NI_OK : (int)e;
}

static int gt_slices(int K) { return (K + GT_BK * GT_SLICE - 1) / (GT_BK * GT_SLICE); }

// Whether K can be cut over `splits` blocks: a slice for each, room in tensor memory for a block's sums and in the ring for those
// that arrive.
template <int BT>
static bool gt_can_split(int M, int K, int splits) {
    if (splits == 1) return true;
    const int slices = gt_slices(K), rows = M < BT ? M : BT;
    return splits <= 8 && splits <= slices && (slices + splits - 1) / splits <= GtSizes<BT>::REGIONS &&
           (long long)slices * ((rows + splits - 1) / splits) * GT_ROWS * 4 <= GtSizes<BT>::RING;
}

typedef CUresult (*GtEncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static GtEncodeTiledFn gt_encode_tiled() {
    static GtEncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<GtEncodeTiledFn>(sym);
    });
    return fn;
}

// 32 columns (128 bytes, 128-byte swizzle) of `box_rows` rows: of the weights [rows, K], or of one head of x [M, H, K].
static int gt_map_w(CUtensorMap* map, const float* w, long long rows, int K) {
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)K * 4};
    const cuuint32_t box[2] = {GT_HALF, GT_ROWS}, elem[2] = {1, 1};
    GtEncodeTiledFn enc = gt_encode_tiled();
    if (!enc) return NI_ERR_BAD_ARGUMENT;
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(w), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
               ? NI_OK : NI_ERR_BAD_ARGUMENT;
}
static int gt_map_x(CUtensorMap* map, const float* x, int M, int H, int K, int ldx, int box_rows) {
    const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)H, (cuuint64_t)M}, strides[2] = {(cuuint64_t)K * 4, (cuuint64_t)ldx * 4};
    const cuuint32_t box[3] = {GT_HALF, 1, (cuuint32_t)box_rows}, elem[3] = {1, 1, 1};
    GtEncodeTiledFn enc = gt_encode_tiled();
    if (!enc) return NI_ERR_BAD_ARGUMENT;
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(x), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
               ? NI_OK : NI_ERR_BAD_ARGUMENT;
}

template <int BT, bool TMA>
static int gt_launch(const GtParams& p, cudaStream_t stream) {
    if (!gt_can_split<BT>(p.M, p.K, p.splits)) return NI_ERR_BAD_ARGUMENT;
    const long long units = (long long)((p.M + BT - 1) / BT) * ((p.N + GT_ROWS - 1) / GT_ROWS) * p.H;
    if (units * p.splits > 0x7fffffff || (long long)p.N * p.H > 0x7fffffff) return NI_ERR_UNSUPPORTED_SIZE;
    CUtensorMap mw = {}, mx = {};
    if (TMA && (gt_map_w(&mw, p.w, (long long)p.N * p.H, p.K) != NI_OK || gt_map_x(&mx, p.x, p.M, p.H, p.K, p.ldx, BT) != NI_OK))
        return gt_launch<BT, false>(p, stream);                     // sizes that a tensor map does not take
    auto kernel = gemm_f32_tc_kernel<BT, TMA>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GtSizes<BT>::SMEM);
    if (e != cudaSuccess) return (int)e;
    const long long resident = (long long)ni_sm_count();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(p.splits > 1 ? units * p.splits : units < resident ? units : resident));
    cfg.blockDim = dim3(GtSizes<BT>::THREADS);
    cfg.dynamicSmemBytes = GtSizes<BT>::SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = p.splits;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p.splits > 1 ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, kernel, mw, mx, p);
    return e == cudaSuccess ? NI_OK : (int)e;
}

template <int BT>
static int gt_launch_loads(const GtParams& p, cudaStream_t stream) {
    const bool tma = p.K % 4 == 0 && p.ldx % 4 == 0 && ((uintptr_t)p.x | (uintptr_t)p.w) % 16 == 0;
    return tma ? gt_launch<BT, true>(p, stream) : gt_launch<BT, false>(p, stream);
}

// Clusters of this many blocks that the device runs at once (a block takes an SM for itself; asked for once per device).
static int gt_clusters(int splits) {
    static int cached[64][9];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    if (cached[dev][splits] <= 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(splits);
        cfg.blockDim = dim3(GtSizes<16>::THREADS);
        cfg.dynamicSmemBytes = GtSizes<16>::SMEM;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = splits;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaFuncSetAttribute(gemm_f32_tc_kernel<16, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, GtSizes<16>::SMEM) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, gemm_f32_tc_kernel<16, true>, &cfg) != cudaSuccess || n <= 0)
            n = ni_sm_count() / splits > 0 ? ni_sm_count() / splits : 1;
        cached[dev][splits] = n;
    }
    return cached[dev][splits];
}

// The tile and the split of K that are done first by what they measured: a k-block of 64 takes a block 0.65, 0.95, 1.10 and 1.62 us
// with 16, 32, 64 and 128 rows of x (128 weight rows; 0.74 us is what memory gives every SM for its 32 KB), a launch 6 us besides, and
// a cluster 1.7 us and 0.02 us for every row and slice of a block's sums.  [2048, 2048] and 177 rows: 30.9 us in two slices of 64-row
// tiles, 43 whole; [2048, 8192] and 1 row: 24.5 in six slices, 29.7 in four, 89 whole.
static void gt_choose(const GtParams& p, int& bt, int& splits) {
    const int slices = gt_slices(p.K);
    const long long n_tiles = (long long)((p.N + GT_ROWS - 1) / GT_ROWS) * p.H;
    double best = 0.0;
    const int want_bt = bt, want_splits = splits;
    bt = 0;
    for (int i = 0; i < 4; ++i) {
        const int b = 16 << i;
        if (want_bt ? b != want_bt : (b > 16 && b >= 2 * p.M)) continue;
        const double per_block = i == 0 ? 0.65 : i == 1 ? 0.95 : i == 2 ? 1.10 : 1.62;
        const long long units = n_tiles * ((p.M + b - 1) / b);
        for (int sp = 1; sp <= 8; ++sp) {
            if (want_splits ? sp != want_splits : sp > 1 && units * sp > 4LL * ni_sm_count()) continue;
            if (!(b == 16 ? gt_can_split<16>(p.M, p.K, sp) : b == 32 ? gt_can_split<32>(p.M, p.K, sp)
                  : b == 64 ? gt_can_split<64>(p.M, p.K, sp) : gt_can_split<128>(p.M, p.K, sp))) continue;
            const long long at_once = sp == 1 ? ni_sm_count() : gt_clusters(sp), waves = (units + at_once - 1) / at_once;
            const int mine = (slices + sp - 1) / sp, rows = p.M < b ? p.M : b;
            const double once = sp == 1 ? 0.0 : 1.7 + 0.02 * rows * mine;
            const double us = 6.0 + waves * (once + per_block * GT_SLICE * mine);
            if (!bt || us < best) { best = us; bt = b; splits = sp; }
        }
    }
}

// One product per head: out[m, h, :] = x[m, h, :] . w[h]^T with x [M, H, K] (rows ldx floats apart), w [H, N, K], out [M, H, N].
// bt (16, 32, 64, 128) and splits (blocks that share K): 0 leaves the choice to the sizes; every choice gives the same bits.
NI_EXPORT int ni_gemm_f32_tc(const float* x, int ldx, const float* w, float* out, int M, int N, int K, int H, int bt, int splits,
                             int* error, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || H <= 0) return NI_OK;
    if (K <= 0 || error == nullptr || (long long)ldx < (long long)H * K || bt < 0 || splits < 0) return NI_ERR_BAD_ARGUMENT;
    GtParams p = {x, w, out, M, N, K, H, ldx, H * N, splits, error};
    gt_choose(p, bt, p.splits);
    switch (bt) {
        case 16: return gt_launch_loads<16>(p, stream);
        case 32: return gt_launch_loads<32>(p, stream);
        case 64: return gt_launch_loads<64>(p, stream);
        case 128: return gt_launch_loads<128>(p, stream);
    }
    return NI_ERR_BAD_ARGUMENT;
}
