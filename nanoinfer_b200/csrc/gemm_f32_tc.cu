// out[M, N] = x[M, K] . w[N, K]^T of FP32 matrices with long rows on the fifth-generation tensor cores, with errors smaller than
// those of a chain of FP32 multiply-adds.  Every FP32 number is the sum of three bfloat16 numbers, each what is left rounded to nearest
// (24 bits in all, so none is lost), and six of the nine products of parts are taken:
//
//     x w = xa wa + (xa wb + xb wa + xb wb + xa wc + xc wa)     [+ xb wc + xc wb + xc wc: 2^-23 of x w at most, 2^-25 in the mean square]
//
// The tensor core adds into its FP32 accumulator by cutting, a bias that grows with the number of additions.  So the accumulator of the
// large products (xa wa) is emptied every 64 columns into registers, where it is added with rounding to nearest, and the small ones,
// 2^-8 of the large, have an accumulator of their own that is emptied every 256:
//     slice s of 256:  sum_s = (((hh_0 + hh_1) + hh_2) + hh_3) + small          result = (sum_0 + sum_1) + ...
// This order is the same for every tile size, number of rows and split of K, so an element's bits depend on its two rows alone.
// Relative error against 64 bits, here / of the chain: normal numbers 0.9e-7 / 5.7e-7 at 1,024 columns, 1.3e-7 / 1.6e-6 at 8,192;
// positive ones 0.9e-7 / 4.9e-7 and 1.2e-7 / 1.4e-6; rows of ten terms 0.56e-7 / 0.65e-7, of one 2.6e-8 / 2.5e-8; a number that meets
// ones and zeros comes back bit for bit.  (Two tf32 parts and three products, which lose two of the 24 bits: 3.0e-7 and 3.7e-7,
// rows of ten terms 1.8e-7, of one 1.7e-7.)
//
// What bounds it: at many rows cutting and multiplying, which have two boxes to hand over (tensor pipe busy 53 % of the time, ALU
// 47 %): 1,087 rows and [16384, 2048] 408 us (179 TFLOP/s; two tf32 parts 418, chains on CUDA cores 1,419), 177 rows 106 (116); at few the weights,
// [128256, 2048] 169 us (6.2 TB/s; 174; the ring of chains 177, at 8 rows 239), and for small matrices the way of one block: 6 us
// of start, first load and last sum, 0.66 us for 64 columns ([2048, 2048] 12.5 us alone (12.1; one row as a chain 8.0, whose bits a row among
// many would not have), less behind a kernel that lets it start early).
//
// The 128 lanes of the tcgen05 tile are weight rows, its columns BT rows of x (16 .. 128): few rows read the weights once, at
// many rows 128 x 128 tiles.  Blocks are persistent; a block's warps:
//   0 - ..  cut: GROUPS groups of four take turns at the boxes of 32 columns that TMA has filled.  The weights' parts go to tensor memory,
//           from where the MMAs read them (in shared memory they are written and read five times by MMAs of few columns: 230 us for
//           the vocabulary); those of x to shared memory, so that xa and xb, or xb and xa, are 2 BT rows of one operand
//   then    empty the accumulators, 4 to 16 warps
//   last    two: the MMAs, and TMA
// A product with few weight rows cuts the slices of K over the blocks of a cluster; their sums go to the block that owns the row
// of x (through its shared memory, once all MMAs are done) and are added there in the order of the slices.
//
// A sum that is not finite, not below 2^100, or below 2^-80 (but no zero) is computed once more as one chain of fused multiply-adds:
// inf - inf among the parts of an infinite operand, a part that rounds beyond FP32's range, or third parts that bfloat16 cannot hold
// (of numbers below 2^-110), do not show.  Beside ordinary numbers such small ones lose 2^-133 at most.
#include <cuda.h>

#include <mutex>

#include "common.cuh"

#define GT_ROWS 128            // weight rows of a tile
#define GT_BOX 32              // columns of a box as TMA brings it: 128 bytes of FP32, 64 of a part
#define GT_BK 64               // k-block: what the accumulator of large products adds up
#define GT_SLICE 4             // k-blocks of a slice
#define GT_ERR_LOAD 51
#define GT_ERR_CUT 52
#define GT_ERR_MMA 53
#define GT_ERR_SUMS 54

// RAW boxes as loaded; STAGES of cut ones, the weights' parts in tensor memory, those of x in shared memory; GROUPS of four cutting
// warps; ACC warps that empty accumulators; HH accumulators of large products
template <int BT> struct GtCfg;
template <> struct GtCfg<16> { static constexpr int RAW = 11, STAGES = 4, GROUPS = 4, ACC = 4, HH = 2; };
template <> struct GtCfg<32> { static constexpr int RAW = 9, STAGES = 4, GROUPS = 4, ACC = 4, HH = 2; };
template <> struct GtCfg<64> { static constexpr int RAW = 6, STAGES = 4, GROUPS = 4, ACC = 8, HH = 1; };
template <> struct GtCfg<128> { static constexpr int RAW = 4, STAGES = 2, GROUPS = 2, ACC = 16, HH = 1; };
template <int BT> struct GtSizes {
    using C = GtCfg<BT>;
    static constexpr int A = GT_ROWS * 128, B = BT * 128, BOX = A + B;               // bytes of a box of weights and of x
    static constexpr int PART = BT * 64, XRING = C::RAW * BOX;                       // of a part of a box of x; where those begin
    static constexpr int RING = XRING + C::STAGES * 3 * PART, SMEM = 1024 + RING + 512;
    // tensor memory: accumulators (the first of large products, small ones, the other of large ones), sums of slices, weights
    static constexpr int SUMS = (1 + C::HH) * BT, WSTAGE = 3 * GT_BOX / 2, WPARTS = 512 - C::STAGES * WSTAGE;
    static constexpr int REGIONS = (WPARTS - SUMS) / BT;                             // sums of slices that a block can keep, but for its last
    static constexpr int CUT = 4 * C::GROUPS, THREADS = (CUT + C::ACC + 2) * 32;
    static_assert(C::GROUPS <= C::STAGES && C::RAW >= C::STAGES, "see the cutting warps' waits");
    static_assert(REGIONS >= 1 && BOX % 1024 == 0 && PART % 1024 == 0, "the swizzle goes by the address");
    static_assert((2 * C::RAW + 2 * C::STAGES + 6) * 8 <= 512 && SMEM <= 232448, "shared memory");
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
__device__ __forceinline__ uint64_t gt_desc(const void* tile) {              // K-major, 64-byte swizzle, 8-row groups 512 bytes apart
    const uint32_t addr = gt_smem(tile);
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;
    return d;
}
__host__ __device__ constexpr uint32_t gt_idesc(int n) {          // BF16 x BF16 -> FP32, M = 128, N = n
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(GT_ROWS >> 4) << 24);
}
__device__ __forceinline__ void gt_mma(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
        ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(acc) : "memory");
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
__device__ __forceinline__ void gt_st4(uint32_t taddr, const uint4& a) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%4], {%0,%1,%2,%3};\n" ::"r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(taddr) : "memory");
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

// The three parts of eight numbers, in pairs of bfloat16.  Each is what is left rounded to nearest, so that three hold all 24 bits.  What
// is not finite, or rounds beyond bfloat16's range, has a NaN among its parts.  What is left comes from multiply-adds that read a
// bfloat16 number as it lies: fewer instructions than packed subtractions of it as FP32, same bits (2 rows and [16384, 2048] 30.4 us
// instead of 31.7, 1,087 rows 449 instead of 470 in turn).
__device__ __forceinline__ void gt_cut(const float4& a, const float4& b, uint4 part[3]) {
    float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        uint32_t h[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float &lo = v[2 * j], &hi = v[2 * j + 1];
            asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(h[j]) : "f"(hi), "f"(lo));
            if (i < 2)
                asm("{\n.reg .b16 l, h, m;\n"
                    "mov.b32 {l, h}, %2;\n"
                    "mov.b16 m, 0xBF80;\n"                          // -1
                    "fma.rn.f32.bf16 %0, l, m, %0;\n"
                    "fma.rn.f32.bf16 %1, h, m, %1;\n}\n" : "+f"(lo), "+f"(hi) : "r"(h[j]));
        }
        part[i] = make_uint4(h[0], h[1], h[2], h[3]);
    }
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

// Whether a sum stands as it is: zero, or from 2^-80 to 2^100.
__device__ __forceinline__ bool gt_stands(float v) {
    const uint32_t magnitude = __float_as_uint(v) & 0x7fffffffu;
    return magnitude == 0u || magnitude - (47u << 23) < (180u << 23);
}
// Up to four sums of one weight row (out, ldo apart) as chains where they do not stand.  VEC: rows lie on 16 bytes, K is a multiple of 4.
// (Number by number, with one sum at a time: 143 ms for 1,087 rows of infinities and [16384, 2048].)
template <bool VEC>
__device__ __forceinline__ void gt_chains(const float* __restrict__ x, int ldx, int rows, const float* __restrict__ w, int K, float* out, int ldo) {
    float a[4] = {0.f, 0.f, 0.f, 0.f};
    for (int k = 0; k < K; k += 4) {
        float xs[4][4], ws[4];
        auto load = [&](const float* from, float v[4]) {
            const float4 q = VEC ? *reinterpret_cast<const float4*>(from + k) : gt_load4(from, k, K, true);
            v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
        };
        load(w, ws);
#pragma unroll
        for (int i = 0; i < 4; ++i) load(x + (size_t)(i < rows ? i : 0) * ldx, xs[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (VEC || k + j < K) {
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = fmaf(xs[i][j], ws[j], a[i]);
            }
        if (a[0] != a[0] && a[1] != a[1] && a[2] != a[2] && a[3] != a[3]) break;         // NaN stays NaN
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (i < rows && !gt_stands(out[(size_t)i * ldo])) out[(size_t)i * ldo] = a[i];
}

struct GtParams {
    const float* x;
    const float* w;
    float* out;
    int M, N, K, H, ldx, ldo, splits, early;
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
    using C = GtCfg<BT>;
    constexpr int RAW = C::RAW, STAGES = C::STAGES, GROUPS = C::GROUPS, ACC = C::ACC, HH = C::HH;
    constexpr int P = GT_BK / GT_BOX;                                                        // boxes of a k-block
    constexpr int CPT = BT * 4 / ACC;                                                        // columns of an emptying thread
    extern __shared__ uint8_t gt_smem_raw[];
    uint8_t* ring = reinterpret_cast<uint8_t*>(((uintptr_t)gt_smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* loaded = reinterpret_cast<uint64_t*>(ring + S::RING);
    uint64_t* raw_empty = loaded + RAW;
    uint64_t* full = raw_empty + RAW;
    uint64_t* empty = full + STAGES;
    uint64_t* hh_full = empty + STAGES;
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

    const int steps = (b1 - b0) * P;                                                         // boxes of a unit
    auto tma_load = [&](int i, int n0, int m0, int head, int k, bool weights, bool x) {
        uint8_t* box = ring + i % RAW * S::BOX;
        uint64_t* bar = &loaded[i % RAW];
        if (weights) gt_expect_tx(bar, S::BOX);
        if (weights) gt_tma_2d(box, &map_w, k, head * p.N + n0, bar);                       // (columns beyond K are zeros)
        if (x) gt_tma_3d(box + S::A, &map_x, k, head, m0, bar);
    };
    // boxes whose weights are asked for at once
    const int ahead = !TMA || !p.early || unit0 >= n_units ? 0 : steps < RAW ? steps : RAW;
    if (threadIdx.x == (S::CUT + ACC + 1) * 32) {
        for (int s = 0; s < RAW; ++s) { gt_init(&loaded[s], 1); gt_init(&raw_empty[s], 4); }
        for (int s = 0; s < STAGES; ++s) { gt_init(&full[s], 4); gt_init(&empty[s], 1); }
        for (int a = 0; a < 2; ++a) { gt_init(&hh_full[a], 1); gt_init(&hh_empty[a], ACC); }
        gt_init(small_empty, ACC);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        // Weights that the caller says the kernel in front does not write are asked for before that kernel has ended, and before the
        // block is set up.
        const GtUnit<BT> u(p, unit0);
        for (int j = 0; j < ahead; ++j) tma_load(j, u.n0, u.m0, u.head, b0 * GT_BK + j * GT_BOX, true, false);
    }
    if (warp == S::CUT + ACC) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n"
                     ::"r"(gt_smem(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    gt_fence_before();
    __syncthreads();
    gt_fence_after();
    const uint32_t tmem = *tmem_slot;
    bool stands = true;                                             // every sum that this thread has written
    gt_pdl_wait();                                                  // x is there, and nobody reads what out was

    if (warp < S::CUT) {
        // ---- cut: box number i of this block is group i % GROUPS's.  Of the weights a warp has the 32 rows of its quarter of tensor
        // memory, a lane one row; of x eight columns of a row (eight lanes next to each other have different rows: no two meet in a
        // bank) ----
        const int group = warp >> 2, quarter = warp & 3, row = quarter * 32 + lane, r = lane & 7, c = lane >> 3;
        const uint32_t wparts = tmem + ((uint32_t)(quarter * 32) << 16) + S::WPARTS;
        int first = 0;                                             // number of the unit's first box
        bool ok = true;
        for (int unit = unit0; unit < n_units && ok; unit += step, first += steps) {
            const GtUnit<BT> u(p, unit);
            for (int i = first + (group + GROUPS - first % GROUPS) % GROUPS; i < first + steps; i += GROUPS) {
                const int s = i % STAGES, buf = HH > 1 ? i / P & 1 : 0;
                // (In this order: MMAs end in order, so every box up to i - STAGES has been cut, and the loaded one cannot be
                // waiting for number i - RAW still, whose phase has the other parity.)
                ok = gt_wait(&empty[s], ((i / STAGES) & 1) ^ 1, p.error, GT_ERR_CUT);
                if (TMA) ok = ok && gt_wait(&loaded[i % RAW], (i / RAW) & 1, p.error, GT_ERR_CUT);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                gt_fence_after();
                const uint8_t* raw = ring + i % RAW * S::BOX;
                const int k0 = b0 * GT_BK + (i - first) * GT_BOX;
#pragma unroll
                for (int k = 0; k < GT_BOX; k += 8) {
                    float4 a, b;
                    if (TMA) {
                        a = *reinterpret_cast<const float4*>(raw + row * 128 + (((k / 4) ^ r) << 4));
                        b = *reinterpret_cast<const float4*>(raw + row * 128 + (((k / 4 + 1) ^ r) << 4));
                    } else {
                        const float* from = p.w + ((size_t)u.head * p.N + u.n0 + row) * K;
                        a = gt_load4(from, k0 + k, K, u.n0 + row < p.N);
                        b = gt_load4(from, k0 + k + 4, K, u.n0 + row < p.N);
                    }
                    uint4 part[3];
                    gt_cut(a, b, part);
#pragma unroll
                    for (int j = 0; j < 3; ++j) gt_st4(wparts + s * S::WSTAGE + j * (GT_BOX / 2) + k / 2, part[j]);
                }
                uint8_t* parts = ring + S::XRING + s * 3 * S::PART;
                uint8_t* x0 = parts + (buf ? S::PART : 0);                                   // (first parts before second ones, or behind them)
                uint8_t* x1 = parts + (buf ? 0 : S::PART);
#pragma unroll
                for (int j = 0; j < (BT / 8 + 3) / 4; ++j) {
                    const int eight = quarter + 4 * j, row = 8 * eight + r;
                    if (BT / 8 % 4 && eight >= BT / 8) break;
                    if (BT == 16 && u.m0 + 8 * eight >= p.M) break;                          // rows that nobody has; up to 8: 26.3 us instead of 26.7
                    float4 a, b;
                    if (TMA) {
                        a = *reinterpret_cast<const float4*>(raw + S::A + row * 128 + (((2 * c) ^ r) << 4));
                        b = *reinterpret_cast<const float4*>(raw + S::A + row * 128 + (((2 * c + 1) ^ r) << 4));
                    } else {
                        const float* x = p.x + (size_t)u.head * K + (size_t)(u.m0 + row) * p.ldx;
                        const int k = k0 + 8 * c;
                        a = gt_load4(x, k, K, u.m0 + row < p.M);
                        b = gt_load4(x, k + 4, K, u.m0 + row < p.M);
                    }
                    uint4 part[3];
                    gt_cut(a, b, part);
                    const int at = row * 64 + ((c ^ (r >> 1)) << 4);
                    *reinterpret_cast<uint4*>(x0 + at) = part[0];
                    *reinterpret_cast<uint4*>(x1 + at) = part[1];
                    *reinterpret_cast<uint4*>(parts + 2 * S::PART + at) = part[2];
                }
                asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");     // the MMAs read through the other proxy
                gt_fence_before();
                __syncwarp();
                if (lane == 0) {
                    gt_arrive(&full[s]);
                    if (TMA) gt_arrive(&raw_empty[i % RAW]);
                }
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
                for (int j = 0; j < ahead; ++j) tma_load(j, u.n0, u.m0, u.head, b0 * GT_BK + j * GT_BOX, false, true);
            }
            for (int unit = unit0; unit < n_units && ok; unit += step) {
                const GtUnit<BT> u(p, unit);
                for (int j = 0; j < steps; ++j, ++i) {
                    if (i < ahead) continue;
                    if (!gt_wait(&raw_empty[i % RAW], ((i / RAW) & 1) ^ 1, p.error, GT_ERR_LOAD)) { ok = false; break; }
                    tma_load(i, u.n0, u.m0, u.head, b0 * GT_BK + j * GT_BOX, true, true);
                }
            }
            for (int j = i < RAW ? 0 : i - RAW; j < i; ++j)         // loads in flight end before the block may
                gt_wait(&loaded[j % RAW], (j / RAW) & 1, p.error, GT_ERR_LOAD);
        }
        __syncwarp();
    } else if (warp == S::CUT + ACC) {
        // ---- MMAs: warp-uniform loop, one elected lane issues ----
        constexpr uint32_t one = gt_idesc(BT), two = gt_idesc(2 * BT);
        uint32_t elected;
        asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.b32 %0, 1, 0, p;\n}\n" : "=r"(elected));
        const bool leader = elected != 0;
        const uint64_t x0 = gt_desc(ring + S::XRING);
        constexpr uint64_t PART = S::PART >> 4;
        int stage = 0, buf = 0, last = -1;
        uint32_t phase = 0, small_phase = 1, hh_phase = 1;         // (two accumulators alternate: one phase for the pair)
        bool ok = true;
        for (int unit = unit0; unit < n_units && ok; unit += step) {
            for (int i = 0; i < steps; ++i) {
                const bool begins = i % P == 0, ends = i % P == P - 1, first = i % (P * GT_SLICE) == 0, hh = begins && HH > 1;
                // (A box in the middle of a k-block asks for one barrier three times rather than for three.)
                ok = gt_ended(&full[stage], phase, hh ? &hh_empty[buf] : &full[stage], hh ? hh_phase : phase,
                              first ? small_empty : &full[stage], first ? small_phase : phase);
                if (!__all_sync(0xffffffffu, ok)) {
                    ok = !hh || gt_wait(&hh_empty[buf], hh_phase, p.error, GT_ERR_MMA);
                    ok = ok && (!first || gt_wait(small_empty, small_phase, p.error, GT_ERR_MMA));
                    ok = __all_sync(0xffffffffu, ok && gt_wait(&full[stage], phase, p.error, GT_ERR_MMA));
                }
                if (first) small_phase ^= 1;
                if (!ok) break;
                gt_fence_after();
                const uint32_t w = tmem + S::WPARTS + stage * S::WSTAGE, d_small = tmem + BT, d_hh = tmem + (buf ? 2 * BT : 0);
                const uint64_t x = x0 + (uint64_t)stage * 3 * PART;
                if (leader) {
#pragma unroll
                    for (int k = 0; k < GT_BOX / 16; ++k) {
                        const uint32_t wa = w + 8 * k, wb = wa + GT_BOX / 2, wc = wb + GT_BOX / 2;                  // parts of the weights
                        const uint64_t xa = x + 2 * k + (buf ? PART : 0), xb = x + 2 * k + (buf ? 0 : PART), xc = x + 2 * k + 2 * PART;
                        if (HH == 1) {                              // the large ones follow below
                            gt_mma(d_small, wa, xb, one, k == 0 && first ? 0u : 1u);
                        } else if (k == 0 && begins && !first) {    // the large ones begin anew, the small ones go on
                            gt_mma(d_hh, wa, xa, one, 0u);
                            gt_mma(d_small, wa, xb, one, 1u);
                        } else {
                            gt_mma(tmem + (buf ? BT : 0), wa, x + 2 * k, two, k == 0 && first ? 0u : 1u);
                        }
                        gt_mma(d_small, wb, xa, one, 1u);
                        gt_mma(d_small, wb, xb, one, 1u);
                        gt_mma(d_small, wa, xc, one, 1u);
                        gt_mma(d_small, wc, xa, one, 1u);
                    }
                }
                if (HH == 1) {                                      // (the one accumulator has been emptied meanwhile)
                    __syncwarp();
                    if (begins) {
                        ok = __all_sync(0xffffffffu, gt_wait(&hh_empty[0], hh_phase, p.error, GT_ERR_MMA));
                        gt_fence_after();
                    }
                    if (leader && ok) {
#pragma unroll
                        for (int k = 0; k < GT_BOX / 16; ++k) gt_mma(d_hh, w + 8 * k, x + 2 * k, one, k == 0 && begins ? 0u : 1u);
                    }
                }
                if (leader) {
                    gt_commit(&empty[stage]);
                    if (ends) gt_commit(&hh_full[buf]);
                }
                __syncwarp();
                last = 2 * stage + (int)phase;
                if (!ok) break;
                if (ends) {
                    hh_phase ^= HH > 1 ? buf : 1;
                    if (HH > 1) buf ^= 1;
                }
                if (++stage == STAGES) { stage = 0; phase ^= 1; }
            }
        }
        if (last >= 0) gt_wait(&empty[last >> 1], last & 1, p.error, GT_ERR_MMA);           // nor do MMAs outlive their tensor memory
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
                const int buf = HH > 1 ? i & 1 : 0, slice = kb / GT_SLICE;
                const bool first = kb % GT_SLICE == 0, end = kb == b1 - 1, last = end || kb % GT_SLICE == GT_SLICE - 1;
                ok = __all_sync(0xffffffffu, gt_wait(&hh_full[buf], (HH > 1 ? i >> 1 : i) & 1, p.error, GT_ERR_SUMS));
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
                if (splits > 1) {                                   // kept until the cluster's MMAs are all done (the last where
                                                                    // large products were: this block's have ended)
#pragma unroll
                    for (int c = 0; c < CPT; c += 16) gt_st16(t + (end ? 0 : S::SUMS + (slice - s0) * BT) + c, s + c);
                    asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                    continue;
                }
                // the sum so far lies in tensor memory
                if (slice > 0) {
#pragma unroll
                    for (int c = 0; c < CPT; c += 16) {
                        gt_ld16(t + S::SUMS + c, v);
#pragma unroll
                        for (int j = 0; j < 16; ++j) s[c + j] = __uint_as_float(v[j]) + s[c + j];
                    }
                }
                if (!end) {
#pragma unroll
                    for (int c = 0; c < CPT; c += 16) gt_st16(t + S::SUMS + c, s + c);
                    asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                }
            }
            const int n = u.n0 + quarter * 32 + lane;
            if (splits == 1 && ok && n < p.N) {
                float* out = p.out + (size_t)u.head * p.N + n;
#pragma unroll
                for (int c = 0; c < CPT; ++c) {
                    const int m = u.m0 + c0 + c;
                    if (m < p.M) {
                        out[(size_t)m * p.ldo] = s[c];
                        stands = stands && gt_stands(s[c]);
                    }
                }
            }
        }
        if (gt_extra_wait) gt_wait(&hh_full[HH > 1 ? i & 1 : 0], (HH > 1 ? i >> 1 : i) & 1, p.error, GT_ERR_SUMS);       // tests: a wait that runs out
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
                    gt_ld16(t + (s == s1 - 1 ? 0 : S::SUMS + (s - s0) * BT) + c, v);
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
                    p.out[(size_t)u.head * p.N + n + (size_t)m * p.ldo] = v;
                    stands = stands && gt_stands(v);
                }
            }
        }
    }
    gt_fence_before();
    const bool again = __syncthreads_or(!stands);
    if (warp == S::CUT + ACC) {
        gt_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512) : "memory");
    }
    if (again) {                                                    // all warps look through what the block has written, four rows of x at a time
        for (int unit = unit0; unit < n_units; unit += step) {
            const GtUnit<BT> u(p, unit);
            const int all = p.M - u.m0 < BT ? p.M - u.m0 : BT, per = (all + splits - 1) / splits;
            const int m0 = u.m0 + rank * per, m1 = m0 + per < u.m0 + all ? m0 + per : u.m0 + all;
            for (int item = warp; item < (per + 3) / 4 * 4; item += S::THREADS / 32) {
                const int m = m0 + item / 4 * 4, rows = m1 - m < 4 ? m1 - m : 4, n = u.n0 + (item & 3) * 32 + lane;
                if (n >= p.N) continue;
                float* out = p.out + (size_t)u.head * p.N + n + (size_t)m * p.ldo;
                bool four = true;
                for (int i = 0; i < rows; ++i) four = four && gt_stands(out[(size_t)i * p.ldo]);
                if (!four)
                    gt_chains<TMA>(p.x + (size_t)u.head * K + (size_t)m * p.ldx, p.ldx, rows, p.w + ((size_t)u.head * p.N + n) * K, K, out, p.ldo);
            }
        }
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
    return splits <= 8 && splits <= slices && (slices + splits - 1) / splits <= GtSizes<BT>::REGIONS + 1 &&
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
    const cuuint32_t box[2] = {GT_BOX, GT_ROWS}, elem[2] = {1, 1};
    GtEncodeTiledFn enc = gt_encode_tiled();
    if (!enc) return NI_ERR_BAD_ARGUMENT;
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(w), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
               ? NI_OK : NI_ERR_BAD_ARGUMENT;
}
static int gt_map_x(CUtensorMap* map, const float* x, int M, int H, int K, int ldx, int box_rows) {
    const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)H, (cuuint64_t)M}, strides[2] = {(cuuint64_t)K * 4, (cuuint64_t)ldx * 4};
    const cuuint32_t box[3] = {GT_BOX, 1, (cuuint32_t)box_rows}, elem[3] = {1, 1, 1};
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

// The tile and the split of K that are done first by what they measured: a k-block of 64 takes a block 0.66, 0.77, 1.02 and 1.50 us
// with 16, 32, 64 and 128 rows of x (128 weight rows; 0.74 us is what memory gives every SM for its 32 KB), a launch 6 us besides, and
// a cluster 1.5 us, 0.045 us for every row and 0.01 for every row and slice of a block's sums.  [2048, 2048] and 120 rows: 18.9 us in
// four slices of 64-row tiles, 38 whole; [2048, 8192] and 2 rows: 24.4 in six slices, 30 in four, 91 whole.
static void gt_choose(const GtParams& p, int& bt, int& splits) {
    const int slices = gt_slices(p.K);
    const long long n_tiles = (long long)((p.N + GT_ROWS - 1) / GT_ROWS) * p.H;
    double best = 0.0;
    const int want_bt = bt, want_splits = splits;
    bt = 0;
    for (int i = 0; i < 4; ++i) {
        const int b = 16 << i;
        if (want_bt ? b != want_bt : (b > 16 && b >= 2 * p.M)) continue;
        const double per_block = i == 0 ? 0.66 : i == 1 ? 0.77 : i == 2 ? 1.02 : 1.50;
        const long long units = n_tiles * ((p.M + b - 1) / b);
        for (int sp = 1; sp <= 8; ++sp) {
            if (want_splits ? sp != want_splits : sp > 1 && units * sp > 4LL * ni_sm_count()) continue;
            if (!(b == 16 ? gt_can_split<16>(p.M, p.K, sp) : b == 32 ? gt_can_split<32>(p.M, p.K, sp)
                  : b == 64 ? gt_can_split<64>(p.M, p.K, sp) : gt_can_split<128>(p.M, p.K, sp))) continue;
            const long long at_once = sp == 1 ? ni_sm_count() : gt_clusters(sp), waves = (units + at_once - 1) / at_once;
            const int mine = (slices + sp - 1) / sp, rows = p.M < b ? p.M : b;
            const double once = sp == 1 ? 0.0 : 1.5 + 0.045 * rows + 0.01 * rows * mine;
            const double us = 6.0 + waves * (once + per_block * GT_SLICE * mine);
            if (!bt || us < best) { best = us; bt = b; splits = sp; }
        }
    }
}

// One product per head: out[m, h, :] = x[m, h, :] . w[h]^T with x [M, H, K] (rows ldx floats apart), w [H, N, K], out [M, H, N].
// bt (16, 32, 64, 128) and splits (blocks that share K): 0 leaves the choice to the sizes; every choice gives the same bits.
NI_EXPORT int ni_gemm_f32_tc(const float* x, int ldx, const float* w, float* out, int M, int N, int K, int H, int bt, int splits,
                             int early, int* error, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || H <= 0) return NI_OK;
    if (K <= 0 || error == nullptr || (long long)ldx < (long long)H * K || bt < 0 || splits < 0) return NI_ERR_BAD_ARGUMENT;
    GtParams p = {x, w, out, M, N, K, H, ldx, H * N, splits, early, error};
    gt_choose(p, bt, p.splits);
    switch (bt) {
        case 16: return gt_launch_loads<16>(p, stream);
        case 32: return gt_launch_loads<32>(p, stream);
        case 64: return gt_launch_loads<64>(p, stream);
        case 128: return gt_launch_loads<128>(p, stream);
    }
    return NI_ERR_BAD_ARGUMENT;
}
