// C[M, N] = A[M, K] * W[N, K]^T (+ residual) at float32 precision: the matrix product of the true 32-bit path, of
// an operand at least that is stored in float32, on the 5th-generation tensor cores.
// It stands in for the reference's dense fp32 GEMM (src/kernel/cuda/mat_mul.cu:151-660).
//
// A float32 number from 2^-110 on is the sum of three bfloat16 terms x = h + m + l, exactly: each is what is left, rounded to
// 8 bits, so that |m| <= 2^-8 and |l| <= 2^-17 of x's power of two (below 2^-110 what l loses is at most 2^-134).  Of the nine products
// of two such sums six are computed, those down to 2^-16 of the largest; the other three (ml, lm, ll) come to at most half a
// unit in the last place of the product of the two elements, of either sign.  Products of equal size are summed in accumulators
// of their own in tensor memory (S0: hh; S1: hm, mh; S2: hl, mm, lh), for a chunk of K at a time: the tensor core cuts off where it
// adds, which drifts over a long sum, so the chunks' sums S0 + (S1 + S2) are added rounded to nearest, in ascending order.
//
// Every output element goes through the same sequence of operations whatever M is, which tile it falls in and how the
// K range was shared out (a product of few rows writes every chunk's sum to a workspace and a second kernel adds
// them in the same order): its value does not depend on what else is in the batch.  An element whose result is not
// finite is computed once more as a plain sum of products, since a split of an infinity has no meaning.
//
// What bounds it.  Few rows: 128 weight rows x 64 of K (32 KB) take a CTA 0.87 us where the memory would give them in 0.74, so the walk
// through registers to tensor memory does not quite keep up, and some 5 us go to the start, the last units and the sum of the
// chunks (4 rows, weights beyond the L2: 12,288 x 2,048 in 23 us, the 8B shape's gate/up product, 403 MB, in 77 = 5.2 TB/s, its down product in
// 55; with the weights' loads in registers and their terms in shared memory 87 and 58).  Many rows: the six products, 1,152 clocks a K block of 96 rows
// at their own rate and about 1,900 here, of which some 150 are the issuing warp's wait and the rest the warps that split beside it
// (536 rows of q/k/v 134 us, of the output projection 107, against 222 and 200 before: both operands' terms then went through shared memory,
// 96 KB written and 160 KB read a K block of 128 rows, two stages of them).  So the weights' terms are the A operand in
// TENSOR MEMORY, which costs shared memory nothing, and from 64 rows on the activations' terms are made once, by a kernel of their own
// (3 us), and come by TMA.  Off 64-bit arithmetic
// (2-norm, random operands) by 2.6e-8 at K = 1, 3.1e-8 at 8, 7.0e-8 at 64, 2.3e-7 at 512, 4.8e-7 at 1,024 and 4,096; a chain of FMAs over
// all of K is by 2.6e-8, 5.4e-8, 1.4e-7, 3.9e-7, 5.7e-7 and 1.1e-6.
//
//   warp 0       loads: the weights as they are stored, and the activations' terms, by TMA (ragged rows: the warps below read for themselves)
//   warp 1       issues the products (M = 128 weight rows on the lanes of tensor memory, BN activation rows as columns; the
//                terms of the activations lie one behind the other, so one instruction takes a term of the weights
//                times up to 256 columns of them)
//   next 8 or 16 split the weights: a thread takes 16 of K of a row at a time to the lane of tensor memory that is the row's
//   next 4       (few rows, ragged rows) split the activations into 128-byte-swizzled K-major tiles
//   last 4 to 16 add the chunks' sums in registers, 32 columns a warp, and write the result
#define TFF_SUSPENDED_WAITS
#include "tcgen05.cuh"

namespace {

using namespace tc5;

// K blocks of 64 whose products meet in tensor memory.  What the tensor core cuts off grows with their number: with 8 an element is
// off by 4.8e-7 from K = 512 on (2-norm of random operands), a chain of FMAs by 4.0e-7 at 512 and 5.7e-7 at 1,024; with 4 by
// 2.3e-7 from K = 256 on, the chain by 2.9e-7 at 256.  Short sums so take chunks of 4, long ones half as many drains.
__host__ __device__ constexpr int chunk_blocks(int kbt) { return kbt < 16 ? 4 : 8; }

template <int BN, int NA, int NW, bool VEC> struct F32Cfg {
    static_assert(NA == 3 || NW == 3, "a split operand");
    static constexpr int kRawBytes = BM * BK * (NW == 3 ? 4 : 2);   // a K block of the weights as they are stored
    static constexpr int kAPlane = BN * BK * 2, kABytes = NA * kAPlane;
    static constexpr int kAStages = BN <= 32 ? 6 : BN <= 96 ? 3 : 2;
    // activations that come as their terms, by TMA: bfloat16 ones of whole rows are their own, else tiles of many rows have them made by a kernel ahead
    // (split in here they were split again for every 128 weight rows, from loads of which only one K block was on its way)
    static constexpr bool kPlanes = BN >= 64 || (VEC && NA == 1);
    static constexpr int kRawFit = (220 * 1024 - kAStages * kABytes) / kRawBytes;
    static constexpr int kRawStages = kRawFit > 6 ? 6 : kRawFit;
    // tensor memory: buffers of the levels' sums, then a ring of the weights' terms, a slot a K block (half a one when BN = 128) and in
    // it 16 of K in 8 columns, a term's behind one another.  A wait of the issuing warp costs the tensor core some 150 clocks, so it
    // waits once a slot.
    static constexpr int kLevels = 3, kBufCols = kLevels * BN, kBufs = BN <= 32 ? 2 : 1;
    static constexpr int kSlotsABlock = BN <= 96 ? 1 : 2, kSlotSteps = BK / UMMA_K / kSlotsABlock;
    static constexpr int kTermCols = 8 * kSlotSteps, kSlotCols = NW * kTermCols, kRingCol = kBufs * kBufCols;
    static constexpr int kFit = (512 - kRingCol) / kSlotCols, kSlots = kFit > 4 ? 4 : kFit;
    static constexpr int kNeedCols = kRingCol + kSlots * kSlotCols;
    static constexpr int kTmemCols = kNeedCols <= 128 ? 128 : kNeedCols <= 256 ? 256 : 512;
    static constexpr int kAWarps = kPlanes ? 0 : 4;                 // split the activations
    static constexpr int kCols = BN < 32 ? BN : 32;                 // columns of an epilogue warp
    static constexpr int kEpiWarps = BN / kCols * 4;
    // Groups of four warps that split the weights, each a quarter or a half of EVERY K block: a barrier tells a phase from the one
    // before only, so a group that left K blocks out could take a stage whose load of before is still on its way for its own.
    static constexpr int kWGroups = 30 - kAWarps - kEpiWarps >= 16 && kSlotsABlock == 1 ? 4 : 2, kGroupSteps = BK / UMMA_K / kWGroups;
    static constexpr int kWWarps = 4 * kWGroups;
    static constexpr int kFirstA = 2 + kWWarps, kFirstEpi = kFirstA + kAWarps, kThreads = 32 * (kFirstEpi + kEpiWarps);
    static constexpr int kSmemBytes = kRawStages * kRawBytes + kAStages * kABytes + 1024 /*alignment slack*/ + 512 /*barriers*/;
    static_assert(kRawStages >= 2 && kSlots >= 2 && kNeedCols <= 512 && kThreads <= 1024, "the configuration does not fit an SM");
};

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st1(uint32_t taddr, uint32_t r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%1], {%0};" ::"r"(r), "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr) : "memory");
}
// Two products of 16 of K: A from tensor memory (lane = row, one 32-bit column = two consecutive K elements), B from shared memory.
__device__ __forceinline__ void umma2_ts(uint32_t d0, uint32_t a0, uint64_t b0, uint32_t idesc0, uint32_t acc0,
                                         uint32_t d1, uint32_t a1, uint64_t b1, uint32_t idesc1, uint32_t acc1) {
    asm volatile(
        "{\n\t.reg .pred p, q, e;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %9, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%5], [%6], %7, %8, q;\n\t}"
        ::"r"(d0), "r"(a0), "l"(b0), "r"(idesc0), "r"(acc0), "r"(d1), "r"(a1), "l"(b1), "r"(idesc1), "r"(acc1) : "memory");
}
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void tma_prefetch_2d_elected(const CUtensorMap* tm, int x, int y) {
    asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
                 "@e cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];\n\t}" ::"l"(tm), "r"(x), "r"(y) : "memory");
}

// 8 consecutive elements of a row; elements at or behind ``left`` are zeros (left counts from p).  The activations may have
// been written by the kernel ahead and are read past the first-level cache.
template <typename T, bool VEC>
__device__ __forceinline__ void load8(const T* p, int left, uint32_t* r) {
    if constexpr (VEC) {                             // rows are multiples of 8 elements and aligned: all of the 8 or none
        if (left <= 0) {
#pragma unroll
            for (int i = 0; i < (sizeof(T) == 4 ? 8 : 4); ++i) r[i] = 0u;
        } else if constexpr (sizeof(T) == 4) {
            asm volatile("ld.global.cg.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                         : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                         : "l"(p) : "memory");
        } else {
            asm volatile("ld.global.cg.v4.b32 {%0,%1,%2,%3}, [%4];"
                         : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "l"(p) : "memory");
        }
    } else {
        auto one = [&](int i) { return i < left ? __float_as_uint(ldcg_f32(p + i)) : 0u; };
        if constexpr (sizeof(T) == 4) {
#pragma unroll
            for (int i = 0; i < 8; ++i) r[i] = one(i);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) r[i] = (one(2 * i) >> 16) | one(2 * i + 1);
        }
    }
}

__device__ __forceinline__ void st_shared16(uint32_t dst, const uint32_t* v) {
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {      // rounded to nearest
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// a and b less the two bfloat16 numbers of t
__device__ __forceinline__ void less2(uint32_t t, float& a, float& b) {
    asm("{\n\t.reg .b16 x, y, minus_one;\n\t"
        "mov.b32 {x, y}, %2;\n\t"
        "mov.b16 minus_one, 0xBF80;\n\t"
        "fma.rn.f32.bf16 %0, x, minus_one, %0;\n\t"
        "fma.rn.f32.bf16 %1, y, minus_one, %1;\n\t}" : "+f"(a), "+f"(b) : "r"(t));
}
// The terms of two elements, a and b, each term's two side by side.
__device__ __forceinline__ void split2(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    h = pack2(a, b);                                 // (the differences are exact)
    less2(h, a, b);
    m = pack2(a, b);
    less2(m, a, b);
    l = pack2(a, b);
}

// The terms of 8 elements, 16 bytes a plane, ``plane`` bytes apart.
template <typename T>
__device__ __forceinline__ void split_store(const uint32_t* r, uint32_t dst, uint32_t plane) {
    if constexpr (sizeof(T) == 2) {
        st_shared16(dst, r);
    } else {
        uint32_t h[4], m[4], l[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) split2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]), h[i], m[i], l[i]);
        st_shared16(dst, h);
        st_shared16(dst + plane, m);
        st_shared16(dst + 2 * plane, l);
    }
}

// Elements whose sum of split products is not finite, as plain sums of products: the warp takes the lanes that hold one in
// turn.  All lanes call it, with the rows of their own element.  (Four products' loads together and no more: with a loop that the
// compiler unrolled as it liked the kernels that call this spilled up to 200 bytes in place of 50 to 105.)
template <typename TA, typename TW>
__device__ __noinline__ float plain_dots(float v, bool mine, const TA* a, const TW* w, int K) {
    const int lane = threadIdx.x & 31;
    for (unsigned todo = __ballot_sync(0xffffffffu, mine); todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1;
        const TA* ra = (const TA*)__shfl_sync(0xffffffffu, (unsigned long long)a, src);
        const TW* rw = (const TW*)__shfl_sync(0xffffffffu, (unsigned long long)w, src);
        float s = 0.f;
        int k = lane;
#pragma unroll 1
        for (; k + 96 < K; k += 128) {
            const float a0 = ldcg_f32(ra + k), w0 = ldcg_f32(rw + k), a1 = ldcg_f32(ra + k + 32), w1 = ldcg_f32(rw + k + 32);
            const float a2 = ldcg_f32(ra + k + 64), w2 = ldcg_f32(rw + k + 64), a3 = ldcg_f32(ra + k + 96), w3 = ldcg_f32(rw + k + 96);
            s = fmaf(a0, w0, s); s = fmaf(a1, w1, s); s = fmaf(a2, w2, s); s = fmaf(a3, w3, s);
        }
#pragma unroll 1
        for (; k < K; k += 32) s = fmaf(ldcg_f32(ra + k), ldcg_f32(rw + k), s);
        s = warp_sum(s);
        if (lane == src) v = s;
    }
    return v;
}
__device__ __forceinline__ bool not_finite(float v) { return (__float_as_uint(v) & 0x7f800000u) == 0x7f800000u; }

__device__ __forceinline__ float tmem_ld1(uint32_t taddr) {
    uint32_t r;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n\ttcgen05.wait::ld.sync.aligned;" : "=r"(r) : "r"(taddr) : "memory");
    return __uint_as_float(r);
}
__device__ __forceinline__ void store_result(void* out, int out_bf16, const float* residual, size_t at, float v) {
    if (residual) v = __ldcg(residual + at) + v;
    if (out_bf16) ((bf16*)out)[at] = from_f32<bf16>(v);
    else ((float*)out)[at] = v;
}

// Which part of the product a unit is.  Units of one weight tile and K slice lie together, activation tiles fastest, and go
// round-robin to the CTAs: those that run together read the same weights.
struct Share { int slices, blocks, chunk; };      // in how many slices K is cut, K blocks a slice and a chunk
struct Unit {
    int n0, m0, kb0, kb1;
    __device__ Unit(int u, int tiles_m, const Share& sh, int kbt, int bn) {
        const int tm = u % tiles_m, v = u / tiles_m;
        n0 = v / sh.slices * BM;
        m0 = tm * bn;
        kb0 = v % sh.slices * sh.blocks;                              // (the launcher has checked that no slice is empty)
        kb1 = min(kb0 + sh.blocks, kbt);
    }
};

template <int BN, typename TA, typename TW, bool VEC>
__global__ void __launch_bounds__(F32Cfg<BN, sizeof(TA) == 4 ? 3 : 1, sizeof(TW) == 4 ? 3 : 1, VEC>::kThreads, 1)
gemm_f32_kernel(const __grid_constant__ CUtensorMap tm_w,     // weights, boxes of 128 bytes x 128 rows (VEC only)
                const __grid_constant__ CUtensorMap tm_a,     // the activations' terms, boxes of 64 x BN, one behind the other (kPlanes only)
                const TA* A, const TW* W, void* out, int out_bf16, const float* residual,
                float* __restrict__ ws, int M, int N, int K, const Share sh, int* error_flag) {
    constexpr int NA = sizeof(TA) == 4 ? 3 : 1, NW = sizeof(TW) == 4 ? 3 : 1;
    using Cfg = F32Cfg<BN, NA, NW, VEC>;
    constexpr int RAW = Cfg::kRawStages, ASTAGES = Cfg::kAStages, SLOTS = Cfg::kSlots, BUFS = Cfg::kBufs;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gen_base = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t a_base = base + RAW * Cfg::kRawBytes, bars = a_base + ASTAGES * Cfg::kABytes;
    auto raw_full = [&](int s) { return bars + 8u * s; };
    auto raw_empty = [&](int s) { return bars + 8u * (RAW + s); };
    auto a_full = [&](int s) { return bars + 8u * (2 * RAW + s); };
    auto a_empty = [&](int s) { return bars + 8u * (2 * RAW + ASTAGES + s); };
    auto w_full = [&](int s) { return bars + 8u * (2 * (RAW + ASTAGES) + s); };
    auto w_empty = [&](int s) { return bars + 8u * (2 * (RAW + ASTAGES) + SLOTS + s); };
    auto tfull_bar = [&](int a) { return bars + 8u * (2 * (RAW + ASTAGES + SLOTS) + a); };
    auto tempty_bar = [&](int a) { return bars + 8u * (2 * (RAW + ASTAGES + SLOTS) + 2 + a); };
    volatile uint32_t* tmem_slot = (volatile uint32_t*)(gen_base + (bars - base) + 8 * (2 * (RAW + ASTAGES + SLOTS) + 4));
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    static_assert(8 * (2 * (RAW + ASTAGES + SLOTS) + 4) + 8 <= 512, "room for the barriers");

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kbt = (K + BK - 1) / BK;
    const int tiles_m = (M + BN - 1) / BN;
    const int units = (N + BM - 1) / BM * sh.slices * tiles_m;             // the launcher has checked that it fits

    if (threadIdx.x == 0) {
        for (int s = 0; s < RAW; ++s) { mbar_init(raw_full(s), 1); mbar_init(raw_empty(s), Cfg::kWWarps); }
        for (int s = 0; s < ASTAGES; ++s) { mbar_init(a_full(s), Cfg::kPlanes ? 1 : Cfg::kAWarps); mbar_init(a_empty(s), 1); }
        for (int s = 0; s < SLOTS; ++s) { mbar_init(w_full(s), Cfg::kWWarps / Cfg::kSlotsABlock); mbar_init(w_empty(s), 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(tfull_bar(a), 1); mbar_init(tempty_bar(a), Cfg::kEpiWarps); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (VEC) asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_w) : "memory");
        if (Cfg::kPlanes) asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_a) : "memory");
    }
    if (warp == 1) tmem_alloc(smem_u32((const void*)tmem_slot), Cfg::kTmemCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t ring = tmem_base + Cfg::kRingCol;
    pdl_launch_dependents();

    if (warp == 0) {
        if constexpr (VEC || Cfg::kPlanes) {
            // ------------------------------------------------- the weights as they are, the activations' terms
            constexpr int HALF = 128 / (int)sizeof(TW), BOXES = BK / HALF;
            int u = blockIdx.x, kb = -1;
            uint32_t n = 0;
            // The L2 may fetch the first weights while the kernel ahead still runs; they are read behind it, since an operand of this
            // path may have been written by whatever came just before.
            for (int ahead = 0; VEC && ahead < RAW && u < units; ++ahead) {
                const Unit it(u, tiles_m, sh, kbt, BN);
                if (kb < 0) kb = it.kb0;
#pragma unroll
                for (int b = 0; b < BOXES; ++b) tma_prefetch_2d_elected(&tm_w, kb * BK + b * HALF, it.n0);
                if (++kb >= it.kb1) { u += gridDim.x; kb = -1; }
            }
            pdl_wait();
            bool ok = true;
            for (u = blockIdx.x; ok && u < units; u += gridDim.x) {
                const Unit it(u, tiles_m, sh, kbt, BN);
                for (kb = it.kb0; kb < it.kb1; ++kb, ++n) {
                    if constexpr (VEC) {
                        const int s = n % RAW;
                        const uint32_t round = n / RAW;
                        if (round > 0 && !mbar_wait_warp(raw_empty(s), (round - 1) & 1, abort_flag)) { ok = false; break; }
                        mbar_expect_tx_elected(raw_full(s), Cfg::kRawBytes);
#pragma unroll
                        for (int b = 0; b < BOXES; ++b)
                            tma_load_2d_elected(base + s * Cfg::kRawBytes + b * (BM * 128), &tm_w, raw_full(s), kb * BK + b * HALF, it.n0);
                    }
                    if constexpr (Cfg::kPlanes) {
                        const int t = n % ASTAGES;
                        const uint32_t a_round = n / ASTAGES;
                        if (a_round > 0 && !mbar_wait_warp(a_empty(t), (a_round - 1) & 1, abort_flag)) { ok = false; break; }
                        mbar_expect_tx_elected(a_full(t), Cfg::kABytes);
                        // (rows of a box behind the last one are the next term's: columns that nobody reads)
#pragma unroll
                        for (int j = 0; j < NA; ++j)
                            tma_load_2d_elected(a_base + t * Cfg::kABytes + j * Cfg::kAPlane, &tm_a, a_full(t), kb * BK, j * M + it.m0);
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ products
        uint32_t n = 0, chunk_no = 0;
        bool ok = true;
        for (int u = blockIdx.x; ok && u < units; u += gridDim.x) {
            const Unit it(u, tiles_m, sh, kbt, BN);
            for (int c0 = it.kb0; ok && c0 < it.kb1; c0 += sh.chunk, ++chunk_no) {
                const uint32_t buf = chunk_no % BUFS, use = chunk_no / BUFS;
                if (use > 0 && !mbar_wait_warp(tempty_bar(buf), (use - 1) & 1, abort_flag)) { ok = false; break; }
                tc_fence_after();
                const uint32_t d = tmem_base + buf * Cfg::kBufCols;
                const int c1 = min(c0 + sh.chunk, it.kb1);
                for (int kb = c0; ok && kb < c1; ++kb, ++n) {
                    const int s = n % ASTAGES;
                    const uint64_t adesc = make_smem_desc(a_base + s * Cfg::kABytes);
#pragma unroll
                    for (int part = 0; part < Cfg::kSlotsABlock; ++part) {
                        const uint32_t slot_no = n * Cfg::kSlotsABlock + part, slot = slot_no % SLOTS;
                        // (the warps that fill a slot have waited for the activations of its K block)
                        if (!mbar_wait_warp(w_full(slot), (slot_no / SLOTS) & 1, abort_flag)) { ok = false; break; }
                        tc_fence_after();
#pragma unroll
                        for (int step = 0; step < Cfg::kSlotSteps; ++step) {
                            const int kk = part * Cfg::kSlotSteps + step;
                            const uint32_t w0 = ring + slot * Cfg::kSlotCols + step * 8, w1 = w0 + Cfg::kTermCols, w2 = w1 + Cfg::kTermCols;
                            const uint32_t more = kb > c0 || kk > 0 ? 1u : 0u;       // the first product on a level starts it from zero
                            // term i of the weights times terms 0 .. of the activations, which lie one behind the other: levels i ..
                            const uint64_t ad = adesc + (uint64_t)(kk * 2);
                            if constexpr (NA == 3) {
                                constexpr int PART = 3 * BN <= 256 ? 3 * BN : 3 * BN / 2;
                                // the largest come last of a K block, so that the tensor core is busy for longer while the next slot is waited for
                                if (NW == 3 && kk == 3)
                                    umma2_ts(d + 2 * BN, w2, ad, make_idesc(BM, BN), 1u, d + BN, w1, ad, make_idesc(BM, 2 * BN), 1u);
                                if constexpr (PART < 3 * BN)
                                    umma2_ts(d, w0, ad, make_idesc(BM, PART), more,
                                             d + PART, w0, ad + (uint64_t)(PART * 128 >> 4), make_idesc(BM, PART), more);
                                else
                                    umma_ts(d, w0, ad, make_idesc(BM, PART), more);
                                if (NW == 3 && kk < 3)
                                    umma2_ts(d + BN, w1, ad, make_idesc(BM, 2 * BN), 1u, d + 2 * BN, w2, ad, make_idesc(BM, BN), 1u);
                            } else {
                                umma_ts(d, w0, ad, make_idesc(BM, BN), more);
                                umma2_ts(d + BN, w1, ad, make_idesc(BM, BN), more, d + 2 * BN, w2, ad, make_idesc(BM, BN), more);
                            }
                        }
                        umma_commit_elected(w_empty(slot));
                    }
                    if (ok) umma_commit_elected(a_empty(s));
                }
                if (ok) umma_commit_elected(tfull_bar(buf));
            }
        }
    } else if (warp < Cfg::kFirstA) {
        // ------------------------------------------------- the weights' terms
        // A warp holds the 32 rows whose lanes of tensor memory it reaches, a thread one row.
        constexpr int STEPS = Cfg::kGroupSteps, WR = NW == 3 ? 16 : 8;
        const int group = (warp - 2) >> 2, row = (warp & 3) * 32 + lane;
        const uint32_t t_row = ring + ((uint32_t)((warp & 3) * 32) << 16) + (Cfg::kSlotsABlock == 1 ? group * STEPS * 8 : 0);
        const uint32_t my = (uint32_t)row * 128u, sw = (uint32_t)(row & 7);
        uint32_t n = 0;                                              // K block of the CTA
        bool ok = true;
        if constexpr (!VEC) pdl_wait();
        for (int u = blockIdx.x; ok && u < units; u += gridDim.x) {
            const Unit it(u, tiles_m, sh, kbt, BN);
            for (int kb = it.kb0; kb < it.kb1; ++kb, ++n) {
                if (VEC && !mbar_wait_warp(raw_full(n % RAW), (n / RAW) & 1, abort_flag)) { ok = false; break; }
                const uint32_t slot_no = n * Cfg::kSlotsABlock + (Cfg::kSlotsABlock == 1 ? 0 : group), slot = slot_no % SLOTS;
#pragma unroll
                for (int step = 0; ok && step < STEPS; ++step) {
                    const int kk = group * STEPS + step;
                    uint32_t r[WR], t[NW][8];
                    const uint32_t src = base + (VEC ? n % RAW : 0u) * Cfg::kRawBytes + my + (NW == 3 ? (uint32_t)(kk >> 1) * (BM * 128) : 0u);
                    if constexpr (!VEC) {
                        // the warp's 32 rows, two at a time, into the cells where a load by TMA would put them
                        const int col = lane & 15, k = kb * BK + kk * UMMA_K + col, r0 = (warp & 3) * 32 + (lane >> 4);
                        const uint32_t byte = (uint32_t)(NW == 3 ? ((kk & 1) * 16 + col) * 4 : (kk * 16 + col) * 2);
                        float v[16];
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            v[i] = it.n0 + r0 + 2 * i < N && k < K ? ldcg_f32(W + ((size_t)(it.n0 + r0 + 2 * i) * K + k)) : 0.f;
                        __syncwarp();                                // (what was there has been read)
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const int r = r0 + 2 * i;
                            const uint32_t at = src - my + (uint32_t)r * 128u + ((((byte >> 4) ^ (uint32_t)(r & 7)) << 4) | (byte & 15u));
                            if constexpr (NW == 3) asm volatile("st.shared.f32 [%0], %1;" ::"r"(at), "f"(v[i]) : "memory");
                            else asm volatile("st.shared.b16 [%0], %1;" ::"r"(at), "h"((unsigned short)(__float_as_uint(v[i]) >> 16)) : "memory");
                        }
                        __syncwarp();
                    }
#pragma unroll
                    for (int c = 0; c < WR / 4; ++c) {
                        const uint32_t chunk = NW == 3 ? (uint32_t)((kk & 1) * 4 + c) : (uint32_t)(kk * 2 + c);
                        asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];"
                                     : "=r"(r[4 * c]), "=r"(r[4 * c + 1]), "=r"(r[4 * c + 2]), "=r"(r[4 * c + 3])
                                     : "r"(src + ((chunk ^ sw) << 4)) : "memory");
                    }
                    if constexpr (NW == 3) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) split2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]), t[0][i], t[1][i], t[2][i]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 8; ++i) t[0][i] = r[i];
                    }
                    if (step == 0) {
                        const uint32_t use = slot_no / SLOTS;
                        if (use > 0 && !mbar_wait_warp(w_empty(slot), (use - 1) & 1, abort_flag)) { ok = false; break; }
                        tc_fence_after();
                    }
#pragma unroll
                    for (int i = 0; i < NW; ++i) tmem_st8(t_row + slot * Cfg::kSlotCols + i * Cfg::kTermCols + step * 8, t[i]);
                }
                // the issuing warp then need not wait for the activations too
                if (!ok || !mbar_wait_warp(a_full(n % ASTAGES), (n / ASTAGES) & 1, abort_flag)) { ok = false; break; }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(w_full(slot));
                    if (VEC) mbar_arrive(raw_empty(n % RAW));
                }
            }
        }
    } else if (warp < Cfg::kFirstEpi) {
        if constexpr (!Cfg::kPlanes) {
        // ------------------------------------------------- the activations' terms
        constexpr int CT = Cfg::kAWarps * 32, STRIDE = CT / 8;               // rows between a thread's items of 8 elements
        constexpr int ITEMS = (BN * 8 + CT - 1) / CT, AR = NA == 3 ? 8 : 4;  // and registers an item
        constexpr int DEPTH = BN == 16 ? 4 : BN == 32 ? 2 : 1;               // K blocks on their way from memory
        const int t = threadIdx.x - 32 * Cfg::kFirstA;
        const int row = t >> 3, oct = t & 7;                                 // item q: row + STRIDE * q
        const uint32_t cell = (uint32_t)row * 128u + (uint32_t)((oct ^ (row & 7)) << 4);
        uint32_t ar[DEPTH][ITEMS][AR];
        int u = blockIdx.x, kb = 0, kb1 = 0, m0 = 0;                         // of the K block that is read next
        uint32_t asked = 0;
        auto begin = [&]() {
            if (u >= units) return;
            const Unit it(u, tiles_m, sh, kbt, BN);
            kb = it.kb0; kb1 = it.kb1; m0 = it.m0;
        };
        auto load = [&](int q, uint32_t* r) {
            const int m = m0 + row + STRIDE * q, k = kb * BK + oct * 8;
            load8<TA, VEC>(A + ((size_t)m * K + k), m < M && row + STRIDE * q < BN ? K - k : 0, r);
        };
        auto step = [&]() {
            ++asked;
            if (++kb >= kb1) { u += gridDim.x; begin(); }
        };
        begin();
        pdl_wait();
#pragma unroll
        for (int d = 0; d < DEPTH; ++d) {
            if (u < units) {
#pragma unroll
                for (int q = 0; q < ITEMS; ++q) load(q, ar[d][q]);
                step();
            }
        }
        bool ok = true;
        for (uint32_t n = 0; ok && n < asked;) {
#pragma unroll
            for (int d = 0; d < DEPTH; ++d, ++n) {
                if (n >= asked) break;
                const int s = n % ASTAGES;
                const uint32_t round = n / ASTAGES;
                if (round > 0 && !mbar_wait_warp(a_empty(s), (round - 1) & 1, abort_flag)) { ok = false; break; }
                const uint32_t dst = a_base + s * Cfg::kABytes + cell;
                // an item's registers are filled again as soon as they are stored
#pragma unroll
                for (int q = 0; q < ITEMS; ++q) {
                    if ((q + 1) * STRIDE <= BN || row + q * STRIDE < BN) split_store<TA>(ar[d][q], dst + q * STRIDE * 128, Cfg::kAPlane);
                    if (u < units) load(q, ar[d][q]);
                }
                if (u < units) step();
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(a_full(s));
            }
        }
        }
    } else {
        // ------------------------------------------------------------ sums
        constexpr int COLS = Cfg::kCols;
        const int q = warp & 3, first_col = ((warp - Cfg::kFirstEpi) >> 2) * COLS;
        const uint32_t t_lane = tmem_base + ((uint32_t)(q * 32) << 16) + first_col;
        float sum[COLS];
        uint32_t chunk_no = 0;
        bool ok = true;
        pdl_wait();
        for (int u = blockIdx.x; ok && u < units; u += gridDim.x) {
            const Unit it(u, tiles_m, sh, kbt, BN);
            const int n = it.n0 + q * 32 + lane, m1 = it.m0 + first_col;
            const int cols = min(M - m1, COLS);                              // columns that are rows of the result (may be none)
            for (int c0 = it.kb0; c0 < it.kb1; c0 += sh.chunk, ++chunk_no) {
                const uint32_t buf = chunk_no % BUFS, use = chunk_no / BUFS;
                if (!mbar_wait_warp(tfull_bar(buf), use & 1, abort_flag)) { ok = false; break; }
                tc_fence_after();
                const uint32_t t_addr = t_lane + buf * Cfg::kBufCols;
                const bool first = sh.slices > 1 || c0 == it.kb0, last = sh.slices > 1 || c0 + sh.chunk >= it.kb1;
#pragma unroll
                for (int j0 = 0; j0 < COLS; j0 += 8) {
                    uint32_t s0[8], s1[8], s2[8];
                    tmem_ld8(t_addr + j0, s0);
                    tmem_ld8(t_addr + BN + j0, s1);
                    tmem_ld8(t_addr + 2 * BN + j0, s2);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 8; ++j) asm volatile("" : "+r"(s0[j]), "+r"(s1[j]), "+r"(s2[j]));    // nothing below moves ahead of the wait
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float p = __uint_as_float(s0[j]) + (__uint_as_float(s1[j]) + __uint_as_float(s2[j]));
                        sum[j0 + j] = first ? p : sum[j0 + j] + p;
                    }
                }
                if (last && sh.slices == 1) {
                    bool bad = false;
#pragma unroll
                    for (int j = 0; j < COLS; ++j) bad |= not_finite(sum[j]) && j < cols;
                    if (__any_sync(0xffffffffu, bad && n < N)) {             // those are written here, from tensor memory
#pragma unroll
                        for (int j = 0; j < COLS; ++j) tmem_st1(t_addr + j, __float_as_uint(sum[j]));
                        tmem_st_wait();
#pragma unroll 1
                        for (int j = 0; j < cols; ++j) {
                            const float x = tmem_ld1(t_addr + j);
                            const bool mine = n < N && not_finite(x);
                            const float v = plain_dots<TA, TW>(x, mine, A + (size_t)(m1 + j) * K, W + (size_t)n * K, K);
                            if (mine) store_result(out, out_bf16, residual, (size_t)(m1 + j) * N + n, v);
                        }
                        __syncwarp();
#pragma unroll
                        for (int j0 = 0; j0 < COLS; j0 += 8) {               // (so that no sum is held in a register over the call)
                            uint32_t s0[8];
                            tmem_ld8(t_addr + j0, s0);
                            tmem_ld_wait();
#pragma unroll
                            for (int j = 0; j < 8; ++j) { asm volatile("" : "+r"(s0[j])); sum[j0 + j] = __uint_as_float(s0[j]); }
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty_bar(buf));
                if (!last || n >= N) {
                } else if (sh.slices > 1) {
                    float* p = ws + ((size_t)(c0 / sh.chunk) * M + m1) * N + n;
#pragma unroll
                    for (int j = 0; j < COLS; ++j)
                        if (j < cols) p[(size_t)j * N] = sum[j];
                } else {
                    // eight residuals on their way together (they may lie where the results go)
#pragma unroll
                    for (int j0 = 0; j0 < COLS; j0 += 8) {
                        if (j0 >= cols) break;
                        const size_t at = (size_t)(m1 + j0) * N + n;
                        float r[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) r[j] = residual && j0 + j < cols ? __ldcg(residual + at + (size_t)j * N) : 0.f;
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            if (j0 + j >= cols || not_finite(sum[j0 + j])) continue;
                            const float v = residual ? r[j] + sum[j0 + j] : sum[j0 + j];
                            if (out_bf16) ((bf16*)out)[at + (size_t)j * N] = from_f32<bf16>(v);
                            else ((float*)out)[at + (size_t)j * N] = v;
                        }
                    }
                }
                __syncwarp();
            }
        }
    }
    // ------------------------------------------------------------------ teardown
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        for (int i = 0; i < 64; ++i) __nanosleep(1000);      // copies and products still in flight end before their memory goes
        if (threadIdx.x == 0) atomicExch(error_flag, 1);
        __syncthreads();
    }
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem_base, Cfg::kTmemCols);
    }
}

// The terms of the activations, [3 or 1][M][pitch] bfloat16, pitch = K rounded up to 8 with zeros behind K.
template <typename TA, bool VEC>
__global__ void __launch_bounds__(256)
gemm_f32_terms_kernel(const TA* A, uint4* __restrict__ terms, int M, int K) {
    pdl_launch_dependents();
    pdl_wait();
    const int octs = (K + 7) / 8;
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x, plane = (long long)M * octs;
    if (i >= plane) return;
    const long long row = i / octs;
    const int k = (int)(i - row * octs) * 8;
    uint32_t r[8];
    load8<TA, VEC>(A + row * K + k, K - k, r);
    if constexpr (sizeof(TA) == 2) {
        terms[i] = make_uint4(r[0], r[1], r[2], r[3]);
    } else {
        uint32_t h[4], m[4], l[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) split2(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]), h[j], m[j], l[j]);
        terms[i] = make_uint4(h[0], h[1], h[2], h[3]);
        terms[plane + i] = make_uint4(m[0], m[1], m[2], m[3]);
        terms[2 * plane + i] = make_uint4(l[0], l[1], l[2], l[3]);
    }
}

// out = sum of the chunks' partial results, in ascending order (+ residual).
template <typename TA, typename TW>
__global__ void __launch_bounds__(256)
gemm_f32_sum_kernel(const TA* A, const TW* W, const float* ws, void* out, int out_bf16,
                    const float* residual, int M, int N, int K, int chunks) {
    pdl_launch_dependents();
    pdl_wait();
    const long long total = (long long)M * N, i = ((long long)blockIdx.x * 256 + threadIdx.x) * 4;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    const bool vec = (total & 3) == 0;                       // chunks then start 16-byte aligned
    const int cnt = i >= total ? 0 : (int)(total - i < 4 ? total - i : 4);
    if (vec && cnt > 0) {
        // (eight chunks' loads on their way together: one behind the other, four rows of the 8B shape's down product took 73 us, so 58)
        for (int s0 = 0; s0 < chunks; s0 += 8) {
            float4 f[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (s0 + u < chunks) f[u] = __ldcg((const float4*)(ws + (size_t)(s0 + u) * total + i));
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (s0 + u >= chunks) continue;
                if (s0 + u == 0) { v[0] = f[u].x; v[1] = f[u].y; v[2] = f[u].z; v[3] = f[u].w; }
                else { v[0] += f[u].x; v[1] += f[u].y; v[2] += f[u].z; v[3] += f[u].w; }
            }
        }
    } else {
        for (int s = 0; s < chunks; ++s) {
            float t[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) t[j] = j < cnt ? __ldcg(ws + (size_t)s * total + i + j) : 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = s == 0 ? t[j] : v[j] + t[j];
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const bool mine = j < cnt;
        const long long at = i + j;
        float x = v[j];
        if (__any_sync(0xffffffffu, mine && not_finite(x)))
            x = plain_dots<TA, TW>(x, mine && not_finite(x), A + (size_t)(at / N) * K, W + (size_t)(at % N) * K, K);
        if (mine) store_result(out, out_bf16, residual, (size_t)at, x);
    }
}

// ------------------------------------------------------------------- host side
struct F32Plan { int bn, slices; };
int chunk_count(int K) {
    const int kbt = (K + BK - 1) / BK;
    return (kbt + chunk_blocks(kbt) - 1) / chunk_blocks(kbt);
}

// Tile width and whether the K range is shared out, from M, N, K and the SM count.  A K block of a tile takes about the
// clocks below (128 weight rows split, their products with bn activation rows: fitted to 130 times of the products of the 8B shape at 4 to
// 1,000 rows), with 5,000 for the kernel that makes the activations' terms; tiles run in rounds of one a SM.  Over the four products of a
// layer at 17 row counts from 1 to 1,000 the pick takes longer than the best of all plans by nothing to 0.5 % at widths of 2,560 and
// 4,096, by 0.6 % on average and 10 % at most at 2,048 (65 rows of 12,288 x 2,048), by 0.8 % and 12 % at 1,024 (65 to 100 rows of
// 4,096 x 1,024).
F32Plan f32_plan(int M, int N, int K) {
    const int sms = tff_num_sms() > 0 ? tff_num_sms() : 148;
    const int kbt = (K + BK - 1) / BK, chunks = chunk_count(K);
    const long long tiles_n = (N + BM - 1) / BM;
    const int bns[5] = {16, 32, 64, 96, 128};
    const double clocks[5] = {1350., 1400., 1550., 1900., 2230.};
    F32Plan best = {16, 1};
    double best_cost = 1e30;
    for (int b = 0; b < 5; ++b) {
        if (b > 0 && bns[b - 1] >= M) break;
        const long long tiles = tiles_n * ((M + bns[b] - 1) / bns[b]);
        for (int split = 0; split < (chunks > 1 ? 2 : 1); ++split) {
            const int slices = split ? chunks : 1;
            const long long rounds = (tiles * slices + sms - 1) / sms;
            // a round also starts up and drains; the partial results are written and read once more
            double cost = (double)rounds * (split ? chunk_blocks(kbt) : kbt) * clocks[b] + 3000. + (bns[b] >= 64 ? 5000. : 0.);
            if (split) cost += 6000. + 2.0 * slices * (double)M * N * 4. / 2600.;
            if (cost < best_cost) { best_cost = cost; best = {bns[b], slices}; }
        }
    }
    return best;
}

// Rows whose terms are made at a time: they take 256 MB at most (or 384 rows).
int rows_at_a_time(int K) {
    const long long rows = (256ll << 20) / (6ll * ((K + 7) / 8 * 8)) / 384 * 384;              // whole tiles of every width
    return rows < 384 ? 384 : rows > (1 << 30) ? (1 << 30) : (int)rows;
}
// Floats of the chunks' partial results, in whole lines of 128 bytes.
long long partial_floats(int M, int N, int K, int slices) {
    return slices > 1 ? ((long long)chunk_count(K) * M * N + 31) / 32 * 32 : 0;
}

template <int BN, typename TA, typename TW, bool VEC>
int launch(const TA* A, const TW* W, void* C, int out_bf16, const float* residual, float* ws, int M, int N, int K,
           int slices, cudaStream_t stream) {
    using Cfg = F32Cfg<BN, sizeof(TA) == 4 ? 3 : 1, sizeof(TW) == 4 ? 3 : 1, VEC>;
    auto kern = gemm_f32_kernel<BN, TA, TW, VEC>;
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes) != cudaSuccess)
            return TFF_ERR_LAUNCH;
        configured = true;
    }
    const long long units = (long long)((N + BM - 1) / BM) * slices * ((M + BN - 1) / BN);
    long long ctas = tff_num_sms();
    if (ctas <= 0 || tff_device_error_flag() == nullptr) return TFF_ERR_LAUNCH;
    if (units + ctas >= (1ll << 31)) return TFF_ERR_UNSUPPORTED;
    if (ctas > units) ctas = units;
    CUtensorMap tm_w = {}, tm_a = {};
    if (VEC && !tff_tensor_map_2d(W, N, K, BM, 128 / (int)sizeof(TW), (int)sizeof(TW), &tm_w)) return TFF_ERR_DRIVER;
    int st = TFF_OK;
    if (Cfg::kPlanes) {
        const void* terms = A;
        const int pitch = (K + 7) / 8 * 8;
        if constexpr (sizeof(TA) == 4 || !VEC) {
            uint4* t = (uint4*)(ws + partial_floats(M, N, K, slices));
            const long long blocks = ((long long)M * (pitch / 8) + 255) / 256;
            st = tff_launch_pdl(gemm_f32_terms_kernel<TA, VEC>, dim3((unsigned)blocks), dim3(256), (size_t)0, stream, A, t, M, K);
            if (st != TFF_OK) return st;
            terms = t;
        }
        if (!tff_tensor_map_2d(terms, (long long)M * (sizeof(TA) == 4 ? 3 : 1), pitch, BN, BK, 2, &tm_a)) return TFF_ERR_DRIVER;
    }
    const int chunk = chunk_blocks((K + BK - 1) / BK);
    const Share sh = {slices, (chunk_count(K) + slices - 1) / slices * chunk, chunk};
    st = tff_launch_pdl(kern, dim3((unsigned)ctas), dim3(Cfg::kThreads), (size_t)Cfg::kSmemBytes, stream, tm_w, tm_a, A, W, C,
                        out_bf16, residual, ws, M, N, K, sh, tff_device_error_flag());
    if (st == TFF_OK && slices > 1) {
        const long long blocks = ((long long)M * N + 1023) / 1024;
        st = tff_launch_pdl(gemm_f32_sum_kernel<TA, TW>, dim3((unsigned)blocks), dim3(256), (size_t)0, stream, A, W,
                            (const float*)ws, C, out_bf16, residual, M, N, K, chunk_count(K));
    }
    return st;
}

template <typename TA, typename TW, bool VEC>
int dispatch(const F32Plan& p, const TA* A, const TW* W, void* C, int out_bf16, const float* residual, float* ws, int M,
             int N, int K, cudaStream_t s) {
    switch (p.bn) {
        case 16: return launch<16, TA, TW, VEC>(A, W, C, out_bf16, residual, ws, M, N, K, p.slices, s);
        case 32: return launch<32, TA, TW, VEC>(A, W, C, out_bf16, residual, ws, M, N, K, p.slices, s);
        case 64: return launch<64, TA, TW, VEC>(A, W, C, out_bf16, residual, ws, M, N, K, p.slices, s);
        case 96: return launch<96, TA, TW, VEC>(A, W, C, out_bf16, residual, ws, M, N, K, p.slices, s);
        default: return launch<128, TA, TW, VEC>(A, W, C, out_bf16, residual, ws, M, N, K, p.slices, s);
    }
}

// What the operands of a call decide: whether their rows can be read 8 elements at a time and by TMA (rows of a multiple of 8 elements
// that start at multiples of 8 elements' bytes), whether the activations' terms are made in the workspace (not of bfloat16 rows that TMA
// takes as they are), and how many rows a pass has (the terms of very many rows are made, and used, for some of them at a time).
struct Passes { bool vec, terms; int part; };
Passes passes_of(const F32Plan& p, const void* A, int a_dt, const void* W, int w_dt, int M, int K) {
    Passes c;
    c.vec = K % 8 == 0 && (uintptr_t)A % (a_dt == 0 ? 32 : 16) == 0 && (uintptr_t)W % (w_dt == 0 ? 32 : 16) == 0;
    c.terms = p.bn >= 64 && (a_dt == 0 || !c.vec);
    c.part = c.terms && rows_at_a_time(K) < M ? rows_at_a_time(K) : M;
    return c;
}
long long workspace_floats(const F32Plan& p, const Passes& c, int a_dt, int N, int K) {
    return partial_floats(c.part, N, K, p.slices) + (c.terms ? (long long)c.part * ((K + 7) / 8 * 4) * (a_dt == 0 ? 3 : 1) : 0);
}

template <typename TA, typename TW>
int dispatch_vec(const F32Plan& p, const Passes& c, const TA* A, const TW* W, void* C, int out_bf16, const float* residual, float* ws,
                 int M, int N, int K, cudaStream_t s) {
    const int part = c.part;
    for (int m = 0; m < M; m += part) {
        const size_t at = (size_t)m * N;
        void* out = out_bf16 ? (void*)((bf16*)C + at) : (void*)((float*)C + at);
        const float* r = residual ? residual + at : nullptr;
        const TA* a = A + (size_t)m * K;
        const int rows = M - m < part ? M - m : part;
        const int st = c.vec ? dispatch<TA, TW, true>(p, a, W, out, out_bf16, r, ws, rows, N, K, s)
                             : dispatch<TA, TW, false>(p, a, W, out, out_bf16, r, ws, rows, N, K, s);
        if (st != TFF_OK || M - m <= part) return st;
    }
    return TFF_OK;
}

}  // namespace

// How tff_gemm_f32 runs a shape: tile width (activation rows) | slices of the K range << 16.
TFF_API int tff_gemm_f32_plan(int M, int N, int K) {
    if (M <= 0 || N <= 0 || K <= 0) return 16 | (1 << 16);
    const F32Plan p = f32_plan(M, N, K);
    return p.bn | (p.slices << 16);
}

// What tff_gemm_f32 takes for these operands and this plan, as launches << 48 | floats of workspace: the chunks' partial results where
// the K range is shared out, the activations' terms (of rows_at_a_time at most) where tiles of many rows read them and the
// activations are not their own terms; a kernel each for the product, the terms and the sum of the chunks, in every pass.
TFF_API long long tff_gemm_f32_needs(const void* A, int a_dt, const void* W, int w_dt, int M, int N, int K, int plan) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    const F32Plan p = {plan & 0xffff, plan >> 16};
    const Passes c = passes_of(p, A, a_dt, W, w_dt, M, K);
    const long long launches = ((M + (long long)c.part - 1) / c.part) * (1 + (c.terms ? 1 : 0) + (p.slices > 1 ? 1 : 0));
    return launches << 48 | workspace_floats(p, c, a_dt, N, K);
}

// dtype codes: 0 = float32, 1 = bfloat16 (one operand at most).  ``residual`` (float32 [M, N], may alias C
// when C is float32) is added to the product when it is not null.  ``plan`` as tff_gemm_f32_plan gives it (slices of
// as many whole chunks each, none empty); ``ws`` holds the floats of tff_gemm_f32_needs and is 16-byte aligned (null when there are none).
TFF_API int tff_gemm_f32(const void* A, int a_dt, const void* W, int w_dt, void* C, int c_dt, const float* residual,
                         float* ws, int M, int N, int K, int plan, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return TFF_OK;
    if (K <= 0 || (a_dt & ~1) || (w_dt & ~1) || (c_dt & ~1)) return TFF_ERR_BAD_ARGUMENT;
    const F32Plan p = {plan & 0xffff, plan >> 16};
    const int chunks = chunk_count(K);
    if ((p.bn != 16 && p.bn != 32 && p.bn != 64 && p.bn != 96 && p.bn != 128) || p.slices < 1 || p.slices > chunks ||
        (long long)(p.slices - 1) * ((chunks + p.slices - 1) / p.slices) >= chunks)
        return TFF_ERR_BAD_ARGUMENT;
    const Passes c = passes_of(p, A, a_dt, W, w_dt, M, K);
    if (workspace_floats(p, c, a_dt, N, K) > 0 && (ws == nullptr || (uintptr_t)ws % 16 != 0)) return TFF_ERR_BAD_ARGUMENT;
    switch (a_dt * 2 + w_dt) {
        case 0: return dispatch_vec<float, float>(p, c, (const float*)A, (const float*)W, C, c_dt, residual, ws, M, N, K, stream);
        case 1: return dispatch_vec<float, bf16>(p, c, (const float*)A, (const bf16*)W, C, c_dt, residual, ws, M, N, K, stream);
        case 2: return dispatch_vec<bf16, float>(p, c, (const bf16*)A, (const float*)W, C, c_dt, residual, ws, M, N, K, stream);
    }
    return TFF_ERR_UNSUPPORTED;                  // two bfloat16 operands: gemm_tc.cu, gemm_simt.cu
}
