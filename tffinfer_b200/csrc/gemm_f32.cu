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
// What bounds it.  Few rows: the latency of the memory, since registers hold only the two K blocks (64 KB) on their way while the
// threads split, and not all of them: at 72 to 80 registers a thread the float32 forms spill 50 to 105 bytes (4 rows of the 8B shape's
// gate/up product, 403 MB: 91 us = 4.4 TB/s; down 58 us; as float32 FMAs, one order of summation a thread, 1.4 ms each).  Asking the L2 for the weights one chunk ahead made it slower (102 us).  Many rows: shared memory, which
// takes 6 bytes an element from the split and feeds six products, beside the products themselves (512 rows of gate/up 0.71 ms,
// 145 TFLOP/s; without the products 0.48, without the loads 0.45; FMAs at most 70).  Off 64-bit arithmetic
// (2-norm, random operands) by 2.6e-8 at K = 1, 3.1e-8 at 8, 7.0e-8 at 64, 2.3e-7 at 512, 4.8e-7 at 1,024 and 4,096; a chain of FMAs over
// all of K is by 2.6e-8, 5.4e-8, 1.4e-7, 3.9e-7, 5.7e-7 and 1.1e-6.
//
//   warps 1-16   read 8 elements of a row at a time from global memory, one or two K blocks ahead, split them and write
//                the terms to shared memory as 128-byte-swizzled K-major tiles
//   warp 0       issues the products (M = 128 weight rows on the lanes of tensor memory, BN activation rows as columns; the
//                terms of the activations lie one behind the other, so one instruction takes a term of the weights
//                times up to 256 columns of them)
//   warps 17-20  (17-24 when BN = 128) add the chunks' sums, in tensor memory again, and write the result
#define TFF_SUSPENDED_WAITS
#include "tcgen05.cuh"

namespace {

using namespace tc5;

// K blocks of 64 whose products meet in tensor memory.  What the tensor core cuts off grows with their number: with 8 an element is
// off by 4.8e-7 from K = 512 on (2-norm of random operands), a chain of FMAs by 4.0e-7 at 512 and 5.7e-7 at 1,024; with 4 by
// 2.3e-7 from K = 256 on, the chain by 2.9e-7 at 256.  Short sums so take chunks of 4, long ones half as many drains.
__host__ __device__ constexpr int chunk_blocks(int kbt) { return kbt < 16 ? 4 : 8; }

template <int BN, int NA, int NW> struct F32Cfg {
    static constexpr int kWPlane = BM * BK * 2, kAPlane = BN * BK * 2;
    static constexpr int kStageBytes = NW * kWPlane + NA * kAPlane;
    static constexpr int kFit = (220 * 1024) / kStageBytes;
    static constexpr int kStages = kFit > 4 ? 4 : kFit;
    static constexpr int kLevels = 3;               // one operand at least has three terms
    static_assert(NA == 3 || NW == 3, "a split operand");
    // tensor memory: one or two buffers of the levels' sums, then the running sum of the chunks
    static constexpr int kBufCols = kLevels * BN;
    static constexpr int kBufs = 2 * kBufCols + BN <= 512 ? 2 : 1;
    static constexpr int kSumCol = kBufs * kBufCols;
    static constexpr int kNeedCols = kSumCol + BN;
    static constexpr int kTmemCols = kNeedCols <= 32 ? 32 : kNeedCols <= 64 ? 64 : kNeedCols <= 128 ? 128 : kNeedCols <= 256 ? 256 : 512;
    // 512 threads read and split.  Few activation rows: two groups of 256 take K blocks in turn, so that two blocks are on
    // their way from memory; many: all 512 share a block, whose registers would not fit 256.
    static constexpr int kGroups = BN <= 32 ? 2 : 1, kConv = 512 / kGroups;
    static constexpr int kEpiGroups = BN >= 128 ? 2 : 1;           // groups of 4 epilogue warps; each takes BN / kEpiGroups columns
    static constexpr int kThreads = 32 + 512 + 128 * kEpiGroups;
    static constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*alignment slack*/ + 256 /*barriers*/;
    static_assert(kStages >= 2 && kNeedCols <= 512, "the configuration does not fit an SM");
};

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};"
        ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 8 consecutive elements of a row as float32; elements at or behind ``left`` are zeros (left counts from p).  The activations may have
// been written by the kernel ahead and are read past the first-level cache.  CONST: the weights, which no kernel of a step writes, on
// the read-only path, where they take no room in that cache.
template <typename T, bool VEC, bool CONST>
__device__ __forceinline__ void load8(const T* p, int left, uint32_t* r) {
    if constexpr (VEC) {                             // rows are multiples of 8 elements and aligned: all of the 8 or none
        if (left <= 0) {
#pragma unroll
            for (int i = 0; i < (sizeof(T) == 4 ? 8 : 4); ++i) r[i] = 0u;
        } else if constexpr (sizeof(T) == 4) {
            if constexpr (CONST)
                asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                             : "l"(p));
            else
                asm volatile("ld.global.cg.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                             : "l"(p) : "memory");
        } else {
            if constexpr (CONST)
                asm volatile("ld.global.nc.L1::no_allocate.v4.b32 {%0,%1,%2,%3}, [%4];"
                             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "l"(p));
            else
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

// The terms of 8 elements, 16 bytes a plane, ``plane`` bytes apart.
template <typename T>
__device__ __forceinline__ void split_store(const uint32_t* r, uint32_t dst, uint32_t plane) {
    if constexpr (sizeof(T) == 2) {
        st_shared16(dst, r);
    } else {
        uint32_t h[4], m[4], l[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {                // (the differences are exact)
            const float a = __uint_as_float(r[2 * i]), b = __uint_as_float(r[2 * i + 1]);
            h[i] = pack2(a, b);
            const float ra = a - __uint_as_float(h[i] << 16), rb = b - __uint_as_float(h[i] & 0xffff0000u);
            m[i] = pack2(ra, rb);
            l[i] = pack2(ra - __uint_as_float(m[i] << 16), rb - __uint_as_float(m[i] & 0xffff0000u));
        }
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
__global__ void __launch_bounds__(F32Cfg<BN, sizeof(TA) == 4 ? 3 : 1, sizeof(TW) == 4 ? 3 : 1>::kThreads, 1)
gemm_f32_kernel(const TA* A, const TW* W, void* out, int out_bf16, const float* residual,
                float* __restrict__ ws, int M, int N, int K, const Share sh, int* error_flag) {
    constexpr int NA = sizeof(TA) == 4 ? 3 : 1, NW = sizeof(TW) == 4 ? 3 : 1;
    using Cfg = F32Cfg<BN, NA, NW>;
    constexpr int STAGES = Cfg::kStages, BUFS = Cfg::kBufs;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gen_base = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t bars = base + STAGES * Cfg::kStageBytes;
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
    auto tfull_bar = [&](int a) { return bars + 8u * (2 * STAGES + a); };
    auto tempty_bar = [&](int a) { return bars + 8u * (2 * STAGES + 2 + a); };
    volatile uint32_t* tmem_slot = (volatile uint32_t*)(gen_base + STAGES * Cfg::kStageBytes + 8 * (2 * STAGES + 4));
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kbt = (K + BK - 1) / BK;
    const int tiles_m = (M + BN - 1) / BN;
    const int units = (N + BM - 1) / BM * sh.slices * tiles_m;             // the launcher has checked that it fits

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar(s), Cfg::kConv / 32); mbar_init(empty_bar(s), 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(tfull_bar(a), 1); mbar_init(tempty_bar(a), 4 * Cfg::kEpiGroups); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(smem_u32((const void*)tmem_slot), Cfg::kTmemCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();

    if (warp == 0) {
        if (lane == 0) {
            // -------------------------------------------------------- products
            uint32_t n = 0, chunk_no = 0;
            bool ok = true;
            for (int u = blockIdx.x; ok && u < units; u += gridDim.x) {
                const Unit it(u, tiles_m, sh, kbt, BN);
                for (int c0 = it.kb0; ok && c0 < it.kb1; c0 += sh.chunk, ++chunk_no) {
                    const uint32_t buf = chunk_no % BUFS, use = chunk_no / BUFS;
                    if (use > 0 && !mbar_wait(tempty_bar(buf), (use - 1) & 1, abort_flag)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t d = tmem_base + buf * Cfg::kBufCols;
                    const int c1 = min(c0 + sh.chunk, it.kb1);
                    for (int kb = c0; kb < c1; ++kb, ++n) {
                        const int s = n % STAGES;
                        if (!mbar_wait(full_bar(s), (n / STAGES) & 1, abort_flag)) { ok = false; break; }
                        tc_fence_after();
                        const uint32_t w_addr = base + s * Cfg::kStageBytes, a_addr = w_addr + NW * Cfg::kWPlane;
#pragma unroll
                        for (int kk = 0; kk < BK / UMMA_K; ++kk) {
                            // term i of the weights times terms 0 .. count-1 of the activations: levels i .. i+count-1
#pragma unroll
                            for (int i = 0; i < NW; ++i) {
                                constexpr int kCols = Cfg::kLevels * BN;
                                const int cols = (kCols - i * BN) < NA * BN ? (kCols - i * BN) : NA * BN;
                                const uint64_t wd = make_smem_desc(w_addr + i * Cfg::kWPlane) + (uint64_t)(kk * 2);
#pragma unroll
                                for (int c = 0; c < cols; c += 256) {
                                    const int w = (cols - c) < 256 ? (cols - c) : 256;
                                    const uint64_t ad = make_smem_desc(a_addr + c * BK * 2) + (uint64_t)(kk * 2);
                                    // the first product on a level starts it from zero: with three terms of the activations all
                                    // levels with i = 0, with one term every level with its own i
                                    const bool fresh = kb == c0 && kk == 0 && (NA == 1 || i == 0);
                                    umma_bf16(d + (uint32_t)(i * BN + c), wd, ad, make_idesc(BM, w), fresh ? 0u : 1u);
                                }
                            }
                        }
                        umma_commit(empty_bar(s));
                    }
                    if (ok) umma_commit(tfull_bar(buf));
                }
            }
        }
    } else if (warp <= 16) {
        // ------------------------------------------------- loads and splits
        constexpr int CT = Cfg::kConv, GROUPS = Cfg::kGroups, STRIDE = CT / 8;   // rows between a thread's items
        constexpr int W_ITEMS = BM * 8 / CT;                                 // 8-element items of a K block a thread
        constexpr int A_ITEMS = (BN * 8 + CT - 1) / CT;
        constexpr int WR = NW == 3 ? 8 : 4, AR = NA == 3 ? 8 : 4;            // registers an item
        const int group = (threadIdx.x - 32) / CT, t = (threadIdx.x - 32) % CT;
        const int row = t >> 3, oct = t & 7;                                 // item q: row + STRIDE * q
        const uint32_t cell = (uint32_t)row * 128u + (uint32_t)((oct ^ (row & 7)) << 4);
        uint32_t wr[W_ITEMS][WR], ar[A_ITEMS][AR];
        int u = blockIdx.x;
        Unit it(u, tiles_m, sh, kbt, BN);
        int kb = it.kb0;
        const TW* wp;                                                        // this thread's first item of the K block, and how many
        const TA* ap;                                                        // rows and elements of the operands lie from there on
        int w_rows, a_rows, left;
        auto aim = [&]() {
            left = K - (kb * BK + oct * 8);
            wp = W + ((size_t)(it.n0 + row) * K + (kb * BK + oct * 8));
            ap = A + ((size_t)(it.m0 + row) * K + (kb * BK + oct * 8));
            w_rows = N - it.n0 - row;
            a_rows = min(M - it.m0, BN) - row;
        };
        const size_t pitch = (size_t)STRIDE * K;
        auto load_w = [&](int q) { load8<TW, VEC, true>(wp + q * pitch, STRIDE * q < w_rows ? left : 0, wr[q]); };
        auto load_a = [&](int q) { load8<TA, VEC, false>(ap + q * pitch, STRIDE * q < a_rows ? left : 0, ar[q]); };
        auto has_a = [&](int q) { return (q + 1) * STRIDE <= BN || row + q * STRIDE < BN; };
        auto step = [&]() {                                                  // to the next K block of the CTA
            if (++kb >= it.kb1) {
                u += gridDim.x;
                if (u < units) { it = Unit(u, tiles_m, sh, kbt, BN); kb = it.kb0; }
            }
        };
        for (int g = 0; g < group; ++g) if (u < units) step();
        if (u < units) {
            // The L2 may fetch the first weights while the kernel ahead still runs; they are read behind it, since an operand of this
            // path may have been written by whatever came just before.
            aim();
#pragma unroll
            for (int q = 0; q < W_ITEMS; ++q)
                if (STRIDE * q < w_rows && left > 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(wp + q * pitch));
            pdl_wait();
#pragma unroll
            for (int q = 0; q < W_ITEMS; ++q) load_w(q);
#pragma unroll
            for (int q = 0; q < A_ITEMS; ++q) load_a(q);
            for (uint32_t n = group;; n += GROUPS) {
                const int s = n % STAGES;
                const uint32_t round = n / STAGES;
                if (round > 0 && !mbar_wait(empty_bar(s), (round - 1) & 1, abort_flag)) break;
                const uint32_t w_dst = base + s * Cfg::kStageBytes + cell, a_dst = w_dst + NW * Cfg::kWPlane;
                // the group's next K block: an item's registers are filled again as soon as they are stored
#pragma unroll
                for (int g = 0; g < GROUPS; ++g) if (u < units) step();
                const bool more = u < units;
                if (more) aim();
#pragma unroll
                for (int q = 0; q < W_ITEMS; ++q) {
                    split_store<TW>(wr[q], w_dst + q * STRIDE * 128, Cfg::kWPlane);
                    if (more) load_w(q);
                }
#pragma unroll
                for (int q = 0; q < A_ITEMS; ++q) {
                    if (has_a(q)) {
                        split_store<TA>(ar[q], a_dst + q * STRIDE * 128, Cfg::kAPlane);
                        if (more) load_a(q);
                    }
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(full_bar(s));
                if (!more) break;
            }
        }
    } else {
        // ------------------------------------------------------------ sums
        constexpr int COLS = BN / Cfg::kEpiGroups;
        const int q = warp & 3, first_col = ((warp - 17) >> 2) * COLS;
        const uint32_t t_lane = tmem_base + ((uint32_t)(q * 32) << 16) + first_col;
        pdl_wait();
        uint32_t chunk_no = 0;
        bool ok = true;
        for (int u = blockIdx.x; ok && u < units; u += gridDim.x) {
            const Unit it(u, tiles_m, sh, kbt, BN);
            const int n = it.n0 + q * 32 + lane;
            for (int c0 = it.kb0; c0 < it.kb1; c0 += sh.chunk, ++chunk_no) {
                const uint32_t buf = chunk_no % BUFS, use = chunk_no / BUFS;
                if (!mbar_wait(tfull_bar(buf), use & 1, abort_flag)) { ok = false; break; }
                tc_fence_after();
                const uint32_t t_addr = t_lane + buf * Cfg::kBufCols;
                const bool first = sh.slices > 1 || c0 == it.kb0, last = sh.slices > 1 || c0 + sh.chunk >= it.kb1;
#pragma unroll 1
                for (int j0 = 0; j0 < COLS; j0 += 16) {
                    uint32_t s0[16], s1[16], s2[16], sum[16];
                    tmem_ld16(t_addr + j0, s0);
                    tmem_ld16(t_addr + BN + j0, s1);
                    tmem_ld16(t_addr + 2 * BN + j0, s2);
                    if (!first) tmem_ld16(t_lane + Cfg::kSumCol + j0, sum);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) {                 // nothing below may move ahead of the wait
                        asm volatile("" : "+r"(s0[j]), "+r"(sum[j]), "+r"(s1[j]), "+r"(s2[j]));
                    }
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const float p = __uint_as_float(s0[j]) + (__uint_as_float(s1[j]) + __uint_as_float(s2[j]));
                        sum[j] = __float_as_uint(first ? p : __uint_as_float(sum[j]) + p);
                    }
                    if (!last) {
                        tmem_st16(t_lane + Cfg::kSumCol + j0, sum);
                    } else {
                        const int m1 = it.m0 + first_col + j0;
                        if (sh.slices > 1) {
                            float* p = ws + ((size_t)(c0 / sh.chunk) * M + m1) * N + n;
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                if (m1 + j < M && n < N) p[(size_t)j * N] = __uint_as_float(sum[j]);
                        } else {
                            bool bad = false;
#pragma unroll
                            for (int j = 0; j < 16; ++j) bad |= not_finite(__uint_as_float(sum[j])) && m1 + j < M;
                            if (__any_sync(0xffffffffu, bad && n < N)) {      // those are written here, from tensor memory
                                tmem_st16(t_lane + Cfg::kSumCol + j0, sum);
                                tmem_st_wait();
#pragma unroll 1
                                for (int j = 0; j < 16 && m1 + j < M; ++j) {
                                    const float x = tmem_ld1(t_lane + Cfg::kSumCol + j0 + j);
                                    const bool mine = n < N && not_finite(x);
                                    const float v = plain_dots<TA, TW>(x, mine, A + (size_t)(m1 + j) * K, W + (size_t)n * K, K);
                                    if (mine) store_result(out, out_bf16, residual, (size_t)(m1 + j) * N + n, v);
                                }
                            }
                            if (n < N) {
#pragma unroll
                                for (int j = 0; j < 16; ++j)
                                    if (m1 + j < M && !not_finite(__uint_as_float(sum[j])))
                                        store_result(out, out_bf16, residual, (size_t)(m1 + j) * N + n, __uint_as_float(sum[j]));
                            }
                        }
                    }
                    __syncwarp();
                }
                if (!last) tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty_bar(buf));
            }
        }
    }
    // ------------------------------------------------------------------ teardown
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        for (int i = 0; i < 64; ++i) __nanosleep(1000);      // products still in flight end before their operands go
        if (threadIdx.x == 0) atomicExch(error_flag, 1);
        __syncthreads();
    }
    if (warp == 0) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem_base, Cfg::kTmemCols);
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
// clocks below (reading and splitting 128 weight rows and bn activation rows, their products: fitted to 60 times of the products of the
// 8B shape at 1 to 2,048 rows); tiles run in rounds of one a SM.
F32Plan f32_plan(int M, int N, int K) {
    const int sms = tff_num_sms() > 0 ? tff_num_sms() : 148;
    const int kbt = (K + BK - 1) / BK, chunks = chunk_count(K);
    const long long tiles_n = (N + BM - 1) / BM;
    const int bns[4] = {16, 32, 64, 128};
    const double clocks[4] = {1720., 1720., 2300., 3300.};
    F32Plan best = {16, 1};
    double best_cost = 1e30;
    for (int b = 0; b < 4; ++b) {
        if (b > 0 && bns[b - 1] >= M) break;
        const long long tiles = tiles_n * ((M + bns[b] - 1) / bns[b]);
        for (int split = 0; split < (chunks > 1 ? 2 : 1); ++split) {
            const int slices = split ? chunks : 1;
            const long long rounds = (tiles * slices + sms - 1) / sms;
            // a round also starts up and drains; the partial results are written and read once more
            double cost = (double)rounds * (split ? chunk_blocks(kbt) : kbt) * clocks[b] + 3000.;
            if (split) cost += 6000. + 2.0 * slices * (double)M * N * 4. / 2600.;
            if (cost < best_cost) { best_cost = cost; best = {bns[b], slices}; }
        }
    }
    return best;
}

template <int BN, typename TA, typename TW, bool VEC>
int launch(const void* A, const void* W, void* C, int out_bf16, const float* residual, float* ws, int M, int N, int K,
           int slices, cudaStream_t stream) {
    using Cfg = F32Cfg<BN, sizeof(TA) == 4 ? 3 : 1, sizeof(TW) == 4 ? 3 : 1>;
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
    const int chunk = chunk_blocks((K + BK - 1) / BK);
    const Share sh = {slices, (chunk_count(K) + slices - 1) / slices * chunk, chunk};
    int st = tff_launch_pdl(kern, dim3((unsigned)ctas), dim3(Cfg::kThreads), (size_t)Cfg::kSmemBytes, stream, (const TA*)A,
                            (const TW*)W, C, out_bf16, residual, ws, M, N, K, sh, tff_device_error_flag());
    if (st == TFF_OK && slices > 1) {
        const long long blocks = ((long long)M * N + 1023) / 1024;
        st = tff_launch_pdl(gemm_f32_sum_kernel<TA, TW>, dim3((unsigned)blocks), dim3(256), (size_t)0, stream, (const TA*)A,
                            (const TW*)W, (const float*)ws, C, out_bf16, residual, M, N, K, chunk_count(K));
    }
    return st;
}

template <typename TA, typename TW, bool VEC>
int dispatch(const F32Plan& p, const void* A, const void* W, void* C, int out_bf16, const float* residual, float* ws, int M,
             int N, int K, cudaStream_t s) {
    switch (p.bn) {
        case 16: return launch<16, TA, TW, VEC>(A, W, C, out_bf16, residual, ws, M, N, K, p.slices, s);
        case 32: return launch<32, TA, TW, VEC>(A, W, C, out_bf16, residual, ws, M, N, K, p.slices, s);
        case 64: return launch<64, TA, TW, VEC>(A, W, C, out_bf16, residual, ws, M, N, K, p.slices, s);
        default: return launch<128, TA, TW, VEC>(A, W, C, out_bf16, residual, ws, M, N, K, p.slices, s);
    }
}

template <typename TA, typename TW>
int dispatch_vec(const F32Plan& p, const void* A, const void* W, void* C, int out_bf16, const float* residual, float* ws,
                 int M, int N, int K, cudaStream_t s) {
    // 8 elements are read at a time: rows must be multiples of 8 elements and start at multiples of 8 elements' bytes
    const bool vec = K % 8 == 0 && ((uintptr_t)A % (8 * sizeof(TA))) == 0 && ((uintptr_t)W % (8 * sizeof(TW))) == 0;
    return vec ? dispatch<TA, TW, true>(p, A, W, C, out_bf16, residual, ws, M, N, K, s)
               : dispatch<TA, TW, false>(p, A, W, C, out_bf16, residual, ws, M, N, K, s);
}

}  // namespace

// How tff_gemm_f32 runs a shape: tile width (activation rows) | slices of the K range << 16.
TFF_API int tff_gemm_f32_plan(int M, int N, int K) {
    if (M <= 0 || N <= 0 || K <= 0) return 16 | (1 << 16);
    const F32Plan p = f32_plan(M, N, K);
    return p.bn | (p.slices << 16);
}

// How many chunks of the K range have a partial result of their own (with more than one slice).
TFF_API int tff_gemm_f32_chunks(int K) { return K <= 0 ? 1 : chunk_count(K); }

// dtype codes: 0 = float32, 1 = bfloat16 (one operand at most).  ``residual`` (float32 [M, N], may alias C
// when C is float32) is added to the product when it is not null.  ``plan`` as tff_gemm_f32_plan gives it; with more than
// one slice (each of as many whole chunks, none empty) ``ws`` holds tff_gemm_f32_chunks(K) * M * N floats.
TFF_API int tff_gemm_f32(const void* A, int a_dt, const void* W, int w_dt, void* C, int c_dt, const float* residual,
                         float* ws, int M, int N, int K, int plan, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return TFF_OK;
    if (K <= 0 || (a_dt & ~1) || (w_dt & ~1) || (c_dt & ~1)) return TFF_ERR_BAD_ARGUMENT;
    const F32Plan p = {plan & 0xffff, plan >> 16};
    const int chunks = chunk_count(K);
    if ((p.bn != 16 && p.bn != 32 && p.bn != 64 && p.bn != 128) || p.slices < 1 || p.slices > chunks ||
        (long long)(p.slices - 1) * ((chunks + p.slices - 1) / p.slices) >= chunks || (p.slices > 1 && ws == nullptr))
        return TFF_ERR_BAD_ARGUMENT;
    switch (a_dt * 2 + w_dt) {
        case 0: return dispatch_vec<float, float>(p, A, W, C, c_dt, residual, ws, M, N, K, stream);
        case 1: return dispatch_vec<float, bf16>(p, A, W, C, c_dt, residual, ws, M, N, K, stream);
        case 2: return dispatch_vec<bf16, float>(p, A, W, C, c_dt, residual, ws, M, N, K, stream);
    }
    return TFF_ERR_UNSUPPORTED;                  // two bfloat16 operands: gemm_tc.cu, gemm_simt.cu
}
