// Prompt-portion attention over the paged cache on the 5th-generation tensor cores.
//
// A CTA takes one or two tiles of 128 packed query rows (row R of a request = token R / G, head
// kvh*G + R % G) of one (request, kv head) and walks the keys in blocks of 64, once for its tiles.
// Per tile:
//   S = Q K^T     tcgen05.mma, M = 128, N = 64, K = head size; both operands K-major in 128-byte-swizzled
//                 shared memory; S (float32) in tensor memory, one buffer
//   softmax       two groups of four warps, one thread per row, which take the blocks in turn: S row from
//                 TMEM (the buffer is given back as soon as the row is in registers), causal/window mask by
//                 position, running maximum and sum in float32, probabilities to tensor memory as bfloat16
//                 pairs, a buffer a group
//   O += P V      tcgen05.mma, M = 128, N = head size, K = 64; P is the A operand in TENSOR MEMORY, V the B
//                 operand in MN-major form, exactly as TMA lays the pages down; O (float32) stays in
//                 tensor memory for the whole key walk
// O is rescaled only when a row's maximum has grown by more than 2^8 since the value the
// exponentials use (the probabilities then stay below 2^8, harmless in float32/bfloat16), so
// the read-modify-write of O in tensor memory is rare.  That reference goes from block to block through shared
// memory; each group sums its own blocks' probabilities, and the two sums meet at the end.
//   warps 0-7    softmax, rescale, epilogue of the first tile (TMEM lane quarter = warp % 4)
//   warps 8-15   the same for the second tile
//   then         TMA producer: one box a page brings its keys and values (both halves of 64 columns) into a ring of stages;
//                an issuing warp for each tile, the first of which owns the tensor memory (512 columns: of tile x, S at
//                256 x, P of the groups at 256 x + 64 and + 96, O at 256 x + 128)
// What it rests on (cycles counted in the kernel on a B200, two tiles a CTA unless said otherwise):
//   - A TMA box costs its producer about 110 cycles to issue.  With a box of 2 KB for every page, half, K and V, sixteen a
//     block, the producer alone took 1,900 cycles a block and bound the kernel whatever the rest did (8,192 tokens of 32/8
//     heads: 564 us); with one box a page, 496.
//   - S runs two blocks ahead of PV, so a group that has written P(j) finds S(j + 2) finished; P in tensor memory leaves
//     PV only V to read from shared memory (62 cycles for 128 x 128 x 16; with P there too 107).
//   - The issuing warps go through their loops with all lanes, one elected lane issuing four products at a time, and with
//     the tile's number as a constant: issued from a branch of one lane, a product cost 80 cycles instead of 48.
//   - Queries and outputs go by whole rows: a thread that took its own row touched 32 lines with every access, 10,000 of
//     the 20,000 cycles that a CTA spends around its walk (2,048 tokens 52 -> 46 us).
//   - Masked or capped scores go back through tensor memory, so that the usual block has no second path whose registers
//     meet the first one's, and a wait is one poll and one vote (1,800 -> 1,590 cycles a block; 8,192 tokens 484 -> 454 us).
// A block of two tiles then takes 1,590 cycles, of one tile 1,050, for 1,280 (640) of products and 1,024 (512) of exponentials
// at the 16 a cycle that the special-function unit gives; four softmax warps a scheduler hide each other's waits.  Tried
// without gain: blocks of 128 keys whose columns two groups share, P over S (tiles fall into step: 772 us at the time against 638);
// part of the exponentials as a polynomial on the FMA pipe (an eighth -1 %, a quarter and more slower).
// CTAs are handed out longest walk first over all kv heads.
// Same contract as the rows mode of attention_bf16.cu, which it replaces when the page size
// is 8/16/32/64.
// The dense form (tff_attention_dense) takes the keys and values of the step's own tokens from plain rows instead of the
// cache, for steps whose requests all start at position 0 (a latent attention that has made per-head keys and values of
// a whole prompt): keys of up to 192 elements, values of up to 128, one box of 64 rows per 64 columns.  A key may lie in
// two tensors: columns of its own head, and a part that all heads share (the rotated part of a latent attention), which is
// then read where it is.
// Every mbarrier wait is bounded; a timeout raises the library's error word.
// Every wait lets the hardware suspend the warp: the waiting warps share their schedulers with the softmax warps
// of the other tile, and polled they took issue slots from those (5 % of the kernel's time).
#define TFF_SUSPENDED_WAITS
#include "tcgen05.cuh"
#include "attention_common.h"
#include <type_traits>

namespace {

// mbarrier, TMA and tensor-memory wrappers shared with the product kernels
using tc5::smem_u32;
using tc5::mbar_init;
using tc5::mbar_expect_tx;
using tc5::mbar_arrive;
using tc5::mbar_wait_warp;
using tc5::umma4_bf16_elected;
using tc5::umma_commit_elected;
using tc5::tma_load_2d;
using tc5::fence_async_smem;
using tc5::tmem_alloc;
using tc5::tmem_dealloc;
using tc5::tc_fence_before;
using tc5::tc_fence_after;
using tc5::tmem_ld16;
using tc5::tmem_ld_wait;


constexpr int BLOCK_M = 128;
constexpr int BLOCK_N = 64;
constexpr int BARS_PER_TILE = 16;
constexpr float RESCALE_THRESHOLD = 8.0f;       // in log2 units

// A box of tff_tensor_map_kv_groups: a page's keys and values of a kv head, from its first group of 8 rows.
__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap* tm, uint32_t bar, int group) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %3, %3, %3, %4}], [%2];"
        ::"r"(dst), "l"(tm), "r"(bar), "r"(0), "r"(group) : "memory");
}
// 2^x on the special-function unit (float32 in and out; 2^-inf = 0)
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Four products as umma4_bf16_elected's with the A operand from tensor memory (lane = row, one 32-bit column = two consecutive K elements), B from shared memory, STEP from
// 16 of its K to the next.
template <int STEP>
__device__ __forceinline__ void umma4_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t.reg .b64 b;\n\t.reg .b32 a;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "setp.eq.b32 p, 0, 0;\n\t"
        "add.u32 a, %1, 8;\n\tadd.u64 b, %2, %5;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, p;\n\t"
        "add.u32 a, %1, 16;\n\tadd.u64 b, b, %5;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, p;\n\t"
        "add.u32 a, %1, 24;\n\tadd.u64 b, b, %5;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate), "n"(STEP) : "memory");
}
// Pairs of float32 in a 64-bit register: fma and add on a pair issue as one instruction on sm_100.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// maximum of three (one instruction on sm_100)
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Shared-memory matrix descriptor, 128-byte swizzle, 8-row groups ``sbo_bytes`` apart.  ``lbo_bytes`` is
// the distance between successive 64-element blocks along the M/N extent of an MN-major operand
// (not used by K-major operands).
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)(sbo_bytes >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// kind::f16 instruction descriptor: float32 accumulate, bfloat16 operands, A K-major; B K-major or MN-major.
__host__ __device__ constexpr uint32_t make_idesc(int m, int n, int b_mn_major) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)b_mn_major << 16) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

struct PrefillParams {
    int companion;                               // the decoded tokens' kernel follows and runs beside this one
    int requests;                                // FLAT: whose CTAs lie one behind the other in the grid
    const bf16* q; int q_row_stride;
    const int* q_start; const int* pos_start; const int* req_ids;
    const int* block_table; int table_width;
    int cache_layers, layer, page_shift;
    bf16* out;
    int nq, nkv; float scale_log2; int window;
    float scale_over_cap, cap_log2; int sink; const float* gate; const float* sink_val;   // AttnExtra, ready for the kernel
    int keep;
    int* error_flag;
    int d, dv;                           // elements of a query row and of an output row (DENSE; at most DK and DV)
    int k_halves, k_head;                // DENSE: 64-column halves of a key that come from tm_k, columns between its heads
    int r_col;                           // DENSE: first column of the shared part in tm_r
};

template <int DK, int DV, int QT>
struct PrefillCfg {
    static constexpr int kQBytes = BLOCK_M * DK * 2;                // [64-column half][128 rows][128 B]
    static constexpr int kStageBytes = BLOCK_N * (DK + DV) * 2;     // a block's keys and values
    static constexpr int kStages = DK > 128 ? (QT == 2 ? 3 : 4) : DK > 64 ? 5 : 8;
    static constexpr int kExchange = QT * 2 * BLOCK_M * 4;          // a float of every row from either group
    // Keys of more than 128 elements leave room for three stages, which S two blocks ahead of PV would hold all: their keys are then
    // given back when S has read them and their values when PV has, each with barriers of its own (2,355 tokens of 32 heads
    // of 192: 88 us a layer's attention, 108 with one barrier for both).
    static constexpr bool kApart = DK > 128;
    static constexpr int kRingBars = (kApart ? 4 : 2) * kStages;
    static constexpr int kBars = kRingBars + BARS_PER_TILE * QT;
    static constexpr int kSmem = QT * kQBytes + kStages * kStageBytes + kExchange + 8 * kBars + 16;
    static constexpr int kThreads = (8 * QT + 1 + QT) * 32;
    static_assert(kSmem <= 227 * 1024, "shared memory of the prompt attention kernel");
};

// QT: query tiles per CTA.  One while single tiles all run at once, two as soon as they are more than the SMs (launch_prefill_tiles).
// DK, DV: elements of a key and of a value (DENSE: rounded up; the query's columns beyond its own are zeros, the output's
// are not stored).  tm_cache is the cache, or the keys' rows when DENSE; tm_v and tm_r are read by the dense form only.
// FLAT: the requests' CTAs lie one behind the other in the grid's y (launch_prefill), else z is the request.
template <int DK, int DV, int QT, bool DENSE, bool FLAT>
__global__ void __launch_bounds__(PrefillCfg<DK, DV, QT>::kThreads, 1)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap tm_cache, const __grid_constant__ CUtensorMap tm_v,
                       const __grid_constant__ CUtensorMap tm_r, const PrefillParams p) {
    using Cfg = PrefillCfg<DK, DV, QT>;
    static_assert(DENSE || DK == DV, "a slot of the cache holds a key or a value");
    constexpr int KH = DK / 64, VH = DV / 64;                    // 64-column halves of a key and of a value
    constexpr int CH = DV / 8;                                   // 16-byte chunks of a value row
    constexpr int NSTAGES = Cfg::kStages, STAGE_BYTES = Cfg::kStageBytes;
    // A stage, in atoms of 8 keys x 64 columns (1 KB).  From the cache, a box a page brings keys and values: [8 keys][K, V][64-column
    // half].  DENSE: K then V, each [half][8 keys].
    constexpr int GROUP = DENSE ? 1024 : (KH + VH) * 1024;                // from 8 keys to the next 8
    constexpr int K_HALF = DENSE ? BLOCK_N * 128 : 1024, V_HALF = K_HALF;  // from a half to the next
    constexpr int V_AT = DENSE ? KH * K_HALF : KH * 1024;                  // of the stage's first values
    constexpr int TMEM_COLS = 512;                               // all of it: the allocation starts at column 0
    constexpr int LOAD_WARP = 8 * QT, ISSUE_WARP = LOAD_WARP + 1;              // behind the softmax warps
    extern __shared__ __align__(1024) uint8_t smem[];            // (the only shared memory of the kernel: it starts 1024-byte aligned)
    const uint32_t sQ = smem_u32(smem);
    const uint32_t sKV = sQ + QT * Cfg::kQBytes;
    constexpr int BARS_AT = QT * Cfg::kQBytes + NSTAGES * STAGE_BYTES + Cfg::kExchange;
    const uint32_t bars = sQ + BARS_AT;
    uint8_t* gKV = smem + QT * Cfg::kQBytes;
    volatile float* exchange = (volatile float*)(gKV + NSTAGES * STAGE_BYTES);       // [tile][group][row]
    auto kv_full = [&](int s) { return bars + 8u * s; };
    auto kv_empty = [&](int s) { return bars + 8u * (NSTAGES + s); };
    constexpr bool APART = Cfg::kApart;                          // (kv_full and kv_empty are then the keys' alone)
    auto v_full = [&](int s) { return bars + 8u * ((APART ? 2 * NSTAGES : 0) + s); };
    auto v_empty = [&](int s) { return bars + 8u * ((APART ? 3 : 1) * NSTAGES + s); };
    auto tile_bar = [&](int x, int i) { return bars + 8u * (Cfg::kRingBars + BARS_PER_TILE * x + i); };
    // S(j), P(j), PV(j) and the reference of block j report to a barrier of the group that has block j (group j % 2): who waits
    // for a barrier then waits for every one of its completions in turn, or knows that the one before is in the past, which a
    // parity wait needs.
    auto s_full = [&](int x, int g) { return tile_bar(x, g); };
    auto s_free = [&](int x) { return tile_bar(x, 2); };
    auto p_full = [&](int x, int g) { return tile_bar(x, 3 + g); };
    auto pv_done = [&](int x, int g) { return tile_bar(x, 5 + g); };
    auto q_ready = [&](int x) { return tile_bar(x, 7); };
    auto ref_bar = [&](int x, int g, int q) { return tile_bar(x, 8 + 4 * g + q); };
    volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem + BARS_AT + 8 * Cfg::kBars);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // CTAs are handed out in the order x, y, z: all kv heads of the last rows (which see the most keys)
    // first, the shortest walks last, so that the SMs finish together
    const int kvh = blockIdx.x;
    const int G = p.nq / p.nkv;

    if (tid == 0) {
        for (int s = 0; s < NSTAGES; ++s) { mbar_init(kv_full(s), 1); if (APART) mbar_init(v_full(s), 1); }
        for (int x = 0; x < QT; ++x) {
            for (int g = 0; g < 2; ++g) {
                mbar_init(s_full(x, g), 1); mbar_init(p_full(x, g), 4); mbar_init(pv_done(x, g), 1);
                for (int q = 0; q < 4; ++q) mbar_init(ref_bar(x, g, q), 1);
            }
            mbar_init(s_free(x), 4); mbar_init(q_ready(x), 8);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_cache) : "memory");
        if (DENSE) asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_v) : "memory");
    }
    if (warp == ISSUE_WARP) tmem_alloc(smem_u32((const void*)tmem_slot), TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    constexpr uint32_t tmem_base = 0;
    if (p.companion) {            // the kernel behind may read what the one ahead of both wrote
        pdl_wait();
        pdl_launch_dependents();
    } else {
        pdl_launch_dependents();
        pdl_wait();
    }

    // request geometry (q_start and pos_start come with the step's batch, read after the dependency wait all the same)
    int at = blockIdx.z, pair = (int)gridDim.y - 1 - (int)blockIdx.y;      // request and CTA of it
    if constexpr (FLAT) {
        // every warp looks for the CTA's request by itself: the tiles of 128 requests a turn, 32 in a scan
        int left = blockIdx.y;
        at = -1;
        for (int r0 = 0; r0 < p.requests && at < 0; r0 += 128) {
            int n[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int r = r0 + u * 32 + lane;
                n[u] = 0;
                if (r < p.requests) {
                    const int* start = p.q_start + (p.req_ids ? p.req_ids[r] : r);
                    n[u] = ((start[1] - start[0]) * G + QT * BLOCK_M - 1) / (QT * BLOCK_M);
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                int sum = n[u];
#pragma unroll
                for (int o = 1; o < 32; o *= 2) {
                    const int before = __shfl_up_sync(0xffffffffu, sum, o);
                    if (lane >= o) sum += before;
                }
                const unsigned behind = __ballot_sync(0xffffffffu, left < sum);
                if (behind && at < 0) {
                    const int src = __ffs(behind) - 1;
                    at = r0 + u * 32 + src;
                    pair = __shfl_sync(0xffffffffu, sum, src) - 1 - left;  // the request's last rows first, as in a grid row of its own
                }
                left -= __shfl_sync(0xffffffffu, sum, 31);
            }
        }
        if (at < 0) { at = 0; pair = 1 << 20; }                    // the grid holds a CTA a request more than there may be tiles: no rows
    }
    const int b = p.req_ids ? p.req_ids[at] : at;
    const int q0 = p.q_start[b];
    const int q_len = p.q_start[b + 1] - q0;
    const int rows_total = q_len * G;
    const int row0 = pair * QT * BLOCK_M;                         // first packed row of the CTA
    const bool active = row0 < rows_total;                        // uniform over the CTA
    const int n_act = !active ? 0 : (row0 + BLOCK_M < rows_total ? QT : 1);   // query tiles of the CTA that have rows
    const int pos0 = p.pos_start[b];
    const int first_tok = row0 / G;
    const int last_tok = min(q_len - 1, (row0 + QT * BLOCK_M - 1) / G);
    const int hi = pos0 + last_tok;                               // last key any row of the CTA sees
    const int lo_cta = p.window > 0 ? max(0, pos0 + first_tok - p.window + 1) : 0;   // first key any row sees
    const KeyWalk walk(p.keep, BLOCK_N, lo_cta / BLOCK_N, hi / BLOCK_N);
    const int nb = active ? walk.count : 0;
    const int* table = DENSE ? nullptr : p.block_table + (size_t)b * p.table_width;
    // a stage is free again when the products of every tile that has rows have read it
    if (tid == 0) {
        for (int s = 0; s < NSTAGES; ++s) {
            mbar_init(kv_empty(s), (uint32_t)(n_act > 0 ? n_act : 1));
            if (APART) mbar_init(v_empty(s), (uint32_t)(n_act > 0 ? n_act : 1));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (warp == LOAD_WARP) {
        // ------------------------------------------------------------ TMA producer
        // the block table's entries of 32 pages, one a lane, and those of the next 32: a lookup a block would be a read from
        // global memory on the way to every load
        const int ppb = DENSE ? 0 : BLOCK_N >> p.page_shift;
        const int table_end = hi >> p.page_shift;
        int chunk = -1, held = -1, ahead = -1;
        auto entry = [&](int c) {
            const int at = c * 32 + lane;
            return at <= table_end ? table[at] : -1;
        };
        for (int i = 0; i < nb; ++i) {
            const int s = i % NSTAGES;
            const uint32_t round = i / NSTAGES;
            if (round > 0 && !mbar_wait_warp(kv_empty(s), (round - 1) & 1, abort_flag)) break;
            // the queries are on their way before more than two blocks are asked for: every CTA of a wave starts with both
            if (i == 2 && !mbar_wait_warp(q_ready(0), 0, abort_flag)) break;
            const uint32_t stage = sKV + s * STAGE_BYTES;
            const int n_first = walk.block(i) * BLOCK_N;
            if constexpr (DENSE) {
                // key n of the request is row q0 + n; rows beyond the request's are another's or zeros, and masked
                if (lane == 0) mbar_expect_tx(kv_full(s), (uint32_t)(APART ? KH * K_HALF : STAGE_BYTES));
                __syncwarp();
                const int row = q0 + n_first;
                if (lane < KH) {
                    const uint32_t dst = stage + lane * K_HALF;
                    if (lane < p.k_halves) tma_load_2d(dst, &tm_cache, kv_full(s), kvh * p.k_head + lane * 64, row);
                    else tma_load_2d(dst, &tm_r, kv_full(s), p.r_col + (lane - p.k_halves) * 64, row);
                }
                if constexpr (APART) {
                    if (round > 0 && !mbar_wait_warp(v_empty(s), (round - 1) & 1, abort_flag)) break;
                    if (lane == 0) mbar_expect_tx(v_full(s), (uint32_t)(VH * V_HALF));
                    __syncwarp();
                }
                if (lane >= KH && lane < KH + VH)
                    tma_load_2d(stage + V_AT + (lane - KH) * V_HALF, &tm_v, v_full(s), kvh * p.dv + (lane - KH) * 64, row);
            } else {
                const int first = n_first >> p.page_shift;               // (a block's pages lie in one run of 32)
                if (first >> 5 != chunk) {
                    held = first >> 5 == chunk + 1 && chunk >= 0 ? ahead : entry(first >> 5);
                    chunk = first >> 5;
                    ahead = entry(chunk + 1);
                }
                const bool valid = lane >= (first & 31) && lane < (first & 31) + ppb && held >= 0;
                const unsigned mask = __ballot_sync(0xffffffffu, valid);
                if (lane == 0) mbar_expect_tx(kv_full(s), (uint32_t)__popc(mask) * (uint32_t)(GROUP << (p.page_shift - 3)));
                __syncwarp();
                if (valid) {
                    const long long row = ((((long long)held * p.cache_layers + p.layer) * 2) * p.nkv + kvh) << p.page_shift;
                    tma_load_5d(stage + (uint32_t)((lane - (first & 31)) * (GROUP << (p.page_shift - 3))), &tm_cache, kv_full(s), (int)(row >> 3));
                }
            }
        }
    } else if (warp >= ISSUE_WARP) {
        // -------------------------------------------------------------- MMA issuers, one per tile
        auto issue = [&](auto tile) {
            constexpr int x = decltype(tile)::value;
            if (x >= n_act || nb == 0) return;
            const uint32_t t_s = tmem_base + x * 256, t_o = t_s + 128;
            // descriptors are built once; a product costs one 64-bit add on each (the low bits of a
            // descriptor are the shared-memory address in units of 16 bytes)
            const uint64_t qdesc = make_smem_desc(sQ + x * Cfg::kQBytes, 16, 1024);
            const uint64_t kdesc = make_smem_desc(sKV, 16, GROUP);             // + stage * STAGE_BYTES
            const uint64_t vdesc = make_smem_desc(sKV + V_AT, V_HALF, GROUP);
            constexpr uint32_t idesc_pv = make_idesc(BLOCK_M, DV, 1);
            constexpr uint32_t idesc_s = make_idesc(BLOCK_M, BLOCK_N, 0);
            bool ok = mbar_wait_warp(q_ready(x), 0, abort_flag);
            // S runs two blocks ahead of PV: a group that has written P(j) finds S(j + 2) finished
            uint32_t phase = 0, phase_pv = 0;
            int st = 0, st_pv = 0;                                 // stages of S(n) and of PV(n - 2)
            for (int n = 0; n < nb + 2 && ok; ++n) {
                if (n < nb) {
                    ok = mbar_wait_warp(kv_full(st), phase, abort_flag);
                    if (ok && n > 0) ok = mbar_wait_warp(s_free(x), (uint32_t)(n - 1) & 1, abort_flag);   // S(n - 1) is in registers
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t kd = kdesc + (uint64_t)(st * (STAGE_BYTES >> 4));
#pragma unroll
                    for (int h = 0; h < KH; ++h)
                        umma4_bf16_elected(t_s, qdesc + (uint64_t)(h * (BLOCK_M * 128) >> 4), kd + (uint64_t)(h * K_HALF >> 4), idesc_s, h > 0 ? 1u : 0u);
                    umma_commit_elected(s_full(x, n & 1));
                    if constexpr (APART) umma_commit_elected(kv_empty(st));    // this tile has read the keys
                    if (++st == NSTAGES) { st = 0; phase ^= 1; }
                }
                const int j = n - 2;
                if (j >= 0) {
                    ok = mbar_wait_warp(p_full(x, j & 1), (uint32_t)(j >> 1) & 1, abort_flag);    // P(j) is in tensor memory
                    if constexpr (APART) { if (ok) ok = mbar_wait_warp(v_full(st_pv), phase_pv, abort_flag); }
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t vd = vdesc + (uint64_t)(st_pv * (STAGE_BYTES >> 4));
                    umma4_ts<(2 * GROUP >> 4)>(t_o, t_s + 64 + (j & 1) * 32, vd, idesc_pv, j > 0 ? 1u : 0u);
                    umma_commit_elected(pv_done(x, j & 1));                    // O holds block j; that P buffer is free
                    umma_commit_elected(v_empty(st_pv));                   // and this tile has read the stage's values (and keys)
                    if (++st_pv == NSTAGES) { st_pv = 0; phase_pv ^= 1; }
                }
            }
        };
        // (a copy of the loop a tile: with its number known, a product's operands are constants and one register a stage)
        if (warp == ISSUE_WARP) issue(std::integral_constant<int, 0>());
        else if constexpr (QT == 2) issue(std::integral_constant<int, 1>());
    } else {
        // ------------------------------------------------- softmax / rescale / epilogue
        const int x = warp >> 3, g = (warp >> 2) & 1;              // query tile and group of this warp: it has blocks g, g + 2, ...
        const int q = warp & 3;                                    // TMEM lane quarter this warp may touch
        const int r = q * 32 + lane;                               // row of the tile = TMEM lane
        const int tt = tid & 127;                                  // within the group
        const int R = row0 + x * BLOCK_M + r;
        const bool tile_active = x < n_act;
        const bool rv = tile_active && R < rows_total;
        const int pr = pos0 + R / G;
        const int lo_r = p.window > 0 ? max(0, pr - p.window + 1) : 0;
        const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + x * 256;
        const uint32_t t_s = t_row, t_p = t_row + 64 + g * 32, t_o = t_row + 128;
        // the two warps that have a row between them
        auto pair_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + x * 4 + q) : "memory"); };
        volatile float* mine = exchange + (x * 2 + g) * BLOCK_M + r;
        volatile float* other = exchange + (x * 2 + (g ^ 1)) * BLOCK_M + r;
        // Rows of 32 go to and from global memory by whole rows: a lane that took its own row would touch 32 lines with every
        // access (the queries in and the outputs out were 10,000 of a CTA's 20,000 cycles around the key walk).
        const int tok = R / G, head = kvh * G + R % G;
        const int rows_left = min(32, rows_total - (R - lane));            // rows of this warp's 32 that exist
        // the query tile: half of the columns of this warp's rows into shared memory, K-major rows of 128 bytes, swizzled
        if (tile_active) {
            constexpr int RC = DK / 16;                            // 16-byte chunks of a row that a group has
            uint4 u[RC];
#pragma unroll
            for (int i = 0; i < RC; ++i) {
                const int row = (i * 32 + lane) / RC, c = g * RC + (i * 32 + lane) % RC;
                const int t = __shfl_sync(0xffffffffu, tok, row), h = __shfl_sync(0xffffffffu, head, row);
                u[i] = make_uint4(0u, 0u, 0u, 0u);
                if (row < rows_left && (!DENSE || c * 8 < p.d))
                    u[i] = __ldcg(reinterpret_cast<const uint4*>(p.q + (size_t)(q0 + t) * p.q_row_stride + (size_t)h * (DENSE ? p.d : DK) + c * 8));
            }
            uint8_t* dst = smem + x * Cfg::kQBytes + q * 32 * 128;
#pragma unroll
            for (int i = 0; i < RC; ++i) {
                const int row = (i * 32 + lane) / RC, c = g * RC + (i * 32 + lane) % RC;
                *reinterpret_cast<uint4*>(dst + (c >> 3) * (BLOCK_M * 128) + row * 128 + (((c & 7) ^ (row & 7)) << 4)) = u[i];
            }
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(q_ready(x));
        }
        const float scale_log2 = p.cap_log2 > 0.f ? p.cap_log2 : p.scale_log2;
        float m_used = -INFINITY, l = 0.f;
        bool ok = true;
        const int nb_x = tile_active ? nb : 0;
        for (int j = g; j < nb_x && ok; j += 2) {
            ok = mbar_wait_warp(s_full(x, g), (uint32_t)(j >> 1) & 1, abort_flag);
            if (!ok) break;
            tc_fence_after();
            const int n_first = walk.block(j) * BLOCK_N;
            // Masked or capped scores are written back over the raw ones, so that the pass below is the same for every block (with the
            // scores of two paths meeting in registers, 64 moves a block).  Rows beyond the last token have queries of zeros and
            // are not stored: they need no mask.  With a cap the scores become tanh(s * scale / cap) and the multiplier of the
            // exponent cap * log2(e).
            const bool masked = !__all_sync(0xffffffffu, !rv || (n_first + BLOCK_N - 1 <= pr && (n_first >= lo_r || n_first + BLOCK_N <= p.keep)));
            if (masked || p.cap_log2 > 0.f) {
                // (in the block's own numbers, which are constants of the unrolled loops)
                const int last = rv ? pr - n_first : BLOCK_N, low = lo_r - n_first, kept = p.keep - n_first;
                uint32_t v[BLOCK_N];
#pragma unroll
                for (int h = 0; h < BLOCK_N / 16; ++h) tmem_ld16(t_s + h * 16, v + h * 16);
                tmem_ld_wait();
                if (p.cap_log2 > 0.f) {
#pragma unroll
                    for (int i = 0; i < BLOCK_N; ++i) v[i] = __float_as_uint(attn_tanh(__uint_as_float(v[i]) * p.scale_over_cap));
                }
                if (p.window == 0) {
#pragma unroll
                    for (int i = 0; i < BLOCK_N; ++i) v[i] = i <= last ? v[i] : 0xff800000u;                             // -infinity
                } else if (masked) {
#pragma unroll
                    for (int i = 0; i < BLOCK_N; ++i) v[i] = i <= last && (i >= low || i < kept) ? v[i] : 0xff800000u;
                }
#pragma unroll
                for (int h = 0; h < BLOCK_N / 16; ++h) tmem_st16(t_s + h * 16, v + h * 16);
                tmem_st_wait();
            }
            uint32_t s[BLOCK_N];
#pragma unroll
            for (int h = 0; h < BLOCK_N / 16; ++h) tmem_ld16(t_s + h * 16, s + h * 16);       // the four loads are in flight together
            tmem_ld_wait();
            tc_fence_before();                                     // the scores are in registers: the buffer may
            __syncwarp();                                          // take the next block's
            if (lane == 0) mbar_arrive(s_free(x));
            // Scores stay unscaled in registers; the scale (> 0) is folded into the exponent below.
            // (four running maxima and, below, four partial sums: chains of 16 dependent operations, not 64)
            float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int i = 0; i < BLOCK_N; i += 2) m4[(i >> 1) & 3] = fmax3(m4[(i >> 1) & 3], __uint_as_float(s[i]), __uint_as_float(s[i + 1]));
            const float m_blk = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * scale_log2;
            // The reference that the exponentials use goes from block to block, and so from group to group.  It is moved, and O and the
            // sums with it, only when the maximum has grown by more than the threshold: a decision of the whole warp.
            float m_prev = m_used;
            if (j > 0) {
                ok = mbar_wait_warp(ref_bar(x, g ^ 1, q), (uint32_t)((j - 1) >> 1) & 1, abort_flag);
                if (!ok) break;
                m_prev = *other;
            }
            const bool grow = m_blk > m_prev + RESCALE_THRESHOLD || (m_prev == -INFINITY && m_blk > -INFINITY);
            const float m_new = grow ? m_blk : m_prev;
            *mine = m_new;
            const bool moved = __any_sync(0xffffffffu, m_new != m_used);
            __syncwarp();                                          // (a vote orders no memory: every lane's reference, then the arrival)
            if (lane == 0) mbar_arrive(ref_bar(x, g, q));
            // the product of the block before last must have read the P buffer that this block writes
            if (j > 1) {
                ok = mbar_wait_warp(pv_done(x, g), (uint32_t)((j >> 1) - 1) & 1, abort_flag);
                if (!ok) break;
                tc_fence_after();
            }
            if (walk.ragged(j)) {
                // value rows no query row of the CTA may see (beyond the last key, between the kept ones and the first
                // window) are cleared, since page slots and unfetched shared memory may hold anything; the warps of both tiles
                // do it (the same zeros), so that each tile's products wait for its own warps only.
                // (S(j) has read the stage's keys: its values have landed with them, or are waited for)
                if constexpr (APART) {
                    ok = mbar_wait_warp(v_full(j % NSTAGES), (uint32_t)(j / NSTAGES) & 1, abort_flag);
                    if (!ok) break;
                }
                uint8_t* rows = gKV + (j % NSTAGES) * STAGE_BYTES + V_AT;
                for (int idx = tt; idx < BLOCK_N * CH; idx += 128) {
                    const int kr = idx / CH, c = idx % CH;
                    const int n = n_first + kr;
                    if (n > hi || (n < lo_cta && n >= p.keep))
                        *reinterpret_cast<uint4*>(rows + (c >> 3) * V_HALF + (kr >> 3) * GROUP + (kr & 7) * 128 + (((c & 7) ^ (kr & 7)) << 4)) =
                            make_uint4(0u, 0u, 0u, 0u);
                }
                fence_async_smem();
            }
            if (moved) {
                const bool any_grow = __any_sync(0xffffffffu, grow);
                if (any_grow && j > 0) {
                    // O must hold every earlier block before it is rescaled
                    ok = mbar_wait_warp(pv_done(x, g ^ 1), (uint32_t)((j - 1) >> 1) & 1, abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                    const float alpha = !grow ? 1.f : m_prev == -INFINITY ? 0.f : exp2f(m_prev - m_new);
#pragma unroll 1
                    for (int c0 = 0; c0 < DV; c0 += 16) {
                        uint32_t v[16];
                        tmem_ld16(t_o + c0, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
                        tmem_st16(t_o + c0, v);
                    }
                }
                if (m_new != m_used) l = m_used == -INFINITY ? 0.f : l * exp2f(m_used - m_new);
                m_used = m_new;
            }
            const float ms = m_used == -INFINITY ? 0.f : m_used;
            // scale, subtraction and the row's sum work on pairs of float32 (one instruction a pair)
            uint64_t lsum2[2] = {0ull, 0ull};
            const uint64_t scale2 = pack2(scale_log2, scale_log2), negms2 = pack2(-ms, -ms);
            // the probabilities, two a column
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                uint32_t w[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    float a0, a1;
                    unpack2(fma2(pack2(__uint_as_float(s[c * 32 + 2 * i]), __uint_as_float(s[c * 32 + 2 * i + 1])), scale2, negms2), a0, a1);
                    const float e0 = ex2_approx(a0), e1 = ex2_approx(a1);
                    __nv_bfloat162 b2 = __floats2bfloat162_rn(e0, e1);
                    lsum2[i & 1] = add2(lsum2[i & 1], pack2(e0, e1));
                    w[i] = *reinterpret_cast<uint32_t*>(&b2);
                }
                tmem_st16(t_p + c * 16, w);
            }
            {
                float s0, s1;
                unpack2(add2(lsum2[0], lsum2[1]), s0, s1);
                l += s0 + s1;
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full(x, g));
        }
        // ---------------------------------------------------------------- epilogue: half of the columns a group
        // the group that does not have the last block takes the last reference; the groups' sums then meet in shared memory
        const int gl = (nb_x - 1) & 1;                             // the group of the last block
        if (ok && nb_x > 0 && g != gl) {
            ok = mbar_wait_warp(ref_bar(x, gl, q), (uint32_t)((nb_x - 1) >> 1) & 1, abort_flag);
            const float m_last = *other;
            if (m_used != m_last) l = m_used == -INFINITY ? 0.f : l * exp2f(m_used - m_last);
            m_used = m_last;
            // (its own last product first: the other barrier's completion before the one that is waited for is then in the past)
            if (ok && nb_x > 1) ok = mbar_wait_warp(pv_done(x, g), (uint32_t)((nb_x - 2) >> 1) & 1, abort_flag);
        }
        if (ok && nb_x > 0) ok = mbar_wait_warp(pv_done(x, gl), (uint32_t)((nb_x - 1) >> 1) & 1, abort_flag);
        pair_sync();                                               // both have read the last references
        *mine = l;
        pair_sync();
        l = g == 0 ? l + *other : *other + l;
        if (ok && nb_x > 0) {
            tc_fence_after();
            if (p.sink && l > 0.f) l += exp2f(attn_sink_log2(p.sink_val, head) - m_used);   // the sink: a key without a value
            float inv = l > 0.f ? 1.f / l : 0.f;
            if (p.gate && rv) inv *= __ldcg(p.gate + (size_t)(q0 + tok) * p.nq + head);
            // through shared memory, where the queries lay (every S is finished), 32 rows of half a row's columns a warp
            constexpr int RC = DV / 16;
            uint8_t* rows = smem + x * Cfg::kQBytes + (g * 4 + q) * (32 * DV);
            auto cell = [&](int row, int c) { return rows + row * DV + ((c ^ (RC == 8 ? row & 7 : (row >> 1) & 3)) << 4); };
#pragma unroll
            for (int half = 0; half < RC / 4; ++half) {
                uint32_t v[32];
                tmem_ld16(t_o + g * (DV / 2) + half * 32, v);
                tmem_ld16(t_o + g * (DV / 2) + half * 32 + 16, v + 16);
                tmem_ld_wait();
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t w[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        __nv_bfloat162 b2 = __floats2bfloat162_rn(__uint_as_float(v[8 * c + 2 * i]) * inv, __uint_as_float(v[8 * c + 2 * i + 1]) * inv);
                        w[i] = *reinterpret_cast<uint32_t*>(&b2);
                    }
                    *reinterpret_cast<uint4*>(cell(lane, half * 4 + c)) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
            __syncwarp();
            const int dv = DENSE ? p.dv : DV;
#pragma unroll
            for (int i = 0; i < RC; ++i) {
                const int row = (i * 32 + lane) / RC, c = (i * 32 + lane) % RC;
                const int t = __shfl_sync(0xffffffffu, tok, row), h = __shfl_sync(0xffffffffu, head, row);
                const int col = (g * RC + c) * 8;
                if (row < rows_left && (!DENSE || col < dv))
                    *reinterpret_cast<uint4*>(p.out + ((size_t)(q0 + t) * p.nq + h) * dv + col) =
                        *reinterpret_cast<const uint4*>(cell(row, c));
            }
        }
    }
    // ------------------------------------------------------------------ teardown
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
        if (tid == 0) atomicExch(p.error_flag, 1);
        __syncthreads();
    }
    if (warp == ISSUE_WARP) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

template <int DK, int DV, int QT, bool DENSE, bool FLAT>
int launch_prefill(const CUtensorMap& tm, const CUtensorMap& tv, const CUtensorMap& tr, const PrefillParams& p, const dim3 grid,
                   cudaStream_t stream) {
    constexpr int NTHREADS = PrefillCfg<DK, DV, QT>::kThreads;
    constexpr int smem = PrefillCfg<DK, DV, QT>::kSmem;
    auto kern = attn_prefill_tc_kernel<DK, DV, QT, DENSE, FLAT>;
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
            return TFF_ERR_LAUNCH;
        configured = true;
    }
    return tff_launch_pdl(kern, grid, dim3(NTHREADS), (size_t)smem, stream, tm, tv, tr, p);
}

// The grid has a row of CTAs for every request, as many as the longest one has, or, where the step's tokens need less than three quarters
// of those, the requests' CTAs one behind the other.  A CTA without rows takes an SM for 2.6 us, one that looks for its request half a
// microsecond more: 200 prompts of 18 tokens and one of 1,000 (32/8 heads) 447 us with a row each, 127 so, 64 prompts of which one has
// 4,096 tokens and the others 20 615 and 168.
template <int DK, int DV, int QT, bool DENSE>
int launch_prefill_grid(const CUtensorMap& tm, const CUtensorMap& tv, const CUtensorMap& tr, PrefillParams p, int tiles, int num_tokens,
                        int B, cudaStream_t stream) {
    const int rows = (tiles + QT - 1) / QT;
    const long long most = (long long)num_tokens * (p.nq / p.nkv) / (QT * BLOCK_M) + B;     // every request may have a CTA that is not full
    p.requests = B;
    if (most * 4 <= (long long)rows * B * 3 && most <= 65535)
        return launch_prefill<DK, DV, QT, DENSE, true>(tm, tv, tr, p, dim3(p.nkv, (unsigned)most, 1), stream);
    return launch_prefill<DK, DV, QT, DENSE, false>(tm, tv, tr, p, dim3(p.nkv, rows, B), stream);
}

// Two query tiles a CTA share one walk over the keys: a block takes 1,590 cycles for a pair of tiles, 1,050 for a single one.  So
// single tiles while they all run at once, one an SM; as soon as they would not, pairs, which get through 1.3 times as many
// tiles in the same time.  Where no request has more than one tile a pair would have one too, and twice the warps to start.
template <int DK, int DV, bool DENSE>
int launch_prefill_tiles(const CUtensorMap& tm, const CUtensorMap& tv, const CUtensorMap& tr, const PrefillParams& p,
                         int max_q_len, int num_tokens, int B, cudaStream_t stream) {
    const int tiles = (max_q_len * (p.nq / p.nkv) + BLOCK_M - 1) / BLOCK_M;
    const long long sms = tff_num_sms() > 0 ? tff_num_sms() : 1;
    const long long most = (long long)num_tokens * (p.nq / p.nkv) / BLOCK_M + B, all = (long long)tiles * B;
    if (tiles > 1 && (most < all ? most : all) * p.nkv > sms)
        return launch_prefill_grid<DK, DV, 2, DENSE>(tm, tv, tr, p, tiles, num_tokens, B, stream);
    return launch_prefill_grid<DK, DV, 1, DENSE>(tm, tv, tr, p, tiles, num_tokens, B, stream);
}

}  // namespace

// Prompt-portion attention on tcgen05.  TFF_ERR_UNSUPPORTED when the shape is not one it takes
// (head size 64/128, page size 8/16/32/64).
int tff_attention_prefill_launch(
    const void* q, const int* q_start, const int* pos_start, const int* req_ids, const int* block_table, int table_width,
    const void* cache, long long cache_pages, int cache_layers, int layer, int page_size,
    void* out, int num_tokens, int num_requests, int max_q_len, int nq, int nkv, int d, float scale, int window, AttnExtra extra,
    cudaStream_t stream, bool companion) {
    if (d != 64 && d != 128) return TFF_ERR_UNSUPPORTED;
    if (page_size != 8 && page_size != 16 && page_size != 32 && page_size != 64) return TFF_ERR_UNSUPPORTED;
    if (cache_pages <= 0 || !(scale > 0.f)) return TFF_ERR_UNSUPPORTED;     // the kernel folds a positive scale into the exponent
    if (((uintptr_t)cache & 15) || ((uintptr_t)q & 15) || ((uintptr_t)out & 15) || (nq * d) % 8) return TFF_ERR_UNSUPPORTED;
    const long long rows = cache_pages * cache_layers * 2 * nkv * page_size;
    if (rows >= (1ll << 31) || num_requests > 65535 || (long long)max_q_len * (nq / nkv) > 65535ll * 256) return TFF_ERR_UNSUPPORTED;
    CUtensorMap tm;
    if (!tff_tensor_map_kv_groups(cache, rows, d, page_size, nkv, &tm)) return TFF_ERR_DRIVER;
    PrefillParams p;
    p.q = (const bf16*)q; p.q_row_stride = nq * d;
    p.q_start = q_start; p.pos_start = pos_start; p.req_ids = req_ids;
    p.block_table = block_table; p.table_width = table_width;
    p.cache_layers = cache_layers; p.layer = layer;
    p.page_shift = page_size == 8 ? 3 : page_size == 16 ? 4 : page_size == 32 ? 5 : 6;
    p.out = (bf16*)out;
    p.nq = nq; p.nkv = nkv; p.scale_log2 = scale * 1.4426950408889634f; p.window = window;
    p.scale_over_cap = extra.softcap > 0.f ? scale / extra.softcap : 0.f;
    p.cap_log2 = extra.softcap > 0.f ? extra.softcap * 1.4426950408889634f : 0.f;
    p.sink = extra.sink; p.gate = extra.gate; p.sink_val = extra.sink_val;
    p.keep = window > 0 ? extra.keep : 0;
    p.error_flag = tff_device_error_flag();
    if (p.error_flag == nullptr) return TFF_ERR_LAUNCH;
    p.d = p.dv = d; p.k_halves = p.k_head = p.r_col = 0;
    p.companion = companion ? 1 : 0;
    return d == 128 ? launch_prefill_tiles<128, 128, false>(tm, tm, tm, p, max_q_len, num_tokens, num_requests, stream)
                    : launch_prefill_tiles<64, 64, false>(tm, tm, tm, p, max_q_len, num_tokens, num_requests, stream);
}

// The dense form: every request of the step starts at position 0, and the keys and values of its tokens are the rows
// q_start .. of k [tokens, k_ld] (head h at columns h * k_head ..) and v [tokens, nkv * dv].  d elements of a query row
// [nq * d]: with ``shared`` (bfloat16 [tokens, shared_ld], columns r_col .. of it) a key's last d - k_head elements are the
// same for all heads and lie there, and k_head is a multiple of 64; without it k_head = d.  out [tokens, nq * dv].
// TFF_ERR_UNSUPPORTED for sizes it does not take (d <= 192, dv <= 128, all multiples of 8).
TFF_API int tff_attention_dense(const void* q, const int* q_start, const int* pos_start, const void* k, int k_ld, int k_head,
                                const void* shared, int shared_ld, int r_col, const void* v, void* out, int num_tokens,
                                int num_requests, int max_q_len, int nq, int nkv, int d, int dv, float scale, int window,
                                float softcap, const float* sink, cudaStream_t stream) {
    if (num_requests <= 0 || max_q_len <= 0 || num_tokens <= 0) return TFF_OK;
    if (!q || !k || !v || !out || nq <= 0 || nkv <= 0 || nq % nkv || d <= 0 || dv <= 0 || window < 0 || k_head <= 0 || k_head > d)
        return TFF_ERR_BAD_ARGUMENT;
    const int rest = d - k_head;
    if ((rest > 0) != (shared != nullptr) || k_ld < nkv * k_head || (shared && (r_col < 0 || r_col + rest > shared_ld)))
        return TFF_ERR_BAD_ARGUMENT;
    if (d > 192 || dv > 128 || (d & 7) || (dv & 7) || (k_ld & 7) || (k_head & 7) || !(scale > 0.f) || num_requests > 65535)
        return TFF_ERR_UNSUPPORTED;
    if (shared && (k_head % 64 || rest > 64 || (shared_ld & 7) || (r_col & 7))) return TFF_ERR_UNSUPPORTED;
    if (((uintptr_t)q & 15) || ((uintptr_t)k & 15) || ((uintptr_t)v & 15) || ((uintptr_t)out & 15) || ((uintptr_t)shared & 15))
        return TFF_ERR_UNSUPPORTED;
    if ((long long)max_q_len * (nq / nkv) > 65535ll * 256) return TFF_ERR_UNSUPPORTED;
    CUtensorMap tk, tv, tr;
    if (!tff_tensor_map_2d(k, num_tokens, k_ld, BLOCK_N, 64, 2, &tk)) return TFF_ERR_DRIVER;
    if (!tff_tensor_map_2d(v, num_tokens, (long long)nkv * dv, BLOCK_N, 64, 2, &tv)) return TFF_ERR_DRIVER;
    tr = tk;
    if (shared && !tff_tensor_map_2d(shared, num_tokens, shared_ld, BLOCK_N, 64, 2, &tr)) return TFF_ERR_DRIVER;
    PrefillParams p = {};
    p.q = (const bf16*)q; p.q_row_stride = nq * d; p.q_start = q_start; p.pos_start = pos_start;
    p.out = (bf16*)out; p.nq = nq; p.nkv = nkv; p.scale_log2 = scale * 1.4426950408889634f; p.window = window;
    p.scale_over_cap = softcap > 0.f ? scale / softcap : 0.f;
    p.cap_log2 = softcap > 0.f ? softcap * 1.4426950408889634f : 0.f;
    p.sink = sink ? 1 : 0; p.sink_val = sink;
    p.d = d; p.dv = dv; p.k_head = k_head; p.r_col = r_col;
    p.error_flag = tff_device_error_flag();
    if (p.error_flag == nullptr) return TFF_ERR_LAUNCH;
    if (d > 128) {
        p.k_halves = shared ? k_head / 64 : 3;
        return launch_prefill_tiles<192, 128, true>(tk, tv, tr, p, max_q_len, num_tokens, num_requests, stream);
    }
    p.k_halves = shared ? k_head / 64 : 2;
    return launch_prefill_tiles<128, 128, true>(tk, tv, tr, p, max_q_len, num_tokens, num_requests, stream);
}
