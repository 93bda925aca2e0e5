// Causal grouped-query attention over the paged cache for flat token rows in float32 arithmetic: any head size up to 512,
// any numbers of heads and groups, optional sliding window.  It is the attention of the true 32-bit path and takes every size
// the faster bfloat16 kernels refuse.
//
// For the token at position p of request b and query head h (kv head h / (nq/nkv),
// src/kernel/cuda/paged_flash_attention.cu:891-892):
//   s[n] = (q . k[n]) * scale for lo <= n <= p, lo = window ? max(0, p-window+1) : 0; with ``keep`` > 0 also for n < keep
//   s[n] = softcap * tanh(s[n] / softcap)                      when softcap > 0
//   out  = sum_n softmax(s)[n] * v[n]
// With ``sink`` the softmax has one more term in its denominator, a key that has no value and whose score (neither
// scaled nor capped) is sink_val[h], or 0 when sink_val is null: weights exp(s[n]) / (exp(sink) + sum exp(s)).  With ``gate`` (float32 [tokens, nq]) the head's output is multiplied by
// gate[t, h].  Keys have d elements and values dv; both lie in cache slots of dc >= max(d, dv) elements.
//
// A CTA takes a tile of packed rows (token, query head of the group) of one request and kv head and walks the keys in
// blocks of 32, which come to shared memory once for all its rows; a warp has up to 4 rows: for the scores a lane is
// a key, for the values a lane has 4 (8, 16) columns.  The running-maximum ("online") softmax of the reference
// (paged_flash_attention.cu:696-792) starts afresh every CHUNK keys, at absolute positions, and the chunks' results are
// joined in ascending order: a step of few rows behind long contexts shares the chunks out to several CTAs, of which the first
// joins its own as it goes and the others leave theirs to a second kernel, with the same operations in the same order.  A token's
// result so depends neither on how the batch was cut nor on what else is in it.
//
// What bounds it: the latency of its chains of shared-memory loads and FMAs (with 8 rows a warp and 8 warps an SM an instruction was
// issued in a third of the cycles), then those loads; for one token behind a context the chain of its chunk's blocks.  A warp a
// (token, head) that read the keys from the second-level cache, a lane a key, took 750 us for four prompts of 134 tokens
// of the 8B shape; this takes 77 (145 with 8 rows a warp).
#include "common.cuh"
#include "attention_common.h"

namespace {

constexpr int BLOCK = 32, CHUNK = 64, PER_CHUNK = CHUNK / BLOCK, JOIN_THREADS = 128;

struct GenericParams {
    const int *q_start, *pos_start, *block_table;
    int table_width, row_stride, layer, nq, nkv, d, dv, window, sink, keep, splits, slots, stages, vec, q_vec;
    float scale, softcap;
    const float *sink_val, *gate;
    float *part_o, *part_ml;
    KvLayout L;
};

// Joins a chunk's (maximum, sum) to the running ones; what the running and the chunk's outputs are to be multiplied by.
__device__ __forceinline__ void join(float& m, float& l, float mc, float lc, float& a, float& b) {
    if (mc == -INFINITY && lc == 0.f) { a = 1.f; b = 0.f; return; }      // no key of the chunk is visible
    const float mn = fmaxf(m, mc);
    a = m == -INFINITY ? 0.f : expf(m - mn);
    b = expf(mc - mn);
    l = __fmaf_rn(l, a, __fmul_rn(lc, b));
    m = mn;
}
__device__ __forceinline__ float join_value(float o, float a, float oc, float b) { return __fmaf_rn(o, a, __fmul_rn(oc, b)); }

// (what the kernels ahead wrote is read past the first-level cache)
__device__ __forceinline__ float4 load4(const float* p) { return __ldcg((const float4*)p); }
__device__ __forceinline__ float4 load4(const bf16* p) {
    const uint2 u = __ldcg((const uint2*)p);
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16),
                       __uint_as_float(u.y & 0xffff0000u));
}

// Which of a request's ``count`` chunks a share takes: the first share the first ``first`` of them, whose joined result is partial
// result 0, the others ``per`` each, every chunk a partial result of its own.  Where there is room for fewer than an even cut takes,
// the first share takes what is left.
struct Shares {
    int first, per;
    __device__ Shares(int count, int splits, int slots) {
        first = splits > 1 ? max((count + splits - 1) / splits, count - (slots - 1)) : count;
        per = splits > 1 ? (count - first + splits - 2) / (splits - 1) : 0;
    }
};

// RW rows a warp, ND groups of 128 value columns (4 a lane).
template <typename T, int WARPS, int RW, int ND>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 8 ? 2 : 1)
attention_generic_kernel(const T* q_in, const T* cache, T* __restrict__ out, const GenericParams p) {
    extern __shared__ float4 smem4[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int G = p.nq / p.nkv, kvh = blockIdx.y, split = blockIdx.z % p.splits, b = blockIdx.z / p.splits;
    const int k4 = (p.d + 3) / 4, v4 = (p.dv + 3) / 4;        // groups of 4 elements a row
    const int ks = k4 | 1;                                    // an odd pitch: 8 lanes read 8 rows' groups in all banks
    const int stage4 = BLOCK * (ks + v4);
    float4* sq = smem4 + p.stages * stage4;                   // [WARPS * RW][k4]
    float* sp = (float*)(sq + WARPS * RW * k4) + warp * RW * BLOCK;       // the warp's weights [RW][32]
    pdl_launch_dependents();
    pdl_wait();
    const int q0 = p.q_start[b], rows = (p.q_start[b + 1] - q0) * G, row0 = blockIdx.x * WARPS * RW;
    if (row0 >= rows) return;
    const int pos0 = p.pos_start[b];
    const int* table = p.block_table + (size_t)b * p.table_width;
    // what the tile's rows see
    const int first_pos = pos0 + row0 / G, hi = pos0 + (min(row0 + WARPS * RW, rows) - 1) / G;
    const int lo_tile = p.window > 0 ? max(0, first_pos - p.window + 1) : 0;
    const KeyWalk walk(p.keep, CHUNK, lo_tile / CHUNK, hi / CHUNK);
    const Shares sh(walk.count, p.splits, p.slots);
    const int w0 = split > 0 ? sh.first + (split - 1) * sh.per : 0, w1 = split > 0 ? min(walk.count, w0 + sh.per) : sh.first;
    if (w0 >= w1) return;

#pragma unroll 4
    for (int i = threadIdx.x; i < WARPS * RW * k4; i += WARPS * 32) {
        const int r = row0 + i / k4, c = (i % k4) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows) {
            const T* src = q_in + (size_t)(q0 + r / G) * p.row_stride + (size_t)(kvh * G + r % G) * p.d + c;
            if (p.q_vec) {
                v = load4(src);
            } else {
                v.x = ldcg_f32(src);
                if (c + 1 < p.d) v.y = ldcg_f32(src + 1);
                if (c + 2 < p.d) v.z = ldcg_f32(src + 2);
                if (c + 3 < p.d) v.w = ldcg_f32(src + 3);
            }
        }
        sq[i] = v;
    }

    auto live = [&](int n0) { return n0 <= hi && (n0 + BLOCK - 1 >= lo_tile || n0 < p.keep); };
    // Where key n0 + lane lies: null for keys that no row of the tile sees (their slots may hold anything, and their pages may
    // have been given back), whose stage rows become zeros.  Looked up a block ahead of the copies.
    auto locate = [&](int n0) -> const T* {
        const int n = n0 + lane;
        if (n > hi || !(n >= lo_tile || n < p.keep)) return nullptr;
        return cache + (size_t)table[n / p.L.page_size] * p.L.page_stride + (size_t)p.layer * p.L.layer_stride +
               (size_t)kvh * p.L.head_stride + (size_t)(n % p.L.page_size) * p.L.head_dim;
    };
    auto fetch = [&](const T* at, int stage) {
        float4* sk = smem4 + stage * stage4;
        float4* sv = sk + BLOCK * ks;
#pragma unroll 2
        for (int kr = warp; kr < BLOCK; kr += WARPS) {
            const T* kp = (const T*)__shfl_sync(0xffffffffu, (unsigned long long)at, kr);
            const bool ok = kp != nullptr;
            const T* vp = kp + p.L.kv_stride;
            auto row = [&](const T* src, int n4, int len, float4* dst) {
                for (int c = lane; c < n4; c += 32) {
                    if (!ok) dst[c] = make_float4(0.f, 0.f, 0.f, 0.f);
                    else if (p.vec) {                         // rows of whole, aligned groups
                        if constexpr (sizeof(T) == 4)
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                                         ::"r"((uint32_t)__cvta_generic_to_shared(dst + c)), "l"(src + c * 4) : "memory");
                        else dst[c] = load4(src + c * 4);
                    } else {
                        const T* at = src + c * 4;
                        float4 v = make_float4(ldcg_f32(at), 0.f, 0.f, 0.f);
                        if (c * 4 + 1 < len) v.y = ldcg_f32(at + 1);
                        if (c * 4 + 2 < len) v.z = ldcg_f32(at + 2);
                        if (c * 4 + 3 < len) v.w = ldcg_f32(at + 3);
                        dst[c] = v;
                    }
                }
            };
            row(kp, k4, p.d, sk + kr * ks);
            row(vp, v4, p.dv, sv + kr * v4);
        }
    };

    const int wrow = row0 + warp * RW;                        // the warp's first row
    int rp[RW], rlo[RW];                                      // positions of the rows, their windows' first keys
#pragma unroll
    for (int j = 0; j < RW; ++j) {
        rp[j] = wrow + j < rows ? pos0 + (wrow + j) / G : -1;
        rlo[j] = p.window > 0 ? max(0, rp[j] - p.window + 1) : 0;
    }
    const float inv_cap = p.softcap > 0.f ? 1.f / p.softcap : 0.f;
    float m[RW], l[RW], mc[RW], lc[RW], o[RW][4 * ND], oc[RW][4 * ND];
#pragma unroll
    for (int j = 0; j < RW; ++j) {
        // the sink is a key ahead of all others: its score starts the running maximum and the sum
        const int h = kvh * G + (wrow + j) % G;
        m[j] = p.sink ? (p.sink_val ? p.sink_val[h] : 0.f) : -INFINITY;
        l[j] = p.sink ? 1.f : 0.f;
        mc[j] = -INFINITY; lc[j] = 0.f;
#pragma unroll
        for (int c = 0; c < 4 * ND; ++c) { o[j][c] = 0.f; oc[j][c] = 0.f; }
    }

    auto partial = [&](int j, int slot, float mx, float sum, const float (&v)[4 * ND]) {
        const size_t at = ((size_t)(q0 + (wrow + j) / G) * p.nq + kvh * G + (wrow + j) % G) * p.slots + slot;
        if (lane == 0) { p.part_ml[2 * at] = mx; p.part_ml[2 * at + 1] = sum; }
#pragma unroll
        for (int c = 0; c < 4 * ND; ++c) {
            const int col = (lane + 32 * (c / 4)) * 4 + c % 4;
            if (col < p.dv) p.part_o[at * p.dv + col] = v[c];
        }
    };

    const int total = (w1 - w0) * PER_CHUNK;
    auto block_start = [&](int i) { return walk.block(w0 + i / PER_CHUNK) * CHUNK + (i % PER_CHUNK) * BLOCK; };
    const T* at = locate(block_start(0));
    if (p.stages > 1) {
        if (live(block_start(0))) fetch(at, 0);
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (total > 1) at = locate(block_start(1));
    }
    for (int i = 0; i < total; ++i) {
        const int n0 = block_start(i), stage = p.stages > 1 ? (i & 1) : 0;
        if (p.stages > 1) {
            if (i + 1 < total && live(block_start(i + 1))) fetch(at, stage ^ 1);
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (i + 2 < total) at = locate(block_start(i + 2));
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            if (live(n0)) fetch(at, 0);
            asm volatile("cp.async.wait_all;" ::: "memory");
            if (i + 1 < total) at = locate(block_start(i + 1));
        }
        __syncthreads();
        if (live(n0) && wrow < rows) {
            const float4* sk = smem4 + stage * stage4 + lane * ks;
            const float4* sv = smem4 + stage * stage4 + BLOCK * ks;
            const float4* qr = sq + warp * RW * k4;
            // ------------------------------------------------ scores: key n0 + lane against the warp's rows
            float acc[RW][4];
#pragma unroll
            for (int j = 0; j < RW; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
#pragma unroll 4
            for (int c = 0; c < k4; ++c) {
                const float4 k = sk[c];
#pragma unroll
                for (int j = 0; j < RW; ++j) {
                    const float4 q = qr[j * k4 + c];
                    acc[j][0] = fmaf(q.x, k.x, acc[j][0]);
                    acc[j][1] = fmaf(q.y, k.y, acc[j][1]);
                    acc[j][2] = fmaf(q.z, k.z, acc[j][2]);
                    acc[j][3] = fmaf(q.w, k.w, acc[j][3]);
                }
            }
            const int n = n0 + lane;
            bool whole = true;                                // every row sees every key of the block
#pragma unroll
            for (int j = 0; j < RW; ++j) {
                float s = ((acc[j][0] + acc[j][1]) + (acc[j][2] + acc[j][3])) * p.scale;
                if (p.softcap > 0.f) s = p.softcap * tanhf(s * inv_cap);
                const bool valid = n <= rp[j] && (n >= rlo[j] || n < p.keep);
                whole = whole && n0 + BLOCK - 1 <= rp[j] && (n0 >= rlo[j] || n0 + BLOCK <= p.keep);
                s = valid ? s : -INFINITY;
                const float mn = fmaxf(mc[j], warp_max(s));
                const float alpha = mc[j] == -INFINITY ? (mn == -INFINITY ? 1.f : 0.f) : expf(mc[j] - mn);
                // (a score of -infinity has no weight, also in a chunk where no other key is visible)
                const float pr = valid && s != -INFINITY ? expf(s - mn) : 0.f;
                lc[j] = lc[j] * alpha + warp_sum(pr);
                mc[j] = mn;
                if (alpha != 1.f) {
#pragma unroll
                    for (int c = 0; c < 4 * ND; ++c) oc[j][c] *= alpha;
                }
                sp[j * BLOCK + lane] = pr;
            }
            __syncwarp();
            // the keys of the block that a row sees are its first ``to[j]``, those from ``from[j]`` on or among the first ``kept``
            int to[RW], from[RW];
#pragma unroll
            for (int j = 0; j < RW; ++j) { to[j] = rp[j] - n0; from[j] = rlo[j] - n0; }
            const int kept = p.keep - n0;
            // ------------------------------------------------ values: the lane's columns of the warp's rows
#pragma unroll 1
            for (int c = 0; c < BLOCK; c += 4) {
                float4 w[RW];
#pragma unroll
                for (int j = 0; j < RW; ++j) w[j] = *(const float4*)(sp + j * BLOCK + c);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int key = c + e;
                    float4 v[ND];
#pragma unroll
                    for (int g = 0; g < ND; ++g) {
                        const int at = lane + 32 * g;
                        v[g] = at < v4 ? sv[(c + e) * v4 + at] : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
#pragma unroll
                    for (int j = 0; j < RW; ++j) {
                        // a key that the row does not see adds nothing, whatever its value is
                        if (whole || (key <= to[j] && (key >= from[j] || key < kept))) {
                        const float x = e == 0 ? w[j].x : e == 1 ? w[j].y : e == 2 ? w[j].z : w[j].w;
#pragma unroll
                        for (int g = 0; g < ND; ++g) {
                            oc[j][4 * g] = fmaf(x, v[g].x, oc[j][4 * g]);
                            oc[j][4 * g + 1] = fmaf(x, v[g].y, oc[j][4 * g + 1]);
                            oc[j][4 * g + 2] = fmaf(x, v[g].z, oc[j][4 * g + 2]);
                            oc[j][4 * g + 3] = fmaf(x, v[g].w, oc[j][4 * g + 3]);
                        }
                        }
                    }
                }
            }
            __syncwarp();
        }
        if (i % PER_CHUNK == PER_CHUNK - 1) {                 // the chunk's end
            const int slot = w0 + i / PER_CHUNK - sh.first + 1;
#pragma unroll
            for (int j = 0; j < RW; ++j) {
                if (split > 0) {
                    if (wrow + j < rows) partial(j, slot, mc[j], lc[j], oc[j]);
                } else {
                    float a, bb;
                    join(m[j], l[j], mc[j], lc[j], a, bb);
#pragma unroll
                    for (int c = 0; c < 4 * ND; ++c) o[j][c] = join_value(o[j][c], a, oc[j][c], bb);
                }
                mc[j] = -INFINITY; lc[j] = 0.f;
#pragma unroll
                for (int c = 0; c < 4 * ND; ++c) oc[j][c] = 0.f;
            }
        }
        __syncthreads();
    }
    if (split > 0) return;
#pragma unroll
    for (int j = 0; j < RW; ++j) {
        if (wrow + j >= rows) continue;
        if (p.splits > 1) { partial(j, 0, m[j], l[j], o[j]); continue; }
        const int h = kvh * G + (wrow + j) % G;
        const size_t t = q0 + (wrow + j) / G;
        const float inv = (p.gate ? __ldcg(p.gate + t * p.nq + h) : 1.f) / l[j];
#pragma unroll
        for (int c = 0; c < 4 * ND; ++c) {
            const int col = (lane + 32 * (c / 4)) * 4 + c % 4;
            if (col < p.dv) out[(t * p.nq + h) * p.dv + col] = from_f32<T>(o[j][c] * inv);
        }
    }
}

// Joins the chunks of the other shares to the first share's result, in ascending order: a block per (token, head), a thread a column (of every JOIN_THREADS), eight chunks' loads
// on their way together.  The rows of a request are one tile.
template <typename T>
__global__ void __launch_bounds__(JOIN_THREADS)
attention_generic_join_kernel(T* __restrict__ out, const int* __restrict__ tok_req, const GenericParams p) {
    pdl_launch_dependents();
    pdl_wait();
    const int item = blockIdx.x, t = item / p.nq, h = item % p.nq, b = tok_req[t];
    const int pos0 = p.pos_start[b], q_len = p.q_start[b + 1] - p.q_start[b];
    const int lo_tile = p.window > 0 ? max(0, pos0 - p.window + 1) : 0;
    const KeyWalk walk(p.keep, CHUNK, lo_tile / CHUNK, (pos0 + q_len - 1) / CHUNK);
    const int count = walk.count - Shares(walk.count, p.splits, p.slots).first + 1;
    const float* ml = p.part_ml + (size_t)item * p.slots * 2;
    for (int col = threadIdx.x; col < p.dv; col += JOIN_THREADS) {
        const float* po = p.part_o + (size_t)item * p.slots * p.dv + col;
        float m = __ldcg(ml), l = __ldcg(ml + 1), o = __ldcg(po);
        for (int w0 = 1; w0 < count; w0 += 8) {
            float2 x[8];
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (w0 + u >= count) continue;
                x[u] = __ldcg((const float2*)(ml + 2 * (w0 + u)));
                v[u] = __ldcg(po + (size_t)(w0 + u) * p.dv);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (w0 + u >= count) continue;
                float a, bb;
                join(m, l, x[u].x, x[u].y, a, bb);
                o = join_value(o, a, v[u], bb);
            }
        }
        out[(size_t)item * p.dv + col] = from_f32<T>(o * ((p.gate ? __ldcg(p.gate + item) : 1.f) / l));
    }
}

template <typename T, int WARPS, int RW, int ND>
int launch(const void* q, const void* cache, void* out, GenericParams p, int num_requests, int max_q_len, cudaStream_t s) {
    auto kern = attention_generic_kernel<T, WARPS, RW, ND>;
    const int k4 = (p.d + 3) / 4, v4 = (p.dv + 3) / 4;
    const size_t stage = (size_t)BLOCK * ((k4 | 1) + v4) * 16;
    const size_t rest = (size_t)WARPS * RW * k4 * 16 + (size_t)WARPS * RW * BLOCK * 4;
    p.stages = 2 * stage + rest <= 200 * 1024 ? 2 : 1;
    const size_t smem = p.stages * stage + rest;
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess) return TFF_ERR_LAUNCH;
        configured = true;
    }
    const long long rows = (long long)max_q_len * (p.nq / p.nkv);
    if (smem > 200 * 1024 || (p.splits > 1 && (long long)num_requests * p.splits > 65535) || p.nkv > 65535) return TFF_ERR_UNSUPPORTED;
    int st = TFF_OK;
    for (int done = 0; done < num_requests && st == TFF_OK; done += 65535) {        // (a grid is 65,535 deep)
        const int n = num_requests - done < 65535 ? num_requests - done : 65535;
        st = tff_launch_pdl(kern, dim3((unsigned)((rows + WARPS * RW - 1) / (WARPS * RW)), p.nkv, (unsigned)(n * p.splits)), dim3(WARPS * 32),
                            smem, s, (const T*)q, (const T*)cache, (T*)out, p);
        p.q_start += n; p.pos_start += n; p.block_table += (size_t)n * p.table_width;
    }
    return st;
}

template <typename T>
int dispatch(const void* q, const void* cache, void* out, const GenericParams& p, int num_requests, int max_q_len, cudaStream_t s) {
    // The warps share the keys in shared memory; a warp takes as many rows as the step has and as its registers hold columns.  32 rows
    // are 8 warps of 4 and not 4 of 8: two shared-memory wavefronts for 4 FMAs instead of 1.5, but twice the warps in flight.
    const long long rows = (long long)max_q_len * (p.nq / p.nkv);
    if (p.dv <= 128) {
        if (rows <= 4) return launch<T, 4, 1, 1>(q, cache, out, p, num_requests, max_q_len, s);
        if (rows <= 8) return launch<T, 8, 1, 1>(q, cache, out, p, num_requests, max_q_len, s);
        if (rows <= 16) return launch<T, 8, 2, 1>(q, cache, out, p, num_requests, max_q_len, s);
        return launch<T, 8, 4, 1>(q, cache, out, p, num_requests, max_q_len, s);
    }
    if (p.dv <= 256) {
        if (rows <= 4) return launch<T, 4, 1, 2>(q, cache, out, p, num_requests, max_q_len, s);
        return launch<T, 8, 2, 2>(q, cache, out, p, num_requests, max_q_len, s);
    }
    if (rows <= 4) return launch<T, 4, 1, 4>(q, cache, out, p, num_requests, max_q_len, s);
    return launch<T, 8, 1, 4>(q, cache, out, p, num_requests, max_q_len, s);
}

// Rows that may be one tile whatever the head size is: what a step's chunks may be shared out for.
int tile_rows(int dv) { return dv <= 128 ? 32 : dv <= 256 ? 16 : 8; }

}  // namespace

// What the partial results of a step may take at most.  A step captured for block tables of 40,960 tokens would want 85 MB for 16 requests of 32
// heads of 128, of a memory that the cache's budget leaves to graphs and activations; the first share then takes 389 of the 640 chunks.
constexpr long long MOST_PARTIALS = 64ll << 20;

// In how many shares (low 16 bits) the chunks of a step's keys go to different CTAs, and for how many partial results of dv + 2
// floats per (token, head) there must be room (above).  One share and no room for steps of long
// portions and for steps with enough requests: two CTAs an SM.  ``max_kv`` bounds the contexts.
TFF_API int tff_attention_generic_plan(int num_requests, int max_q_len, int max_kv, int nq, int nkv, int dv, int window, int keep,
                                       int sms) {
    if (num_requests <= 0 || max_q_len <= 0 || max_kv <= 0 || nkv <= 0 || nq % nkv || sms <= 0) return 1;
    if ((long long)max_q_len * (nq / nkv) > tile_rows(dv)) return 1;
    long long chunks = (max_kv + CHUNK - 1) / CHUNK;
    if (window > 0) {
        const long long seen = ((long long)window + max_q_len + CHUNK - 1) / CHUNK + 1 + (keep > 0 ? (keep + CHUNK - 1) / CHUNK : 0);
        chunks = chunks < seen ? chunks : seen;
    }
    const long long ctas = (long long)num_requests * nkv;
    long long splits = 2ll * sms / ctas;
    if (splits > chunks) splits = chunks;
    if (splits < 2 || num_requests * splits > 65535) return 1;
    long long slots = chunks - (chunks + splits - 1) / splits + 1;
    const long long most = MOST_PARTIALS / ((long long)num_requests * max_q_len * nq * (dv + 2) * 4);
    if (slots > most) slots = most;
    if (slots > 32767) slots = 32767;
    return slots < 2 ? 1 : (int)(splits | (slots << 16));
}

// Keys of d and values of dv elements in cache slots of dc, score cap, sink, head gates.  ``plan`` as
// tff_attention_generic_plan gives it; with more than one share ``ws`` holds tokens * nq * slots * (dv + 2) floats.
TFF_API int tff_attention_generic(
    const void* qkv, int is_bf16, int row_stride, const int* tok_req, const int* q_start, const int* pos_start, int num_requests,
    int max_q_len, const int* block_table, int table_width,
    const void* cache, int cache_layers, int layer, int page_size,
    void* out, int num_tokens, int nq, int nkv, int d, int dv, int dc, float scale, int window,
    float softcap, int sink, const float* sink_val, const float* gate, int keep, int plan, float* ws, cudaStream_t stream) {
    if (num_tokens <= 0 || num_requests <= 0) return TFF_OK;
    if (nq <= 0 || nkv <= 0 || nq % nkv != 0 || d <= 0 || dv <= 0 || dc < d || dc < dv || page_size <= 0 || softcap < 0.f || keep < 0 || max_q_len <= 0)
        return TFF_ERR_BAD_ARGUMENT;
    if (d > 512 || dv > 512) return TFF_ERR_UNSUPPORTED;
    GenericParams p = {};
    p.q_start = q_start; p.pos_start = pos_start; p.block_table = block_table; p.table_width = table_width;
    p.row_stride = row_stride; p.layer = layer; p.nq = nq; p.nkv = nkv; p.d = d; p.dv = dv;
    p.window = window > 0 ? window : 0; p.keep = window > 0 ? keep : 0;
    p.sink = sink; p.sink_val = sink_val; p.gate = gate; p.scale = scale; p.softcap = softcap;
    p.L = make_kv_layout(cache_layers, nkv, page_size, dc);
    p.splits = plan & 0xffff; p.slots = plan >> 16;
    if (p.splits < 1 || (p.splits > 1 && (ws == nullptr || p.slots < 1 || (long long)max_q_len * (nq / nkv) > tile_rows(dv))))
        return TFF_ERR_BAD_ARGUMENT;
    if (p.splits > 1) { p.part_ml = ws; p.part_o = ws + (size_t)num_tokens * nq * p.slots * 2; }
    // 4 elements are read at a time where rows and slots are whole groups at aligned addresses
    p.q_vec = d % 4 == 0 && row_stride % 4 == 0 && ((uintptr_t)qkv & 15) == 0;
    p.vec = d % 4 == 0 && dv % 4 == 0 && dc % 4 == 0 && ((uintptr_t)cache & 15) == 0;
    int st = is_bf16 ? dispatch<bf16>(qkv, cache, out, p, num_requests, max_q_len, stream)
                     : dispatch<float>(qkv, cache, out, p, num_requests, max_q_len, stream);
    if (st == TFF_OK && p.splits > 1) {
        const unsigned blocks = (unsigned)((long long)num_tokens * nq);
        st = is_bf16 ? tff_launch_pdl(attention_generic_join_kernel<bf16>, dim3(blocks), dim3(JOIN_THREADS), (size_t)0, stream, (bf16*)out, tok_req, p)
                     : tff_launch_pdl(attention_generic_join_kernel<float>, dim3(blocks), dim3(JOIN_THREADS), (size_t)0, stream, (float*)out, tok_req, p);
    }
    return st;
}
