// Causal attention over the paged cache for any mix of prompt portions and
// single decoded tokens, any head size up to 256 and any number of heads and
// key/value groups, with all arithmetic in 32-bit.
//
// This is the 32-bit engine's attention and the fallback of the bfloat16 engine
// for shapes its tensor-core kernels refuse.  One block serves one (token, head).
// The token's visible keys are cut into tiles of 32 from the first visible key;
// tile i goes to warp i mod W (W, the warps of a block, is fixed by the head size),
// every warp keeps a running softmax over its tiles in ascending order, and the
// warps' states are merged in warp order.  So the order of every sum depends on
// the token's position only, never on the batch or on where its pages lie (the
// reference cuts a token's keys into spans by its position alone for the same
// reason and merges the spans in order: src/core/transformer.cpp:2130-2144,
// 2225-2227, 2367-2385).  Scores s_j = (q . k_j) * scale, running maximum,
// p = exp(s - m), o = sum p_j v_j, out = o / sum p (src/core/transformer.cpp:2303-2313,
// 2327-2341, 2344-2358).
#include "api.h"
#include "common.cuh"

#include <math_constants.h>

namespace {

constexpr int kTile = 32;       // keys per step, one per lane
constexpr int kMaxHeadDim = 256;
constexpr long long kFewPairs = 1024;   // up to this many (token, head) pairs take the latency-arranged float32 kernel

// Four consecutive elements as floats with one load (the address is aligned to the four of them).
__device__ __forceinline__ float4 lb_load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 lb_load4(const __nv_bfloat16* p) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&raw.x), hi = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
    const float2 a = __bfloat1622float2(lo), b = __bfloat1622float2(hi);
    return make_float4(a.x, a.y, b.x, b.y);
}

// Copies the rows of up to 32 keys (lane i knows the row of key i: `base`, negative if there is none) into
// the warp's tile as floats.  Eight loads are issued before any is used, so a lone warp (a decode step of
// one request) still keeps several requests to memory in flight.
template <typename T>
__device__ __forceinline__ void load_tile(const T* __restrict__ cache, long long base, long long offset, float* tile,
                                          int tile_stride, int head_dim, int lane) {
    constexpr int kBatch = 8;
    if (head_dim % 4 == 0) {
        // Four values per load (rows of the cache start on 16-byte, or for 2-byte types 8-byte, boundaries).
        constexpr int kQuadBatch = 4;
        const int quads = head_dim / 4, total4 = kTile * quads;     // a multiple of 32
        for (int idx0 = lane; idx0 < total4; idx0 += 32 * kQuadBatch) {
            float4 r[kQuadBatch];
#pragma unroll
            for (int u = 0; u < kQuadBatch; ++u) {
                const int idx = idx0 + 32 * u;
                r[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (idx < total4) {            // uniform across the warp
                    const int key = idx / quads, d = (idx - key * quads) * 4;
                    const long long b = __shfl_sync(0xffffffffu, base, key);
                    if (b >= 0) r[u] = lb_load4(cache + b + offset + d);
                }
            }
#pragma unroll
            for (int u = 0; u < kQuadBatch; ++u) {
                const int idx = idx0 + 32 * u;
                if (idx < total4) {
                    const int key = idx / quads;
                    float* dst = tile + key * tile_stride + (idx - key * quads) * 4;
                    dst[0] = r[u].x; dst[1] = r[u].y; dst[2] = r[u].z; dst[3] = r[u].w;
                }
            }
        }
        return;
    }
    const int total = kTile * head_dim;        // a multiple of 32: every lane makes the same number of trips
    for (int idx0 = lane; idx0 < total; idx0 += 32 * kBatch) {
        float r[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int idx = idx0 + 32 * u;
            r[u] = 0.0f;
            if (idx < total) {                 // uniform across the warp
                const int key = idx / head_dim, d = idx - key * head_dim;
                const long long b = __shfl_sync(0xffffffffu, base, key);
                if (b >= 0) r[u] = lb_to_float(cache[b + offset + d]);
            }
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int idx = idx0 + 32 * u;
            if (idx < total) {
                const int key = idx / head_dim;
                tile[key * tile_stride + (idx - key * head_dim)] = r[u];
            }
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(512)
paged_attention_generic_kernel(const T* __restrict__ q, int64_t q_stride, const T* __restrict__ cache,
                               const int32_t* __restrict__ tok_seq, const int32_t* __restrict__ positions,
                               const int32_t* __restrict__ block_table, int table_stride, T* __restrict__ out,
                               int64_t out_stride, int n_tokens, int n_head, int n_kv_head, int head_dim,
                               int page_size, float scale, int window, const float* __restrict__ distance, const float* __restrict__ sink,
                               float soft_cap) {
    extern __shared__ float smem[];
    lb_wait_for_predecessor();
    lb_dependents_may_launch();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_warps = blockDim.x >> 5;
    const int pair = blockIdx.x;
    const int t = pair / n_head, h = pair - t * n_head;
    const int kvh = h / (n_head / n_kv_head);
    const int pos = positions[t];
    const int32_t* table = block_table + (size_t)tok_seq[t] * table_stride;
    // The head's pair (r1, r2) of the penalty by distance; r1 = 0 without one.
    const float r1 = distance != nullptr ? distance[h] : 0.0f, r2 = distance != nullptr ? distance[n_head + h] : 0.0f;

    const int tile_stride = head_dim + 1;
    float* q_s = smem + (size_t)warp * (head_dim + kTile * tile_stride + kTile);
    float* tile = q_s + head_dim;
    float* p_s = tile + kTile * tile_stride;

    const T* q_row = q + (size_t)t * q_stride + (size_t)h * head_dim;
    for (int d = lane; d < head_dim; d += 32) q_s[d] = lb_to_float(q_row[d]);

    const size_t plane = (size_t)n_kv_head * page_size * head_dim;
    float m = -CUDART_INF_F, l = 0.0f;
    float acc[kMaxHeadDim / 32];
#pragma unroll
    for (int i = 0; i < kMaxHeadDim / 32; ++i) acc[i] = 0.0f;

    const int first = lb_first_visible(pos, window);
    for (int j0 = first + warp * kTile; j0 <= pos; j0 += n_warps * kTile) {
        const int n_keys = min(kTile, pos + 1 - j0);
        // Each lane resolves its own key's row once; the others fetch it by shuffle.
        long long base = -1;
        if (lane < n_keys) {
            const int j = j0 + lane;
            const int page = table[j / page_size];
            base = (long long)page * 2 * (long long)plane + ((long long)kvh * page_size + (j % page_size)) * head_dim;
        }
        __syncwarp();
        load_tile(cache, base, 0, tile, tile_stride, head_dim, lane);
        __syncwarp();
        float s = -CUDART_INF_F;
        if (lane < n_keys) {
            float dot = 0.0f;
            const float* krow = tile + lane * tile_stride;
            for (int d = 0; d < head_dim; ++d) dot = fmaf(q_s[d], krow[d], dot);
            s = dot * scale;
            if (soft_cap > 0.0f) s = soft_cap * tanhf(s / soft_cap);
            if (distance != nullptr) s -= lb_distance_penalty(r1, r2, pos - (j0 + lane));
        }
        const float m_new = fmaxf(m, lb_warp_max(s));
        const float p = lane < n_keys ? expf(s - m_new) : 0.0f;
        const float corr = expf(m - m_new);      // exp(-inf) = 0 on the first tile
        l = l * corr + lb_warp_sum(p);
        m = m_new;
        p_s[lane] = p;
        __syncwarp();
        load_tile(cache, base, (long long)plane, tile, tile_stride, head_dim, lane);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < kMaxHeadDim / 32; ++i) {
            const int d = lane + 32 * i;
            if (d < head_dim) {
                float o = acc[i] * corr;
                for (int j = 0; j < n_keys; ++j) o = fmaf(p_s[j], tile[j * tile_stride + d], o);
                acc[i] = o;
            }
        }
        __syncwarp();
    }
    // The warps' states (m, l, o) meet in shared memory and are merged in warp order.  A warp without a tile
    // has m = -inf, l = 0, o = 0 and weighs nothing.
    float* merge = smem + (size_t)n_warps * (head_dim + kTile * tile_stride + kTile);
    float* mine = merge + (size_t)warp * (head_dim + 2);
    if (lane == 0) { mine[0] = m; mine[1] = l; }
#pragma unroll
    for (int i = 0; i < kMaxHeadDim / 32; ++i) {
        const int d = lane + 32 * i;
        if (d < head_dim) mine[2 + d] = acc[i];
    }
    __syncthreads();
    T* o_row = out + (size_t)t * out_stride + (size_t)h * head_dim;
    for (int d = threadIdx.x; d < head_dim; d += blockDim.x) {
        // A head's sink joins the divisor as a state without values: maximum sink[h], sum 1.
        float top = sink != nullptr ? sink[h] : -CUDART_INF_F;
        for (int w = 0; w < n_warps; ++w) top = fmaxf(top, merge[(size_t)w * (head_dim + 2)]);
        float total = sink != nullptr ? expf(sink[h] - top) : 0.0f, o = 0.0f;
        for (int w = 0; w < n_warps; ++w) {
            const float* st = merge + (size_t)w * (head_dim + 2);
            const float f = expf(st[0] - top);      // exp(-inf) = 0 for a warp without keys
            total = fmaf(st[1], f, total);
            o = fmaf(st[2 + d], f, o);
        }
        o_row[d] = lb_from_float<T>(o / total);
    }
}

// ---- float32, few (token, head) pairs: the same sums in the same order, arranged around memory latency --------
//
// A decode step of a few requests launches fewer blocks than the GPU has SMs, and each warp's chain of round
// trips to memory sets the pace.  Here keys and values have a buffer each and travel by asynchronous 16-byte copies
// (no registers in between): a tile's values are in flight while its scores are computed, the next tile's keys
// while the values are summed, and the page of the next tile is looked up a tile ahead.  Rows lie head_dim + 4
// floats apart, so a lane reads its key's row as 16-byte pieces without meeting a bank twice.  Every product and
// sum is the one paged_attention_generic_kernel makes, in its order: the two kernels agree bit for bit.

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// Which 16-byte pieces of a 32-key tile a lane copies: piece lane + 32 u, u = 0 .. head_dim / 4 - 1, of the tile's
// [key][piece of the row]; (key, piece) advance by fixed steps, so nothing is divided inside the loop.
struct PieceWalk {
    int key0, c0, dk, dc, quads;
};

// The rows of up to 32 keys (row_s[i]: where key i's row starts, negative if there is none) -> the tile, as copies in flight.
__device__ __forceinline__ void tile_in_flight(const float* __restrict__ cache, const long long* row_s, long long offset,
                                               float* tile, int tile_stride, const PieceWalk& w) {
    int key = w.key0, c = w.c0;
    for (int u = 0; u < w.quads; ++u) {
        const long long b = row_s[key];
        if (b >= 0) cp_async16(tile + key * tile_stride + 4 * c, cache + b + offset + 4 * c);
        key += w.dk;
        c += w.dc;
        if (c >= w.quads) { c -= w.quads; ++key; }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

__global__ void __launch_bounds__(256, 1)
paged_attention_f32_few_kernel(const float* __restrict__ q, int64_t q_stride, const float* __restrict__ cache,
                               const int32_t* __restrict__ tok_seq, const int32_t* __restrict__ positions,
                               const int32_t* __restrict__ block_table, int table_stride, float* __restrict__ out,
                               int64_t out_stride, int n_tokens, int n_head, int n_kv_head, int head_dim,
                               int page_size, float scale, int window, const float* __restrict__ distance, const float* __restrict__ sink,
                               float soft_cap) {
    extern __shared__ __align__(16) float smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_warps = blockDim.x >> 5;
    const int pair = blockIdx.x;
    const int t = pair / n_head, h = pair - t * n_head;
    const int kvh = h / (n_head / n_kv_head);
    const int pos = positions[t];
    const int32_t* table = block_table + (size_t)tok_seq[t] * table_stride;
    // The head's pair (r1, r2) of the penalty by distance; r1 = 0 without one.
    const float r1 = distance != nullptr ? distance[h] : 0.0f, r2 = distance != nullptr ? distance[n_head + h] : 0.0f;

    const int tile_stride = head_dim + 4;
    float* q_s = smem + (size_t)warp * (head_dim + 2 * kTile * tile_stride + kTile + 2 * kTile);
    float* k_tile = q_s + head_dim;
    float* v_tile = k_tile + kTile * tile_stride;
    float* p_s = v_tile + kTile * tile_stride;
    long long* row_s = reinterpret_cast<long long*>(p_s + kTile);      // where each key's row of the coming tile starts
    const int quads = head_dim / 4;
    const PieceWalk walk{lane / quads, lane % quads, 32 / quads, 32 % quads, quads};

    const size_t plane = (size_t)n_kv_head * page_size * head_dim;
    const int first = lb_first_visible(pos, window);
    const int step = n_warps * kTile;
    auto row_of = [&](int j0) -> long long {      // this lane's key of the tile that starts at j0
        const int j = j0 + lane;
        if (j0 > pos || j > pos) return -1;
        const int page = __ldg(table + j / page_size);
        return (long long)page * 2 * (long long)plane + ((long long)kvh * page_size + (j % page_size)) * head_dim;
    };
    int j0 = first + warp * kTile;
    row_s[lane] = row_of(j0);            // positions and block table came from the host: looked up before the wait
    lb_wait_for_predecessor();           // queries, and the newest keys and values, come from the kernel before this one
    lb_dependents_may_launch();
    __syncwarp();
    if (j0 <= pos) {
        tile_in_flight(cache, row_s, 0, k_tile, tile_stride, walk);
        tile_in_flight(cache, row_s, (long long)plane, v_tile, tile_stride, walk);
    }
    const float* q_row = q + (size_t)t * q_stride + (size_t)h * head_dim;
    for (int d = lane; d < head_dim; d += 32) q_s[d] = q_row[d];

    float m = -CUDART_INF_F, l = 0.0f;
    float acc[kMaxHeadDim / 32];
#pragma unroll
    for (int i = 0; i < kMaxHeadDim / 32; ++i) acc[i] = 0.0f;

    for (; j0 <= pos; j0 += step) {
        const int n_keys = min(kTile, pos + 1 - j0);
        const bool more = j0 + step <= pos;
        const long long next_base = row_of(j0 + step);           // the next tile's page, asked for a tile ahead
        asm volatile("cp.async.wait_group 1;" ::: "memory");     // this tile's keys have landed (its values may not have)
        __syncwarp();
        float s = -CUDART_INF_F;
        if (lane < n_keys) {
            float dot = 0.0f;
            const float4* krow = reinterpret_cast<const float4*>(k_tile + lane * tile_stride);
            const float4* qv = reinterpret_cast<const float4*>(q_s);
            for (int c = 0; c < head_dim / 4; ++c) {
                const float4 kq = krow[c], qq = qv[c];
                dot = fmaf(qq.x, kq.x, dot);
                dot = fmaf(qq.y, kq.y, dot);
                dot = fmaf(qq.z, kq.z, dot);
                dot = fmaf(qq.w, kq.w, dot);
            }
            s = dot * scale;
            if (soft_cap > 0.0f) s = soft_cap * tanhf(s / soft_cap);
            if (distance != nullptr) s -= lb_distance_penalty(r1, r2, pos - (j0 + lane));
        }
        const float m_new = fmaxf(m, lb_warp_max(s));
        const float p = lane < n_keys ? expf(s - m_new) : 0.0f;
        const float corr = expf(m - m_new);      // exp(-inf) = 0 on the first tile
        l = l * corr + lb_warp_sum(p);
        m = m_new;
        p_s[lane] = p;
        row_s[lane] = next_base;                 // this tile's copies were all issued: the rows of the next one
        __syncwarp();                            // every lane has read the keys: the next tile's go into the buffer
        if (more) tile_in_flight(cache, row_s, 0, k_tile, tile_stride, walk);
        else asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");     // this tile's values have landed
        __syncwarp();
        // Each element's sum runs over the keys in ascending order, as in the plain kernel; the elements of a lane
        // advance side by side and share the weight they read.
#pragma unroll
        for (int i = 0; i < kMaxHeadDim / 32; ++i) acc[i] *= corr;
#pragma unroll 4
        for (int j = 0; j < n_keys; ++j) {
            const float pj = p_s[j];
            const float* vrow = v_tile + j * tile_stride + lane;
#pragma unroll
            for (int i = 0; i < kMaxHeadDim / 32; ++i)
                if (32 * i < head_dim && lane + 32 * i < head_dim) acc[i] = fmaf(pj, vrow[32 * i], acc[i]);
        }
        __syncwarp();
        if (more) tile_in_flight(cache, row_s, (long long)plane, v_tile, tile_stride, walk);
        else asm volatile("cp.async.commit_group;" ::: "memory");
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    float* merge = smem + (size_t)n_warps * (head_dim + 2 * kTile * tile_stride + kTile + 2 * kTile);
    float* mine = merge + (size_t)warp * (head_dim + 2);
    if (lane == 0) { mine[0] = m; mine[1] = l; }
#pragma unroll
    for (int i = 0; i < kMaxHeadDim / 32; ++i) {
        const int d = lane + 32 * i;
        if (d < head_dim) mine[2 + d] = acc[i];
    }
    __syncthreads();
    float* o_row = out + (size_t)t * out_stride + (size_t)h * head_dim;
    for (int d = threadIdx.x; d < head_dim; d += blockDim.x) {
        // A head's sink joins the divisor as a state without values: maximum sink[h], sum 1.
        float top = sink != nullptr ? sink[h] : -CUDART_INF_F;
        for (int w = 0; w < n_warps; ++w) top = fmaxf(top, merge[(size_t)w * (head_dim + 2)]);
        float total = sink != nullptr ? expf(sink[h] - top) : 0.0f, o = 0.0f;
        for (int w = 0; w < n_warps; ++w) {
            const float* st = merge + (size_t)w * (head_dim + 2);
            const float f = expf(st[0] - top);      // exp(-inf) = 0 for a warp without keys
            total = fmaf(st[1], f, total);
            o = fmaf(st[2 + d], f, o);
        }
        o_row[d] = o / total;
    }
}

// ---- float32, many (token, head) pairs of head size 64: the same sums, a tile's keys and values read once for sixteen queries ----
//
// One block a (token, head) reads all the keys that the token sees, and a prompt's neighbouring tokens see nearly the same ones.  Here a
// block serves sixteen neighbouring tokens, run by run: the tokens of a run belong to one request and start at the same key.  A warp still owns the tiles i mod 8:
// it holds a tile's keys (a lane a key) in registers while it makes the scores of all the run's queries, four of them at a time so that
// four chains of products run side by side, and then the tile's values (a lane two of the 64 columns) while it adds them up; the queries'
// states wait in shared memory in between.  Bound by instructions issued: a score or a weighted value costs one product and a fraction of a
// broadcast load.  A warp goes from run to run without waiting for the others.  Every product and sum is the one that
// paged_attention_generic_kernel makes, in its order: the kernels agree bit for bit.
// Measured (12 heads, prompts of 188, 152 and 250 tokens, a layer): 229 us a block a (token, head); 57 us with a block started for every
// (token, head) of which one in sixteen worked; see the product's kernel for the step as a whole.
constexpr int kRun = 16;         // tokens of a block
constexpr int kRunWarps = 8;
constexpr int kRunDim = 64;
constexpr int kRunAcc = kRunDim + 2;       // a state: maximum, sum, weighted values
constexpr size_t kRunSmem = sizeof(float) * (kRun * kRunDim + kRunWarps * kRun * (kTile + 1 + kRunAcc));

__global__ void __launch_bounds__(kRunWarps * 32, 2)
paged_attention_f32_runs_kernel(const float* __restrict__ q, int64_t q_stride, const float* __restrict__ cache, const int32_t* __restrict__ tok_seq,
                                const int32_t* __restrict__ positions, const int32_t* __restrict__ block_table, int table_stride, float* __restrict__ out,
                                int64_t out_stride, int n_tokens, int n_head, int n_kv_head, int page_size, float scale, int window,
                                const float* __restrict__ sink) {
    extern __shared__ __align__(16) float smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t0 = blockIdx.x / n_head * kRun, h = blockIdx.x % n_head;
    const int n_here = min(kRun, n_tokens - t0);
    // Positions and requests came from the host, before any kernel of the step: read ahead of the wait.  Lane i knows token t0 + i.
    const int my_pos = lane < n_here ? positions[t0 + lane] : -1, my_seq = lane < n_here ? tok_seq[t0 + lane] : -1;
    const int my_first = lb_first_visible(max(my_pos, 0), window);
    const int before_pos = __shfl_up_sync(0xffffffffu, my_pos, 1), before_seq = __shfl_up_sync(0xffffffffu, my_seq, 1);
    const int before_first = __shfl_up_sync(0xffffffffu, my_first, 1);
    const uint32_t starts = __ballot_sync(0xffffffffu, lane == 0 || lane >= n_here || my_seq != before_seq || my_pos != before_pos + 1 || my_first != before_first);
    lb_wait_for_predecessor();
    lb_dependents_may_launch();
    const int kvh = h / (n_head / n_kv_head);
    const size_t plane = (size_t)n_kv_head * page_size * kRunDim;

    float* q_s = smem;                                                    // [query][64]
    float* p_s = q_s + kRun * kRunDim + warp * kRun * kTile;              // this warp's weights of the tile, [query][32]
    float* corr_s = q_s + kRun * kRunDim + kRunWarps * kRun * kTile + warp * kRun;
    float* states = q_s + kRun * kRunDim + kRunWarps * kRun * (kTile + 1);          // [warp][query][maximum, sum, 64 values]
    float* mine = states + warp * kRun * kRunAcc;
    for (int i = threadIdx.x; i < kRun * kRunDim; i += blockDim.x) {
        const int u = i / kRunDim;
        q_s[i] = u < n_here ? q[(size_t)(t0 + u) * q_stride + (size_t)h * kRunDim + i % kRunDim] : 0.0f;
    }
    for (int i = lane; i < kRun * kRunAcc; i += 32) mine[i] = i % kRunAcc == 0 ? -CUDART_INF_F : 0.0f;
    __syncthreads();

    // `pos` stands for the position that the block's first token would have in the run's request: query u is at pos + u throughout.
    for (int run = 0, run_end; run < n_here; run = run_end) {
        run_end = min(n_here, run + __ffs(starts >> (run + 1)));            // the lanes from n_here on start runs of their own
        const int first = __shfl_sync(0xffffffffu, my_first, run), pos = __shfl_sync(0xffffffffu, my_pos, run) - run, last = pos + run_end - 1;
        const int32_t* table = block_table + (size_t)__shfl_sync(0xffffffffu, my_seq, run) * table_stride;
        for (int j0 = first + warp * kTile; j0 <= last; j0 += kRunWarps * kTile) {
            const int j = j0 + lane;
            long long base = -1;
            if (j <= last) base = (long long)table[j / page_size] * 2 * (long long)plane + ((long long)kvh * page_size + (j % page_size)) * kRunDim;
            const int u0 = max(run, j0 - pos);                  // the run's first queries may lie before the tile
            {
                float4 key[kRunDim / 4];
#pragma unroll
                for (int c = 0; c < kRunDim / 4; ++c)
                    key[c] = base >= 0 ? __ldg(reinterpret_cast<const float4*>(cache + base) + c) : make_float4(0.f, 0.f, 0.f, 0.f);
                for (int u = u0 & ~3; u < run_end; u += 4) {
                    float dot[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int c = 0; c < kRunDim / 4; ++c)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float4 qq = *reinterpret_cast<const float4*>(q_s + (u + e) * kRunDim + 4 * c);
                            dot[e] = fmaf(qq.x, key[c].x, dot[e]);
                            dot[e] = fmaf(qq.y, key[c].y, dot[e]);
                            dot[e] = fmaf(qq.z, key[c].z, dot[e]);
                            dot[e] = fmaf(qq.w, key[c].w, dot[e]);
                        }
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int n_keys = min(kTile, pos + u + e + 1 - j0);
                        const float s = lane < n_keys ? dot[e] * scale : -CUDART_INF_F;
                        float* state = mine + (u + e) * kRunAcc;
                        const float m = state[0];
                        float l = state[1];
                        const float m_new = fmaxf(m, lb_warp_max(s));
                        const float p = lane < n_keys ? expf(s - m_new) : 0.0f;
                        const float corr = expf(m - m_new);      // exp(-inf) = 0 on the first tile
                        l = l * corr + lb_warp_sum(p);
                        if (u + e >= u0 && u + e < run_end) {    // the others' states are not this run's, or see none of the tile
                            p_s[(u + e) * kTile + lane] = p;
                            if (lane == 0) {
                                state[0] = m_new;
                                state[1] = l;
                                corr_s[u + e] = corr;
                            }
                        }
                    }
                }
            }
            __syncwarp();
            {
                float v0[kTile], v1[kTile];
                const int n_rows = min(kTile, last + 1 - j0);
#pragma unroll
                for (int k = 0; k < kTile; ++k) {
                    const long long b = __shfl_sync(0xffffffffu, base, k);
                    v0[k] = k < n_rows ? __ldg(cache + b + plane + lane) : 0.0f;
                    v1[k] = k < n_rows ? __ldg(cache + b + plane + 32 + lane) : 0.0f;
                }
#pragma unroll 2
                for (int u = u0; u < run_end; ++u) {
                    const int n_keys = min(kTile, pos + u + 1 - j0);
                    float* state = mine + u * kRunAcc + 2;
                    const float corr = corr_s[u];
                    float o0 = state[lane] * corr, o1 = state[lane + 32] * corr;
                    const float4* weights = reinterpret_cast<const float4*>(p_s + u * kTile);
                    if (n_keys == kTile) {
#pragma unroll
                        for (int k = 0; k < kTile / 4; ++k) {
                            const float4 p = weights[k];
                            o0 = fmaf(p.x, v0[4 * k], o0);
                            o1 = fmaf(p.x, v1[4 * k], o1);
                            o0 = fmaf(p.y, v0[4 * k + 1], o0);
                            o1 = fmaf(p.y, v1[4 * k + 1], o1);
                            o0 = fmaf(p.z, v0[4 * k + 2], o0);
                            o1 = fmaf(p.z, v1[4 * k + 2], o1);
                            o0 = fmaf(p.w, v0[4 * k + 3], o0);
                            o1 = fmaf(p.w, v1[4 * k + 3], o1);
                        }
                    } else {                                      // the keys after the query are no terms of its sums
#pragma unroll
                        for (int k = 0; k < kTile; ++k) {
                            const float p = p_s[u * kTile + k];
                            o0 = k < n_keys ? fmaf(p, v0[k], o0) : o0;
                            o1 = k < n_keys ? fmaf(p, v1[k], o1) : o1;
                        }
                    }
                    state[lane] = o0;
                    state[lane + 32] = o1;
                }
            }
            __syncwarp();
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n_here * kRunDim; i += blockDim.x) {
        const int u = i / kRunDim, d = i % kRunDim;
        // A head's sink joins the divisor as a state without values: maximum sink[h], sum 1.
        float top = sink != nullptr ? sink[h] : -CUDART_INF_F;
        for (int w = 0; w < kRunWarps; ++w) top = fmaxf(top, states[(w * kRun + u) * kRunAcc]);
        float total = sink != nullptr ? expf(sink[h] - top) : 0.0f, o = 0.0f;
        for (int w = 0; w < kRunWarps; ++w) {
            const float* st = states + (w * kRun + u) * kRunAcc;
            const float f = expf(st[0] - top);      // exp(-inf) = 0 for a warp without keys
            total = fmaf(st[1], f, total);
            o = fmaf(st[2 + d], f, o);
        }
        out[(size_t)(t0 + u) * out_stride + (size_t)h * kRunDim + d] = o / total;
    }
}

// ---- float32, few pairs of head size 64: the same sums, the streams' steps side by side -------------------------------
//
// The warps of the kernel above each walk a chain: scores, maximum, sum, values, tile after tile.  Only the maxima, the sums and the weighted
// values of a stream (the tiles i mod 8) depend on its tile before; the scores do not.  Here a block of sixteen warps takes sixteen tiles at
// a time: every warp makes the scores of one tile, eight warps carry the streams' maxima and sums over two tiles each, and
// then all sixteen add up the weighted values (two warps a stream, a lane a column).  The tiles' keys travel into shared memory by
// asynchronous copies and their values into registers from the start of the round, the next sixteen tiles' keys under the values of
// these.  Every product and sum is the one paged_attention_generic_kernel makes, in its order: the kernels agree bit for bit.
// Measured (8 requests x 12 heads, contexts of 360 to 880, a layer, cold): 20.8 us with the chains, 14.7 us here; GPT-2 small's step 770 -> 703 us
// with its logits' copy.
constexpr int kWideWarps = 16;
constexpr int kWideStreams = 8;
constexpr int kWideStride = 64 + 4;        // floats between the keys of a tile
constexpr size_t kWideSmem = sizeof(float) * (kWideWarps * kTile * kWideStride + 64 + 2 * kWideWarps * kTile + kWideWarps + kWideStreams * (64 + 2));

__global__ void __launch_bounds__(kWideWarps * 32, 1)
paged_attention_f32_wide_kernel(const float* __restrict__ q, int64_t q_stride, const float* __restrict__ cache, const int32_t* __restrict__ tok_seq,
                                const int32_t* __restrict__ positions, const int32_t* __restrict__ block_table, int table_stride, float* __restrict__ out,
                                int64_t out_stride, int n_head, int n_kv_head, int page_size, float scale, int window, const float* __restrict__ sink) {
    extern __shared__ __align__(16) float smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x / n_head, h = blockIdx.x - t * n_head;
    const int kvh = h / (n_head / n_kv_head);
    const int pos = positions[t];
    const int32_t* table = block_table + (size_t)tok_seq[t] * table_stride;
    const size_t plane = (size_t)n_kv_head * page_size * 64;
    const int first = lb_first_visible(pos, window);
    float* k_tile = smem + (size_t)warp * kTile * kWideStride;            // this warp's tile of keys
    float* q_s = smem + (size_t)kWideWarps * kTile * kWideStride;
    float* s_s = q_s + 64;                                                // [tile][32] scores
    float* p_s = s_s + kWideWarps * kTile;                                // [tile][32] weights
    float* corr_s = p_s + kWideWarps * kTile;                             // [tile] what the stream's sums are multiplied by
    float* merge = corr_s + kWideWarps;                                   // [stream][maximum, sum, 64 values]
    auto row_of = [&](int j) -> long long {                               // where key j's row starts; -1: there is none
        if (j > pos) return -1;
        return (long long)__ldg(table + j / page_size) * 2 * (long long)plane + ((long long)kvh * page_size + (j % page_size)) * 64;
    };
    // The keys of the tile that starts at j0: piece lane % 16 of two rows at a time.
    auto keys_in_flight = [&](long long row) {
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            const int key = 2 * u + (lane >> 4);
            const long long b = __shfl_sync(0xffffffffu, row, key);
            if (b >= 0) cp_async16(k_tile + key * kWideStride + 4 * (lane & 15), cache + b + 4 * (lane & 15));
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // In the second half of a round this warp sums the values of stream `stream`, column `column`.
    const int stream = warp >> 1, column = (warp & 1) * 32 + lane;
    long long key_row = row_of(first + warp * kTile + lane);              // host data: looked up before the wait
    long long value_row[2] = {row_of(first + stream * kTile + lane), row_of(first + (stream + kWideStreams) * kTile + lane)};
    lb_wait_for_predecessor();                                            // queries, and the newest keys and values, come from the kernel before
    lb_dependents_may_launch();
    keys_in_flight(key_row);
    if (threadIdx.x < 64) q_s[threadIdx.x] = q[(size_t)t * q_stride + (size_t)h * 64 + threadIdx.x];
    float m = -CUDART_INF_F, l = 0.0f;                                    // warps 0..7: their stream's
    float acc = 0.0f;
    for (int j0 = first; j0 <= pos; j0 += kWideWarps * kTile) {
        // The values that this thread will weigh, two tiles of its stream: asked for now.
        float v[2][kTile];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int k = 0; k < kTile; ++k) {
                const long long b = __shfl_sync(0xffffffffu, value_row[i], k);
                v[i][k] = b >= 0 ? __ldcg(cache + b + plane + column) : 0.0f;
            }
        const int my_j = j0 + warp * kTile + lane;
        const bool more = j0 + kWideWarps * kTile <= pos;
        if (more) {
            key_row = row_of(my_j + kWideWarps * kTile);
            value_row[0] = row_of(j0 + (kWideWarps + stream) * kTile + lane);
            value_row[1] = row_of(j0 + (kWideWarps + stream + kWideStreams) * kTile + lane);
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                                  // the queries too
        float s = -CUDART_INF_F;
        if (my_j <= pos) {
            float dot = 0.0f;
            const float4* krow = reinterpret_cast<const float4*>(k_tile + lane * kWideStride);
            const float4* qv = reinterpret_cast<const float4*>(q_s);
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                const float4 kq = krow[c], qq = qv[c];
                dot = fmaf(qq.x, kq.x, dot);
                dot = fmaf(qq.y, kq.y, dot);
                dot = fmaf(qq.z, kq.z, dot);
                dot = fmaf(qq.w, kq.w, dot);
            }
            s = dot * scale;
        }
        s_s[warp * kTile + lane] = s;
        __syncthreads();                                                  // every tile's scores; every warp has read its keys
        if (more) keys_in_flight(key_row);
        if (warp < kWideStreams) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int tile = warp + i * kWideStreams;
                const int n_keys = min(kTile, pos + 1 - (j0 + tile * kTile));
                if (n_keys > 0) {
                    const float sc = s_s[tile * kTile + lane];
                    const float m_new = fmaxf(m, lb_warp_max(sc));
                    const float p = lane < n_keys ? expf(sc - m_new) : 0.0f;
                    const float corr = expf(m - m_new);                   // exp(-inf) = 0 on the first tile
                    l = l * corr + lb_warp_sum(p);
                    m = m_new;
                    p_s[tile * kTile + lane] = p;
                    if (lane == 0) corr_s[tile] = corr;
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int tile = stream + i * kWideStreams;
            const int n_keys = min(kTile, pos + 1 - (j0 + tile * kTile));
            if (n_keys > 0) {
                float o = acc * corr_s[tile];
                const float4* weights = reinterpret_cast<const float4*>(p_s + tile * kTile);
                if (n_keys == kTile) {
#pragma unroll
                    for (int k = 0; k < kTile / 4; ++k) {
                        const float4 p = weights[k];
                        o = fmaf(p.x, v[i][4 * k], o);
                        o = fmaf(p.y, v[i][4 * k + 1], o);
                        o = fmaf(p.z, v[i][4 * k + 2], o);
                        o = fmaf(p.w, v[i][4 * k + 3], o);
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < kTile; ++k) o = k < n_keys ? fmaf(p_s[tile * kTile + k], v[i][k], o) : o;
                }
                acc = o;
            }
        }
    }
    if (warp < kWideStreams && lane == 0) {
        merge[warp * 66] = m;
        merge[warp * 66 + 1] = l;
    }
    merge[stream * 66 + 2 + column] = acc;
    __syncthreads();
    if (threadIdx.x < 64) {
        const int d = threadIdx.x;
        // A head's sink joins the divisor as a state without values: maximum sink[h], sum 1.
        float top = sink != nullptr ? sink[h] : -CUDART_INF_F;
        for (int w = 0; w < kWideStreams; ++w) top = fmaxf(top, merge[w * 66]);
        float total = sink != nullptr ? expf(sink[h] - top) : 0.0f, o = 0.0f;
        for (int w = 0; w < kWideStreams; ++w) {
            const float* st = merge + w * 66;
            const float f = expf(st[0] - top);      // exp(-inf) = 0 for a stream without keys
            total = fmaf(st[1], f, total);
            o = fmaf(st[2 + d], f, o);
        }
        out[(size_t)t * out_stride + (size_t)h * 64 + d] = o / total;
    }
}

// What a block of paged_attention_f32_few_kernel needs of an SM's shared memory; launch() takes that kernel for float32, 16-byte rows and few enough pairs that
// latency and not throughput sets the time, where head size 64 and plain scores do not make it the one with the streams' steps side by side.
size_t few_smem(int warps, int head_dim) {
    return (size_t)warps * (head_dim + 2 * kTile * (head_dim + 4) + kTile + 2 * kTile + head_dim + 2) * sizeof(float);
}

// Warps per block, by the head size alone: eight while three such blocks fit the shared memory of an SM (up to head size 64), fewer for larger heads.
int warps_for(int head_dim) {
    const size_t per_warp = (size_t)(head_dim + kTile * (head_dim + 1) + kTile + head_dim + 2) * sizeof(float);
    int w = 8;
    while (w > 1 && 3 * w * per_warp > 220 * 1024) w >>= 1;
    return w;
}

template <typename T>
int launch(const void* q, int64_t q_stride, const void* cache, const int32_t* tok_seq, const int32_t* positions,
           const int32_t* block_table, int table_stride, void* out, int64_t out_stride, int n_tokens, int n_head,
           int n_kv_head, int head_dim, int page_size, float scale, int window, const float* distance, const float* sink, float soft_cap,
           cudaStream_t s) {
    const int warps = warps_for(head_dim);
    const size_t smem = (size_t)warps * (head_dim + kTile * (head_dim + 1) + kTile + head_dim + 2) * sizeof(float);
    static size_t configured = 0;   // largest dynamic shared memory asked for so far
    if (smem > configured) {
        LB_CHECK_CUDA(cudaFuncSetAttribute(paged_attention_generic_kernel<T>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured = smem;
    }
    const long long pairs = (long long)n_tokens * n_head;
    LB_CHECK_ARG(pairs <= 2147483647ll, "attention: %lld (token, head) pairs are too many for one launch", pairs);
    if constexpr (sizeof(T) == 4) {
        // Few pairs: the kernel arranged around latency (the same warps per block, so the same sums).
        const size_t few = few_smem(warps, head_dim);
        if (pairs <= kFewPairs && head_dim == 64 && warps == kWideStreams && distance == nullptr && soft_cap == 0.0f && ((uintptr_t)cache & 15) == 0) {
            LB_CHECK_CUDA(cudaFuncSetAttribute(paged_attention_f32_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWideSmem));
            LB_CHECK_CUDA(lb_launch_overlapped(paged_attention_f32_wide_kernel, dim3((unsigned)pairs), dim3(kWideWarps * 32), kWideSmem, s, (const float*)q,
                                               q_stride, (const float*)cache, tok_seq, positions, block_table, table_stride, (float*)out, out_stride, n_head,
                                               n_kv_head, page_size, scale, window, sink));
            LB_CHECK_LAUNCH();
            return LB_OK;
        }
        if (pairs <= kFewPairs && head_dim % 4 == 0 && q_stride % 4 == 0 && few <= 227 * 1024 && ((uintptr_t)cache & 15) == 0) {
            static size_t few_configured = 0;
            if (few > few_configured) {
                LB_CHECK_CUDA(cudaFuncSetAttribute(paged_attention_f32_few_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)few));
                few_configured = few;
            }
            LB_CHECK_CUDA(lb_launch_overlapped(paged_attention_f32_few_kernel, dim3((unsigned)pairs), dim3(warps * 32), few, s, 
                (const float*)q, q_stride, (const float*)cache, tok_seq, positions, block_table, table_stride, (float*)out, out_stride,
                n_tokens, n_head, n_kv_head, head_dim, page_size, scale, window, distance, sink, soft_cap));
            LB_CHECK_LAUNCH();
            return LB_OK;
        }
    }
    LB_CHECK_CUDA(lb_launch_overlapped(paged_attention_generic_kernel<T>, dim3((unsigned)pairs), dim3(warps * 32), smem, s, 
        (const T*)q, q_stride, (const T*)cache, tok_seq, positions, block_table, table_stride, (T*)out, out_stride,
        n_tokens, n_head, n_kv_head, head_dim, page_size, scale, window, distance, sink, soft_cap));
    LB_CHECK_LAUNCH();
    return LB_OK;
}

}  // namespace

// Whether float32 launches of these sizes take the kernel that shares a tile among neighbouring tokens: head size 64, keys whose first one does
// not move with the token (all earlier ones, or those of a chunk), plain scores, and more pairs than the few that are bound by latency (that
// kernel is the faster one up to there).  A block takes single tokens one after another: whether a step's portions suit it is the host's to say.
extern "C" int lb_paged_attention_f32_runs_supports(const void* cache, int n_tokens, int n_head, int n_kv_head, int head_dim, int window) {
    return head_dim == kRunDim && warps_for(head_dim) == kRunWarps && window <= 0 && n_head > 0 && n_kv_head > 0 && n_head % n_kv_head == 0 &&
           (long long)n_tokens * n_head > kFewPairs && (long long)n_tokens * n_head <= 2147483647ll && ((uintptr_t)cache & 15) == 0;
}

extern "C" int lb_paged_attention_f32_runs(const float* q, int64_t q_stride, const float* cache, const int32_t* tok_seq, const int32_t* positions,
                                           const int32_t* block_table, int table_stride, float* out, int64_t out_stride, int n_tokens, int n_head,
                                           int n_kv_head, int page_size, float scale, int window, const float* sink, void* stream) {
    LB_CHECK_ARG(n_tokens >= 0 && n_head > 0 && n_kv_head > 0 && page_size > 0 && n_head % n_kv_head == 0, "attention: bad sizes");
    LB_CHECK_ARG(window <= 0 && ((uintptr_t)cache & 15) == 0, "attention: runs of queries need a first key that does not move and a cache on a 16-byte boundary");
    const long long blocks = (long long)((n_tokens + kRun - 1) / kRun) * n_head;
    LB_CHECK_ARG(blocks <= 2147483647ll, "attention: %d tokens are too many for one launch", n_tokens);
    if (n_tokens == 0) return LB_OK;
    LB_CHECK_CUDA(cudaFuncSetAttribute(paged_attention_f32_runs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRunSmem));
    LB_CHECK_CUDA(lb_launch_overlapped(paged_attention_f32_runs_kernel, dim3((unsigned)blocks), dim3(kRunWarps * 32), kRunSmem, static_cast<cudaStream_t>(stream), q,
                                       q_stride, cache, tok_seq, positions, block_table, table_stride, out, out_stride, n_tokens, n_head, n_kv_head, page_size,
                                       scale, window, sink));
    LB_CHECK_LAUNCH();
    return LB_OK;
}

extern "C" int lb_paged_attention_generic(int dtype, const void* q, int64_t q_stride, const void* cache,
                                          const int32_t* tok_seq, const int32_t* positions,
                                          const int32_t* block_table, int table_stride, void* out, int64_t out_stride,
                                          int n_tokens, int n_head, int n_kv_head, int head_dim, int page_size,
                                          float scale, int window, void* stream) {
    return lb_paged_attention_generic_biased(dtype, q, q_stride, cache, tok_seq, positions, block_table, table_stride, out, out_stride, n_tokens, n_head,
                                             n_kv_head, head_dim, page_size, scale, window, nullptr, stream);
}

extern "C" int lb_paged_attention_generic_biased(int dtype, const void* q, int64_t q_stride, const void* cache, const int32_t* tok_seq,
                                                 const int32_t* positions, const int32_t* block_table, int table_stride, void* out, int64_t out_stride,
                                                 int n_tokens, int n_head, int n_kv_head, int head_dim, int page_size, float scale, int window,
                                                 const float* distance, void* stream) {
    return lb_paged_attention_generic_sink(dtype, q, q_stride, cache, tok_seq, positions, block_table, table_stride, out, out_stride, n_tokens, n_head,
                                           n_kv_head, head_dim, page_size, scale, window, distance, nullptr, stream);
}

extern "C" int lb_paged_attention_generic_sink(int dtype, const void* q, int64_t q_stride, const void* cache, const int32_t* tok_seq,
                                               const int32_t* positions, const int32_t* block_table, int table_stride, void* out, int64_t out_stride,
                                               int n_tokens, int n_head, int n_kv_head, int head_dim, int page_size, float scale, int window,
                                               const float* distance, const float* sink, void* stream) {
    return lb_paged_attention_generic_capped(dtype, q, q_stride, cache, tok_seq, positions, block_table, table_stride, out, out_stride, n_tokens, n_head,
                                             n_kv_head, head_dim, page_size, scale, window, distance, sink, 0.0f, stream);
}

extern "C" int lb_paged_attention_generic_capped(int dtype, const void* q, int64_t q_stride, const void* cache, const int32_t* tok_seq,
                                                 const int32_t* positions, const int32_t* block_table, int table_stride, void* out, int64_t out_stride,
                                                 int n_tokens, int n_head, int n_kv_head, int head_dim, int page_size, float scale, int window,
                                                 const float* distance, const float* sink, float soft_cap, void* stream) {
    LB_CHECK_ARG(soft_cap >= 0.0f && (soft_cap == 0.0f || distance == nullptr), "attention: a soft cap is positive and goes without a penalty by distance");
    LB_CHECK_ARG(n_tokens >= 0 && n_head > 0 && n_kv_head > 0 && page_size > 0, "attention: bad sizes");
    LB_CHECK_ARG(n_head % n_kv_head == 0, "attention: n_head %d is not a multiple of n_kv_head %d", n_head, n_kv_head);
    LB_CHECK_ARG(head_dim > 0 && head_dim <= kMaxHeadDim, "attention: head_dim %d is outside (0, %d]", head_dim,
                 kMaxHeadDim);
    if (n_tokens == 0) return LB_OK;
    auto s = static_cast<cudaStream_t>(stream);
    if (dtype == LB_F32)
        return launch<float>(q, q_stride, cache, tok_seq, positions, block_table, table_stride, out, out_stride,
                             n_tokens, n_head, n_kv_head, head_dim, page_size, scale, window, distance, sink, soft_cap, s);
    if (dtype == LB_BF16)
        return launch<__nv_bfloat16>(q, q_stride, cache, tok_seq, positions, block_table, table_stride, out,
                                     out_stride, n_tokens, n_head, n_kv_head, head_dim, page_size, scale, window, distance, sink, soft_cap, s);
    return lb_fail(LB_ERR_INVALID_ARGUMENT, "attention: unknown dtype %d", dtype);
}
