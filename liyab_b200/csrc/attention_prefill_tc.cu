// Prefill attention for bfloat16 on the fifth-generation tensor cores (head size
// 64): the step's prompt portions (any lengths, cut anywhere) against their
// requests' paged keys and values.
//
// One block serves 128 consecutive query tokens of one request and one head and
// walks the keys the tile can see in tiles of 128 (eight runs of 16 keys, each
// inside one page):
//   warps 0..7  softmax, two threads per query row (tensor-memory lane = row; warps
//               0..3 take the first 64 keys of a tile, warps 4..7 the others; the two
//               maxima of a row meet in shared memory): scale, causal/window mask,
//               running maximum, exp2, the probabilities as bfloat16 back into tensor
//               memory, where the second product takes its first operand from, and the
//               rescaling of O when a maximum moved.  Runs of 32 keys that no row
//               of a warp sees, and warps without rows, cost nothing.
//   warp 8      TMA producer.  The query tile comes from the activations through
//               one tensor map, key and value tiles from the cache through another
//               ([all rows of all pages][64]): lanes 0..7 fetch the eight 16-key
//               boxes of a key tile, lanes 8..15 those of the value tile, two tiles
//               of each ahead.  A box past the last visible key is asked for at an
//               out-of-range row and arrives as zeros.
//   warp 9      issues tcgen05.mma: S = Q K^T (128 x 128, columns 0..127 of tensor
//               memory) and O += P V (columns 128..191 hold P, two keys a column,
//               192..255 O), the scores of tile j+1 before the update of tile j.  V is
//               used as it lies in the cache ([key][dim], the "MN-major" operand form).
// What bounds it: a tile's 16,384 exponentials take the SM's special-function units
// 1,024 cycles, its products some 500 of the tensor pipe, and a tile is a chain (scores,
// maximum, exponentials, update).  So two blocks share an SM (256 columns of tensor
// memory and 82 KB each): one block's chain and its start hide under the other's
// exponentials, or one where the step's plan says so: where a few long blocks set the time, and above all with capped scores or a penalty by distance, whose two or three
// special functions a score two blocks share (2 requests x 12 heads x 1,024 tokens capped 33.0 / 27.5 us, 1 x 16 x 2,048 70 / 52).  Measured (us a launch, 20 a graph; one block of sixteen softmax warps an SM with the probabilities through shared memory /
// here / the mma.sync kernel): 2 requests x 12 heads x 1,024 tokens 21.1 / 17.4 / 40.3, 5 x 25 x 469 36.7 / 18.5 / 40.5, 1 x 25 x 453
// 12.9 / 8.8 / 19.3, 8 x 12 x 180 14.9 / 7.1 / 10.7, 1 x 12 x 37 7.0 / 3.9 / 4.1.  Long contexts with few blocks are the chain: some 2,600 cycles
// a tile.  On the way: issuing the products and the copies from a branch on the lane's number took 700 cycles for eight products and
// 770 for eight boxes (370 and 310 from an elected lane, see elect_one), so that the copies, not the softmax, set the pace.
// Softmax, sums and both accumulators are 32-bit.  Every wait is bounded; a wait
// that runs out records a code in the device status word and the block drains
// its copies, frees tensor memory and returns.
//
// Reference formulas: scores, causal range, softmax and weighted values
// (src/core/transformer.cpp:2303-2313, 497-510, 2327-2341, 2344-2358).
#include "api.h"
#include "common.cuh"
#include "tcgen05.cuh"

#include <algorithm>
#include <math_constants.h>

namespace {

using namespace lb_tc;

constexpr int kHD = 64;
constexpr int kBM = 128;              // query rows per block
constexpr int kBN = 128;              // keys per tile
constexpr int kStages = 2;            // tiles of keys, and of values, in shared memory
constexpr int kThreads = 320;
constexpr int kParts = 2;             // threads per query row, each with 64 of a tile's 128 keys
constexpr int kKeys = kBN / kParts;
constexpr int kSoftmaxWarps = 4 * kParts;
constexpr int kProducerWarp = kSoftmaxWarps, kProductWarp = kSoftmaxWarps + 1;
constexpr float kLog2e = 1.4426950408889634f;
constexpr int kTileBytes = 128 * 128;          // [128 rows][128 bytes]: Q, a K tile, a V tile
constexpr uint32_t kTmemCols = 256, kPCol = 128, kOCol = 192;

struct Control {
    uint64_t q_full;
    uint64_t k_full[kStages], k_empty[kStages];
    uint64_t v_full[kStages], v_empty[kStages];
    uint64_t s_full, s_free, p_full, o_done;
    uint32_t tmem_base;
    int abort_flag;
    float row_max[2][kParts][kBM];        // [tile parity][key part][row]: the parts' maxima of a tile; NaN: that part gave up
    float row_sum[kParts][kBM];           // [key part][row]: the parts' sums at the end
};

__device__ __forceinline__ void give_up(Control* c, int* status, int site) {
    atomicCAS(status, 0, (0xA << 12) | site);
    *(volatile int*)&c->abort_flag = 1;
}

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
          "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
// 2^x (the exponentials' arguments are at most 0 up to rounding): the hardware approximation alone (results below the normal range become zero).
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// 1 / x for x >= 1 (0 above the normal range), log2 x for x in the normal range: the hardware approximations alone as well.
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float lg2_approx(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// The wait for a load, tied to its registers so that nothing is made of them before it.
__device__ __forceinline__ void tmem_ld_wait32(uint32_t (&v)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]), "+r"(v[10]),
                   "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]), "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]),
                   "+r"(v[21]), "+r"(v[22]), "+r"(v[23]), "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]), "+r"(v[30]), "+r"(v[31])
                 :: "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// The product with its first operand in tensor memory (lane = row, two bfloat16 values of K to a column).
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Descriptor of the value tile as the second operand in its MN-major form: rows of 64 dims (128 bytes, swizzled by
// TMA), eight keys to a 1024-byte group; both offset fields name that group stride.
__device__ __forceinline__ uint64_t umma_desc_mn(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(1024 >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// Instruction descriptor as umma_idesc, with the second operand MN-major (bit 16).
__host__ __device__ constexpr uint32_t umma_idesc_b_mn(int m, int n) { return umma_idesc(m, n) | (1u << 16); }

// The query tile that the block of this number serves: among every 32 requests the last tiles first, which see the most keys.  The grid holds
// no more blocks than tiles can exist among its tokens (a block that finds none still costs a launch: 0.5 us for every 148 with one block
// an SM).  False: no such tile.
__device__ __forceinline__ bool find_tile(const int32_t* __restrict__ q_start, int n_seq, int min_len, int& number, int lane, int* seq, int* tile) {
    for (int s0 = 0; s0 < n_seq; s0 += 32) {
        const int s = s0 + lane, len = s < n_seq ? q_start[s + 1] - q_start[s] : 0;
        const int mine = len >= min_len ? (len + kBM - 1) / kBM : 0;
        for (int t = __reduce_max_sync(0xffffffffu, mine) - 1; t >= 0; --t) {
            const uint32_t with = __ballot_sync(0xffffffffu, mine > t);
            const int count = __popc(with);
            if (number < count) {
                const uint32_t it = __ballot_sync(0xffffffffu, mine > t && __popc(with & ((1u << lane) - 1u)) == number);
                *seq = s0 + __ffs(it) - 1;
                *tile = t;
                return true;
            }
            number -= count;
        }
    }
    return false;
}

// The number-th request of one token; -1: there is none.
__device__ __forceinline__ int find_single(const int32_t* __restrict__ q_start, int n_seq, int number, int lane) {
    for (int s0 = 0; s0 < n_seq; s0 += 32) {
        const int s = s0 + lane;
        const bool single = s < n_seq && q_start[s + 1] - q_start[s] == 1;
        const uint32_t with = __ballot_sync(0xffffffffu, single);
        if (number < __popc(with)) return s0 + __ffs(__ballot_sync(0xffffffffu, single && __popc(with & ((1u << lane) - 1u)) == number)) - 1;
        number -= __popc(with);
    }
    return -1;
}

__device__ __forceinline__ void unpack_bf16(const uint4& u, float (&f)[8]) {
    f[0] = __uint_as_float(u.x << 16); f[1] = __uint_as_float(u.x & 0xffff0000u);
    f[2] = __uint_as_float(u.y << 16); f[3] = __uint_as_float(u.y & 0xffff0000u);
    f[4] = __uint_as_float(u.z << 16); f[5] = __uint_as_float(u.z & 0xffff0000u);
    f[6] = __uint_as_float(u.w << 16); f[7] = __uint_as_float(u.w & 0xffff0000u);
}

// 16 bytes global -> shared; when `valid` is false nothing is read and the destination is filled with zeros.
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}

// A request's one token and one head (with a key/value head of its own) by a whole block on the 32-bit units, as the decode kernel does it
// (attention_decode_mma.cu, SINGLE): a pair of lanes has a key's score, a lane eight dims of four keys of the update.  A lane copies the pieces that it will
// read itself, two tiles of 16 keys ahead, into places of its own (no barrier); all of a block's shared memory is on its way at once.
// A step that mixes a portion with single tokens has blocks without a query tile anyway, and the portion's few blocks leave most of the GPU idle, while
// a launch of their own takes the single tokens as long as the portion: a step of XL with 12 single tokens beside a portion of 453 4.44 -> 4.23 ms (host/kernels.cpp has
// the launches and where they pay).  Bound by the bytes on their way: the two lanes of a key take its pieces in turn, so that a copy of the warp asks for
// whole sectors (halves of 32 dims each: 22.7 us for that attention in place of 20.0, 41.5 in place of 29.9 for 4 tokens on 6000 keys); without the ring, straight to
// registers, that step took 4.68 ms.
template <bool PLAIN>
__device__ void serve_single(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* cache, const int32_t* __restrict__ table, __nv_bfloat16* __restrict__ out,
                             int pos, int head, int n_head, int page_shift, float scale, int window, const float* __restrict__ distance,
                             const float* __restrict__ sink, float soft_cap, float bound, uint8_t* smem) {
    constexpr int kWarps = kThreads / 32, kKeysTile = 16, kState = kHD + 2, kRing = 2;
    static_assert(kWarps * kRing * 8 * 32 * 16 == (1 + 2 * kStages) * kTileBytes, "the rings take the place of the query, key and value tiles");
    static_assert(kHD * sizeof(float) <= sizeof(Control), "the query lies behind them");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint4* ring = reinterpret_cast<uint4*>(smem) + (size_t)warp * kRing * 8 * 32 + lane;      // [stage][piece: 4 of a key, 4 of values][lane]
    float* q_s = reinterpret_cast<float*>(smem + (1 + 2 * kStages) * kTileBytes);               // the query
    float* red = reinterpret_cast<float*>(smem);                                              // at the end: [warp][maximum, sum, 64 values]
    const int page_size = 1 << page_shift, key = lane >> 1, half = lane & 1;
    const int first = lb_first_visible(pos, window), tile0 = first / kKeysTile, n_tiles = pos / kKeysTile + 1 - tile0;
    const int my_tiles = n_tiles > warp ? (n_tiles - warp + kWarps - 1) / kWarps : 0;
    const size_t v_plane = (size_t)n_head * page_size * kHD;
    int page_reg = 0;
    auto tile_at = [&](int i) { return (tile0 + warp + kWarps * i) * kKeysTile; };
    auto load = [&](int i) {                    // the page numbers of 32 tiles are read at once
        if ((i & 31) == 0) page_reg = i + lane < my_tiles ? table[tile_at(i + lane) >> page_shift] : 0;
        const int page = __shfl_sync(0xffffffffu, page_reg, i & 31), j0 = tile_at(i), j = j0 + key;
        const __nv_bfloat16* rows = cache + (((size_t)page * 2 * n_head + head) * page_size + (j0 & (page_size - 1))) * kHD;
        uint4* to = ring + (i % kRing) * 8 * 32;
#pragma unroll
        for (int c = 0; c < 4; ++c) cp_async16(to + c * 32, rows + key * kHD + (2 * c + half) * 8, j >= first && j <= pos);
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4) {
            const int vk = (lane >> 3) * 4 + k4;
            cp_async16(to + (4 + k4) * 32, rows + v_plane + vk * kHD + (lane & 7) * 8, j0 + vk >= first && j0 + vk <= pos);
        }
    };
    // Keys and values of earlier positions are there before the kernel before this one ends; that kernel writes the newest position's.
    bool asked[kRing];
#pragma unroll
    for (int i = 0; i < kRing; ++i) {
        asked[i] = i >= my_tiles || tile_at(i) + kKeysTile <= pos;
        if (asked[i] && i < my_tiles) load(i);
    }
    lb_wait_for_predecessor();
    lb_dependents_may_launch();
#pragma unroll
    for (int i = 0; i < kRing; ++i) {           // a tile held back is the request's last: those before it are asked for already
        if (!asked[i]) load(i);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if (threadIdx.x < kHD) q_s[threadIdx.x] = __bfloat162float(q[threadIdx.x]);
    __syncthreads();
    const lb_soft_cap capped(PLAIN ? 0.0f : soft_cap, bound);
    const bool biased = !PLAIN && distance != nullptr;
    const float r1 = biased ? distance[head] : 0.0f, r2 = biased ? distance[n_head + head] : 0.0f, sc = scale * kLog2e;
    float m = -CUDART_INF_F, l = 0.0f, o[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int i = 0; i < my_tiles; ++i) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        const uint4* from = ring + (i % kRing) * 8 * 32;
        float dot[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            float kf[8];
            unpack_bf16(from[c * 32], kf);
            const float4 qa = *reinterpret_cast<const float4*>(q_s + (2 * c + half) * 8), qb = *reinterpret_cast<const float4*>(q_s + (2 * c + half) * 8 + 4);
            dot[0] = fmaf(qa.x, kf[0], dot[0]); dot[1] = fmaf(qa.y, kf[1], dot[1]);
            dot[2] = fmaf(qa.z, kf[2], dot[2]); dot[3] = fmaf(qa.w, kf[3], dot[3]);
            dot[0] = fmaf(qb.x, kf[4], dot[0]); dot[1] = fmaf(qb.y, kf[5], dot[1]);
            dot[2] = fmaf(qb.z, kf[6], dot[2]); dot[3] = fmaf(qb.w, kf[7], dot[3]);
        }
        const int j = tile_at(i) + key;
        float s1 = (dot[0] + dot[1]) + (dot[2] + dot[3]);
        s1 = (s1 + __shfl_xor_sync(0xffffffffu, s1, 1)) * sc;
        if (capped.on) s1 = capped(s1);
        if (biased) s1 -= lb_distance_penalty_log2(r1, r2, max(pos - j, 0));
        if (j < first || j > pos) s1 = -CUDART_INF_F;
        if (__any_sync(0xffffffffu, s1 > m)) {                    // a maximum moved: rare after the first tiles
            float mx = s1;
#pragma unroll
            for (int d = 2; d < 32; d *= 2) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
            mx = fmaxf(mx, m);
            const float corr = exp2f(m - mx);
            m = mx;
            l *= corr;
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] *= corr;
        }
        const float p = exp2f(s1 - (m == -CUDART_INF_F ? 0.0f : m));
        l += half == 0 ? p : 0.0f;
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4) {
            const float pk = __shfl_sync(0xffffffffu, p, 2 * ((lane >> 3) * 4 + k4));
            float vf[8];
            unpack_bf16(from[(4 + k4) * 32], vf);
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] = fmaf(pk, vf[e], o[e]);
        }
        if (i + kRing < my_tiles) load(i + kRing);          // its place has been read, by this lane alone
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    l = lb_warp_sum(l);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        o[e] += __shfl_xor_sync(0xffffffffu, o[e], 8);
        o[e] += __shfl_xor_sync(0xffffffffu, o[e], 16);
    }
    __syncthreads();                            // the rings have been read
    if (lane < 8) {
        float* st = red + warp * kState;
        if (lane == 0) { st[0] = m; st[1] = l; }
#pragma unroll
        for (int e = 0; e < 8; ++e) st[2 + lane * 8 + e] = o[e];
    }
    __syncthreads();
    if (threadIdx.x < kHD) {
        const int d = threadIdx.x;
        float mm = -CUDART_INF_F, ll = 0.0f, a = 0.0f;
        for (int w = 0; w < kWarps; ++w) mm = fmaxf(mm, red[w * kState]);
        for (int w = 0; w < kWarps; ++w) {
            const float* st = red + w * kState;
            const float f = mm == -CUDART_INF_F ? 0.0f : exp2f(st[0] - mm);
            ll += st[1] * f;
            a += st[2 + d] * f;
        }
        if (sink != nullptr) a *= lb_sink_join_exp2(sink[head] * kLog2e, mm, ll);
        out[d] = __float2bfloat16_rn(a / ll);
    }
}

// PLAIN: no soft cap on the scores and no penalty by distance.
template <bool PLAIN>
__global__ void __launch_bounds__(kThreads, 2)
prefill_attention_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv,
                            const int32_t* __restrict__ q_start, const int32_t* __restrict__ n_past,
                            const int32_t* __restrict__ block_table, int table_stride, __nv_bfloat16* __restrict__ out,
                            int64_t out_stride, int n_head, int n_kv_head, int page_shift, int kv_rows, float scale, int window,
                            const float* __restrict__ distance, const float* __restrict__ sink,
                            float soft_cap, float bound, int n_seq, int min_len, const __nv_bfloat16* __restrict__ q, int64_t q_stride, const __nv_bfloat16* cache,
                            int singles, int* status) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* q_s = base;                                   // 16 KB
    uint8_t* k_s = q_s + kTileBytes;                       // [kStages] 16 KB
    uint8_t* v_s = k_s + kStages * kTileBytes;             // [kStages] 16 KB
    Control* c = reinterpret_cast<Control*>(v_s + kStages * kTileBytes);
    volatile int* abort_flag = &c->abort_flag;

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // one number for the warp
    // Where portions start, how far their requests are and the block tables came from the host before any kernel of the
    // step, keys and values of earlier positions from earlier steps: they are read before this kernel waits for the one
    // before it.  A block without rows ends at once (one of the grid waits all the same, so that this kernel never ends
    // before the one before it).
    const int head = (int)(blockIdx.x % (unsigned)n_head);
    int seq = 0, tile_q = 0, number = (int)(blockIdx.x / (unsigned)n_head);
    if (!find_tile(q_start, n_seq, min_len, number, lane, &seq, &tile_q)) {
        // The blocks past the last query tile take the single tokens, where they are asked to.
        const int single = singles != 0 ? find_single(q_start, n_seq, number, lane) : -1;
        if (single >= 0) {
            const int token = q_start[single];
            serve_single<PLAIN>(q + (size_t)token * q_stride + (size_t)head * kHD, cache, block_table + (size_t)single * table_stride,
                                out + (size_t)token * out_stride + (size_t)head * kHD, n_past[single], head, n_head, page_shift, scale, window, distance, sink,
                                soft_cap, bound, base);
            return;
        }
        if (blockIdx.x == gridDim.x - 1) lb_wait_for_predecessor();
        return;
    }
    const int row0 = q_start[seq], q_len = q_start[seq + 1] - row0;
    const int past = n_past[seq];
    const int kvh = head / (n_head / n_kv_head);
    const int page_size = 1 << page_shift;
    const int rows_here = min(kBM, q_len - tile_q * kBM);
    const int p_min = past + tile_q * kBM, p_max = p_min + rows_here - 1;
    const int kv_lo = lb_first_visible(p_min, window) / kBN * kBN;
    const int n_tiles = (p_max - kv_lo) / kBN + 1;

    if (threadIdx.x == 0) {
        prefetch_tensormap(&map_q);
        prefetch_tensormap(&map_kv);
        mbar_init(&c->q_full, 1);
        for (int i = 0; i < kStages; ++i) {
            mbar_init(&c->k_full[i], 1);
            mbar_init(&c->k_empty[i], 1);
            mbar_init(&c->v_full[i], 1);
            mbar_init(&c->v_empty[i], 1);
        }
        mbar_init(&c->s_full, 1);
        mbar_init(&c->s_free, kSoftmaxWarps);      // one arrival per softmax warp
        mbar_init(&c->p_full, kSoftmaxWarps);
        mbar_init(&c->o_done, 1);
        c->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kProductWarp) {
        tmem_alloc(&c->tmem_base, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, c->tmem_base, 0);

    if (warp == kProducerWarp) {
        // ---- producer: the key and value tiles two ahead, Q as soon as the kernel before this one (whose output it is,
        // like the keys and values of the step's own tokens) has ended.
        const int32_t* table = block_table + (size_t)seq * table_stride;
        int keys = 0, values = 0;                      // tiles asked for
        bool waited = false, ok = true;
        // Lane `sub` of 0..7 finds the rows of the tile's box `sub` of keys, those 8 above it of values; the next tile's while this one's is asked for.
        auto row_of = [&](int tile) -> int {
            const int j0 = kv_lo + tile * kBN + (lane & 7) * 16;
            if (lane >= 16 || j0 > p_max) return kv_rows;                // out of range: the box arrives as zeros
            const int page = table[j0 >> page_shift];
            return page >= 0 ? ((page * 2 + (lane >> 3)) * n_kv_head + kvh) * page_size + (j0 & (page_size - 1)) : kv_rows;
        };
        int row = row_of(0);
        for (int tile = 0; tile < n_tiles; ++tile) {
            const int st = tile % kStages;
            const uint32_t ph = (tile / kStages) & 1;
            const int next_row = tile + 1 < n_tiles ? row_of(tile + 1) : 0;
            if (!waited && (tile >= kStages || kv_lo + (tile + 1) * kBN > past)) {
                lb_wait_for_predecessor();
                waited = true;
                if (elect_one()) {
                    mbar_expect_tx(&c->q_full, kTileBytes);
                    tma_load_2d(q_s, &map_q, &c->q_full, head * kHD, row0 + tile_q * kBM);
                }
                __syncwarp();
            }
            for (int kv = 0; kv < 2; ++kv) {
                uint64_t* empty = kv == 0 ? &c->k_empty[st] : &c->v_empty[st];
                uint64_t* full = kv == 0 ? &c->k_full[st] : &c->v_full[st];
                uint8_t* dst = (kv == 0 ? k_s : v_s) + (size_t)st * kTileBytes;
                ok = __all_sync(0xffffffffu, mbar_wait(empty, ph ^ 1, abort_flag));
                if (!ok) break;
                if (elect_one()) mbar_expect_tx(full, kTileBytes);
                __syncwarp();
#pragma unroll
                for (int sub = 0; sub < 8; ++sub) {          // one lane for all boxes, the operands the warp's: see elect_one
                    const int box_row = __shfl_sync(0xffffffffu, row, kv * 8 + sub);
                    if (elect_one()) tma_load_2d(dst + sub * 2048, &map_kv, full, 0, box_row);
                }
                __syncwarp();
                (kv == 0 ? keys : values) = tile + 1;
            }
            if (!ok) break;
            row = next_row;
        }
        if (lane == 0 && !ok) give_up(c, status, 1);
        if (*abort_flag != 0 && lane == 0) {
            // Leave no copy in flight: the barriers of the last loads issued complete when their bytes landed.
            if (waited) mbar_wait(&c->q_full, 0, nullptr);
            for (int tile = max(keys - kStages, 0); tile < keys; ++tile) mbar_wait(&c->k_full[tile % kStages], (tile / kStages) & 1, nullptr);
            for (int tile = max(values - kStages, 0); tile < values; ++tile) mbar_wait(&c->v_full[tile % kStages], (tile / kStages) & 1, nullptr);
        }
    } else if (warp == kProductWarp) {
        // ---- products: scores of tile j + 1 before the update of tile j.
        lb_wait_for_predecessor();
        lb_dependents_may_launch();
        constexpr uint32_t idesc_s = umma_idesc(kBM, kBN);
        constexpr uint32_t idesc_o = umma_idesc_b_mn(kBM, kHD);
        // Descriptors are made once per operand tile and moved by addition (the start address sits in the low bits
        // in units of 16 bytes, and no tile crosses the field's range).
        const uint64_t dq = umma_desc(smem_u32(q_s));
        bool ok = __all_sync(0xffffffffu, mbar_wait(&c->q_full, 0, abort_flag));
        if (!ok) give_up(c, status, 2);
        auto scores = [&](int tile) -> bool {
            const int st = tile % kStages;
            if (!__all_sync(0xffffffffu, mbar_wait(&c->k_full[st], (tile / kStages) & 1, abort_flag))) { give_up(c, status, 3); return false; }
            if (tile > 0 && !__all_sync(0xffffffffu, mbar_wait(&c->s_free, (tile - 1) & 1, abort_flag))) { give_up(c, status, 4); return false; }
            tc_fence_after();
            const uint64_t dk = umma_desc(smem_u32(k_s + (size_t)st * kTileBytes));
            if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < kHD / kUmmaK; ++kk)
                    umma_bf16(tmem_base, dq + (uint64_t)(kk * 2), dk + (uint64_t)(kk * 2), idesc_s, kk != 0 ? 1u : 0u);
                umma_commit(&c->s_full);
                umma_commit(&c->k_empty[st]);
            }
            __syncwarp();
            return true;
        };
        if (ok) ok = scores(0);
        for (int tile = 0; tile < n_tiles && ok; ++tile) {
            if (tile + 1 < n_tiles) ok = scores(tile + 1);
            if (!ok) break;
            const int st = tile % kStages;
            if (!__all_sync(0xffffffffu, mbar_wait(&c->v_full[st], (tile / kStages) & 1, abort_flag) && mbar_wait(&c->p_full, tile & 1, abort_flag))) {
                give_up(c, status, 5);
                break;
            }
            tc_fence_after();
            const uint64_t dv = umma_desc_mn(smem_u32(v_s + (size_t)st * kTileBytes));
            if (elect_one()) {
#pragma unroll
                for (int ks = 0; ks < kBN / kUmmaK; ++ks)       // 16 keys: eight columns of P, 2048 bytes of V
                    umma_bf16_ts(tmem_base + kOCol, tmem_base + kPCol + ks * 8, dv + (uint64_t)((ks * 2048) >> 4), idesc_o, (tile | ks) != 0 ? 1u : 0u);
                umma_commit(&c->o_done);            // O holds tile `tile`, and its probabilities have been read
                umma_commit(&c->v_empty[st]);
            }
            __syncwarp();
        }
    } else {
        // ---- softmax
        lb_wait_for_predecessor();                  // the output rows may still be read by an earlier kernel
        lb_dependents_may_launch();
        const int quarter = warp & 3, part = warp >> 2;
        const int r = quarter * 32 + lane;                              // row of the tile = lane of tensor memory
        const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16);
        const bool rows = quarter * 32 < rows_here;                     // a warp without rows only keeps the barriers going
        const int pos = p_min + min(r, rows_here - 1);                  // rows past the end copy the last one; not stored
        const int pos_lo = p_min + min(quarter * 32, rows_here - 1), pos_hi = p_min + min(quarter * 32 + 31, rows_here - 1);
        const int first = lb_first_visible(pos, window), first_lo = lb_first_visible(pos_lo, window), first_hi = lb_first_visible(pos_hi, window);
        // With a soft cap the scores are brought to base 2 as they are capped, so nothing is left to multiply.
        const lb_soft_cap capped(PLAIN ? 0.0f : soft_cap, bound);
        const float raw_sc = scale * kLog2e, sc = !PLAIN && capped.on ? 1.0f : raw_sc;
        const float cap_in = raw_sc * capped.in;
        // The head's penalty by distance in the units of the raw scores (which are multiplied by sc later): a key d positions
        // back loses r1 ln(1 + r2 d) / scale = pen log2(1 + r2 d), or, with r2 < 0, r1 d / scale = pen d.
        const float r2 = !PLAIN && distance != nullptr ? distance[n_head + head] : 0.0f;
        const float pen = !PLAIN && distance != nullptr ? distance[head] * (r2 < 0.0f ? 1.0f : 0.6931471805599453f) / scale : 0.0f;
        float m = -CUDART_INF_F, l = 0.0f;                              // l: this thread's part of the row's sum
        bool ok = true;
        for (int tile = 0; tile < n_tiles; ++tile) {
            if (ok) {
                ok = __all_sync(0xffffffffu, mbar_wait(&c->s_full, tile & 1, abort_flag));      // one answer for the warp
                if (!ok) give_up(c, status, 6);
            }
            if (!rows) {
                // Like the others it says that a tile's probabilities are there only after the update of the tile before: the next tile's
                // scores may be there earlier than that, and two arrivals of this warp would count as two warps'.
                if (ok && tile > 0) {
                    ok = __all_sync(0xffffffffu, mbar_wait(&c->o_done, (tile - 1) & 1, abort_flag));
                    if (!ok) give_up(c, status, 8);
                }
                if (!ok) break;
                if (lane == 0) {
                    mbar_arrive(&c->s_free);
                    mbar_arrive(&c->p_full);
                }
                continue;
            }
            tc_fence_after();
            const int t0 = kv_lo + tile * kBN, j0 = t0 + part * kKeys;       // this thread's first key of the tile
            // The maximum of this part of the row.  Its 64 scores are taken 32 at a time (all of them beside one another do not fit the
            // registers of a thread where two blocks share an SM): the second half stays for the exponentials, the first is read again.
            uint32_t v[32];
            bool seen[2];
            float mx0 = -CUDART_INF_F, mx1 = -CUDART_INF_F, mx2 = -CUDART_INF_F, mx3 = -CUDART_INF_F;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int jh = j0 + h * 32;
                seen[h] = ok && jh <= pos_hi && jh + 31 >= first_lo;      // the same for the warp
                if (!seen[h]) continue;
                tmem_ld32(t_row + (uint32_t)(part * kKeys + h * 32), v);
                tmem_ld_wait32(v);
                if (!PLAIN && capped.on && capped.series) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(capped(__uint_as_float(v[i]) * raw_sc));
                } else if (!PLAIN && capped.on) {
                    // The other form of lb_soft_cap, out - 2 out / (1 + 2^(in s)).
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        v[i] = __float_as_uint(fmaf(-2.0f * capped.out, rcp_approx(1.0f + ex2_approx(__uint_as_float(v[i]) * cap_in)), capped.out));
                } else if (!PLAIN && distance != nullptr && r2 < 0.0f) {
                    // pen (pos - jh - i) = b0 - pen i.
                    const float b0 = pen * (float)(pos - jh);
#pragma unroll
                    for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) - fmaf(-pen, (float)i, b0));
                } else if (!PLAIN && distance != nullptr) {
                    // 1 + r2 (pos - jh - i) = a0 - r2 i; keys after the query (masked below) are kept from an argument below zero.
                    const float a0 = fmaf(r2, (float)(pos - jh), 1.0f);
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        v[i] = __float_as_uint(fmaf(-pen, lg2_approx(fmaxf(fmaf(-r2, (float)i, a0), 1e-30f)), __uint_as_float(v[i])));
                }
                const bool masked = jh + 31 > pos_lo || jh < first_hi;
                if (masked) {
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if (jh + i > pos || jh + i < first) v[i] = __float_as_uint(-CUDART_INF_F);
                }
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    mx0 = fmaxf(mx0, __uint_as_float(v[i]));
                    mx1 = fmaxf(mx1, __uint_as_float(v[i + 1]));
                    mx2 = fmaxf(mx2, __uint_as_float(v[i + 2]));
                    mx3 = fmaxf(mx3, __uint_as_float(v[i + 3]));
                }
                if (h == 0 && (!PLAIN || masked)) {             // read again as they are now
#pragma unroll
                    for (int g = 0; g < 2; ++g) tmem_st16(t_row + (uint32_t)(part * kKeys + g * 16), v + g * 16);
                    tmem_st_wait();
                }
            }
            // The two parts of a row meet (64 threads, warps `quarter` and `quarter + 4`), and agree on whether to go on.
            c->row_max[tile & 1][part][r] = ok ? fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)) : CUDART_NAN_F;
            named_barrier(1 + quarter, 32 * kParts);
            const float part0 = c->row_max[tile & 1][0][r], part1 = c->row_max[tile & 1][1][r];
            if (__any_sync(0xffffffffu, isnan(part0) || isnan(part1))) { ok = false; break; }
            // A maximum that lags behind the row's (by up to 2^8, which would leave O alone more often) was 0 to 0.4 us faster a launch and no
            // longer gives the largest key the exact weight 1: relative error 1.92e-3 against 1.75e-3 on mixed portions; so it never lags.
            const float m_new = fmaxf(m, fmaxf(part0, part1) * sc);
            const float base_m = m_new == -CUDART_INF_F ? 0.0f : m_new;
            const float corr = exp2f(m - base_m);
            // Probabilities (masked scores are -inf: weight 0) and their sum: one multiply-add and one MUFU a score.
            float sum0 = 0.0f, sum1 = 0.0f;
#pragma unroll
            for (int h = 1; h >= 0; --h) {
                if (h == 0) {
                    if (seen[0]) {
                        tmem_ld32(t_row + (uint32_t)(part * kKeys), v);
                        tmem_ld_wait32(v);
                    }
                    // The scores have been read: the next tile's may overwrite them.  (One lane arrives for its warp: hundreds of
                    // arrivals on one barrier word would queue up behind one another.)
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&c->s_free);
                }
                uint32_t pk[16];
                if (seen[h]) {
#pragma unroll
                    for (int i = 0; i < 16; i += 2) {
                        const float p0 = ex2_approx(fmaf(__uint_as_float(v[2 * i]), sc, -base_m)), p1 = ex2_approx(fmaf(__uint_as_float(v[2 * i + 1]), sc, -base_m));
                        const float p2 = ex2_approx(fmaf(__uint_as_float(v[2 * i + 2]), sc, -base_m)), p3 = ex2_approx(fmaf(__uint_as_float(v[2 * i + 3]), sc, -base_m));
                        sum0 += p0 + p1;
                        sum1 += p2 + p3;
                        pk[i] = pack2(p0, p1);
                        pk[i + 1] = pack2(p2, p3);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i) pk[i] = 0u;
                }
                // The update of the tile before has read its probabilities, and O may be touched.
                if (h == 1 && tile > 0) {
                    ok = __all_sync(0xffffffffu, mbar_wait(&c->o_done, (tile - 1) & 1, abort_flag));
                    if (!ok) break;
                    tc_fence_after();
                }
                tmem_st16(t_row + kPCol + (uint32_t)(part * (kKeys / 2) + h * 16), pk);
            }
            if (!ok) { give_up(c, status, 8); continue; }              // the other part learns of it at the next tile; neither stores
            l = l * corr + (sum0 + sum1);
            m = m_new;
            // O *= corr where some row of the warp moved its maximum (never for the first tile: O is overwritten).  Each
            // part rescales 32 of the 64 columns.
            if (tile > 0 && __any_sync(0xffffffffu, corr != 1.0f)) {
                uint32_t o[32];
                tmem_ld32(t_row + kOCol + part * 32, o);
                tmem_ld_wait32(o);
#pragma unroll
                for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
#pragma unroll
                for (int h = 0; h < 2; ++h) tmem_st16(t_row + kOCol + part * 32 + h * 16, o + h * 16);
            }
            tmem_st_wait();
            // A 16-key box that straddles the last visible key brings rows of later positions with it: whatever the
            // cache holds there (it may be anything, also NaN) would meet its zero weight in the second product.
            // Those value rows (fewer than 16, in the last tile only) are zeroed here, after the tile has landed, by the
            // first warp (which has rows in every block).
            const int last = p_max - t0;                            // last visible row of the tile
            if (warp == 0 && last + 1 < kBN && (last + 1) % 16 != 0) {
                ok = __all_sync(0xffffffffu, mbar_wait(&c->v_full[tile % kStages], (tile / kStages) & 1, abort_flag));
                if (!ok) { give_up(c, status, 9); continue; }
                const int row = last + 1 + (lane & 15);
                if (row < (last / 16 + 1) * 16) {
                    uint4* dst = reinterpret_cast<uint4*>(v_s + (size_t)(tile % kStages) * kTileBytes + (size_t)row * 128) + (lane >> 4) * 4;
#pragma unroll
                    for (int i = 0; i < 4; ++i) dst[i] = make_uint4(0, 0, 0, 0);
                }
                fence_async_shared();               // those rows, written through the generic proxy, are read by the tensor core
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&c->p_full);
        }
        if (rows) {
            // The parts' sums meet, then each part normalises and stores 32 of the row's 64 values.
            c->row_sum[part][r] = l;
            named_barrier(1 + quarter, 32 * kParts);
            if (ok) {
                ok = __all_sync(0xffffffffu, mbar_wait(&c->o_done, (n_tiles - 1) & 1, abort_flag));
                if (!ok) give_up(c, status, 10);
            }
        }
        if (rows && ok) {
            tc_fence_after();
            const float total = c->row_sum[0][r] + c->row_sum[1][r];
            // A head's sink joins the row's divisor once, after all its keys (m: the row's maximum in the exponentials' base-2 scale).
            float divisor = total;
            const float share = sink != nullptr ? lb_sink_join_exp2(sink[head] * kLbLog2e, m, divisor) : 1.0f;
            const float inv = share / divisor;
            __nv_bfloat16* dst = out + (size_t)(row0 + tile_q * kBM + r) * out_stride + (size_t)head * kHD + part * 32;
            uint32_t o[32];
            tmem_ld32(t_row + kOCol + part * 32, o);
            tmem_ld_wait32(o);
            if (r < rows_here) {
#pragma unroll
                for (int q8 = 0; q8 < 4; ++q8) {
                    uint4 pk;
                    pk.x = pack2(__uint_as_float(o[q8 * 8]) * inv, __uint_as_float(o[q8 * 8 + 1]) * inv);
                    pk.y = pack2(__uint_as_float(o[q8 * 8 + 2]) * inv, __uint_as_float(o[q8 * 8 + 3]) * inv);
                    pk.z = pack2(__uint_as_float(o[q8 * 8 + 4]) * inv, __uint_as_float(o[q8 * 8 + 5]) * inv);
                    pk.w = pack2(__uint_as_float(o[q8 * 8 + 6]) * inv, __uint_as_float(o[q8 * 8 + 7]) * inv);
                    *reinterpret_cast<uint4*>(dst + q8 * 8) = pk;
                }
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == kProductWarp) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

}  // namespace

// Whether the tcgen05 prefill kernel takes the shape: head size 64, pages of 16 positions or more (a power of two).
extern "C" int lb_prefill_attention_tc_supports(int n_head, int n_kv_head, int head_dim, int page_size) {
    return n_kv_head > 0 && n_head % n_kv_head == 0 && head_dim == kHD && page_size >= 16 && (page_size & (page_size - 1)) == 0;
}

extern "C" int lb_prefill_attention_tc(const void* q, int64_t q_stride, int n_tokens, const void* cache, int n_pages,
                                       const int32_t* q_start, const int32_t* n_past, const int32_t* block_table,
                                       int table_stride, void* out, int64_t out_stride, int n_seq, int max_q_len, int n_head,
                                       int n_kv_head, int head_dim, int page_size, float scale, int window, void* stream) {
    return lb_prefill_attention_tc_biased(q, q_stride, n_tokens, cache, n_pages, q_start, n_past, block_table, table_stride, out, out_stride, n_seq, max_q_len,
                                          n_head, n_kv_head, head_dim, page_size, scale, window, nullptr, stream);
}

extern "C" int lb_prefill_attention_tc_biased(const void* q, int64_t q_stride, int n_tokens, const void* cache, int n_pages, const int32_t* q_start,
                                              const int32_t* n_past, const int32_t* block_table, int table_stride, void* out, int64_t out_stride,
                                              int n_seq, int max_q_len, int n_head, int n_kv_head, int head_dim, int page_size, float scale, int window,
                                              const float* distance, void* stream) {
    return lb_prefill_attention_tc_sink(q, q_stride, n_tokens, cache, n_pages, q_start, n_past, block_table, table_stride, out, out_stride, n_seq, max_q_len,
                                        n_head, n_kv_head, head_dim, page_size, scale, window, distance, nullptr, stream);
}

extern "C" int lb_prefill_attention_tc_sink(const void* q, int64_t q_stride, int n_tokens, const void* cache, int n_pages, const int32_t* q_start,
                                            const int32_t* n_past, const int32_t* block_table, int table_stride, void* out, int64_t out_stride,
                                            int n_seq, int max_q_len, int n_head, int n_kv_head, int head_dim, int page_size, float scale, int window,
                                            const float* distance, const float* sink, void* stream) {
    return lb_prefill_attention_tc_capped(q, q_stride, n_tokens, cache, n_pages, q_start, n_past, block_table, table_stride, out, out_stride, n_seq, max_q_len,
                                          n_head, n_kv_head, head_dim, page_size, scale, window, distance, sink, 0.0f, 0.0f, stream);
}

extern "C" int lb_prefill_attention_tc_capped(const void* q, int64_t q_stride, int n_tokens, const void* cache, int n_pages, const int32_t* q_start,
                                              const int32_t* n_past, const int32_t* block_table, int table_stride, void* out, int64_t out_stride,
                                              int n_seq, int max_q_len, int n_head, int n_kv_head, int head_dim, int page_size, float scale, int window,
                                              const float* distance, const float* sink, float soft_cap, float bound, void* stream) {
    return lb_prefill_attention_tc_portions(q, q_stride, n_tokens, cache, n_pages, q_start, n_past, block_table, table_stride, out, out_stride, n_seq, max_q_len,
                                            n_head, n_kv_head, head_dim, page_size, scale, window, distance, sink, soft_cap, bound, 1, stream);
}

extern "C" int lb_prefill_attention_tc_portions(const void* q, int64_t q_stride, int n_tokens, const void* cache, int n_pages, const int32_t* q_start,
                                              const int32_t* n_past, const int32_t* block_table, int table_stride, void* out, int64_t out_stride,
                                              int n_seq, int max_q_len, int n_head, int n_kv_head, int head_dim, int page_size, float scale, int window,
                                              const float* distance, const float* sink, float soft_cap, float bound, int min_len, void* stream) {
    return lb_prefill_attention_tc_mixed(q, q_stride, n_tokens, cache, n_pages, q_start, n_past, block_table, table_stride, out, out_stride, n_seq, max_q_len,
                                         n_head, n_kv_head, head_dim, page_size, scale, window, distance, sink, soft_cap, bound, min_len, 0, stream);
}

extern "C" int lb_prefill_attention_tc_mixed(const void* q, int64_t q_stride, int n_tokens, const void* cache, int n_pages, const int32_t* q_start,
                                              const int32_t* n_past, const int32_t* block_table, int table_stride, void* out, int64_t out_stride,
                                              int n_seq, int max_q_len, int n_head, int n_kv_head, int head_dim, int page_size, float scale, int window,
                                              const float* distance, const float* sink, float soft_cap, float bound, int min_len, int flags, void* stream) {
    LB_CHECK_ARG((flags & ~3) == 0, "prefill attention (tcgen05): unknown flags %d", flags);
    const int singles = flags & 1;
    LB_CHECK_ARG(singles == 0 || (min_len > 1 && n_head == n_kv_head), "prefill attention (tcgen05): single tokens beside the tiles need a key/value head to every query head and min_len above 1");
    LB_CHECK_ARG(soft_cap >= 0.0f && (soft_cap == 0.0f || distance == nullptr), "prefill attention (tcgen05): a soft cap is positive and goes without a penalty by distance");
    LB_CHECK_ARG(distance == nullptr || scale != 0.0f, "prefill attention (tcgen05): a penalty by distance needs a factor on the scores that is not zero");
    LB_CHECK_ARG(n_seq >= 0 && max_q_len >= 0 && n_tokens >= 0 && n_pages > 0, "prefill attention: bad sizes");
    if (!lb_prefill_attention_tc_supports(n_head, n_kv_head, head_dim, page_size))
        return lb_fail(LB_ERR_UNSUPPORTED, "prefill attention (tcgen05): unsupported shape heads %d/%d head_dim %d page_size %d",
                       n_head, n_kv_head, head_dim, page_size);
    LB_CHECK_ARG(q_stride % 8 == 0 && out_stride % 8 == 0 && ((uintptr_t)q & 15) == 0 && ((uintptr_t)out & 15) == 0 &&
                     ((uintptr_t)cache & 15) == 0,
                 "prefill attention (tcgen05): q, out and cache rows must be 16-byte aligned");
    // Every portion ends in a tile that may be partly empty; the others are full of the step's tokens.
    const int per_seq = (max_q_len + kBM - 1) / kBM;
    LB_CHECK_ARG(per_seq <= 65535, "prefill attention: a portion of %d tokens is too long for one launch", max_q_len);
    const long long blocks = n_head * std::min((long long)n_seq * per_seq, (long long)n_tokens / kBM + n_seq);
    LB_CHECK_ARG(blocks < (1ll << 31), "prefill attention: %lld query tiles and heads are too many for one launch", blocks);
    const long long kv_rows = (long long)n_pages * 2 * n_kv_head * page_size;
    LB_CHECK_ARG(kv_rows < (1ll << 31), "prefill attention (tcgen05): the cache has too many rows for one tensor map");
    if (n_seq == 0 || max_q_len == 0 || n_tokens == 0) return LB_OK;
    int page_shift = 0;
    while ((1 << page_shift) < page_size) ++page_shift;
    CUtensorMap map_q, map_kv;
    int rc = lb_tensor_map_2d(&map_q, q, 2, n_tokens, n_head * kHD, q_stride, kBM);
    if (rc == LB_OK) rc = lb_tensor_map_2d(&map_kv, cache, 2, (int)kv_rows, kHD, kHD, 16);
    if (rc != LB_OK) return rc;
    int* status = nullptr;
    rc = lb_tc_status_word(&status);
    if (rc != LB_OK) return rc;
    constexpr size_t kTwo = 1024 + (size_t)(1 + 2 * kStages) * kTileBytes + sizeof(Control), kOne = 114 * 1024;      // the least that keeps a second block out of an SM's 228 KB
    static bool configured = false;
    if (!configured) {
        for (auto* kernel : {prefill_attention_tc_kernel<true>, prefill_attention_tc_kernel<false>})
            LB_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kOne));
        configured = true;
    }
    const size_t smem = (flags & 2) != 0 ? kOne : kTwo;
    dim3 grid((unsigned)blocks);
    auto* kernel = soft_cap == 0.0f && distance == nullptr ? prefill_attention_tc_kernel<true> : prefill_attention_tc_kernel<false>;
    LB_CHECK_CUDA(lb_launch_overlapped(kernel, dim3(grid), dim3(kThreads), smem, static_cast<cudaStream_t>(stream), 
        map_q, map_kv, q_start, n_past, block_table, table_stride, (__nv_bfloat16*)out, out_stride, n_head, n_kv_head, page_shift,
        (int)kv_rows, scale, window, distance, sink, soft_cap, bound, n_seq, min_len,
        (const __nv_bfloat16*)q, q_stride, (const __nv_bfloat16*)cache, singles, status));
    LB_CHECK_LAUNCH();
    return LB_OK;
}
