// out[M, N] = epilogue(A[M, K] . W[N, K]^T) for many tokens: tiles of 256 tokens x BN features that two SMs make together.
//
// The persistent kernel of one block a tile (gemm_tcgen05_persistent.cu) is bound by what the SMs pull from L2: a 128 x 192 tile
// fetches 40 KB a k-block for 3.1 MFLOP.  Here the two blocks of a cluster issue tcgen05.mma with cta_group::2: each brings its
// 128 tokens and half of the tile's features (32 KB a k-block at BN = 256) and keeps the 128 x BN sums of its own tokens, 4.2 MFLOP for
// those 32 KB.  The float32 results and residuals pass through four strips of shared memory instead of a whole tile, which leaves
// room for five stages.
// Measured (B200, 20 launches a graph, TFLOP/s; one block a tile / here / cuBLAS with bfloat16 results and a bare epilogue): 2343 x 6400 x 1600 1062 / 1246 /
// 1347, with GELU 983 / 1147 / -; 2343 x 1600 x 6400 with residual 705 / 1183 / 1337; 2343 x 4800 x 1600 997 / 1221 / 1289.  GPT-2 XL, five prompts of 2,343 tokens: 11.77 -> 9.87 ms
// a step.  A k-block took 0.31 to 0.34 us whatever the tile's features and however few tiles run while a branch on the lane's number issued products and
// copies; from an elected lane (elect_one in tcgen05.cuh) it takes 0.20, 0.25 or 0.32 us at 128, 192 or 256 features until the operands of all
// blocks take longer from L2 (some 13 to 18 TB/s).  Two producer threads instead of one change nothing.
//
// Roles of a block's warps:
//   warp 0      TMA producer of the block's own operands; both blocks' copies count on the first block's barrier.
//   warp 1      (first block) issues the products of both; every commit arrives at both blocks' barriers.
//   warps 2..9  epilogue of the block's 128 tokens, in two groups of four that take alternate 128-byte-wide strips: tcgen05.ld,
//               bias, activation, residual (fetched by TMA a strip ahead into the slot that the result leaves from), one TMA store a strip.
// Two accumulators of up to 256 columns: a tile's epilogue runs under the next tile's products.
//
// Handshakes (mbarriers; waits are bounded, and one that runs out stops both blocks: they drain their copies, free tensor memory and
// return, with a code in the device status word):
//   full[s]        (first block) both blocks' k-block of stage s has landed
//   empty[s]       (both) the products have read stage s
//   acc_full[b]    (both) accumulator b is complete
//   acc_empty[b]   (first block) both blocks' epilogues have read accumulator b
//   res_full       (both) a group's residual strip has landed
//
// Epilogue order as the reference's (src/core/transformer.cpp:111-118, 4903-4912, 5526-5532): bias, activation, then the residual sum,
// all in 32-bit.
#include "api.h"
#include "common.cuh"
#include "gemm_tile.cuh"
#include "tcgen05.cuh"

namespace {

using namespace lb_tc;
using namespace lb_tile;

constexpr int kEpilogueWarps = 8;
constexpr int kThreads = 64 + 32 * kEpilogueWarps;
constexpr int kMaxStages = 8;
constexpr int kStripBytes = 128 * 128;
constexpr int kSlots = 2;                     // strips of a group in shared memory
constexpr int kATileBytes = kLaneTile * kBlockK * (int)sizeof(__nv_bfloat16);
constexpr size_t kSmemLimit = 227 * 1024;

static int g_withhold_next = 0;      // host side: the next launch's pairs leave their first accumulator's barriers unsignalled (tests)

struct Control {
    uint64_t full[kMaxStages];
    uint64_t empty[kMaxStages];
    uint64_t acc_full[2];
    uint64_t acc_empty[2];
    uint64_t res_full[2][kSlots];
    uint32_t tmem_base;
    int abort_flag;
};

__device__ __forceinline__ void give_up(Control* c, int* status, int site, int detail, uint32_t rank) {
    atomicCAS(status, 0, (0xE << 12) | (site << 8) | (detail & 0xff));
    c->abort_flag = 1;
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(peer_address(smem_u32(&c->abort_flag), rank ^ 1u)), "r"(1) : "memory");
}

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A tile of this block's operands; `bar` (an address of the cluster) may lie in the other block.
__device__ __forceinline__ void tma_load_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1)
        : "memory");
}

__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %3};\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %4, p;\n\t}"
        ::"r"(tmem_d), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Arrives at the barrier of this offset in both blocks once the products issued so far are complete.
__device__ __forceinline__ void commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((uint16_t)3) : "memory");
}

// A barrier of `count` threads whose answer is the same for all of them: whether any brought true.
__device__ __forceinline__ bool barrier_any(int id, int count, bool mine) {
    uint32_t any;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.or.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(any) : "r"(mine ? 1u : 0u), "r"(id), "r"(count) : "memory");
    return any != 0;
}

template <typename TO, int ACT, bool HAS_RES, bool KV>
__global__ void __launch_bounds__(kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_res,
                 const __grid_constant__ CUtensorMap map_out, const float* __restrict__ bias, int M, int N, int K, int BN, int n_stages, int* status,
                 int withhold, const KvTarget kv) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t stage_bytes = (uint32_t)(kLaneTile + BN / 2) * kBlockK * sizeof(__nv_bfloat16);
    constexpr int kStripCols = 128 / (int)sizeof(TO);
    uint8_t* staging = base + (size_t)n_stages * stage_bytes;                      // [group][slot] strips
    float* bias_s = reinterpret_cast<float*>(staging + 2 * kSlots * kStripBytes);  // [group][its strips' features]
    Control* c = reinterpret_cast<Control*>(bias_s + 2 * 128);
    volatile int* abort_flag = &c->abort_flag;
    const uint32_t stages_u32 = smem_u32(base), full_u32 = smem_u32(&c->full[0]), empty_u32 = smem_u32(&c->empty[0]);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // one number for the warp: see elect_one
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int m_tiles = (M + 2 * kLaneTile - 1) / (2 * kLaneTile), n_tiles = (N + BN - 1) / BN, total = m_tiles * n_tiles;
    const int pair = (int)(blockIdx.x >> 1), n_pairs = (int)(gridDim.x >> 1);
    const int n_kb = (K + kBlockK - 1) / kBlockK;

    if (threadIdx.x == 0) {
        prefetch_tensormap(&map_a);
        prefetch_tensormap(&map_w);
        prefetch_tensormap(&map_out);
        if (HAS_RES) prefetch_tensormap(&map_res);
        for (int i = 0; i < n_stages; ++i) {
            mbar_init(&c->full[i], 1);
            mbar_init(&c->empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&c->acc_full[i], 1);
            mbar_init(&c->acc_empty[i], 2 * kEpilogueWarps);
            for (int j = 0; j < kSlots; ++j) mbar_init(&c->res_full[i][j], 1);
        }
        c->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&c->tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_barrier();                          // both blocks' barriers and tensor memory exist
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, c->tmem_base, 0);

    if (warp == 0) {
        // The whole warp walks these loops and one lane issues the copies (see elect_one).
        const uint32_t lead_full = peer_address(full_u32, 0);
        uint32_t st = 0, empty_parity = 1;                      // a fresh barrier passes a wait for parity 1
        bool ok = true, first = true;
        uint32_t last_stage = 0, last_parity = 0;
        int issued = 0;
        for (int tile = pair; tile < total && ok; tile += n_pairs) {
            const int m0 = (tile % m_tiles) * 2 * kLaneTile + (int)rank * kLaneTile, n0 = (tile / m_tiles) * BN + (int)rank * (BN / 2);
            int kb = 0;
            if (first) {
                // The first ring: the weights are asked for before the kernel before this one has ended, the activations after.
                first = false;
                const int ahead = n_kb < n_stages ? n_kb : n_stages;
                for (int i = 0; i < ahead; ++i) {
                    if (elect_one()) {
                        if (rank == 0) expect_tx_u32(full_u32 + 8 * i, 2 * stage_bytes);
                        tma_load_pair(stages_u32 + i * stage_bytes + kATileBytes, &map_w, lead_full + 8 * i, i * kBlockK, n0);
                    }
                }
                lb_wait_for_predecessor();
                lb_dependents_may_launch();
                for (int i = 0; i < ahead; ++i)
                    if (elect_one()) tma_load_pair(stages_u32 + i * stage_bytes, &map_a, lead_full + 8 * i, i * kBlockK, m0);
                kb = issued = ahead;
                last_stage = (uint32_t)ahead - 1;
                st = (uint32_t)ahead;
                if (st == (uint32_t)n_stages) {
                    st = 0;
                    empty_parity ^= 1;
                }
            }
            for (; kb < n_kb; ++kb) {
                if (!__all_sync(0xffffffffu, wait_u32(empty_u32 + 8 * st, empty_parity, abort_flag))) {
                    give_up(c, status, 1, st, rank);
                    ok = false;
                    break;
                }
                const uint32_t dst = stages_u32 + st * stage_bytes, bar = lead_full + 8 * st;
                if (elect_one()) {
                    if (rank == 0) expect_tx_u32(full_u32 + 8 * st, 2 * stage_bytes);
                    tma_load_pair(dst, &map_a, bar, kb * kBlockK, m0);
                    tma_load_pair(dst + kATileBytes, &map_w, bar, kb * kBlockK, n0);
                }
                ++issued;
                last_stage = st;
                last_parity = empty_parity ^ 1;
                if (++st == (uint32_t)n_stages) {
                    st = 0;
                    empty_parity ^= 1;
                }
            }
        }
        if (*abort_flag != 0 && issued > 0) {
            // Leave no copy in flight.  The first block's barrier counts both blocks' copies; the other block, which has none of its own
            // to ask, gives its last ones a millisecond, hundreds of times what they take.
            if (rank == 0) mbar_wait(&c->full[last_stage], last_parity, nullptr);
            const long long t0 = clock64();
            while (clock64() - t0 < 2000000) {}
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const uint32_t idesc = umma_idesc(2 * kLaneTile, BN);
            const uint32_t desc_hi = (uint32_t)(1024 >> 4) | (1u << 14) | (2u << 29);
            const uint32_t lo0 = ((stages_u32 & 0x3FFFFu) >> 4) | (1u << 16);
            const uint32_t lo_stage = stage_bytes >> 4, lo_w = kATileBytes >> 4;
            uint32_t st = 0, full_parity = 0;
            int it = 0;
            bool ok = true;
            for (int tile = pair; tile < total && ok; tile += n_pairs, ++it) {
                const int buf = it & 1;
                if (!__all_sync(0xffffffffu, wait_cluster(smem_u32(&c->acc_empty[buf]), (uint32_t)(((it >> 1) & 1) ^ 1), abort_flag))) {
                    give_up(c, status, 5, buf, rank);
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem_base + (uint32_t)buf * 256u;
                for (int kb = 0; kb < n_kb; ++kb) {
                    if (!__all_sync(0xffffffffu, wait_u32(full_u32 + 8 * st, full_parity, abort_flag))) {
                        give_up(c, status, 2, st, rank);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a_lo = lo0 + st * lo_stage, w_lo = a_lo + lo_w;
                    if (elect_one()) {
                        umma_pair(d, a_lo, w_lo, desc_hi, idesc, kb != 0 ? 1u : 0u);
#pragma unroll
                        for (uint32_t k = 1; k < kBlockK / kUmmaK; ++k) umma_pair(d, a_lo + 2 * k, w_lo + 2 * k, desc_hi, idesc, 1u);
                        commit_pair(empty_u32 + 8 * st);
                    }
                    if (++st == (uint32_t)n_stages) {
                        st = 0;
                        full_parity ^= 1;
                    }
                }
                // (`withhold`: a test's launch, whose epilogues find nothing and give up.)
                if (ok && (withhold == 0 || it != 0) && elect_one()) commit_pair(smem_u32(&c->acc_full[buf]));
            }
        }
    } else {
        const int ew = warp - 2, group = ew >> 2, quarter = warp & 3;
        const int row = quarter * 32 + lane;                           // this thread's token within the block's 128
        const int gt = (int)threadIdx.x - 64 - 128 * group;            // 0..127 within the group
        const bool elected = gt == 0;
        const uint32_t swz = (uint32_t)(row & 7);
        uint8_t* slots = staging + (size_t)group * kSlots * kStripBytes;
        const uint32_t row_u32 = smem_u32(slots) + (uint32_t)row * 128u;
        const uint32_t lead_acc_empty = peer_address(smem_u32(&c->acc_empty[0]), 0);
        const lb_act_pair act_pair = lb_act_load(bias, N, ACT);
        lb_wait_for_predecessor();           // before anything this block stores, and before a cache page is written
        lb_dependents_may_launch();
        int it = 0;
        uint32_t turn = 0;                                             // strips that this group has stored so far: slot and parity
        for (int tile = pair; tile < total; tile += n_pairs, ++it) {
            const int m0 = (tile % m_tiles) * 2 * kLaneTile + (int)rank * kLaneTile, n0 = (tile / m_tiles) * BN;
            const int buf = it & 1;
            const int n_strips = min(BN, N - n0 + kStripCols - 1) / kStripCols;          // those with a feature
            // The bias of this group's strips.  (The last tile's readers are past its last barrier.)
            float* bias_here = bias_s + group * 128;
            const int bias_col = n0 + (group + 2 * (gt / kStripCols)) * kStripCols + gt % kStripCols;
            bias_here[gt] = (bias != nullptr && bias_col < N) ? bias[bias_col] : 0.0f;
            if (HAS_RES && elected && group < n_strips) {
                bulk_wait_read();                                      // the slot's last store has read it
                uint64_t* bar = &c->res_full[group][turn & 1];
                mbar_expect_tx(bar, kStripBytes);
                tma_load_2d(slots + (turn & 1) * kStripBytes, &map_res, bar, n0 + group * kStripCols, m0);
            }
            const bool ok = mbar_wait(&c->acc_full[buf], (it >> 1) & 1, abort_flag);
            if (!ok) give_up(c, status, 3, quarter, rank);
            if (barrier_any(2 + group, 128, !ok || *abort_flag != 0)) break;       // one answer for the group; the bias is there
            tc_fence_after();
            const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)buf * 256u;
            const uint32_t bias_u32 = smem_u32(bias_here);
            int slot = -1;                                             // where this thread's token lies in the cache
            if constexpr (KV) slot = m0 + row < M ? __ldg(kv.slot_mapping + m0 + row) : -1;
            for (int sp = group; sp < n_strips; sp += 2) {
                const uint32_t strip = row_u32 + (turn & 1) * kStripBytes;
                const uint32_t b = bias_u32 + (uint32_t)((sp >> 1) * kStripCols) * 4u;
                // A strip of keys or values goes straight from the registers to its page, a strip of queries to `out`.
                bool to_cache = false;
                uint4* cache_row = nullptr;
                if constexpr (KV) {
                    const int col0 = n0 + sp * kStripCols;
                    to_cache = col0 >= kv.q_dim;
                    if (to_cache && slot >= 0) {
                        const int kvd = kv.n_kv_head * kv.head_dim, rel = col0 - kv.q_dim;
                        const int which = rel >= kvd ? 1 : 0, within = rel - which * kvd;
                        const int head = within / kv.head_dim, dd = within - head * kv.head_dim;
                        const int page = slot >> kv.page_shift, off = slot & ((1 << kv.page_shift) - 1);
                        const size_t at = ((((size_t)page * 2 + which) * kv.n_kv_head + head) << kv.page_shift) + off;
                        cache_row = reinterpret_cast<uint4*>(kv.cache + at * kv.head_dim + dd);
                    }
                }
                if constexpr (HAS_RES) {
                    if (elected && sp + 2 < n_strips) {                // the next strip's residual, into the other slot
                        bulk_wait_read();
                        uint64_t* bar = &c->res_full[group][(turn + 1) & 1];
                        mbar_expect_tx(bar, kStripBytes);
                        tma_load_2d(slots + ((turn + 1) & 1) * kStripBytes, &map_res, bar, n0 + (sp + 2) * kStripCols, m0);
                    }
                    if (!mbar_wait(&c->res_full[group][turn & 1], (turn >> 1) & 1, abort_flag)) give_up(c, status, 4, quarter, rank);
                } else if (!to_cache) {
                    // The slot's last store but one has read it: one group of stores a turn, and a strip that goes to the cache takes no turn (a turn
                    // without a store would let the slot be written while that store still reads it).
                    if (elected) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                    named_barrier(2 + group, 128);
                }
                if constexpr (sizeof(TO) == 4) {
                    uint32_t v[32];
                    tmem_ld32(t_row + (uint32_t)(sp * 32), v);
                    tmem_ld_wait();
#pragma unroll
                    for (int ch = 0; ch < 8; ++ch) {
                        const uint32_t at = strip + (((uint32_t)ch ^ swz) << 4);
                        const float4 bb = lds4(b + 16 * ch);
                        float4 y;
                        y.x = activate<ACT, false>(__uint_as_float(v[4 * ch]) + bb.x, act_pair);
                        y.y = activate<ACT, false>(__uint_as_float(v[4 * ch + 1]) + bb.y, act_pair);
                        y.z = activate<ACT, false>(__uint_as_float(v[4 * ch + 2]) + bb.z, act_pair);
                        y.w = activate<ACT, false>(__uint_as_float(v[4 * ch + 3]) + bb.w, act_pair);
                        if constexpr (HAS_RES) {
                            const float4 r = lds4(at);
                            y.x += r.x; y.y += r.y; y.z += r.z; y.w += r.w;
                        }
                        sts4(at, y);
                    }
                } else {
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        uint32_t v[32];
                        tmem_ld32(t_row + (uint32_t)(sp * 64 + half * 32), v);
                        tmem_ld_wait();
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const int ch = half * 4 + q;
                            const float4 b0 = lds4(b + 128 * half + 32 * q), b1 = lds4(b + 128 * half + 32 * q + 16);
                            uint4 y;
                            y.x = pack2(activate<ACT, true>(__uint_as_float(v[8 * q]) + b0.x, act_pair), activate<ACT, true>(__uint_as_float(v[8 * q + 1]) + b0.y, act_pair));
                            y.y = pack2(activate<ACT, true>(__uint_as_float(v[8 * q + 2]) + b0.z, act_pair), activate<ACT, true>(__uint_as_float(v[8 * q + 3]) + b0.w, act_pair));
                            y.z = pack2(activate<ACT, true>(__uint_as_float(v[8 * q + 4]) + b1.x, act_pair), activate<ACT, true>(__uint_as_float(v[8 * q + 5]) + b1.y, act_pair));
                            y.w = pack2(activate<ACT, true>(__uint_as_float(v[8 * q + 6]) + b1.z, act_pair), activate<ACT, true>(__uint_as_float(v[8 * q + 7]) + b1.w, act_pair));
                            if (KV && to_cache) {
                                if (cache_row != nullptr) cache_row[ch] = y;
                            } else {
                                sts4(strip + (((uint32_t)ch ^ swz) << 4), y);
                            }
                        }
                    }
                }
                if (!(KV && to_cache)) {
                    fence_async_shared();
                    named_barrier(2 + group, 128);
                    if (elected) {
                        if (m0 < M) tma_store_2d(&map_out, slots + (turn & 1) * kStripBytes, n0 + sp * kStripCols, m0);
                        bulk_commit();
                    }
                    ++turn;
                }
            }
            // The accumulator has been read: the products of the tile after next may overwrite it.
            tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_at_peer(lead_acc_empty + 8 * buf);
            if constexpr (KV) named_barrier(2 + group, 128);           // strips that went to the cache had no barrier of their own
        }
        if (elected) {
            bulk_wait_all();
            if (HAS_RES && *abort_flag != 0) {                         // a residual still on its way
                const long long t0 = clock64();
                while (clock64() - t0 < 2000000) {}
            }
        }
    }
    __syncwarp();            // the elected lanes rejoin their warps before the block-wide barriers
    tc_fence_before();
    __syncthreads();
    cluster_barrier();       // both blocks are done with each other's barriers and with tensor memory
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }
    cluster_barrier();
}

size_t smem_bytes(int BN, int n_stages) {
    return 1024 + (size_t)n_stages * (kLaneTile + BN / 2) * kBlockK * 2 + (size_t)2 * kSlots * kStripBytes + 2 * 128 * sizeof(float) + sizeof(Control);
}

int stages_for(int BN) {
    int n = 0;
    while (n < kMaxStages && smem_bytes(BN, n + 1) <= kSmemLimit) ++n;
    return n;
}

}  // namespace

// The feature tile (128, 192 or 256) whose rounds over the pairs of SMs cost least, and that cost in nanoseconds: a k-block costs 330 ns, or
// what all active blocks' operands take from L2 at 13.5 TB/s; the first tile's way in and the last one's epilogue about 3.5 us.
extern "C" int lb_gemm_pair_tile(int M, int N, int K, int n_sm, int* cost_ns) {
    const long m_tiles = (M + 2 * kLaneTile - 1) / (2 * kLaneTile), n_kb = (K + kBlockK - 1) / kBlockK, n_pairs = n_sm / 2;
    int best = 0;
    long best_cost = 0;
    for (int bn = 256; bn >= 128; bn -= 64) {
        const long tiles = m_tiles * ((N + bn - 1) / bn), rounds = (tiles + n_pairs - 1) / n_pairs, active = 2 * (tiles < n_pairs ? tiles : n_pairs);
        const long operands = active * (kLaneTile + bn / 2) * 128 / 13500;
        const long cost = rounds * n_kb * (operands > 330 ? operands : 330) + 2500 + 1000 * bn / 256;
        if (best == 0 || cost < best_cost) {
            best = bn;
            best_cost = cost;
        }
    }
    if (cost_ns != nullptr) *cost_ns = (int)best_cost;
    return best;
}

// Operands as lb_gemm_persistent takes them; feature_tile 128, 192 or 256.
extern "C" int lb_gemm_pair(int out_dtype, const void* A, int64_t lda, const void* W, int64_t ldw, const float* bias, const float* residual, int64_t ldr,
                            void* out, int64_t ldo, int M, int N, int K, int act, int feature_tile, void* kv_cache, const int32_t* slot_mapping, int q_dim,
                            int n_kv_head, int head_dim, int page_size, void* stream) {
    LB_CHECK_ARG(M > 0 && N > 0 && K > 0 && (out_dtype == LB_BF16 || out_dtype == LB_F32), "gemm_pair: bad sizes or type M=%d N=%d K=%d", M, N, K);
    LB_CHECK_ARG(feature_tile == 128 || feature_tile == 192 || feature_tile == 256, "gemm_pair: feature tile %d", feature_tile);
    LB_CHECK_ARG(lda >= K && ldw >= K && ldo >= N, "gemm_pair: a row stride is shorter than the row");
    if (lb_gemm_persistent_tile(out_dtype, A, lda, W, ldw, residual, ldr, out, ldo, M, N, K) == 0)
        return lb_fail(LB_ERR_UNSUPPORTED, "gemm_pair: needs more than 64 tokens, K and all row strides on 16-byte boundaries, and float32 output where a residual "
                       "is given (M=%d K=%d lda=%lld ldw=%lld ldo=%lld ldr=%lld)", M, K, (long long)lda, (long long)ldw, (long long)ldo, (long long)ldr);
    KvTarget kv{static_cast<__nv_bfloat16*>(kv_cache), slot_mapping, q_dim, n_kv_head, head_dim, 0};
    if (kv_cache != nullptr) {
        if (!lb_gemm_persistent_kv_supports(out_dtype, N, act, residual != nullptr, q_dim, n_kv_head, head_dim, page_size))
            return lb_fail(LB_ERR_UNSUPPORTED, "gemm_pair: keys and values go to the cache only from a bfloat16 product without activation or residual, with q_dim "
                           "and head_dim multiples of 64 and a power-of-two page (N=%d q_dim=%d kv_heads=%d head_dim=%d page_size=%d)", N, q_dim, n_kv_head,
                           head_dim, page_size);
        LB_CHECK_ARG(slot_mapping != nullptr, "gemm_pair: the slot mapping is missing");
        while ((1 << kv.page_shift) < page_size) ++kv.page_shift;
    }
    const int elem = out_dtype == LB_F32 ? 4 : 2, bn = feature_tile, n_stages = stages_for(bn);
    CUtensorMap map_a, map_w, map_res, map_out;
    int rc = lb_tensor_map_2d(&map_a, A, 2, M, K, lda, kLaneTile);
    if (rc == LB_OK) rc = lb_tensor_map_2d(&map_w, W, 2, N, K, ldw, bn / 2);
    if (rc == LB_OK) rc = lb_tensor_map_2d(&map_out, out, elem, M, N, ldo, kLaneTile);
    if (rc == LB_OK && residual != nullptr) rc = lb_tensor_map_2d(&map_res, residual, 4, M, N, ldr, kLaneTile);
    if (rc != LB_OK) return rc;
    if (residual == nullptr) map_res = map_out;
    int* status = nullptr;
    rc = lb_tc_status_word(&status);
    if (rc != LB_OK) return rc;
    int dev = 0, n_sm = 0;
    LB_CHECK_CUDA(cudaGetDevice(&dev));
    LB_CHECK_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
    const long tiles = (long)((M + 2 * kLaneTile - 1) / (2 * kLaneTile)) * ((N + bn - 1) / bn);
    const int grid = 2 * (int)(tiles < n_sm / 2 ? tiles : n_sm / 2);
    const size_t smem = kSmemLimit;                  // a block has its SM, and all of its tensor memory, to itself
    const int withhold = g_withhold_next;
    g_withhold_next = 0;
    auto s = static_cast<cudaStream_t>(stream);
#define LB_GO(TO, ACT, RES, KV)                                                                                                                    \
    {                                                                                                                                              \
        LB_CHECK_CUDA(cudaFuncSetAttribute(gemm_pair_kernel<TO, ACT, RES, KV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));            \
        LB_CHECK_CUDA(lb_launch_overlapped_cluster(0, 2, gemm_pair_kernel<TO, ACT, RES, KV>, dim3(grid), dim3(kThreads), smem, s, map_a, map_w,     \
                                                   map_res, map_out, bias, M, N, K, bn, n_stages, status, withhold, kv));                                    \
    }
#define LB_GO_ACT(TO, RES)                                                            \
    switch (act) {                                                                    \
        case LB_ACT_NONE: LB_GO(TO, LB_ACT_NONE, RES, false); break;                  \
        case LB_ACT_GELU_TANH: LB_GO(TO, LB_ACT_GELU_TANH, RES, false); break;        \
        case LB_ACT_GELU_ERF: LB_GO(TO, LB_ACT_GELU_ERF, RES, false); break;          \
        case LB_ACT_XIELU: LB_GO(TO, LB_ACT_XIELU, RES, false); break;                \
        case LB_ACT_RELU2: LB_GO(TO, LB_ACT_RELU2, RES, false); break;                \
        default: return lb_fail(LB_ERR_INVALID_ARGUMENT, "gemm_pair: unknown activation %d", act); \
    }
    if (elem == 4) {
        if (residual != nullptr) LB_GO_ACT(float, true) else LB_GO_ACT(float, false)
    } else if (kv_cache != nullptr) {
        LB_GO(__nv_bfloat16, LB_ACT_NONE, false, true)
    } else {
        LB_GO_ACT(__nv_bfloat16, false)
    }
#undef LB_GO_ACT
#undef LB_GO
    LB_CHECK_LAUNCH();
    return LB_OK;
}

// The pairs of the next launch never signal their first accumulator: the epilogues of both blocks wait to their limit (about two seconds), report it in
// the status word and stop the other roles.  A test of the give-up path that faults nothing.
extern "C" int lb_gemm_pair_withhold_next(int on) {
    g_withhold_next = on != 0 ? 1 : 0;
    return LB_OK;
}
