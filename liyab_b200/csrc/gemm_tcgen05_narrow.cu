// out[M, N] = epilogue(A[M, K] . W[N, K]^T) for some dozens of tokens (17 to 512): one launch on tcgen05 whose tiles are 64 or 128 tokens by a few features.
//
// Between the products of single tokens and those that fill 128 x 128 tiles the weights are still most of what has to move, and the tokens no longer fit
// the rows of mma.sync cheaply: a product of 64 tokens spent 3 to 6 us in mma.sync and the rest in staging 128 KB of activations through cp.async and
// ldmatrix (10.3 us of a step for 3072 x 1024), and where the reduction is long a second launch added its parts.  Here a block takes `features` (a multiple of 8, as
// many as give every SM a block) of W and 64 or 128 tokens, which are the lanes of the accumulator; TMA brings both operands' k-blocks, weights before the wait
// for the kernel before, and nothing but descriptors passes through registers.  A block's way in is bound by its activations (8 or 16 KB a
// k-block), so a long reduction is cut between the blocks of a cluster, which hand each other the sums of their share of the features through distributed
// shared memory and finish them in rank order.
// The tensor core's tile is 128 rows by a multiple of 16 features whatever is there: rows past the box of tokens and features past the block's read
// what lies behind in shared memory, and give sums that nobody reads.
//
// Roles: warp 0 TMA producer, warp 1 products, warps 2..9 epilogue (warp % 4 names the 32 lanes, the two warps of those take alternate pieces of eight
// features).  Handshakes and bounded waits as in the other tcgen05 products.
//
// Epilogue order as the reference's (src/core/transformer.cpp:111-118, 4903-4912, 5526-5532): bias, activation, then the residual sum, all in 32-bit.
#include "api.h"
#include "common.cuh"
#include "gemm_tile.cuh"
#include "tcgen05.cuh"

namespace {

using namespace lb_tc;
using namespace lb_tile;

constexpr int kEpilogueWarps = 8;
constexpr int kThreads = 64 + 32 * kEpilogueWarps;
constexpr int kMaxStages = 16;
constexpr int kMaxFeatures = 256;
constexpr int kMaxSplits = 8;
constexpr size_t kSmemLimit = 227 * 1024;

int g_withhold_next = 0;      // the next launch's blocks leave their accumulator-ready barriers unsignalled (tests)

struct Control {
    uint64_t full[kMaxStages];
    uint64_t empty[kMaxStages];
    uint64_t acc_ready;
    uint32_t tmem_base;
    int abort_flag;
};

__device__ __forceinline__ void give_up(Control* c, int* status, int site, int detail) {
    atomicCAS(status, 0, (0xF << 12) | (site << 8) | (detail & 0xff));
    *(volatile int*)&c->abort_flag = 1;
}

// Eight accumulator columns of this thread's lane.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\ttcgen05.wait::ld.sync.aligned;"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(taddr) : "memory");
}

// ROWS: tokens a block's box holds (64 or 128).  gridDim.x = tiles x splits; the splits of a tile are a cluster.
template <int ROWS, typename TO, int ACT>
__global__ void __launch_bounds__(kThreads)
gemm_narrow_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const float* __restrict__ bias, const float* residual,
                   int64_t ldr, TO* out, int64_t ldo, int M, int N, int K, int features, int splits, int alias, int n_stages, int tmem_cols, int withhold, int* status, const KvTarget kv) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    constexpr uint32_t kABytes = ROWS * 128u;
    const uint32_t stage_bytes = kABytes + (uint32_t)features * 128u;
    uint8_t* behind = base + (size_t)n_stages * stage_bytes;
    float* inbox = reinterpret_cast<float*>(alias ? base : behind);                        // [split][share's pieces of 8][2][ROWS][4]: a warp's 16-byte stores side by side
    float* bias_s = reinterpret_cast<float*>(behind) + (splits > 1 && !alias ? ROWS * features : 0);
    Control* c = reinterpret_cast<Control*>(bias_s + kMaxFeatures);
    volatile int* abort_flag = &c->abort_flag;
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int rank = (int)blockIdx.x % splits, n0 = (int)blockIdx.x / splits * features, m0 = (int)blockIdx.y * ROWS;
    const int all_kb = (K + kBlockK - 1) / kBlockK, per = (all_kb + splits - 1) / splits;
    const int kb_lo = min(all_kb, rank * per), n_kb = min(all_kb, kb_lo + per) - kb_lo;     // the host leaves no rank without one
    // Every block of the cluster has started before one of them writes into another's shared memory: arrive now, wait just before.  (Where the
    // sums come to lie over the stages, every block's products have to be complete before that: arrive then.)
    if (splits > 1 && !alias) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");

    if (threadIdx.x == 0) {
        prefetch_tensormap(&map_a);
        prefetch_tensormap(&map_w);
        for (int i = 0; i < n_stages; ++i) {
            mbar_init(&c->full[i], 1);
            mbar_init(&c->empty[i], 1);
        }
        mbar_init(&c->acc_ready, 1);
        c->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        tmem_alloc(&c->tmem_base, tmem_cols);
        tmem_relinquish();
    }
    if (threadIdx.x >= 64 && (int)threadIdx.x - 64 < features) {          // as many epilogue threads as the most features
        const int f = (int)threadIdx.x - 64;
        bias_s[f] = bias != nullptr && n0 + f < N ? bias[n0 + f] : 0.0f;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, c->tmem_base, 0);
    const uint32_t stages_u32 = smem_u32(base), full_u32 = smem_u32(&c->full[0]), empty_u32 = smem_u32(&c->empty[0]);

    if (warp == 0) {
        const int ahead = min(n_kb, n_stages);
        for (int kb = 0; kb < ahead; ++kb)
            if (elect_one()) {
                expect_tx_u32(full_u32 + 8 * kb, stage_bytes);
                tma_load_u32(stages_u32 + kb * stage_bytes + kABytes, &map_w, full_u32 + 8 * kb, (kb_lo + kb) * kBlockK, n0);
            }
        lb_wait_for_predecessor();
        lb_dependents_may_launch();
        for (int kb = 0; kb < ahead; ++kb)
            if (elect_one()) tma_load_u32(stages_u32 + kb * stage_bytes, &map_a, full_u32 + 8 * kb, (kb_lo + kb) * kBlockK, m0);
        int issued = ahead, st = ahead == n_stages ? 0 : ahead;
        uint32_t parity = 0;
        for (int kb = ahead; kb < n_kb; ++kb) {
            if (!__all_sync(0xffffffffu, wait_u32(empty_u32 + 8 * st, parity, abort_flag))) {
                give_up(c, status, 1, st);
                break;
            }
            if (elect_one()) {
                expect_tx_u32(full_u32 + 8 * st, stage_bytes);
                tma_load_u32(stages_u32 + st * stage_bytes, &map_a, full_u32 + 8 * st, (kb_lo + kb) * kBlockK, m0);
                tma_load_u32(stages_u32 + st * stage_bytes + kABytes, &map_w, full_u32 + 8 * st, (kb_lo + kb) * kBlockK, n0);
            }
            issued = kb + 1;
            if (++st == n_stages) {
                st = 0;
                parity ^= 1;
            }
        }
        // Leave no copy in flight: the barriers of the last loads complete when their bytes landed.
        if (*abort_flag != 0)
            for (int kb = max(0, issued - n_stages); kb < issued; ++kb) mbar_wait(&c->full[kb % n_stages], (kb / n_stages) & 1, nullptr);
    } else if (warp == 1) {
        const uint32_t idesc = umma_idesc(kLaneTile, (features + 15) / 16 * 16);
        const uint32_t desc_hi = (uint32_t)(1024 >> 4) | (1u << 14) | (2u << 29);
        const uint32_t lo0 = ((stages_u32 & 0x3FFFFu) >> 4) | (1u << 16);
        int st = 0;
        uint32_t parity = 0;
        bool ok = true;
        for (int kb = 0; kb < n_kb; ++kb) {
            if (!__all_sync(0xffffffffu, wait_u32(full_u32 + 8 * st, parity, abort_flag))) {
                give_up(c, status, 2, st);
                ok = false;
                break;
            }
            tc_fence_after();
            const uint32_t a_lo = lo0 + (uint32_t)st * (stage_bytes >> 4), w_lo = a_lo + (kABytes >> 4);
            if (elect_one()) {
                umma_lo(tmem_base, a_lo, w_lo, desc_hi, idesc, kb != 0 ? 1u : 0u);
#pragma unroll
                for (uint32_t k = 1; k < kBlockK / kUmmaK; ++k) umma_lo(tmem_base, a_lo + 2 * k, w_lo + 2 * k, desc_hi, idesc, 1u);
                commit_u32(empty_u32 + 8 * st);
            }
            if (++st == n_stages) {
                st = 0;
                parity ^= 1;
            }
        }
        // (`withhold`: a test's launch, whose epilogues find nothing and give up.)
        if (ok && withhold == 0 && elect_one()) umma_commit(&c->acc_ready);
        lb_wait_for_predecessor();
        lb_dependents_may_launch();
    }
    const int quarter = warp & 3, group = (warp - 2) >> 2, row = quarter * 32 + lane, token = m0 + row;
    const bool epilogue = warp >= 2 && quarter * 32 < ROWS && m0 + quarter * 32 < M;
    const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const int mine = features / splits, f_lo = rank * mine;                   // this block's share of the tile's features: f_lo .. f_lo + mine - 1
    if (warp >= 2) {
        lb_wait_for_predecessor();           // before the residual is read and anything is written
        lb_dependents_may_launch();
    }
    const lb_act_pair act_pair = lb_act_load(bias, N, ACT);
    bool ok = true;
    // The first piece's residual travels under the products.
    float res[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    auto load_residual = [&](int piece) {
        const int f = n0 + f_lo + piece * 8;
        if (residual != nullptr && token < M && f < N) {
            const float4* r = reinterpret_cast<const float4*>(residual + (size_t)token * ldr + f);
            const float4 a = __ldcg(r), b = __ldcg(r + 1);
            res[0] = a.x; res[1] = a.y; res[2] = a.z; res[3] = a.w;
            res[4] = b.x; res[5] = b.y; res[6] = b.z; res[7] = b.w;
        }
    };
    const int pieces = mine / 8;
    if (epilogue && group < pieces) load_residual(group);
    if (epilogue) {
        ok = __all_sync(0xffffffffu, mbar_wait(&c->acc_ready, 0, abort_flag));
        if (!ok) give_up(c, status, 3, quarter);
        tc_fence_after();
    }
    __syncwarp();
    if (splits > 1) {
        if (alias) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (epilogue && ok) {
            for (int piece = group; piece < features / 8; piece += 2) {
                const int to = piece / pieces, within = piece - to * pieces;
                uint32_t v[8];
                tmem_ld8(t_row + (uint32_t)(piece * 8), v);
                const uint32_t at = peer_address(smem_u32(inbox + ((size_t)(rank * pieces + within) * 2 * ROWS + row) * 4), (uint32_t)to);
                store_at_peer(at, v[0], v[1], v[2], v[3]);
                store_at_peer(at + ROWS * 16, v[4], v[5], v[6], v[7]);
            }
        }
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    if (epilogue && ok) {
        int slot = -1;
        if (kv.cache != nullptr && token < M) slot = __ldg(kv.slot_mapping + token);
        for (int piece = group; piece < pieces; piece += 2) {
            if (piece != group) load_residual(piece);
            float y[8];
            if (splits > 1) {
#pragma unroll
                for (int i = 0; i < 8; ++i) y[i] = 0.0f;
                for (int from = 0; from < splits; ++from) {
                    const float4* p = reinterpret_cast<const float4*>(inbox) + (size_t)(from * pieces + piece) * 2 * ROWS + row;
                    const float4 a = p[0], b = p[ROWS];
                    y[0] += a.x; y[1] += a.y; y[2] += a.z; y[3] += a.w;
                    y[4] += b.x; y[5] += b.y; y[6] += b.z; y[7] += b.w;
                }
            } else {
                uint32_t v[8];
                tmem_ld8(t_row + (uint32_t)(piece * 8), v);
#pragma unroll
                for (int i = 0; i < 8; ++i) y[i] = __uint_as_float(v[i]);
            }
            const int f = n0 + f_lo + piece * 8;
            if (token >= M || f >= N) continue;
#pragma unroll
            for (int i = 0; i < 8; ++i) y[i] = activate<ACT, sizeof(TO) == 2>(y[i] + bias_s[f_lo + piece * 8 + i], act_pair) + res[i];
            if constexpr (sizeof(TO) == 4) {
                float4* dst = reinterpret_cast<float4*>(out + (size_t)token * ldo + f);
                dst[0] = make_float4(y[0], y[1], y[2], y[3]);
                dst[1] = make_float4(y[4], y[5], y[6], y[7]);
            } else {
                uint4 p;
                p.x = pack2(y[0], y[1]);
                p.y = pack2(y[2], y[3]);
                p.z = pack2(y[4], y[5]);
                p.w = pack2(y[6], y[7]);
                if (kv.cache != nullptr && f >= kv.q_dim) {          // keys and values go straight to their pages
                    if (slot < 0) continue;
                    const int kvd = kv.n_kv_head * kv.head_dim, rel = f - kv.q_dim, which = rel >= kvd ? 1 : 0, within = rel - which * kvd;
                    const int head = within / kv.head_dim, dd = within - head * kv.head_dim;
                    const int page = slot >> kv.page_shift, off = slot & ((1 << kv.page_shift) - 1);
                    const size_t at = ((((size_t)page * 2 + which) * kv.n_kv_head + head) << kv.page_shift) + off;
                    *reinterpret_cast<uint4*>(kv.cache + at * kv.head_dim + dd) = p;
                } else {
                    *reinterpret_cast<uint4*>(out + (size_t)token * ldo + f) = p;
                }
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, tmem_cols);
    }
}

struct Plan {
    int features = 0, splits = 1, alias = 0, stages = 0;
    double us = 0;
};

size_t behind_bytes(int rows, int features, int splits, bool alias) {
    // The tensor core reads 128 rows of A and up to a multiple of 16 of W, from the last stage too.
    const size_t reach = 16384 + 1024, kept = (splits > 1 && !alias ? (size_t)rows * features * 4 : 0) + kMaxFeatures * 4 + sizeof(Control);
    return kept > reach ? kept : reach;
}

// Stages of `features` features, with the received sums over them (alias) where too few would fit beside those.
Plan stages_for(int rows, int features, int splits, int n_kb) {
    const size_t stage = (size_t)(rows + features) * 128;
    Plan p;
    p.features = features;
    p.splits = splits;
    for (const bool alias : {false, true}) {
        if (alias && splits == 1) break;
        const size_t n = (kSmemLimit - 1024 - behind_bytes(rows, features, splits, alias)) / stage;
        p.stages = (int)(n < (size_t)n_kb ? n : n_kb);
        if (p.stages > kMaxStages) p.stages = kMaxStages;
        p.alias = alias;
        if (p.stages >= 6 || p.stages == n_kb) break;
    }
    if (p.alias && (size_t)p.stages * stage < (size_t)rows * features * 4) p.stages = 0;      // the sums do not fit over them
    return p;
}

// Columns of tensor memory for the block's sums.
int tmem_columns(int features) { return features <= 32 ? 32 : features <= 64 ? 64 : features <= 128 ? 128 : 256; }

// The blocks of a cluster wait for one another while each holds its columns, so one that waited for columns held by a block of another cluster could wait for
// good, each cluster's other blocks being in the other's place on another SM.  A block that is part of a cluster therefore asks for at least as large a share of
// the SM's 228 KB (1 KB of each block's is the system's) as of its 512 columns: what fits the one fits the other.  Only short parts of a reduction with many
// features are below that (K = 128 in two parts of 144 features: 66 KB and half of the columns); the plan makes none.
size_t smem_bytes(int rows, const Plan& p) {
    const size_t needed = 1024 + (size_t)p.stages * (rows + p.features) * 128 + behind_bytes(rows, p.features, p.splits, p.alias != 0);
    const size_t share = (size_t)tmem_columns(p.features) * (228 * 1024 / 512) - 1024;
    return p.splits > 1 && needed < share ? share : needed;
}

}  // namespace

// Features a block and blocks a reduction for the product, and an estimate in nanoseconds; 0 where this kernel does not take the sizes.
//
// The estimate is a fit to 2,248 launches (20 to 640 tokens, 768 to 6400 features, reductions of 384 to 6400, all of the tiles and parts below with 36 to 148
// blocks): a start, 0.16 us a k-block (four products of 128 rows, a wait and a commit), what all blocks' operands take from L2, and the exchange.  The tile
// it picks is 3 % slower than the best one of those on average, 2 % up to 256 tokens.  Clusters of four and eight blocks that have an SM each do not all
// start at once where they would fill the GPU (a cluster lies within one group of SMs): 136 blocks in fours took 19 us where 104 took 13.
extern "C" int lb_gemm_narrow_plan(int M, int N, int K, int n_sm, int* splits_out, int* cost_ns) {
    if (M < 1 || M > 65535 * 64 || N < 8 || K < 8 || N % 8 != 0 || K % 8 != 0 || n_sm < 1) return 0;
    const int rows = M <= 64 ? 64 : 128, all_kb = (K + kBlockK - 1) / kBlockK, m_tiles = (M + rows - 1) / rows;
    Plan best;
    for (int splits = 1; splits <= kMaxSplits; splits *= 2) {
        const int per = (all_kb + splits - 1) / splits;
        if (splits > 1 && (per < 3 || (splits - 1) * per >= all_kb)) continue;      // short parts, or a block without one
        const int step = 8 * splits;
        for (int f = step; f <= kMaxFeatures; f += step) {
            const Plan p = stages_for(rows, f, splits, per);
            if (p.stages < (per < 3 ? per : 3)) continue;
            const bool two = smem_bytes(rows, p) <= 113 * 1024;
            const long at_once = (long)n_sm * (splits == 4 ? 132 : splits == 8 ? 104 : 148) / 148 * (two ? 2 : 1), most = at_once < n_sm ? at_once : n_sm;
            const long blocks = (long)((N + f - 1) / f) * splits * m_tiles, rounds = (blocks + most - 1) / most, active = blocks < most ? blocks : most;
            const double us = 2.4 + rounds * (0.16 * per + 3.8e-6 * active * per * (rows + f) + 0.037 * per * f / 64 + 0.219 * f / splits * rows / 4096 +
                                              (splits > 1 ? 0.72 * f * rows / 4096 : 0.0) + (splits == 4 ? 0.1 : 0.0));
            if (best.features == 0 || us < best.us) {
                best = p;
                best.us = us;
            }
        }
    }
    if (splits_out != nullptr) *splits_out = best.splits;
    if (cost_ns != nullptr) *cost_ns = (int)(best.us * 1e3);
    return best.features;
}

// Whether a bfloat16 product of these sizes is faster here than by the kernels for single tokens (gemm_rows.cu: up to 32 with a reduction of up to 1024), the split
// tcgen05 product (up to 64 tokens) and the persistent one.  Measured (us, before / here): 40 x 2304 x 768 5.2 / 4.1, 64 x 1024 x 4096 8.2 / 6.1, 64 x 6400 x 1600
// 14.2 / 8.6, 128 x 768 x 3072 10.3 / 6.0, 128 x 1600 x 6400 16.5 / 10.0; 256 x 768 x 768 5.4 / 4.7, 256 x 6400 x 1600 10.5 / 10.1, but 256 x 1280 x 1280 with float32
// results 7.7 / 8.1 (a thread stores 32 bytes of a row at a time, which many float32 results feel: 128 x 2560 x 768 5.7 / 7.0); beyond 256 only long reductions
// gain: 465 x 1024 x 4096 14.0 / 11.1, 330 x 1600 x 6400 20.1 / 16.7, but 465 x 1600 x 6400 20.5 / 20.1 and slower within a step, level or slower at 640.  Up to 32 tokens 20 x 3072 x 768 4.1 / 4.5 but 20 x 1600 x 6400 9.2 / 7.7.
// Up to 48 tokens with reductions of up to 512 and up to 2048 features the kernel for single tokens is through while this one has hardly begun: 40 x 256 x 256 2.5 / 2.8,
// 40 x 1000 x 264 3.6 / 3.9, 33 x 2048 x 512 4.1 / 4.2, but 56 x 1000 x 264 4.2 / 3.8, 48 x 768 x 640 4.4 / 3.6.
// Reductions under 256 and more than 10240 features were not measured.
extern "C" int lb_gemm_narrow_pays(int out_dtype, int M, int N, int K) {
    if (M <= 16 || M > 512 || K < 256 || N < 256 || N > 10240 || N % 8 != 0 || K % 8 != 0) return 0;
    if (M <= 32) return K > 1024;
    if (M <= 48 && K <= 512 && N <= 2048) return 0;
    const bool wide = out_dtype == LB_F32 && N > 2048;
    if (M <= 128) return !wide;
    const bool deep = out_dtype == LB_F32 && K >= 3 * N && K >= 2048 && (M <= 256 || (long)M * N <= 600000);
    if (M <= 256) return out_dtype == LB_F32 ? deep || (N <= 1024 && K >= 512) : 1;
    return deep;
}

// Whether lb_gemm_narrow takes the product: N and K multiples of 8, rows of A, W, out and residual on 16-byte boundaries, a residual
// with float32 output only.
extern "C" int lb_gemm_narrow_supports(int out_dtype, const void* A, int64_t lda, const void* W, int64_t ldw, const float* residual, int64_t ldr, const void* out,
                                       int64_t ldo, int M, int N, int K) {
    const int elem = out_dtype == LB_F32 ? 4 : 2;
    return M >= 1 && M <= 65535 * 64 && N >= 8 && N % 8 == 0 && K >= 8 && K % 8 == 0 && lda % 8 == 0 && ldw % 8 == 0 && (((uintptr_t)A | (uintptr_t)W | (uintptr_t)out) & 15) == 0 &&
           (ldo * elem) % 16 == 0 && (residual == nullptr || (out_dtype == LB_F32 && ((uintptr_t)residual & 15) == 0 && ldr % 4 == 0));
}

// Shared memory of a block of that launch, and its columns of tensor memory; 0: no such launch.
extern "C" int lb_gemm_narrow_block(int M, int K, int features, int splits, int* columns) {
    if (M < 1 || K < 1 || features < 8 || features > kMaxFeatures || splits < 1 || splits > kMaxSplits || features % (8 * splits) != 0) return 0;
    const int rows = M <= 64 ? 64 : 128, all_kb = (K + kBlockK - 1) / kBlockK, per = (all_kb + splits - 1) / splits;
    if ((splits - 1) * per >= all_kb) return 0;
    const Plan plan = stages_for(rows, features, splits, per);
    if (columns != nullptr) *columns = tmem_columns(features);
    return plan.stages >= 1 ? (int)smem_bytes(rows, plan) : 0;
}

// Whether it can put the features from q_dim on into the pages of a cache instead of `out`.
extern "C" int lb_gemm_narrow_kv_supports(int out_dtype, int N, int act, int has_residual, int q_dim, int n_kv_head, int head_dim, int page_size) {
    return out_dtype == LB_BF16 && act == LB_ACT_NONE && !has_residual && q_dim > 0 && q_dim % 8 == 0 && head_dim > 0 && head_dim % 8 == 0 &&
           N == q_dim + 2 * n_kv_head * head_dim && page_size > 0 && (page_size & (page_size - 1)) == 0;
}

// features, splits: 0 for the plan's.
extern "C" int lb_gemm_narrow(int out_dtype, const void* A, int64_t lda, const void* W, int64_t ldw, const float* bias, const float* residual, int64_t ldr, void* out,
                              int64_t ldo, int M, int N, int K, int act, int features, int splits, void* kv_cache, const int32_t* slot_mapping, int q_dim,
                              int n_kv_head, int head_dim, int page_size, void* stream) {
    LB_CHECK_ARG(M > 0 && N > 0 && K > 0 && (out_dtype == LB_BF16 || out_dtype == LB_F32), "gemm_narrow: bad sizes or type M=%d N=%d K=%d", M, N, K);
    LB_CHECK_ARG((M + 63) / 64 <= 65535, "gemm_narrow: M=%d is too large for one launch", M);
    LB_CHECK_ARG(lda >= K && ldw >= K && ldo >= N, "gemm_narrow: a row stride is shorter than the row");
    if (!lb_gemm_narrow_supports(out_dtype, A, lda, W, ldw, residual, ldr, out, ldo, M, N, K))
        return lb_fail(LB_ERR_UNSUPPORTED, "gemm_narrow: takes N and K multiples of 8, rows on 16-byte boundaries and a residual with float32 output "
                       "(M=%d N=%d K=%d lda=%lld ldw=%lld ldo=%lld ldr=%lld)", M, N, K, (long long)lda, (long long)ldw, (long long)ldo, (long long)ldr);
    KvTarget kv{static_cast<__nv_bfloat16*>(kv_cache), slot_mapping, q_dim, n_kv_head, head_dim, 0};
    if (kv_cache != nullptr) {
        if (!lb_gemm_narrow_kv_supports(out_dtype, N, act, residual != nullptr, q_dim, n_kv_head, head_dim, page_size))
            return lb_fail(LB_ERR_UNSUPPORTED, "gemm_narrow: keys and values go to the cache only from a bfloat16 product without activation or residual, with q_dim and "
                           "head_dim multiples of 8 and a power-of-two page (N=%d q_dim=%d kv_heads=%d head_dim=%d page_size=%d)", N, q_dim, n_kv_head, head_dim, page_size);
        LB_CHECK_ARG(slot_mapping != nullptr, "gemm_narrow: the slot mapping is missing");
        while ((1 << kv.page_shift) < page_size) ++kv.page_shift;
    }
    static int n_sm = 0;
    if (n_sm == 0) {
        int dev = 0;
        LB_CHECK_CUDA(cudaGetDevice(&dev));
        LB_CHECK_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
    }
    if (features <= 0 || splits <= 0) features = lb_gemm_narrow_plan(M, N, K, n_sm, &splits, nullptr);
    const int all_kb = (K + kBlockK - 1) / kBlockK, per = (all_kb + splits - 1) / splits;
    LB_CHECK_ARG(features >= 8 && features <= kMaxFeatures && (splits == 1 || splits == 2 || splits == 4 || splits == 8) && features % (8 * splits) == 0 &&
                     (splits - 1) * per < all_kb, "gemm_narrow: %d features in %d parts of K=%d", features, splits, K);
    const int rows = M <= 64 ? 64 : 128;
    const Plan plan = stages_for(rows, features, splits, per);
    LB_CHECK_ARG(plan.stages >= 1, "gemm_narrow: no stage fits %d features in %d parts", features, splits);
    CUtensorMap map_a, map_w;
    int rc = lb_tensor_map_2d(&map_a, A, 2, M, K, lda, rows);
    if (rc == LB_OK) rc = lb_tensor_map_2d(&map_w, W, 2, N, K, ldw, features);
    if (rc != LB_OK) return rc;
    int* status = nullptr;
    rc = lb_tc_status_word(&status);
    if (rc != LB_OK) return rc;
    const size_t smem = smem_bytes(rows, plan);
    const int tmem_cols = tmem_columns(features);
    const dim3 grid((N + features - 1) / features * splits, (M + rows - 1) / rows);
    auto s = static_cast<cudaStream_t>(stream);
    const int withhold = g_withhold_next;
    g_withhold_next = 0;
#define LB_GO(ROWS, TO, ACT)                                                                                                                                     \
    {                                                                                                                                                            \
        LB_CHECK_CUDA(cudaFuncSetAttribute(gemm_narrow_kernel<ROWS, TO, ACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit));                     \
        LB_CHECK_CUDA(lb_launch_overlapped_cluster(1, splits, gemm_narrow_kernel<ROWS, TO, ACT>, grid, dim3(kThreads), smem, s, map_a, map_w, bias, residual, \
                                                   ldr, (TO*)out, ldo, M, N, K, features, splits, plan.alias, plan.stages, tmem_cols, withhold, status, kv));                             \
    }
#define LB_GO_ACT(ROWS, TO)                                                              \
    switch (act) {                                                                       \
        case LB_ACT_NONE: LB_GO(ROWS, TO, LB_ACT_NONE); break;                           \
        case LB_ACT_GELU_TANH: LB_GO(ROWS, TO, LB_ACT_GELU_TANH); break;                 \
        case LB_ACT_GELU_ERF: LB_GO(ROWS, TO, LB_ACT_GELU_ERF); break;                   \
        case LB_ACT_XIELU: LB_GO(ROWS, TO, LB_ACT_XIELU); break;                         \
        case LB_ACT_RELU2: LB_GO(ROWS, TO, LB_ACT_RELU2); break;                         \
        default: return lb_fail(LB_ERR_INVALID_ARGUMENT, "gemm_narrow: unknown activation %d", act); \
    }
    if (out_dtype == LB_F32) {
        if (rows == 64) LB_GO_ACT(64, float) else LB_GO_ACT(128, float)
    } else {
        if (rows == 64) LB_GO_ACT(64, __nv_bfloat16) else LB_GO_ACT(128, __nv_bfloat16)
    }
#undef LB_GO_ACT
#undef LB_GO
    LB_CHECK_LAUNCH();
    return LB_OK;
}

extern "C" int lb_gemm_narrow_withhold_next(int on) {
    g_withhold_next = on != 0 ? 1 : 0;
    return LB_OK;
}
