// out[M, N] = epilogue(A[M, K] . W[N, K]^T) for 1 to 64 tokens (bfloat16
// operands): the products of a decode step, too small to fill a tcgen05 tile row,
// whose reduction is short enough (the host takes it for K up to 1024, and for up
// to 16 tokens up to 8192: gemm_stream_kernel below).
//
// At these sizes a product reads a few MB of weights and does next to no
// arithmetic; what it costs is latency.  The tcgen05 kernel needs K split over
// blocks and a second kernel to add the partial sums (two launches, 8-9 us per
// product).  Here one launch does it: every block takes a slice of the output
// features and the whole reduction length, as the matrix phases of the fused
// decode step do: the activations of all tokens come into shared memory by
// cp.async in chunks of 256 columns (two buffers: the next chunk travels while the
// current one is used), each warp takes 32 columns of every chunk, requests all
// its weights of the pass (up to four groups of eight features) at the start with
// 16-byte loads that go straight into mma.sync m16n8k16 fragments (tokens are the
// rows: one to four tiles of 16), and the eight warps' partial tiles are summed in
// warp order through shared memory.  For up to 16 tokens all columns of the
// activations are staged at once (or made in the kernel by a LayerNorm of the
// float32 rows), and a thread asks for the bias and residual of the elements it
// will finish before its products.  The launch may overlap the kernel before:
// weights are asked for before the wait for it, activations after.
// Every weight byte is read once; a row's result does not depend on the other
// rows.  Accumulators, bias, activation and residual sum are 32-bit, in the
// reference's order (src/core/transformer.cpp:111-118, 4903-4912, 5526-5532).
#include "api.h"
#include "common.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = 8;
constexpr int kChunk = 256;           // columns of the activations per chunk: one k-block of 32 per warp
constexpr int kChunkLd = kChunk + 32; // row stride in a buffer: 64 bytes mod 128, conflict-free 16-byte reads
constexpr int kMaxRows = 64;
constexpr int kWRegs = 16;            // 16-byte weight pieces a thread holds: groups per pass x chunks

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Optional second destination of a fused query/key/value projection: features from q_dim on are keys, then values,
// and go (as bfloat16) to the token's slot of its cache page as well (layout [page][K|V][kv_head][slot][head_dim];
// slot_mapping[token] = page * page_size + slot, negative: not kept).  cache == nullptr: none.
struct KvScatter {
    __nv_bfloat16* cache;
    const int32_t* slot_mapping;
    int q_dim, n_kv_head, head_dim, page_size;
};

// Feature f >= q_dim of token r's fused projection: also into the token's slot of its cache page.
__device__ __forceinline__ void keep_key_or_value(const KvScatter& kv, int r, int f, float y) {
    const int kvf = f - kv.q_dim, kv_dim = kv.n_kv_head * kv.head_dim;
    const int which = kvf >= kv_dim ? 1 : 0, within = kvf - which * kv_dim;
    const int head = within / kv.head_dim, dd = within - head * kv.head_dim;
    const int slot = __ldg(kv.slot_mapping + r);
    if (slot < 0) return;
    const int page = slot / kv.page_size, off = slot - page * kv.page_size;
    const size_t plane = (size_t)kv.n_kv_head * kv.page_size * kv.head_dim;
    kv.cache[(size_t)page * 2 * plane + (size_t)which * plane + ((size_t)head * kv.page_size + off) * kv.head_dim + dd] = __float2bfloat16_rn(y);
}

// Activations made in the kernel from the float32 residual rows by a LayerNorm (two-pass 32-bit statistics,
// (x - mean) / sqrt(var + eps) * gain + offset, as the separate kernel computes them): for up to 16 tokens and a
// reduction length of up to 1024 a block normalises the rows itself, one warp per row with the row in registers (one
// round trip), and keeps them in shared memory for all its passes.  That saves the LayerNorm's launch.  x == nullptr: off.
struct RowNorm {
    const float* x;
    int64_t ldx;
    const float* gain;
    const float* offset;
    float eps;
    int rms;                  // non-zero: no mean is taken off (an RMS norm); gain_offset is added to every gain
    float gain_offset;
};

__device__ void layernorm_rows_to_smem(const RowNorm& n, int M, int K, __nv_bfloat16* act, int ld, int k_pad, int rows) {
    constexpr int kVecs = 8;                       // float4 per lane: rows of up to 1024 values
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_vec = K / 4;
    float4 gain[kVecs], offs[kVecs];
#pragma unroll
    for (int j = 0; j < kVecs; ++j) {              // weights: asked for before the kernel before this one has ended
        const int i = lane + 32 * j;
        gain[j] = (i < n_vec && n.gain != nullptr) ? __ldg(reinterpret_cast<const float4*>(n.gain) + i) : make_float4(1.f, 1.f, 1.f, 1.f);
        if (n.gain != nullptr) {
            gain[j].x += n.gain_offset;
            gain[j].y += n.gain_offset;
            gain[j].z += n.gain_offset;
            gain[j].w += n.gain_offset;
        }
        offs[j] = (i < n_vec && n.offset != nullptr) ? __ldg(reinterpret_cast<const float4*>(n.offset) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    lb_wait_for_predecessor();
    lb_dependents_may_launch();
    for (int r = warp; r < rows; r += kWarps) {
        __nv_bfloat16* dst = act + r * ld;
        if (r >= M) {                              // rows past the step's tokens: zeros
            for (int i = lane * 8; i < k_pad; i += 256) *reinterpret_cast<uint4*>(dst + i) = make_uint4(0, 0, 0, 0);
            continue;
        }
        const float* row = n.x + (size_t)r * n.ldx;
        float4 v[kVecs];
#pragma unroll
        for (int j = 0; j < kVecs; ++j) {
            const int i = lane + 32 * j;
            v[j] = i < n_vec ? __ldcg(reinterpret_cast<const float4*>(row) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        float sum = 0.0f;
#pragma unroll
        for (int j = 0; j < kVecs; ++j) sum += (v[j].x + v[j].y) + (v[j].z + v[j].w);
        const float mean = n.rms ? 0.0f : lb_warp_sum(sum) / (float)K;
        float ss = 0.0f;
#pragma unroll
        for (int j = 0; j < kVecs; ++j) {
            if (lane + 32 * j < n_vec) {
                const float d0 = v[j].x - mean, d1 = v[j].y - mean, d2 = v[j].z - mean, d3 = v[j].w - mean;
                ss = fmaf(d0, d0, ss);
                ss = fmaf(d1, d1, ss);
                ss = fmaf(d2, d2, ss);
                ss = fmaf(d3, d3, ss);
            }
        }
        const float inv = 1.0f / sqrtf(lb_warp_sum(ss) / (float)K + n.eps);
#pragma unroll
        for (int j = 0; j < kVecs; ++j) {
            const int i = lane + 32 * j;
            if (i < n_vec) {
                const float4 g = gain[j], o = offs[j];
                const __nv_bfloat162 lo = __floats2bfloat162_rn((v[j].x - mean) * inv * g.x + o.x, (v[j].y - mean) * inv * g.y + o.y);
                const __nv_bfloat162 hi = __floats2bfloat162_rn((v[j].z - mean) * inv * g.z + o.z, (v[j].w - mean) * inv * g.w + o.w);
                uint2 packed;
                packed.x = *reinterpret_cast<const uint32_t*>(&lo);
                packed.y = *reinterpret_cast<const uint32_t*>(&hi);
                *reinterpret_cast<uint2*>(dst + 4 * i) = packed;
            }
        }
        for (int i = K + lane; i < k_pad; i += 32) dst[i] = __float2bfloat16_rn(0.0f);
    }
}

// MT: tiles of 16 tokens (1 to 4).  NG: feature groups (of 8 features) per pass: 4, 2 or 1, for a reduction length
// of up to 1024, 2048 or 4096 (NG x chunks = the 16 weight pieces a thread holds: all of a pass's weights are
// requested at its start, one DRAM round trip, and used as the chunks of activations come in).
// STAGE: how the activations reach shared memory.  0: chunk by chunk through two buffers (any number of tokens).
// 1 (up to 16 tokens): all columns at once, one round trip, kept for all of the block's passes.  2 (up to 16 tokens,
// K up to 1024): the same, made here from the float32 rows by a LayerNorm.
// FEW (up to 8 tokens, STAGE 1 and 2): two feature groups are the sixteen rows of a product and the tokens its eight columns, where otherwise sixteen
// rows of tokens, half of them empty, meet eight features: half as many products for the same sums (mma.sync is one product in some 32
// cycles a scheduler, 0.3 of the 1.0 us that a pass over 2304 x 768 spends in them).
template <int MT, int NG, typename TO, int STAGE = 0, bool FEW = false>
__global__ void __launch_bounds__(kThreads, 1)
gemm_rows_kernel(const __nv_bfloat16* __restrict__ A, int64_t lda, const __nv_bfloat16* __restrict__ W, int64_t ldw,
                 const float* __restrict__ bias, const float* residual, int64_t ldr, TO* out, int64_t ldo, int M, int N, int K,
                 int act, KvScatter kv, RowNorm norm) {
    static_assert(STAGE == 0 || MT == 1, "all columns at once for up to 16 tokens only");
    static_assert(STAGE != 2 || NG == 4, "rows are normalised in the kernel for K up to 1024");
    static_assert(!FEW || STAGE != 0, "few tokens have all columns at once");
    constexpr bool FULL = STAGE != 0;
    constexpr int kRows = FEW ? 8 : MT * 16, MC = kWRegs / NG, kTileFloats = FEW ? 64 : 128;
    extern __shared__ __align__(16) uint8_t smem_bytes[];
    // The activations: two buffers of one chunk each, [2][kRows][kChunkLd]; or (FULL) all columns at once, [16][ld_full].
    __nv_bfloat16* act_s = reinterpret_cast<__nv_bfloat16*>(smem_bytes);
    const int ld_full = (K + kChunk - 1) / kChunk * kChunk + 32;        // 64 bytes mod 128 as well
    const size_t act_bytes = FULL ? (size_t)kRows * ld_full * sizeof(__nv_bfloat16) : (size_t)2 * kRows * kChunkLd * sizeof(__nv_bfloat16);
    float* red_s = reinterpret_cast<float*>(smem_bytes + act_bytes);   // [kWarps][NG][MT][kTileFloats]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int n_groups = (N + 7) / 8;
    const int per_cta = (n_groups + (int)gridDim.x - 1) / (int)gridDim.x;
    const int g_begin = min(n_groups, (int)blockIdx.x * per_cta), g_end = min(n_groups, g_begin + per_cta);
    const int n_chunks = (K + kChunk - 1) / kChunk;            // at most MC (the host checks)

    // Chunk c of the activations -> buffer c & 1 (rows past M and columns past K as zeros).
    auto stage = [&](int c) {
        __nv_bfloat16* dst = act_s + (size_t)(c & 1) * kRows * kChunkLd;
        const int k0 = c * kChunk;
        constexpr int kPieces = kChunk / 8;
        for (int idx = threadIdx.x; idx < kRows * kPieces; idx += kThreads) {
            const int r = idx / kPieces, p = idx - r * kPieces;
            const bool valid = r < M && k0 + p * 8 < K;
            cp_async16(dst + r * kChunkLd + p * 8, A + (valid ? (size_t)r * lda + k0 + p * 8 : 0), valid);
        }
    };

    for (int gp = g_begin; gp < g_end; gp += NG) {
        const int ng = min(NG, g_end - gp);
        // This warp's k-block of every chunk (columns c * 256 + warp * 32 ...), for every group of the pass.
        uint4 w[kWRegs];
#pragma unroll
        for (int c = 0; c < MC; ++c)
#pragma unroll
            for (int gi = 0; gi < NG; ++gi) {
                const int f = (gp + gi) * 8 + g, k = c * kChunk + warp * 32 + t * 8;
                w[c * NG + gi] = (c < n_chunks && gi < ng && f < N && k < K) ? __ldg(reinterpret_cast<const uint4*>(W + (size_t)f * ldw + k))
                                                                           : make_uint4(0, 0, 0, 0);
            }
        float acc[NG][MT][4];
#pragma unroll
        for (int i = 0; i < NG; ++i)
#pragma unroll
            for (int m = 0; m < MT; ++m) acc[i][m][0] = acc[i][m][1] = acc[i][m][2] = acc[i][m][3] = 0.0f;
        if (gp == g_begin) {
            // The first pass's weights are under way; the activations come from the kernel before this one.
            if constexpr (STAGE == 2) {
                layernorm_rows_to_smem(norm, M, K, act_s, ld_full, n_chunks * kChunk, kRows);
                __syncthreads();
            } else if constexpr (STAGE == 1) {
                lb_wait_for_predecessor();
                lb_dependents_may_launch();
                const int pieces = n_chunks * kChunk / 8;
                for (int idx = threadIdx.x; idx < kRows * pieces; idx += kThreads) {
                    const int r = idx / pieces, p = idx - r * pieces;
                    const bool valid = r < M && p * 8 < K;
                    cp_async16(act_s + r * ld_full + p * 8, A + (valid ? (size_t)r * lda + p * 8 : 0), valid);
                }
                cp_async_commit();
                cp_async_wait<0>();
                __syncthreads();
            } else {
                lb_wait_for_predecessor();
                lb_dependents_may_launch();
            }
        }
        if constexpr (!FULL) {
            stage(0);
            cp_async_commit();
        }
        // A thread finishes at most kEarly elements of a pass (element idx = threadIdx.x + 256 e); their bias and residual
        // are asked for now and arrive under the products instead of after them.
        constexpr int kEarly = (NG * kRows * 8 + kThreads - 1) / kThreads;
        const lb_act_pair act_pair = lb_act_load(bias, N, act);
        float2 early[kEarly];
#pragma unroll
        for (int e = 0; e < kEarly; ++e) {
            early[e] = make_float2(0.f, 0.f);
            const int idx = threadIdx.x + e * kThreads;
            const int gi = idx / (kRows * 8), rest = idx - gi * kRows * 8, r = rest >> 3, f = (gp + gi) * 8 + (rest & 7);
            if (gi < ng && r < M && f < N)
                early[e] = make_float2(bias != nullptr ? __ldg(bias + f) : 0.0f, residual != nullptr ? __ldcg(residual + (size_t)r * ldr + f) : 0.0f);
        }
#pragma unroll
        for (int c = 0; c < MC; ++c) {
            if (c < n_chunks) {                                 // the same for every thread
                if constexpr (!FULL) {
                    if (c + 1 < n_chunks) stage(c + 1);
                    cp_async_commit();
                    cp_async_wait<1>();
                    __syncthreads();
                }
                const int kLd = FULL ? ld_full : kChunkLd;
                const __nv_bfloat16* buf = (FULL ? act_s + c * kChunk : act_s + (size_t)(c & 1) * kRows * kChunkLd) + warp * 32 + t * 8;
                if constexpr (FEW) {
                    if (c * kChunk + warp * 32 < K) {
                        const uint4 x = *reinterpret_cast<const uint4*>(buf + g * kLd);
#pragma unroll
                        for (int gi = 0; gi < NG; gi += 2) {
                            if (gi < ng) {                            // a group that is not there: zeros
                                const uint4 w0 = w[c * NG + gi], w1 = gi + 1 < NG ? w[c * NG + (gi + 1 < NG ? gi + 1 : gi)] : make_uint4(0, 0, 0, 0);
                                mma_bf16(acc[gi][0], w0.x, w1.x, w0.y, w1.y, x.x, x.y);
                                mma_bf16(acc[gi][0], w0.z, w1.z, w0.w, w1.w, x.z, x.w);
                            }
                        }
                    }
                } else if (c * kChunk + warp * 32 < K) {
#pragma unroll
                    for (int m = 0; m < MT; ++m) {
                        const uint4 lo = *reinterpret_cast<const uint4*>(buf + (m * 16 + g) * kLd);
                        const uint4 hi = *reinterpret_cast<const uint4*>(buf + (m * 16 + g + 8) * kLd);
#pragma unroll
                        for (int gi = 0; gi < NG; ++gi) {
                            if (gi < ng) {
                                mma_bf16(acc[gi][m], lo.x, hi.x, lo.y, hi.y, w[c * NG + gi].x, w[c * NG + gi].y);
                                mma_bf16(acc[gi][m], lo.z, hi.z, lo.w, hi.w, w[c * NG + gi].z, w[c * NG + gi].w);
                            }
                        }
                    }
                }
                if constexpr (!FULL) __syncthreads();        // the buffer is free: the chunk after next goes into it
            }
        }
        // Partial tiles of the eight warps -> shared memory -> summed in warp order -> epilogue.
#pragma unroll
        for (int gi = 0; gi < NG; ++gi) {
            if (FEW && gi < ng) {
                // Feature g of the group, tokens 2t and 2t + 1: a pair's first group has the first half of the sums, its second one the other.
                float* tile = red_s + (size_t)(warp * NG + gi) * kTileFloats;
                tile[2 * t * 8 + g] = acc[gi & ~1][0][gi & 1 ? 2 : 0];
                tile[(2 * t + 1) * 8 + g] = acc[gi & ~1][0][gi & 1 ? 3 : 1];
            } else if (gi < ng) {
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    float* tile = red_s + ((size_t)(warp * NG + gi) * MT + m) * 128;
                    tile[g * 8 + 2 * t] = acc[gi][m][0];
                    tile[g * 8 + 2 * t + 1] = acc[gi][m][1];
                    tile[(g + 8) * 8 + 2 * t] = acc[gi][m][2];
                    tile[(g + 8) * 8 + 2 * t + 1] = acc[gi][m][3];
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int e = 0; e < kEarly; ++e) {
            const int idx = threadIdx.x + e * kThreads;
            const int gi = idx / (kRows * 8), rest = idx - gi * kRows * 8, r = rest >> 3, cfeat = rest & 7;
            const int f = (gp + gi) * 8 + cfeat;
            if (gi < ng && r < M && f < N) {
                const int m = r >> 4, rr = r & 15;
                float v = 0.0f;
#pragma unroll
                for (int wp = 0; wp < kWarps; ++wp) v += red_s[((size_t)(wp * NG + gi) * MT + m) * kTileFloats + rr * 8 + cfeat];
                float y = lb_activate(v + early[e].x, act, act_pair);
                if (residual != nullptr) y += early[e].y;
                out[(size_t)r * ldo + f] = lb_from_float<TO>(y);
                if (kv.cache != nullptr && f >= kv.q_dim) keep_key_or_value(kv, r, f, y);
            }
        }
        __syncthreads();
    }
}

template <int MT, int NG, typename TO, int STAGE = 0, bool FEW = false>
int launch(const void* A, int64_t lda, const void* W, int64_t ldw, const float* bias, const float* residual, int64_t ldr,
           void* out, int64_t ldo, int M, int N, int K, int act, KvScatter kv, int n_sm, cudaStream_t s, RowNorm norm = RowNorm{}) {
    const size_t ld_full = (size_t)(K + kChunk - 1) / kChunk * kChunk + 32;
    const size_t act_bytes = STAGE != 0 ? (FEW ? 8 : 16) * ld_full * sizeof(__nv_bfloat16) : (size_t)2 * MT * 16 * kChunkLd * sizeof(__nv_bfloat16);
    const size_t smem = act_bytes + (size_t)kWarps * NG * MT * (FEW ? 64 : 128) * sizeof(float);
    static size_t configured = 0;
    if (smem > configured) {
        LB_CHECK_CUDA(cudaFuncSetAttribute(gemm_rows_kernel<MT, NG, TO, STAGE, FEW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured = smem;
    }
    const int n_groups = (N + 7) / 8;
    const int grid = n_groups < n_sm ? n_groups : n_sm;
    LB_CHECK_CUDA(lb_launch_overlapped(gemm_rows_kernel<MT, NG, TO, STAGE, FEW>, dim3(grid), dim3(kThreads), smem, s, (const __nv_bfloat16*)A, lda,
                                       (const __nv_bfloat16*)W, ldw, bias, residual, ldr, (TO*)out, ldo, M, N, K, act, kv, norm));
    return LB_OK;
}

template <int MT, typename TO, int STAGE = 0, bool FEW = false>
int launch_by_k(const void* A, int64_t lda, const void* W, int64_t ldw, const float* bias, const float* residual, int64_t ldr,
                void* out, int64_t ldo, int M, int N, int K, int act, KvScatter kv, int n_sm, cudaStream_t s) {
    if (K <= 4 * kChunk) return launch<MT, 4, TO, STAGE, FEW>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, kv, n_sm, s);
    if (K <= 8 * kChunk) return launch<MT, 2, TO, STAGE, FEW>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, kv, n_sm, s);
    return launch<MT, 1, TO, STAGE, FEW>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, kv, n_sm, s);
}

// ---- up to 16 tokens, a slice of weights that does not fit a pass's registers -----------------------------------------
//
// gemm_rows_kernel asks for the weights of a pass at its start and for the next pass's after it, a round trip to memory a pass; the
// split tcgen05 product that served longer reductions before needs a second launch to add its parts, and a third where the rows
// have to be normalised first.  Here the block's weights run through a ring in shared memory instead: a lane copies by cp.async the
// very 16 bytes that it will feed to its products and reads them back itself, so the ring needs no barrier, and it is kept full from
// before the wait for the kernel before until the last chunk is asked for.  The activations of a chunk travel with its weights, or
// (NORMED) are made here from the float32 rows as gemm_rows_kernel makes them.  Bound by the weights' way from memory:
// 148 blocks with some 64 KB in flight each.  A block takes 74 to 138 KB of shared memory for up to 8 tokens (more beyond), so that small launches
// start beside the one before; GPT-2 XL's do not (138 KB where rows are normalised, 98 KB elsewhere, and an SM has 228), and ask for their weights as
// the blocks before them leave.
// Measured (GPT-2 XL, 8 requests, contexts of 360 to 880): the step's 243 launches took 483 before; 2.38 -> 2.31 ms with its logits'
// copy, 1.98 ms since the norm is short code.  Alone with cold caches, 8 tokens: 1600 -> 6400 normed 10 us (before: norm 3.6, split product 9.2 and
// second half 4.1), 6400 -> 1600 7.5 us (9.2 and 3.6).
constexpr int kStreamGroups = 8;       // the most feature groups of eight a block takes
constexpr int kStreamMaxK = 8192;
constexpr int kStreamNormedMaxK = 2048;
// Chunks in flight: GB groups of weights (and the activations' one or two pieces) of 4 KB each a chunk.
constexpr int stream_depth(int gb, bool normed, bool wide) {
    const int pieces = normed ? 19 : 24, a = normed ? 0 : wide ? 2 : 1, d = pieces / (gb + a);
    return d < 2 ? 2 : d > 12 ? 12 : d;
}

// Bytes between the rows that are normalised: room for a float32 row, and 64 bytes mod 128 for the bfloat16 one that takes its place.
__host__ __device__ constexpr int stream_row_bytes(int K) {
    const int whole = 4 * K, padded = 2 * ((K + kChunk - 1) / kChunk * kChunk), most = whole > padded ? whole : padded;
    return (most - 64 + 127) / 128 * 128 + 64;
}

// The rows' norm with gains and offsets in shared memory (gain_s, offset_s), for K up to kStreamNormedMaxK; one warp a row.  A launch
// runs this code once, among other kernels, so the code is kept short: a lane puts its pieces of the row into shared memory as they come and
// walks them there in loops.  Unrolled over registers it was half a microsecond faster launched again and again by itself, and
// slower in a step, where its instructions came from memory each time: GPT-2 XL, 8 requests, 2.08 -> 1.98 ms a step.
__device__ void stream_norm_rows(const RowNorm& n, int M, int K, uint8_t* rows_s, int k_pad, int rows, const float* gain_s, const float* offset_s) {
    constexpr int kVecs = kStreamNormedMaxK / 128;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_vec = K / 4, stride = stream_row_bytes(K);
    for (int r = warp; r < rows; r += kWarps) {
        float4* x_s = reinterpret_cast<float4*>(rows_s + (size_t)r * stride);
        uint8_t* dst = rows_s + (size_t)r * stride;
        if (r >= M) {
            for (int i = lane * 16; i < 2 * k_pad; i += 512) *reinterpret_cast<uint4*>(dst + i) = make_uint4(0, 0, 0, 0);
            continue;
        }
        const float4* row = reinterpret_cast<const float4*>(n.x + (size_t)r * n.ldx);
        float sum = 0.0f;
        {
            float4 v[kVecs];
#pragma unroll
            for (int j = 0; j < kVecs; ++j) v[j] = lane + 32 * j < n_vec ? __ldcg(row + lane + 32 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < kVecs; ++j) {
                if (lane + 32 * j < n_vec) x_s[lane + 32 * j] = v[j];
                sum += (v[j].x + v[j].y) + (v[j].z + v[j].w);
            }
        }
        const float mean = n.rms ? 0.0f : lb_warp_sum(sum) / (float)K;
        float ss = 0.0f;
#pragma unroll 4
        for (int i = lane; i < n_vec; i += 32) {                         // the lane's own pieces
            const float4 v = x_s[i];
            const float d0 = v.x - mean, d1 = v.y - mean, d2 = v.z - mean, d3 = v.w - mean;
            ss = fmaf(d0, d0, ss);
            ss = fmaf(d1, d1, ss);
            ss = fmaf(d2, d2, ss);
            ss = fmaf(d3, d3, ss);
        }
        const float inv = 1.0f / sqrtf(lb_warp_sum(ss) / (float)K + n.eps);
#pragma unroll 2
        for (int i0 = 0; i0 < n_vec; i0 += 32) {
            const int i = i0 + lane;
            const bool in = i < n_vec;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f), g = make_float4(1.f, 1.f, 1.f, 1.f), o = v;
            if (in) v = x_s[i];
            if (in && n.gain != nullptr) {
                g = reinterpret_cast<const float4*>(gain_s)[i];
                g.x += n.gain_offset;
                g.y += n.gain_offset;
                g.z += n.gain_offset;
                g.w += n.gain_offset;
            }
            if (in && n.offset != nullptr) o = reinterpret_cast<const float4*>(offset_s)[i];
            const __nv_bfloat162 lo = __floats2bfloat162_rn((v.x - mean) * inv * g.x + o.x, (v.y - mean) * inv * g.y + o.y);
            const __nv_bfloat162 hi = __floats2bfloat162_rn((v.z - mean) * inv * g.z + o.z, (v.w - mean) * inv * g.w + o.w);
            uint2 packed;
            packed.x = *reinterpret_cast<const uint32_t*>(&lo);
            packed.y = *reinterpret_cast<const uint32_t*>(&hi);
            __syncwarp();                                                // all have read: the 256 bytes of these 32 pieces lie over pieces read by now
            if (in) *reinterpret_cast<uint2*>(dst + 8 * i) = packed;
        }
        __syncwarp();
        for (int i = 2 * K + 2 * lane; i < 2 * k_pad; i += 64) *reinterpret_cast<uint16_t*>(dst + i) = 0;
    }
}

// GB: the most groups a block has.  WIDE: more than 8 tokens.  K, the row strides and the bases as for gemm_rows_kernel.
template <int GB, bool NORMED, bool WIDE, typename TO>
__global__ void __launch_bounds__(kThreads, 2)
gemm_stream_kernel(const __nv_bfloat16* __restrict__ A, int64_t lda, const __nv_bfloat16* __restrict__ W, int64_t ldw, const float* __restrict__ bias,
                   const float* residual, int64_t ldr, TO* out, int64_t ldo, int M, int N, int K, int act, KvScatter kv, RowNorm norm) {
    constexpr int DEPTH = stream_depth(GB, NORMED, WIDE), ROWS = WIDE ? 16 : 8, APIECES = NORMED ? 0 : WIDE ? 2 : 1;
    extern __shared__ __align__(16) uint8_t smem_bytes[];
    uint4* ring = reinterpret_cast<uint4*>(smem_bytes);                      // [DEPTH][GB + APIECES][256 lanes]; at the end the warps' sums
    float* red_s = reinterpret_cast<float*>(smem_bytes);                     // [kWarps][GB][ROWS][8]
    static_assert((size_t)kWarps * GB * ROWS * 8 * sizeof(float) <= (size_t)DEPTH * (GB + APIECES) * kThreads * 16, "the sums fit the ring");
    float* gain_s = reinterpret_cast<float*>(ring + DEPTH * (GB + APIECES) * kThreads);     // NORMED: gains and offsets, then the rows
    float* offset_s = gain_s + K;
    const int ld = stream_row_bytes(K) / 2;
    __nv_bfloat16* act_s = reinterpret_cast<__nv_bfloat16*>(offset_s + K);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int n_groups = (N + 7) / 8, n_chunks = (K + kChunk - 1) / kChunk;
    const int share = n_groups / (int)gridDim.x, more = n_groups % (int)gridDim.x;      // the first `more` blocks have a group more
    const int g_begin = (int)blockIdx.x * share + min((int)blockIdx.x, more), ng = share + ((int)blockIdx.x < more ? 1 : 0);
    const int k_lane = warp * 32 + t * 8;
    const __nv_bfloat16* w_lane = W + (size_t)(g_begin * 8 + g) * ldw + k_lane;

    auto weights = [&](int c) {                                              // chunk c's weights -> its place in the ring
        uint4* to = ring + (c % DEPTH) * (GB + APIECES) * kThreads + threadIdx.x;
        const bool there = c * kChunk + k_lane < K;
#pragma unroll
        for (int gi = 0; gi < GB; ++gi)
            if (gi < ng) {
                const bool valid = there && (g_begin + gi) * 8 + g < N;
                cp_async16(to + gi * kThreads, valid ? w_lane + (size_t)gi * 8 * ldw + c * kChunk : W, valid);
            }
    };
    auto activations = [&](int c) {
        uint4* to = ring + ((c % DEPTH) * (GB + APIECES) + GB) * kThreads + threadIdx.x;
        const int k = c * kChunk + k_lane;
#pragma unroll
        for (int p = 0; p < APIECES; ++p) {
            const bool valid = k < K && g + 8 * p < M;
            cp_async16(to + p * kThreads, valid ? A + (size_t)(g + 8 * p) * lda + k : A, valid);
        }
    };

    // Before the wait: what does not depend on the kernel before.
    if constexpr (NORMED) {
        for (int i = threadIdx.x; i < K / 4; i += kThreads) {
            if (norm.gain != nullptr) cp_async16(gain_s + 4 * i, norm.gain + 4 * i, true);
            if (norm.offset != nullptr) cp_async16(offset_s + 4 * i, norm.offset + 4 * i, true);
        }
        cp_async_commit();
    }
#pragma unroll
    for (int c = 0; c < DEPTH; ++c) {
        if (c < n_chunks) weights(c);
        cp_async_commit();
    }
    if constexpr (NORMED) cp_async_wait<DEPTH>();
    const lb_act_pair act_pair = lb_act_load(bias, N, act);
    lb_wait_for_predecessor();
    lb_dependents_may_launch();
    if constexpr (NORMED) {
        __syncthreads();                                                     // every thread's gains and offsets
        stream_norm_rows(norm, M, K, reinterpret_cast<uint8_t*>(act_s), n_chunks * kChunk, ROWS, gain_s, offset_s);
        __syncthreads();
    } else {
#pragma unroll
        for (int c = 0; c < DEPTH; ++c) {
            if (c < n_chunks) activations(c);
            cp_async_commit();
        }
    }
    // The elements this thread will finish: their bias and residual travel under the products.
    constexpr int kElements = GB * ROWS * 8, kEarly = (kElements + kThreads - 1) / kThreads;
    float2 early[kEarly];
#pragma unroll
    for (int e = 0; e < kEarly; ++e) {
        early[e] = make_float2(0.f, 0.f);
        const int idx = threadIdx.x + e * kThreads, gi = idx / (ROWS * 8), r = idx / 8 % ROWS, f = (g_begin + gi) * 8 + (idx & 7);
        if (gi < ng && r < M && f < N)
            early[e] = make_float2(bias != nullptr ? __ldg(bias + f) : 0.0f, residual != nullptr ? __ldcg(residual + (size_t)r * ldr + f) : 0.0f);
    }
    // Up to 8 tokens a pair of groups is the sixteen rows of a product, the tokens its columns (see FEW above): acc[gi] has both groups' sums, gi even.
    float acc[GB][4];
#pragma unroll
    for (int gi = 0; gi < GB; ++gi) acc[gi][0] = acc[gi][1] = acc[gi][2] = acc[gi][3] = 0.0f;
    // Groups of copies are counted alike in both forms: DEPTH - 1 later chunks may be on their way when chunk c is used.
    for (int c = 0; c < n_chunks; ++c) {
        cp_async_wait<DEPTH - 1>();
        const uint4* from = ring + (c % DEPTH) * (GB + APIECES) * kThreads + threadIdx.x;
        uint4 lo, hi = make_uint4(0, 0, 0, 0);
        if constexpr (NORMED) {
            const __nv_bfloat16* row = act_s + g * ld + c * kChunk + k_lane;
            lo = *reinterpret_cast<const uint4*>(row);
            if constexpr (WIDE) hi = *reinterpret_cast<const uint4*>(row + 8 * ld);
        } else {
            lo = from[GB * kThreads];
            if constexpr (WIDE) hi = from[(GB + 1) * kThreads];
        }
        if constexpr (!WIDE) {
#pragma unroll
            for (int gi = 0; gi < GB; gi += 2)
                if (gi < ng) {
                    const uint4 w0 = from[gi * kThreads];
                    // (The place of a group that the block does not have holds anything: its sums are rows of their own, which nobody reads.)
                    const uint4 w1 = gi + 1 < GB ? from[(gi + 1 < GB ? gi + 1 : gi) * kThreads] : make_uint4(0, 0, 0, 0);
                    mma_bf16(acc[gi], w0.x, w1.x, w0.y, w1.y, lo.x, lo.y);
                    mma_bf16(acc[gi], w0.z, w1.z, w0.w, w1.w, lo.z, lo.w);
                }
        }
#pragma unroll
        for (int gi = 0; gi < GB; ++gi)
            if (WIDE && gi < ng) {
                const uint4 w = from[gi * kThreads];
                mma_bf16(acc[gi], lo.x, hi.x, lo.y, hi.y, w.x, w.y);
                mma_bf16(acc[gi], lo.z, hi.z, lo.w, hi.w, w.z, w.w);
            }
        // The pieces are in the products: the chunk DEPTH further on may take their place.
        if (c + DEPTH < n_chunks) {
            weights(c + DEPTH);
            if constexpr (!NORMED) activations(c + DEPTH);
        }
        cp_async_commit();
    }
    cp_async_wait<0>();
    __syncthreads();                                                         // the ring turns into the warps' sums
#pragma unroll
    for (int gi = 0; gi < GB; ++gi)
        if (gi < ng) {
            float* tile = red_s + (size_t)(warp * GB + gi) * ROWS * 8;
            if constexpr (WIDE) {
                *reinterpret_cast<float2*>(tile + g * 8 + 2 * t) = make_float2(acc[gi][0], acc[gi][1]);
                *reinterpret_cast<float2*>(tile + (g + 8) * 8 + 2 * t) = make_float2(acc[gi][2], acc[gi][3]);
            } else {
                tile[2 * t * 8 + g] = acc[gi & ~1][gi & 1 ? 2 : 0];
                tile[(2 * t + 1) * 8 + g] = acc[gi & ~1][gi & 1 ? 3 : 1];
            }
        }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < kEarly; ++e) {
        const int idx = threadIdx.x + e * kThreads, gi = idx / (ROWS * 8), r = idx / 8 % ROWS, f = (g_begin + gi) * 8 + (idx & 7);
        if (gi >= ng || r >= M || f >= N) continue;
        float v = 0.0f;
#pragma unroll
        for (int wp = 0; wp < kWarps; ++wp) v += red_s[(size_t)(wp * GB) * ROWS * 8 + idx];
        float y = lb_activate(v + early[e].x, act, act_pair);
        if (residual != nullptr) y += early[e].y;
        out[(size_t)r * ldo + f] = lb_from_float<TO>(y);
        if (kv.cache != nullptr && f >= kv.q_dim) keep_key_or_value(kv, r, f, y);
    }
}

template <int GB, bool NORMED, bool WIDE, typename TO>
int launch_stream(const void* A, int64_t lda, const void* W, int64_t ldw, const float* bias, const float* residual, int64_t ldr, void* out, int64_t ldo,
                  int M, int N, int K, int act, KvScatter kv, RowNorm norm, int grid, cudaStream_t s) {
    size_t smem = (size_t)stream_depth(GB, NORMED, WIDE) * (GB + (NORMED ? 0 : WIDE ? 2 : 1)) * kThreads * 16;
    if (NORMED) smem += (size_t)2 * K * sizeof(float) + (size_t)(WIDE ? 16 : 8) * stream_row_bytes(K);
    static size_t configured = 0;
    if (smem > configured) {
        LB_CHECK_CUDA(cudaFuncSetAttribute(gemm_stream_kernel<GB, NORMED, WIDE, TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured = smem;
    }
    LB_CHECK_CUDA(lb_launch_overlapped(gemm_stream_kernel<GB, NORMED, WIDE, TO>, dim3(grid), dim3(kThreads), smem, s, (const __nv_bfloat16*)A, lda,
                                       (const __nv_bfloat16*)W, ldw, bias, residual, ldr, (TO*)out, ldo, M, N, K, act, kv, norm));
    return LB_OK;
}

template <bool NORMED, bool WIDE, typename TO>
int stream_by_groups(const void* A, int64_t lda, const void* W, int64_t ldw, const float* bias, const float* residual, int64_t ldr, void* out, int64_t ldo,
                     int M, int N, int K, int act, KvScatter kv, RowNorm norm, int n_sm, cudaStream_t s) {
    const int n_groups = (N + 7) / 8, grid = n_groups < n_sm ? n_groups : n_sm, most = (n_groups + grid - 1) / grid;
#define LB_GO(GB) return launch_stream<GB, NORMED, WIDE, TO>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, kv, norm, grid, s)
    if (most <= 1) LB_GO(1);
    if (most <= 2) LB_GO(2);
    if (most <= 4) LB_GO(4);
    if (most <= 6) LB_GO(6);
    if (most <= kStreamGroups) LB_GO(8);
#undef LB_GO
    return lb_fail(LB_ERR_UNSUPPORTED, "gemm_rows: %d features are too many for one launch", N);
}

template <bool NORMED>
int stream(int out_dtype, const void* A, int64_t lda, const void* W, int64_t ldw, const float* bias, const float* residual, int64_t ldr, void* out,
           int64_t ldo, int M, int N, int K, int act, KvScatter kv, RowNorm norm, int n_sm, cudaStream_t s) {
    if (out_dtype == LB_F32)
        return M > 8 ? stream_by_groups<NORMED, true, float>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, kv, norm, n_sm, s)
                     : stream_by_groups<NORMED, false, float>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, kv, norm, n_sm, s);
    return M > 8 ? stream_by_groups<NORMED, true, __nv_bfloat16>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, kv, norm, n_sm, s)
                 : stream_by_groups<NORMED, false, __nv_bfloat16>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, kv, norm, n_sm, s);
}

int sm_count() {
    static int n_sm = 0;
    if (n_sm == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n_sm = 148;
    }
    return n_sm;
}

}  // namespace

// The kernel that takes a product of these sizes on n_sm SMs: 2 the ring (gemm_stream_kernel), 1 the one that holds a pass's weights in registers
// (gemm_rows_kernel), 0 none.  Up to 16 tokens the ring takes over where one pass of registers does not hold a block's weights, while
// a block has at most eight groups; the register kernel takes reductions of up to 4096 (normed: 1024) and at most four passes over the feature groups of
// 148 blocks (the head's vocabulary is left to the tcgen05 kernel, whose tiles suit it).
// Where either could take 9 to 16 tokens with K up to 1024, the ring's two pieces of activations (or its norm, which walks shared memory) leave less
// to gain.  Measured with cold weights, registers / ring in us: 12 tokens, normed, 4744 x 512 6.9 / 6.6, 9472 x 512 7.9 / 8.0, 4744 x 1024 8.1 / 9.1, 9472 x
// 1024 9.7 / 11.3; not normed, 9472 x 768 7.3 / 6.6, 6400 x 1024 7.0 / 5.9, 8192 x 1024 7.8 / 7.8.
extern "C" int lb_gemm_rows_kind(int M, int N, int K, int n_sm, int normed) {
    if (M <= 0 || N <= 0 || K <= 0 || n_sm <= 0 || M > (normed ? 16 : kMaxRows)) return 0;
    const int n_groups = (N + 7) / 8, grid = n_groups < n_sm ? n_groups : n_sm, most = (n_groups + grid - 1) / grid;
    const int pass = K <= 4 * kChunk ? 4 : K <= 8 * kChunk ? 2 : K <= 16 * kChunk ? 1 : 0;       // groups whose weights a pass's registers hold
    const bool registers = (normed ? pass == 4 : pass != 0) && n_groups <= 148 * 4 * pass;
    const bool ring = M <= 16 && K <= (normed ? kStreamNormedMaxK : kStreamMaxK) && most <= kStreamGroups;
    if (!registers) return ring ? 2 : 0;
    bool faster = most > pass;
    if (M > 8 && K <= 4 * kChunk) {
        const bool few = most <= 6;
        faster = faster && (normed ? K <= kChunk || (K <= 2 * kChunk && few) : K <= 3 * kChunk + kChunk / 2 || few);
    }
    return ring && faster ? 2 : 1;
}

// Whether the kernels take the product: sizes as above, K and the row strides of A and W multiples of 8, 16-byte aligned bases.
extern "C" int lb_gemm_rows_supports(const void* A, int64_t lda, const void* W, int64_t ldw, int M, int N, int K) {
    if (K % 8 != 0 || lda % 8 != 0 || ldw % 8 != 0 || ((uintptr_t)A & 15) != 0 || ((uintptr_t)W & 15) != 0) return 0;
    return lb_gemm_rows_kind(M, N, K, sm_count(), 0) != 0;
}

// The same product for up to 16 tokens and a reduction length of up to 2048 with the activations made in the kernel:
// LayerNorm (two-pass 32-bit statistics, eps, gain and offset or null) of the float32 rows x, normalised by every
// block for itself.  lb_gemm_rows_normed_supports says whether the kernel takes the operands.
extern "C" int lb_gemm_rows_normed_supports(const void* x, int64_t ldx, const void* W, int64_t ldw, int M, int N, int K) {
    if (K % 8 != 0 || ldx % 4 != 0 || ldw % 8 != 0 || ((uintptr_t)x & 15) != 0 || ((uintptr_t)W & 15) != 0) return 0;
    return lb_gemm_rows_kind(M, N, K, sm_count(), 1) != 0;
}

// Whether a step's rows are better normalised by every block of the product than by a launch of their own before it.  Every block reads and normalises
// all rows: with long rows (the ring's form) sixteen of them take longer than the launch that it saves, and the wait for them is exposed.
// Measured (GPT-2 XL, contexts of 300 to 1000, a step with the norm inside / in a launch): 8 requests 1.93 ms / -, 9 requests 2.60 / 2.23,
// 12 requests 2.67 / 2.27, 16 requests 2.73 / 2.42.
extern "C" int lb_gemm_rows_normed_pays(int M, int K) { return K <= 4 * kChunk || M <= 8; }

extern "C" int lb_gemm_rows_normed(int out_dtype, const float* x, int64_t ldx, const float* gain, const float* offset, float eps,
                                   const void* W, int64_t ldw, const float* bias, const float* residual, int64_t ldr, void* out,
                                   int64_t ldo, int M, int N, int K, int act, void* kv_cache, const int32_t* slot_mapping, int q_dim,
                                   int n_kv_head, int head_dim, int page_size, void* stream) {
    return lb_gemm_rows_normed_kind(out_dtype, x, ldx, gain, offset, eps, 0, 0.0f, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, kv_cache,
                                    slot_mapping, q_dim, n_kv_head, head_dim, page_size, stream);
}

// The same with the kind of norm as an argument: rms != 0 divides by sqrt(mean(x^2) + eps) without taking a mean off, and gain_offset is
// added to every gain.
extern "C" int lb_gemm_rows_normed_kind(int out_dtype, const float* x, int64_t ldx, const float* gain, const float* offset, float eps, int rms,
                                        float gain_offset, const void* W, int64_t ldw, const float* bias, const float* residual, int64_t ldr,
                                        void* out, int64_t ldo, int M, int N, int K, int act, void* kv_cache, const int32_t* slot_mapping,
                                        int q_dim, int n_kv_head, int head_dim, int page_size, void* stream_handle) {
    LB_CHECK_ARG(out_dtype == LB_BF16 || out_dtype == LB_F32, "gemm_rows_normed: unknown output dtype %d", out_dtype);
    if (!lb_gemm_rows_normed_supports(x, ldx, W, ldw, M, N, K) || ((uintptr_t)gain & 15) != 0 || ((uintptr_t)offset & 15) != 0)
        return lb_fail(LB_ERR_UNSUPPORTED, "gemm_rows_normed: takes 1 to 16 tokens, K up to 2048 and a multiple of 8, 16-byte aligned bases "
                       "(M=%d N=%d K=%d ldx=%lld ldw=%lld)", M, N, K, (long long)ldx, (long long)ldw);
    LB_CHECK_ARG(ldx >= K && ldw >= K && ldo >= N, "gemm_rows_normed: a row stride is shorter than the row");
    const int n_sm = sm_count();
    KvScatter kv{static_cast<__nv_bfloat16*>(kv_cache), slot_mapping, q_dim, n_kv_head, head_dim, page_size};
    if (kv_cache != nullptr)
        LB_CHECK_ARG(slot_mapping != nullptr && q_dim >= 0 && n_kv_head > 0 && head_dim > 0 && page_size > 0 &&
                         q_dim + 2 * n_kv_head * head_dim == N,
                     "gemm_rows_normed: the cache destination needs N = q_dim + 2 * n_kv_head * head_dim (N=%d q_dim=%d heads %d x %d)", N,
                     q_dim, n_kv_head, head_dim);
    const RowNorm norm{x, ldx, gain, offset, eps, rms, gain_offset};
    auto s = static_cast<cudaStream_t>(stream_handle);
    if (lb_gemm_rows_kind(M, N, K, n_sm, 1) == 2) return stream<true>(out_dtype, nullptr, 0, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, kv, norm, n_sm, s);
    if (out_dtype == LB_F32)
        return (M <= 8 ? launch<1, 4, float, 2, true> : launch<1, 4, float, 2>)(nullptr, 0, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, kv, n_sm, s, norm);
    return (M <= 8 ? launch<1, 4, __nv_bfloat16, 2, true> : launch<1, 4, __nv_bfloat16, 2>)(nullptr, 0, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, kv, n_sm, s, norm);
}

extern "C" int lb_gemm_rows(int out_dtype, const void* A, int64_t lda, const void* W, int64_t ldw, const float* bias,
                            const float* residual, int64_t ldr, void* out, int64_t ldo, int M, int N, int K, int act,
                            void* kv_cache, const int32_t* slot_mapping, int q_dim, int n_kv_head, int head_dim, int page_size,
                            void* stream_handle) {
    LB_CHECK_ARG(out_dtype == LB_BF16 || out_dtype == LB_F32, "gemm_rows: unknown output dtype %d", out_dtype);
    if (!lb_gemm_rows_supports(A, lda, W, ldw, M, N, K))
        return lb_fail(LB_ERR_UNSUPPORTED, "gemm_rows: takes 1 to 64 tokens, K and row strides multiples of 8 and 16-byte aligned "
                       "bases (M=%d N=%d K=%d lda=%lld ldw=%lld)", M, N, K, (long long)lda, (long long)ldw);
    LB_CHECK_ARG(lda >= K && ldw >= K && ldo >= N, "gemm_rows: a row stride is shorter than the row");
    const int n_sm = sm_count();
    KvScatter kv{static_cast<__nv_bfloat16*>(kv_cache), slot_mapping, q_dim, n_kv_head, head_dim, page_size};
    if (kv_cache != nullptr)
        LB_CHECK_ARG(slot_mapping != nullptr && q_dim >= 0 && n_kv_head > 0 && head_dim > 0 && page_size > 0 &&
                         q_dim + 2 * n_kv_head * head_dim == N,
                     "gemm_rows: the cache destination needs N = q_dim + 2 * n_kv_head * head_dim (N=%d q_dim=%d heads %d x %d)", N,
                     q_dim, n_kv_head, head_dim);
    auto s = static_cast<cudaStream_t>(stream_handle);
    if (lb_gemm_rows_kind(M, N, K, n_sm, 0) == 2) return stream<false>(out_dtype, A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, kv, RowNorm{}, n_sm, s);
    const int mt = (M + 15) / 16;
    if (M <= 8)
        return out_dtype == LB_F32 ? launch_by_k<1, float, 1, true>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, kv, n_sm, s)
                                   : launch_by_k<1, __nv_bfloat16, 1, true>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, kv, n_sm, s);
#define LB_GO(MT)                                                                                                          \
    return out_dtype == LB_F32 ? launch_by_k<MT, float>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, kv, n_sm, s)   \
                               : launch_by_k<MT, __nv_bfloat16>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, kv, n_sm, s)
    if (mt <= 1)           // up to 16 tokens: all columns of the activations at once
        return out_dtype == LB_F32 ? launch_by_k<1, float, 1>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, kv, n_sm, s)
                                   : launch_by_k<1, __nv_bfloat16, 1>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, kv, n_sm, s);
    if (mt == 2) LB_GO(2);
    if (mt == 3) LB_GO(3);
    LB_GO(4);
#undef LB_GO
}
