// out[M, N] = epilogue(A[M, K] . W[N, K]^T) on the ordinary 32-bit units.
//
// This is the true 32-bit matrix product of the engine (no tensor cores, no
// reduced-precision mode), and the fallback for 16-bit operands whose sizes the
// tensor-core kernel refuses.  The order in which an output element's products
// are summed is a function of K alone, whatever the kernel, the tile shape and
// whatever else is in the batch, so a row's result never depends on how many
// other rows share the launch (the reference promises the same of its matmul:
// include/liyab/backend.h:40-42):
//
//   K is cut into chunks of 64 (the last may be shorter); a chunk's products are one
//   chain of fused multiply-adds in ascending k starting from zero; G = ceil(chunks /
//   32) consecutive chunks form a group whose chunk sums are added in ascending
//   order; the (at most 32) group sums are added in ascending order.
//
// Four kernels follow that order.  The tiled one (any number of tokens) cuts the groups among
// four slices of a block and adds their sums in order.  The one for up to 16 tokens (decoding)
// is bound by reading the weights once: a block owns eight features and all of K,
// each of its 32 (warp, slot) pairs owns one group of chunks for those features,
// a thread fetches its 64 weights of a chunk as 16-byte pieces that are all in
// flight together and multiplies them with the tokens' activations from the warp's
// buffer in shared memory; the group sums meet in shared memory and are added in
// order.  The third takes some products of 9 to 16 tokens in float32: the weights come into
// shared memory by whole rows of a chunk as well.  The fourth takes most of up to 8 tokens in float32: whole rows of
// weights by bulk copies, the activations once a block.
//
// Epilogue, in the reference's order (src/core/transformer.cpp:111-118, 4903-4912,
// 5526-5532): + bias[n], activation, + residual[m, n].
#include "api.h"
#include "common.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int kChunk = 64;           // products per chain
constexpr int kGroups = 32;          // at most this many group sums per output

__host__ __device__ inline int chunks_per_group(int K) {
    const int chunks = (K + kChunk - 1) / kChunk;
    return (chunks + kGroups - 1) / kGroups;
}

// ---- more than 16 tokens: 64 x 64 outputs a block, four slices of K side by side -------------------------------
//
// Bound by the FMA units.  A thread makes 8 x 8 outputs, so a tile of 64 x 64 is the work of two warps, and an SM wants at least eight:
// four slices of the block (two warps each) take four consecutive groups of chunks at a time, put their group sums into shared
// memory, and every thread adds them to its sixteen running totals in ascending order.  That keeps the order of the sums and the
// small tile, which the narrow products need to fill the SMs (590 tokens x 768 features: 120 blocks).  Products come in pairs along
// the features (fma.rn.f32x2, which rounds each half as fmaf does), half as many instructions as single ones, so that the loads
// from shared memory and the copies of a token's value into both halves find issue slots beside them.
// Measured (GPT-2 small in float32, three prompts of 590 tokens together): the step's products took 8.5 of 12.9 ms with 4 x 4 outputs a
// thread and operands loaded element by element (8 TFLOP/s); with this kernel and the attention of runs the step takes 4.1 ms.  590 x 3072
// x 768 alone, on the way: 210 us before; 115 us with two pieces of a row a warp (23 TFLOP/s; 123 us with single products, 139 us with
// a second copy of W in shared memory instead of the copies into both halves), the load unit 80 % busy with uncoalesced rows.
constexpr int kTile = 64;            // tokens and features of a block
constexpr int kSlices = 4;           // slices of K
constexpr int kSliceThreads = 64;
constexpr int kStepK = 32;           // products between two synchronisations of a slice: 128 bytes of a float32 row
constexpr int kOperandFloats = kStepK * kTile;      // [k][token or feature], its pieces of four permuted by k / 4
constexpr size_t kTiledSmem = (size_t)kSlices * (4 * kOperandFloats + kTile * kTile) * sizeof(float);

__device__ __forceinline__ uint64_t both_halves(float v) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ uint64_t fma_pair(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float2 halves(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

// The four elements at `at` as floats, of which the first `left` belong to the row; zeros for the others (and for a row that is not there).
// VECTORS: K and the strides are whole pieces of four and the bases are aligned to them, so a piece is either whole or not there.
template <typename T, bool VECTORS>
__device__ __forceinline__ float4 four_of(const T* __restrict__ at, int left, bool live) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!live || left <= 0) return v;
    if constexpr (VECTORS && sizeof(T) == 4) {
        v = *reinterpret_cast<const float4*>(at);
    } else if constexpr (VECTORS) {
        const uint2 u = *reinterpret_cast<const uint2*>(at);
        v = make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
    } else {
        v.x = lb_to_float(at[0]);
        if (left > 1) v.y = lb_to_float(at[1]);
        if (left > 2) v.z = lb_to_float(at[2]);
        if (left > 3) v.w = lb_to_float(at[3]);
    }
    return v;
}

// GROUPED: a group has more than one chunk (K > 2048).
template <typename TI, typename TO, bool VECTORS, bool GROUPED>
__global__ void __launch_bounds__(kSlices* kSliceThreads, 1)
gemm_ffma_kernel(const TI* __restrict__ A, int64_t lda, const TI* __restrict__ W, int64_t ldw, const float* __restrict__ bias, const float* residual,
                 int64_t ldr, TO* out, int64_t ldo, int M, int N, int K, int act) {
    extern __shared__ __align__(16) float tiled_smem[];
    lb_wait_for_predecessor();
    lb_dependents_may_launch();
    const int slice = threadIdx.x / kSliceThreads, tid = threadIdx.x % kSliceThreads;
    const int tx = tid % 8, ty = tid / 8;
    const int m0 = blockIdx.y * kTile, n0 = blockIdx.x * kTile;
    float* operands = tiled_smem + (size_t)slice * 4 * kOperandFloats;          // two buffers of A's and W's [32][64]
    float* sums = tiled_smem + (size_t)kSlices * 4 * kOperandFloats;            // [slice][64][64] group sums
    const int n_chunks = (K + kChunk - 1) / kChunk, G = chunks_per_group(K);
    const int n_groups = (n_chunks + G - 1) / G, rounds = (n_groups + kSlices - 1) / kSlices;

    // A thread fetches eight pieces of four of an operand a step: rows row0, row0 + 8, .. and the k piece kq of eight, so that eight lanes
    // read 128 bytes of a row in one go (two pieces of a row a warp instead took 31 passes of the load unit an instruction, as
    // many as all the rest together).  Row r of k lies at column r ^ (4 (k / 4 mod 8)): the lanes of a store fall into 32 banks and a
    // piece of four rows stays one.
    const int kq = tid & 7, row0 = (tid >> 5) * 4 + ((tid >> 3) & 3);
    const TI* a_row = A + (size_t)(m0 + row0) * lda + 4 * kq;
    const TI* w_row = W + (size_t)(n0 + row0) * ldw + 4 * kq;
    const int a_rows = M - m0 - row0, w_rows = N - n0 - row0;          // rows 8 i below these are there
    float4 piece[8];
    auto fetch = [&](const TI* rows, int64_t ld, int n_rows, int k) {
#pragma unroll
        for (int i = 0; i < 8; ++i) piece[i] = four_of<TI, VECTORS>(rows + 8 * i * ld + k, K - k - 4 * kq, 8 * i < n_rows);
    };
    auto keep = [&](float* operand) {
        float* to = operand + 4 * kq * kTile;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int column = (row0 + 8 * i) ^ (4 * kq);
            to[column] = piece[i].x;
            to[column + kTile] = piece[i].y;
            to[column + 2 * kTile] = piece[i].z;
            to[column + 3 * kTile] = piece[i].w;
        }
    };

    // This thread's share of the block's totals: 16-byte pieces threadIdx.x + 256 i of the tile's [64][16 pieces].
    float4 tot[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) tot[i] = make_float4(0.f, 0.f, 0.f, 0.f);

    // Half a step's products run between the loads of an operand's next step and its stores: A's under the first half, W's under the second.
    const int group_k = G * kChunk;
    int turn = 0;
    if (slice < n_groups) {
        fetch(a_row, lda, a_rows, slice * group_k);
        keep(operands);
        fetch(w_row, ldw, w_rows, slice * group_k);
        keep(operands + kOperandFloats);
    }
    for (int round = 0; round < rounds; ++round) {
        const int group = round * kSlices + slice;
        uint64_t grp[8][4];
        if (group < n_groups) {
            const int k_begin = group * group_k, k_end = min(K, k_begin + group_k);
            uint64_t acc[8][4];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = 0;
            for (int k0 = k_begin; k0 < k_end; k0 += kStepK) {
                const float* buffer = operands + turn * 2 * kOperandFloats;
                turn ^= 1;
                float* coming = operands + turn * 2 * kOperandFloats;
                // The slice's two warps: this step's operands are there, and nobody reads the buffer that the next step's go to.
                asm volatile("bar.sync %0, 64;" ::"r"(slice + 1) : "memory");
                const int next = k0 + kStepK < k_end ? k0 + kStepK : (group + kSlices) * group_k;      // from K on: zeros
                auto products = [&](int half) {
#pragma unroll
                    for (int kk = half * (kStepK / 2); kk < (half + 1) * (kStepK / 2); ++kk) {
                        const int turned = 4 * (kk / 4 % 8);
                        const float* a_s = buffer + kk * kTile + ((4 * ty) ^ turned);
                        const float* w_s = buffer + kOperandFloats + kk * kTile + ((4 * tx) ^ turned);
                        const float4 a0 = *reinterpret_cast<const float4*>(a_s), a1 = *reinterpret_cast<const float4*>(a_s + 32);
                        const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(w_s), w1 = *reinterpret_cast<const ulonglong2*>(w_s + 32);
                        const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const uint64_t aa = both_halves(a[i]);
                            acc[i][0] = fma_pair(aa, w0.x, acc[i][0]);
                            acc[i][1] = fma_pair(aa, w0.y, acc[i][1]);
                            acc[i][2] = fma_pair(aa, w1.x, acc[i][2]);
                            acc[i][3] = fma_pair(aa, w1.y, acc[i][3]);
                        }
                    }
                };
                if (next < K) fetch(a_row, lda, a_rows, next);
                products(0);
                if (next < K) {
                    keep(coming);
                    fetch(w_row, ldw, w_rows, next);
                }
                products(1);
                if (next < K) keep(coming + kOperandFloats);
                const int done = k0 + kStepK;
                if constexpr (GROUPED) {
                    if (done % kChunk == 0 || done >= k_end) {                     // a chunk ends: into the group's sum
                        const bool first = (done - 1) / kChunk * kChunk == k_begin;
#pragma unroll
                        for (int i = 0; i < 8; ++i)
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                if (first) {
                                    grp[i][j] = acc[i][j];
                                } else {
                                    const float2 g = halves(grp[i][j]), c = halves(acc[i][j]);
                                    asm("mov.b64 %0, {%1, %2};" : "=l"(grp[i][j]) : "f"(g.x + c.x), "f"(g.y + c.y));
                                }
                                acc[i][j] = 0;
                            }
                    }
                }
            }
            if constexpr (!GROUPED) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) grp[i][j] = acc[i][j];
            }
        }
        if (round > 0) __syncthreads();              // the sums of the round before have been read
        if (group < n_groups) {
            float* mine = sums + (size_t)slice * kTile * kTile;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float* row = mine + (size_t)((i < 4 ? 0 : 32) + ty * 4 + (i & 3)) * kTile + tx * 4;
                *reinterpret_cast<ulonglong2*>(row) = make_ulonglong2(grp[i][0], grp[i][1]);
                *reinterpret_cast<ulonglong2*>(row + 32) = make_ulonglong2(grp[i][2], grp[i][3]);
            }
        }
        __syncthreads();
        for (int s2 = 0; s2 < kSlices && round * kSlices + s2 < n_groups; ++s2) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 g = reinterpret_cast<const float4*>(sums + (size_t)s2 * kTile * kTile)[threadIdx.x + 256 * i];
                if (round == 0 && s2 == 0) {
                    tot[i] = g;
                } else {
                    tot[i].x += g.x;
                    tot[i].y += g.y;
                    tot[i].z += g.z;
                    tot[i].w += g.w;
                }
            }
        }
    }
    const lb_act_pair act_pair = lb_act_load(bias, N, act);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int piece = threadIdx.x + 256 * i, gm = m0 + piece / 16;
        if (gm >= M) continue;
        const float t[4] = {tot[i].x, tot[i].y, tot[i].z, tot[i].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + (piece % 16) * 4 + j;
            if (gn >= N) continue;
            float v = t[j];
            if (bias != nullptr) v += bias[gn];
            v = lb_activate(v, act, act_pair);
            if (residual != nullptr) v += residual[(size_t)gm * ldr + gn];
            out[(size_t)gm * ldo + gn] = lb_from_float<TO>(v);
        }
    }
}

template <typename TI, typename TO, bool VECTORS, bool GROUPED>
int launch_tiled(const void* A, int64_t lda, const void* W, int64_t ldw, const float* bias, const float* residual, int64_t ldr, void* out, int64_t ldo,
                 int M, int N, int K, int act, cudaStream_t s) {
    LB_CHECK_CUDA(cudaFuncSetAttribute(gemm_ffma_kernel<TI, TO, VECTORS, GROUPED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTiledSmem));
    const dim3 grid((N + kTile - 1) / kTile, (M + kTile - 1) / kTile);
    LB_CHECK_CUDA(lb_launch_overlapped(gemm_ffma_kernel<TI, TO, VECTORS, GROUPED>, grid, dim3(kSlices * kSliceThreads), kTiledSmem, s, (const TI*)A, lda,
                                       (const TI*)W, ldw, bias, residual, ldr, (TO*)out, ldo, M, N, K, act));
    LB_CHECK_LAUNCH();
    return LB_OK;
}

// ---- up to 16 tokens: the weights are read once, everything else is arranged around that -----------------

constexpr int kSkinnyFeatures = 8;       // features per block
constexpr int kSkinnyTokens = 16;        // the most tokens; the kernel is also built for 8 (half the products and buffers)
// Floats between the buffers of a warp's four slots: banks 8 apart.
__host__ __device__ constexpr int skinny_pitch(int tokens) { return tokens * kChunk + 8; }

__device__ __forceinline__ void cp_async16_zfill(void* dst, const void* src, bool valid) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

// 64 weights of one feature as floats: sixteen (float) or eight (bfloat16) 16-byte loads, all issued before use.
template <typename TI>
struct WeightChunk;
template <>
struct WeightChunk<float> {
    float4 v[16];
    __device__ __forceinline__ void load(const float* row, int k0, int K, bool live) {
#pragma unroll
        for (int i = 0; i < 16; ++i)
            v[i] = (live && k0 + 4 * i < K) ? __ldg(reinterpret_cast<const float4*>(row + k0 + 4 * i)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __device__ __forceinline__ float4 quad(int i) const { return v[i]; }
};
template <>
struct WeightChunk<__nv_bfloat16> {
    uint4 v[8];
    __device__ __forceinline__ void load(const __nv_bfloat16* row, int k0, int K, bool live) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
            v[i] = (live && k0 + 8 * i < K) ? __ldg(reinterpret_cast<const uint4*>(row + k0 + 8 * i)) : make_uint4(0, 0, 0, 0);
    }
    __device__ __forceinline__ float4 quad(int i) const {
        const uint4 u = v[i >> 1];
        const uint32_t lo = (i & 1) ? u.z : u.x, hi = (i & 1) ? u.w : u.y;
        return make_float4(__uint_as_float(lo << 16), __uint_as_float(lo & 0xffff0000u), __uint_as_float(hi << 16),
                           __uint_as_float(hi & 0xffff0000u));
    }
};

// K, lda and ldw are multiples of the 16-byte vector (4 floats, 8 bfloat16) and the bases 16-byte aligned.
// The block has as many warps as the reduction length has groups of chunks to give them (four groups a warp).
template <typename TI, typename TO, int TOKENS>
__global__ void __launch_bounds__(256)
gemm_ffma_skinny_kernel(const TI* __restrict__ A, int64_t lda, const TI* __restrict__ W, int64_t ldw,
                        const float* __restrict__ bias, const float* residual, int64_t ldr, TO* out, int64_t ldo, int M,
                        int N, int K, int act) {
    constexpr int VEC = 16 / (int)sizeof(TI);                   // elements per 16-byte piece
    constexpr int kPitch = skinny_pitch(TOKENS);
    extern __shared__ __align__(16) float skinny_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int fi = lane & 7, slot = lane >> 3;                   // feature within the block, chunk slot within the warp
    const int f = blockIdx.x * kSkinnyFeatures + fi;
    const int group = warp * 4 + slot;                           // this thread's group of chunks
    const int n_chunks = (K + kChunk - 1) / kChunk, G = chunks_per_group(K);
    const int c_begin = min(n_chunks, group * G), c_end = min(n_chunks, c_begin + G);
    // The warp's buffers: [slot][token][64] floats of activations (as stored: float or bfloat16 widened on use).
    float* my_buf = skinny_smem + (size_t)warp * 4 * kPitch;
    const TI* w_row = W + (size_t)min(f, N - 1) * ldw;
    float grp[TOKENS];
#pragma unroll
    for (int r = 0; r < TOKENS; ++r) grp[r] = 0.0f;
    for (int ci = 0; ci < G; ++ci) {                             // the same trip count for the whole warp
        const int c = c_begin + ci;
        const bool live = c < c_end;
        const int k0 = c * kChunk;
        WeightChunk<TI> w;
        w.load(w_row, k0, K, live && f < N);
        if (ci == 0) {
            // The first chunk's weights are under way; the activations come from the kernel before this one.
            lb_wait_for_predecessor();
            lb_dependents_may_launch();
        }
        // The warp's four slots bring their chunks of the tokens' activations: slot s2's chunk, token r, piece q.
        __syncwarp();
        for (int idx = lane; idx < 4 * TOKENS * (kChunk / VEC); idx += 32) {
            const int s2 = idx / (TOKENS * (kChunk / VEC)), rem = idx - s2 * (TOKENS * (kChunk / VEC));
            const int r = rem / (kChunk / VEC), q = rem - r * (kChunk / VEC);
            const int c2 = min(n_chunks, (warp * 4 + s2) * G) + ci;
            const int kk = c2 * kChunk + q * VEC;
            const bool valid = c2 < min(n_chunks, min(n_chunks, (warp * 4 + s2) * G) + G) && r < M && kk < K;
            TI* dst = reinterpret_cast<TI*>(my_buf + (size_t)s2 * kPitch) + r * kChunk + q * VEC;
            cp_async16_zfill(dst, A + (size_t)(valid ? r : 0) * lda + (valid ? kk : 0), valid);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        const TI* a_s = reinterpret_cast<const TI*>(my_buf + (size_t)slot * kPitch);
        float acc[TOKENS];
#pragma unroll
        for (int r = 0; r < TOKENS; ++r) acc[r] = 0.0f;
#pragma unroll
        for (int i = 0; i < kChunk / 4; ++i) {
            const float4 wq = w.quad(i);
#pragma unroll
            for (int r = 0; r < TOKENS; ++r) {
                float4 aq;
                if constexpr (sizeof(TI) == 4) {
                    aq = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(a_s) + r * kChunk + 4 * i);
                } else {
                    const uint2 u = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(a_s) + r * kChunk + 4 * i);
                    aq = make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16),
                                     __uint_as_float(u.y & 0xffff0000u));
                }
                acc[r] = fmaf(aq.x, wq.x, acc[r]);
                acc[r] = fmaf(aq.y, wq.y, acc[r]);
                acc[r] = fmaf(aq.z, wq.z, acc[r]);
                acc[r] = fmaf(aq.w, wq.w, acc[r]);
            }
        }
        if (live) {
#pragma unroll
            for (int r = 0; r < TOKENS; ++r) grp[r] = ci == 0 ? acc[r] : grp[r] + acc[r];
        }
    }
    // The group sums of the block meet in shared memory (over the activation buffers) and are added in ascending order.
    __syncthreads();
    float* red = skinny_smem;                                    // [group][token][feature]
#pragma unroll
    for (int r = 0; r < TOKENS; ++r) red[(group * TOKENS + r) * kSkinnyFeatures + fi] = grp[r];
    __syncthreads();
    const lb_act_pair act_pair = lb_act_load(bias, N, act);
    for (int idx = threadIdx.x; idx < TOKENS * kSkinnyFeatures; idx += blockDim.x) {
        const int r = idx / kSkinnyFeatures, ff = idx % kSkinnyFeatures;
        const int gn = blockIdx.x * kSkinnyFeatures + ff;
        if (r < M && gn < N) {
            const int n_groups = (n_chunks + G - 1) / G;
            float v = red[(0 * TOKENS + r) * kSkinnyFeatures + ff];
            for (int g2 = 1; g2 < n_groups; ++g2) v += red[(g2 * TOKENS + r) * kSkinnyFeatures + ff];
            if (bias != nullptr) v += bias[gn];
            v = lb_activate(v, act, act_pair);
            if (residual != nullptr) v += residual[(size_t)r * ldr + gn];
            out[(size_t)r * ldo + gn] = lb_from_float<TO>(v);
        }
    }
}

// The same for 9 to 16 tokens in float32, with the weights brought into shared memory by whole rows of a chunk: sixteen lanes copy a chunk's 256 bytes, where the
// kernel above has every lane read 16 bytes of a chunk of its own (32 lines an instruction) and hold all sixteen pieces of it beside its sixteen sums (214
// registers: nine warps an SM).  A thread has FPT features, eight apart, so that a piece of the activations that it reads serves FPT times four products.
// Sums as above, in their order.  Which products take it: lb_gemm_ffma_row_features.  (Without the loop over chunks, which most of them go
// through once, the compiler keeps 72 registers instead of 214, and the kernel is up to a tenth slower.)  GPT-2 small, a decode step of 12 requests: 910 -> 791 us; of 16: 946 -> 858 us.
constexpr int kRowPitch = kChunk + 4;          // floats between the chunks of neighbouring features: eight lanes' pieces fall into 32 banks

constexpr size_t skinny_rows_smem(int warps, int fpt) {
    return ((size_t)warps * 4 * fpt * 8 * kRowPitch + (size_t)warps * 4 * skinny_pitch(kSkinnyTokens)) * sizeof(float);
}

template <int FPT>
__global__ void __launch_bounds__(256)
gemm_ffma_skinny_rows_kernel(const float* __restrict__ A, int64_t lda, const float* __restrict__ W, int64_t ldw, const float* __restrict__ bias,
                             const float* residual, int64_t ldr, float* out, int64_t ldo, int M, int N, int K, int act) {
    constexpr int TOKENS = kSkinnyTokens, kPitch = skinny_pitch(TOKENS), F = 8 * FPT;
    extern __shared__ __align__(16) float skinny_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_slots = (int)(blockDim.x >> 5) * 4;
    const int fi = lane & 7, slot = lane >> 3, group = warp * 4 + slot;
    const int f0 = blockIdx.x * F;
    const int n_chunks = (K + kChunk - 1) / kChunk, G = chunks_per_group(K);
    float* w_s = skinny_smem;                                            // [group][feature][64 + 4]
    float* my_buf = skinny_smem + (size_t)n_slots * F * kRowPitch + (size_t)warp * 4 * kPitch;      // the warp's [slot][token][64] activations
    auto weights = [&](int ci) {                                         // chunk ci of every group
        for (int idx = threadIdx.x; idx < n_slots * F * 16; idx += blockDim.x) {
            const int q = idx & 15, row = idx >> 4, f = row % F, g = row / F;
            const int c = g * G + ci, k = c * kChunk + 4 * q;
            const bool valid = c < n_chunks && k < K && f0 + f < N;
            cp_async16_zfill(w_s + (size_t)row * kRowPitch + 4 * q, valid ? W + (size_t)(f0 + f) * ldw + k : W, valid);
        }
    };
    auto activations = [&](int ci) {                                     // the chunks of the warp's four groups
        for (int idx = lane; idx < 4 * TOKENS * 16; idx += 32) {
            const int q = idx & 15, r = (idx >> 4) % TOKENS, s2 = (idx >> 4) / TOKENS;
            const int c = (warp * 4 + s2) * G + ci, k = c * kChunk + 4 * q;
            const bool valid = c < n_chunks && k < K && r < M;
            cp_async16_zfill(my_buf + (size_t)s2 * kPitch + r * kChunk + 4 * q, valid ? A + (size_t)r * lda + k : A, valid);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    weights(0);
    lb_wait_for_predecessor();               // the weights are under way; the activations come from the kernel before this one
    lb_dependents_may_launch();
    activations(0);
    float grp[FPT][TOKENS];
#pragma unroll
    for (int p = 0; p < FPT; ++p)
#pragma unroll
        for (int r = 0; r < TOKENS; ++r) grp[p][r] = 0.0f;
    for (int ci = 0; ci < G; ++ci) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        const float* a_s = my_buf + (size_t)slot * kPitch;
        const float* w_row = w_s + (size_t)(group * F + fi) * kRowPitch;
        float acc[FPT][TOKENS];
#pragma unroll
        for (int p = 0; p < FPT; ++p)
#pragma unroll
            for (int r = 0; r < TOKENS; ++r) acc[p][r] = 0.0f;
#pragma unroll 4
        for (int i = 0; i < kChunk / 4; ++i) {
            float4 w[FPT];
#pragma unroll
            for (int p = 0; p < FPT; ++p) w[p] = *reinterpret_cast<const float4*>(w_row + (size_t)p * 8 * kRowPitch + 4 * i);
#pragma unroll
            for (int r = 0; r < TOKENS; ++r) {
                const float4 a = *reinterpret_cast<const float4*>(a_s + r * kChunk + 4 * i);
#pragma unroll
                for (int p = 0; p < FPT; ++p) {
                    acc[p][r] = fmaf(a.x, w[p].x, acc[p][r]);
                    acc[p][r] = fmaf(a.y, w[p].y, acc[p][r]);
                    acc[p][r] = fmaf(a.z, w[p].z, acc[p][r]);
                    acc[p][r] = fmaf(a.w, w[p].w, acc[p][r]);
                }
            }
        }
        if (group * G + ci < n_chunks) {
#pragma unroll
            for (int p = 0; p < FPT; ++p)
#pragma unroll
                for (int r = 0; r < TOKENS; ++r) grp[p][r] = ci == 0 ? acc[p][r] : grp[p][r] + acc[p][r];
        }
        __syncthreads();                                                 // the buffers are free: for the next chunks, or for the group sums
        if (ci + 1 < G) {
            weights(ci + 1);
            activations(ci + 1);
        }
    }
    float* red = skinny_smem;                                            // [group][token][feature]
#pragma unroll
    for (int p = 0; p < FPT; ++p)
#pragma unroll
        for (int r = 0; r < TOKENS; ++r) red[(group * TOKENS + r) * F + 8 * p + fi] = grp[p][r];
    __syncthreads();
    const lb_act_pair act_pair = lb_act_load(bias, N, act);
    const int n_groups = (n_chunks + G - 1) / G;
    for (int idx = threadIdx.x; idx < M * F; idx += blockDim.x) {
        const int r = idx / F, ff = idx % F, gn = f0 + ff;
        if (gn >= N) continue;
        float v = red[r * F + ff];
        for (int g2 = 1; g2 < n_groups; ++g2) v += red[(g2 * TOKENS + r) * F + ff];
        if (bias != nullptr) v += bias[gn];
        v = lb_activate(v, act, act_pair);
        if (residual != nullptr) v += residual[(size_t)r * ldr + gn];
        out[(size_t)r * ldo + gn] = v;
    }
}

template <int FPT>
int launch_skinny_rows(const void* A, int64_t lda, const void* W, int64_t ldw, const float* bias, const float* residual, int64_t ldr, void* out, int64_t ldo,
                       int M, int N, int K, int act, int warps, cudaStream_t s) {
    const size_t smem = skinny_rows_smem(warps, FPT);
    LB_CHECK_CUDA(cudaFuncSetAttribute(gemm_ffma_skinny_rows_kernel<FPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    LB_CHECK_CUDA(lb_launch_overlapped(gemm_ffma_skinny_rows_kernel<FPT>, dim3((N + 8 * FPT - 1) / (8 * FPT)), dim3(warps * 32), smem, s, (const float*)A,
                                       lda, (const float*)W, ldw, bias, residual, ldr, (float*)out, ldo, M, N, K, act));
    LB_CHECK_LAUNCH();
    return LB_OK;
}

// ---- up to 8 tokens in float32, whole rows of weights by bulk copies --------------------------------------------
//
// Both kernels above bring their weights and, again for every eight or sixteen features, the activations: as many bytes from L2 as the weights are, which
// is what the logits' product was bound by (76 us for 50257 x 768 at eight tokens, 24 for its bytes), and lane by lane, 32 lines an instruction.  Here the
// activations of all tokens stay in a block's shared memory, and the block walks groups of eight features whose rows come whole, by one bulk copy each, a ring of
// them ahead and the first ones before the wait for the kernel before.  A thread has a feature and a group of chunks, as above, and the sums are made in the same order:
// the same bits.  A long reduction (K = 3072) has a block's eight rows at once instead of a chunk after the other.
// Bound by shared memory now: a warp reads nine pieces for 32 products, and few warps fit beside the rows.  With 9 to 16 tokens that was slower than the kernel
// above (50257 x 768 107 us against 89).
// Measured (us, before / here): 8 tokens 50257 x 768 68 / 48, 4800 x 1600 22.2 / 14.0, 1600 x 1600 8.5 / 7.1, and within a step of GPT-2 small 2304 x 768 6.2 / 4.9,
// 768 x 3072 11.4 / 8.3, but 768 x 768 3.8 / 4.8 and 3072 x 768 6.6 / 6.9: see stream_takes.
constexpr int kStreamFeatures = 8, kStreamTokens = 8;
constexpr int kStreamChunkPitch = kChunk + 8;       // floats between the chunks of a token: the four chunks a warp reads fall into banks 8 apart
__host__ __device__ constexpr int stream_row_pitch(int K) { return (K + 31) / 32 * 32 + 4; }      // eight features' pieces fall into 32 banks

struct StreamShape {
    int warps, stages;
    size_t smem;
};
// Stages that fit (up to `most`; 0: not even one), two blocks an SM where that leaves each two stages.
inline StreamShape stream_shape(int K, int most) {
    const int n_chunks = (K + kChunk - 1) / kChunk, G = chunks_per_group(K), n_groups = (n_chunks + G - 1) / G;
    constexpr int kFinishing = kStreamTokens * kStreamFeatures / 32;          // a thread an element at the end
    StreamShape s{(n_groups + 3) / 4 > kFinishing ? (n_groups + 3) / 4 : kFinishing, 0, 0};
    const size_t fixed = ((size_t)kStreamTokens * n_chunks * kStreamChunkPitch + (size_t)2 * s.warps * 4 * kStreamTokens * kStreamFeatures) * sizeof(float) + 80;
    const size_t stage = (size_t)kStreamFeatures * stream_row_pitch(K) * sizeof(float), half = 113 * 1024, whole = 227 * 1024;
    if (fixed + stage > whole) return s;
    const int in_half = fixed < half ? (int)((half - fixed) / stage) : 0, in_whole = (int)((whole - fixed) / stage);
    s.stages = in_half >= 2 || in_half >= most ? in_half : in_whole;
    if (s.stages > most) s.stages = most;
    if (s.stages > 8) s.stages = 8;
    s.smem = fixed + s.stages * stage;
    return s;
}

int g_withhold_next = 0;      // the next launch's blocks leave their first stage's barrier one arrival short (tests)

// Whether a product goes that way: a block has at least two stages or no second group of features.  Short reductions (one chunk a group, which the kernel of
// eight features a block brings in one go as well) stay with that one where they have no more groups than SMs, and where the last round of blocks would be less
// than two fifths full.
inline bool stream_takes(int N, int K, int n_sm, StreamShape* shape, int* grid) {
    const int groups = (N + kStreamFeatures - 1) / kStreamFeatures;
    *shape = stream_shape(K, (groups + n_sm - 1) / n_sm);
    if (shape->stages < 1 || (shape->stages < 2 && groups > n_sm)) return false;
    const int slots = n_sm * (shape->smem <= 113 * 1024 ? 2 : 1), last = groups % slots;
    *grid = groups < slots ? groups : slots;
    if (K <= 1024 && (groups <= n_sm || (groups > slots && groups < 4 * slots && last != 0 && 5 * last < 2 * slots))) return false;
    return true;
}

__device__ __forceinline__ uint32_t ffma_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__global__ void __launch_bounds__(256)
gemm_ffma_stream_kernel(const float* __restrict__ A, int64_t lda, const float* __restrict__ W, int64_t ldw, const float* __restrict__ bias,
                        const float* residual, int64_t ldr, float* out, int64_t ldo, int M, int N, int K, int act, int stages, int withhold, int* status) {
    constexpr int TOKENS = kStreamTokens;
    extern __shared__ __align__(16) float stream_smem[];
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31, n_warps = blockDim.x >> 5;
    const int fi = lane & 7, group = warp * 4 + (lane >> 3);
    const int n_chunks = (K + kChunk - 1) / kChunk, G = chunks_per_group(K), n_groups = (n_chunks + G - 1) / G;
    const int w_pitch = stream_row_pitch(K), a_pitch = n_chunks * kStreamChunkPitch;
    float* w_s = stream_smem;                                            // [stage][8][w_pitch]
    float* a_s = w_s + (size_t)stages * kStreamFeatures * w_pitch;       // [token][chunk][64 + 8]
    float* red = a_s + (size_t)TOKENS * a_pitch;                         // [2][group][token][8]
    const int red_floats = n_warps * 4 * TOKENS * kStreamFeatures;
    uint64_t* full = reinterpret_cast<uint64_t*>(red + 2 * red_floats);
    volatile int* gave_up = reinterpret_cast<int*>(full + 8);             // a wait ran out: the later ones end at once
    const int n_feature_groups = (N + kStreamFeatures - 1) / kStreamFeatures, step = gridDim.x;
    if (threadIdx.x == 0) {
        *gave_up = 0;
        for (int i = 0; i < stages; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(ffma_smem(full + i)), "r"(i == 0 && withhold != 0 ? 2 : 1));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // Eight rows of weights -> a stage (by the first warp).
    auto rows = [&](int fg, int stage) {
        const int here = min(kStreamFeatures, N - fg * kStreamFeatures);
        const uint32_t bar = ffma_smem(full + stage), bytes = (uint32_t)K * 4u;
        if (lb_tc::elect_one()) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)here * bytes) : "memory");
        __syncwarp();
        for (int i = 0; i < here; ++i)
            if (lb_tc::elect_one())
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             ::"r"(ffma_smem(w_s + ((size_t)stage * kStreamFeatures + i) * w_pitch)), "l"(W + (size_t)(fg * kStreamFeatures + i) * ldw), "r"(bytes), "r"(bar)
                             : "memory");
        __syncwarp();
    };
    if (warp == 0)
        for (int s = 0; s < stages; ++s)
            if ((int)blockIdx.x + s * step < n_feature_groups) rows((int)blockIdx.x + s * step, s);
    const lb_act_pair act_pair = lb_act_load(bias, N, act);
    lb_wait_for_predecessor();               // the weights are under way; the activations come from the kernel before this one
    lb_dependents_may_launch();
    for (int idx = threadIdx.x; idx < M * n_chunks * 16; idx += blockDim.x) {
        const int q = idx & 15, c = (idx >> 4) % n_chunks, r = (idx >> 4) / n_chunks, k = c * kChunk + 4 * q;
        cp_async16_zfill(a_s + (size_t)r * a_pitch + c * kStreamChunkPitch + 4 * q, k < K ? A + (size_t)r * lda + k : A, k < K);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const int c_begin = min(n_chunks, group * G), c_end = min(n_chunks, c_begin + G);
    int it = 0;
    for (int fg = blockIdx.x; fg < n_feature_groups; fg += step, ++it) {
        const int stage = it % stages;
        // The element that this thread finishes: its bias and residual travel under the products.
        const int er = threadIdx.x / kStreamFeatures, ef = fg * kStreamFeatures + threadIdx.x % kStreamFeatures;
        const bool finishes = threadIdx.x < TOKENS * kStreamFeatures && er < M && ef < N;
        const float early_b = finishes && bias != nullptr ? __ldg(bias + ef) : 0.0f, early_r = finishes && residual != nullptr ? __ldcg(residual + (size_t)er * ldr + ef) : 0.0f;
        {
            // Bounded, once for the block: a copy that never lands leaves a code in the status word and wrong results instead of a hang, and the groups
            // after it are not waited for.
            if (!lb_tc::mbar_wait(full + stage, (uint32_t)(it / stages) & 1u, gave_up)) {
                atomicCAS(status, 0, (0x9 << 12) | 1);
                *gave_up = 1;
            }
        }
        const float* w_row = w_s + ((size_t)stage * kStreamFeatures + fi) * w_pitch;
        float grp[TOKENS];
#pragma unroll
        for (int r = 0; r < TOKENS; ++r) grp[r] = 0.0f;
        for (int c = c_begin; c < c_end; ++c) {
            const float* w = w_row + c * kChunk;
            const float* a = a_s + (size_t)c * kStreamChunkPitch;
            const int quads = min(kChunk, K - c * kChunk) / 4;
            float acc[TOKENS];
#pragma unroll
            for (int r = 0; r < TOKENS; ++r) acc[r] = 0.0f;
#pragma unroll 4
            for (int i = 0; i < quads; ++i) {
                const float4 wq = *reinterpret_cast<const float4*>(w + 4 * i);
#pragma unroll
                for (int r = 0; r < TOKENS; ++r) {
                    const float4 aq = *reinterpret_cast<const float4*>(a + (size_t)r * a_pitch + 4 * i);
                    acc[r] = fmaf(aq.x, wq.x, acc[r]);
                    acc[r] = fmaf(aq.y, wq.y, acc[r]);
                    acc[r] = fmaf(aq.z, wq.z, acc[r]);
                    acc[r] = fmaf(aq.w, wq.w, acc[r]);
                }
            }
#pragma unroll
            for (int r = 0; r < TOKENS; ++r) grp[r] = c == c_begin ? acc[r] : grp[r] + acc[r];
        }
        float* here = red + (it & 1) * red_floats;
#pragma unroll
        for (int r = 0; r < TOKENS; ++r) here[(group * TOKENS + r) * kStreamFeatures + fi] = grp[r];
        __syncthreads();                                                 // the group sums are there, and the stage has been read
        if (warp == 0 && fg + stages * step < n_feature_groups && __shfl_sync(0xffffffffu, *gave_up, 0) == 0) rows(fg + stages * step, stage);
        if (finishes) {
            float v = here[threadIdx.x];
            for (int g2 = 1; g2 < n_groups; ++g2) v += here[g2 * TOKENS * kStreamFeatures + threadIdx.x];
            if (bias != nullptr) v += early_b;
            v = lb_activate(v, act, act_pair);
            if (residual != nullptr) v += early_r;
            out[(size_t)er * ldo + ef] = v;
        }
    }
    // Leave no copy in flight: what was asked for has its time once more.  (Before the limit nothing is: every stage asked for was waited for.)
    __syncthreads();
    if (warp == 0 && *gave_up != 0) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {}              // a millisecond, hundreds of times what a copy takes
    }
}

int launch_stream(const void* A, int64_t lda, const void* W, int64_t ldw, const float* bias, const float* residual, int64_t ldr, void* out, int64_t ldo,
                  int M, int N, int K, int act, const StreamShape& shape, int grid, cudaStream_t s) {
    int* status = nullptr;
    const int rc = lb_tc_status_word(&status);
    if (rc != LB_OK) return rc;
    LB_CHECK_CUDA(cudaFuncSetAttribute(gemm_ffma_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    LB_CHECK_CUDA(lb_launch_overlapped(gemm_ffma_stream_kernel, dim3(grid), dim3(shape.warps * 32), shape.smem, s, (const float*)A, lda,
                                       (const float*)W, ldw, bias, residual, ldr, (float*)out, ldo, M, N, K, act, shape.stages, g_withhold_next, status));
    g_withhold_next = 0;
    LB_CHECK_LAUNCH();
    return LB_OK;
}

template <typename TI, typename TO>
int launch(const void* A, int64_t lda, const void* W, int64_t ldw, const float* bias, const float* residual,
           int64_t ldr, void* out, int64_t ldo, int M, int N, int K, int act, cudaStream_t s) {
    constexpr int VEC = 16 / (int)sizeof(TI);
    const bool vectors = K % VEC == 0 && lda % VEC == 0 && ldw % VEC == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0;
    // The tiled kernel loads four elements at a time where no such piece crosses a row's end and all are aligned.
    const uintptr_t quad_mask = 4 * sizeof(TI) - 1;
    const bool quads = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & quad_mask) == 0;
    if (M <= kSkinnyTokens && vectors) {
        // Few tokens: bound by reading the weights once (see the head of the file).  A warp serves four groups of
        // chunks, so a short reduction length makes small blocks, of which several share an SM.
        const int n_chunks = (K + kChunk - 1) / kChunk, per_group = chunks_per_group(K);
        const int n_groups = (n_chunks + per_group - 1) / per_group, warps = (n_groups + 3) / 4;
        if constexpr (sizeof(TI) == 4 && sizeof(TO) == 4) {
            StreamShape shape;
            int grid = 0;
            static const int n_sm = [] {
                int dev = 0, n = 0;
                return cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess ? n : 148;
            }();
            if (M <= kStreamTokens && stream_takes(N, K, n_sm, &shape, &grid)) return launch_stream(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, shape, grid, s);
        }
        if constexpr (sizeof(TI) == 4) {
            if (M > 8) {
                const int features = lb_gemm_ffma_row_features(M, N, K);
                if (features == 16) return launch_skinny_rows<2>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, warps, s);
                if (features == 8) return launch_skinny_rows<1>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, warps, s);
            }
        }
        const dim3 grid((N + kSkinnyFeatures - 1) / kSkinnyFeatures);
        if (M <= 8) {
            const size_t smem = (size_t)warps * 4 * skinny_pitch(8) * sizeof(float);
            static bool configured = false;
            if (!configured) {
                LB_CHECK_CUDA(cudaFuncSetAttribute(gemm_ffma_skinny_kernel<TI, TO, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)(8 * 4 * skinny_pitch(8) * sizeof(float))));
                configured = true;
            }
            LB_CHECK_CUDA(lb_launch_overlapped(gemm_ffma_skinny_kernel<TI, TO, 8>, dim3(grid), dim3(warps * 32), smem, s, (const TI*)A, lda, (const TI*)W, ldw, bias, residual, ldr,
                                                                             (TO*)out, ldo, M, N, K, act));
        } else {
            const size_t smem = (size_t)warps * 4 * skinny_pitch(16) * sizeof(float);
            static bool configured = false;
            if (!configured) {
                LB_CHECK_CUDA(cudaFuncSetAttribute(gemm_ffma_skinny_kernel<TI, TO, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)(8 * 4 * skinny_pitch(16) * sizeof(float))));
                configured = true;
            }
            LB_CHECK_CUDA(lb_launch_overlapped(gemm_ffma_skinny_kernel<TI, TO, 16>, dim3(grid), dim3(warps * 32), smem, s, (const TI*)A, lda, (const TI*)W, ldw, bias, residual, ldr,
                                                                              (TO*)out, ldo, M, N, K, act));
        }
    } else {
        const bool grouped = chunks_per_group(K) > 1;
        if (quads) return grouped ? launch_tiled<TI, TO, true, true>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, s)
                                  : launch_tiled<TI, TO, true, false>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, s);
        return grouped ? launch_tiled<TI, TO, false, true>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, s)
                       : launch_tiled<TI, TO, false, false>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, s);
    }
    LB_CHECK_LAUNCH();
    return LB_OK;
}

}  // namespace

// The features a block has in the kernel whose weights come by whole rows, for float32 products of whole 16-byte pieces: 16, 8, or 0 where the kernel that
// brings them lane by lane is the faster one.  Measured with cold weights, lane by lane / by rows in us (12 tokens): 9.8 / 8.4 for 3072 x 768, 110 / 91 for
// 50257 x 768, 15.9 / 12.5 for 4096 x 1024; 4.7 / 5.5 for 768 x 64 and 22.3 / 24.7 for 256 x 6400 (bound by latency: the rows' form has a barrier more), 19.0 /
// 25.6 for 2304 x 3072 (a block's chunks fill an SM by themselves, as do those of K = 1280).  So: two to four warps (K of 257 to 1024; one warp with 193 to
// 256 and two rounds of blocks), enough blocks to fill the GPU, and with four warps, whose blocks of sixteen features have an SM each, rounds over the SMs
// that are at least two thirds full (3072 x 1024: 11.5 / 12.0).  Fewer features than a wave of such blocks go by rows, eight a block, from 768 on, with 11 to 16
// chunks, or 33 to 48 below 1536 features: alone such a product is level (768 x 3072 13.4 / 13.0), within a step it is not (GPT-2 small, 12
// requests: 878 / 803 us with its down products by rows; medium, 9 requests: 1677 / 1647 with its output products).  Up to eight tokens it was behind
// throughout (a step of 8 requests 615 against 632 us); most of those products have bulk copies now (stream_takes).
extern "C" int lb_gemm_ffma_row_features(int M, int N, int K) {
    const int n_chunks = (K + kChunk - 1) / kChunk, warps = (n_chunks + 3) / 4;
    const int round = 16 * 148, rounds = (N + round - 1) / round;
    if (M <= 8 || M > kSkinnyTokens || n_chunks < 4) return 0;
    if (N < round) return (N >= 768 && n_chunks > 10 && n_chunks <= 16) || (N >= 768 && N < 1536 && n_chunks > 32 && n_chunks <= 48) ? 8 : 0;
    if (warps == 1) return N >= 2 * round ? 16 : 0;
    return warps < 4 || (warps == 4 && 3ll * N >= 2ll * rounds * round) ? 16 : 0;
}

// The stages of a block in the kernel whose weights come by whole rows and bulk copies, for float32 products of whole 16-byte pieces on n_sm SMs; 0 where another kernel
// takes the product.  *blocks: the launch's.
extern "C" int lb_gemm_ffma_stream_stages(int M, int N, int K, int n_sm, int* blocks) {
    StreamShape shape{};
    int grid = 0;
    if (M < 1 || M > kStreamTokens || N < 1 || K < 4 || K % 4 != 0 || n_sm < 1 || !stream_takes(N, K, n_sm, &shape, &grid)) return 0;
    if (blocks != nullptr) *blocks = grid;
    return shape.stages;
}

extern "C" int lb_gemm_ffma(int in_dtype, int out_dtype, const void* A, int64_t lda, const void* W, int64_t ldw,
                            const float* bias, const float* residual, int64_t ldr, void* out, int64_t ldo, int M, int N,
                            int K, int act, void* stream) {
    LB_CHECK_ARG(M >= 0 && N > 0 && K > 0, "gemm: bad sizes M=%d N=%d K=%d", M, N, K);
    LB_CHECK_ARG(lda >= K && ldw >= K && ldo >= N, "gemm: a row stride is shorter than the row");
    LB_CHECK_ARG((M + 63) / 64 <= 65535, "gemm: M=%d is too large for one launch", M);
    if (M == 0) return LB_OK;
    auto s = static_cast<cudaStream_t>(stream);
    if (in_dtype == LB_F32 && out_dtype == LB_F32)
        return launch<float, float>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, s);
    if (in_dtype == LB_BF16 && out_dtype == LB_BF16)
        return launch<__nv_bfloat16, __nv_bfloat16>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, s);
    if (in_dtype == LB_BF16 && out_dtype == LB_F32)
        return launch<__nv_bfloat16, float>(A, lda, W, ldw, bias, residual, ldr, out, ldo, M, N, K, act, s);
    return lb_fail(LB_ERR_INVALID_ARGUMENT, "gemm: unsupported dtypes in=%d out=%d", in_dtype, out_dtype);
}

extern "C" int lb_gemm_ffma_withhold_next(int on) {
    g_withhold_next = on != 0 ? 1 : 0;
    return LB_OK;
}
