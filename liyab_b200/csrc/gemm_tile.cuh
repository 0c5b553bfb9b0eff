// What the two persistent tcgen05 products share: waits and copies on 32-bit shared-memory addresses, handshakes between the
// two blocks of a cluster, the activation in the epilogue and the cache as a second destination.
#pragma once

#include "common.cuh"
#include "tcgen05.cuh"

namespace lb_tile {

using namespace lb_tc;

// The loops of the two issuing warps (one elected lane of each) run once per k-block while the tensor pipe waits for them: they work on
// 32-bit shared-memory addresses and a running stage index, with no division and no 64-bit pointer arithmetic.
__device__ __forceinline__ bool try_wait_u32(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}

__device__ __forceinline__ bool wait_u32(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    if (try_wait_u32(bar, parity)) return true;
#pragma unroll 1
    for (int i = 0; i < 256; ++i)
        if (try_wait_u32(bar, parity)) return true;
    const long long t0 = clock64();
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 64; ++i)
            if (try_wait_u32(bar, parity)) return true;
        if (abort_flag != nullptr && *abort_flag != 0) return false;
        if (clock64() - t0 > kWaitLimitCycles) return false;
    }
}

// Handshakes between the two blocks of a pair (a cluster): the address of a barrier or of a piece of the staging
// buffer in the other block, an arrival there that publishes this thread's (and, after a warp barrier, its warp's)
// writes to the cluster, a wait that sees what the other block published, and a float32 addition into the other
// block's shared memory.
__device__ __forceinline__ uint32_t peer_address(uint32_t local, uint32_t rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
    return remote;
}
__device__ __forceinline__ void arrive_at_peer(uint32_t remote_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote_bar) : "memory");
}
__device__ __forceinline__ bool try_wait_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool wait_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
#pragma unroll 1
    for (int i = 0; i < 256; ++i)
        if (try_wait_cluster(bar, parity)) return true;
    const long long t0 = clock64();
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 64; ++i)
            if (try_wait_cluster(bar, parity)) return true;
        if (abort_flag != nullptr && *abort_flag != 0) return false;
        if (clock64() - t0 > kWaitLimitCycles) return false;
    }
}
__device__ __forceinline__ void store_at_peer(uint32_t remote, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(remote), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

__device__ __forceinline__ void expect_tx_u32(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void tma_load_u32(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1)
        : "memory");
}

__device__ __forceinline__ void commit_u32(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// tcgen05.mma with both shared-memory descriptors given as (low word, common high word).
__device__ __forceinline__ void umma_lo(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc,
                                        uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %3};\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}"
        ::"r"(tmem_d), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ float4 lds4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ void sts4(uint32_t addr, float4 v) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void sts4(uint32_t addr, uint4 v) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// The activation inside the epilogue.  Results that are rounded to bfloat16 take x/2 (1 + tanh u) as x / (1 + exp(-2u)) with
// the fast exponential and division (relative error about 1e-6, far below bfloat16's rounding), seven
// instructions instead of dozens; float32 results take the library functions.
template <int ACT, bool FAST>
__device__ __forceinline__ float activate(float x, const lb_act_pair& p) {
    if constexpr (ACT == LB_ACT_GELU_TANH) {
        if constexpr (FAST) {
            // x / (1 + exp(-2u)), 2u = x (1.5957... + 0.0713... x^2).
            return __fdividef(x, 1.0f + __expf(x * fmaf(-0.07135481282553524f * x, x, -1.5957691216057308f)));
        } else {
            return lb_gelu_tanh(x);
        }
    } else if constexpr (ACT == LB_ACT_GELU_ERF) {
        return lb_gelu_erf(x);
    } else if constexpr (ACT == LB_ACT_XIELU) {
        if constexpr (FAST) {
            // Without a branch: the positive part feeds the square, the negative part the exponential (which then never overflows).
            const float pos = fmaxf(x, 0.0f), neg = fminf(x, 0.0f);
            return fmaf(p.a * pos, pos, fmaf(p.b, __expf(neg) - 1.0f - neg, 0.5f * x));
        }
        else return lb_xielu(x, p.a, p.b);
    } else if constexpr (ACT == LB_ACT_RELU2) {
        const float pos = fmaxf(x, 0.0f);
        return pos * pos;
    } else {
        return x;
    }
}

// Where the features from q_dim on go instead of `out` when the product is a fused query/key/value projection:
// the pages of the cache ([page][K|V][kv_head][slot][head_dim]), row (token) i at slot_mapping[i] (negative: nowhere).
// A 64-feature strip lies inside one head (head_dim and q_dim are multiples of 64): 128 contiguous bytes per token.
struct KvTarget {
    __nv_bfloat16* cache;
    const int32_t* slot_mapping;
    int q_dim, n_kv_head, head_dim, page_shift;
};

}  // namespace lb_tile
