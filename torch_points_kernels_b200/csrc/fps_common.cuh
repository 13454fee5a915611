// What the furthest-point-sampling kernels share: the tie rule of the reference and the
// distributed-shared-memory primitives of a thread-block cluster.
#pragma once

#include <math_constants.h>

#include "packed.cuh"
#include "tpk_common.cuh"

namespace tpk
{

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint32_t cluster_ctarank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_nctarank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t mapa_cluster(uint32_t addr, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync_all()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
                 "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

constexpr unsigned long long kWaitLimitNs = 1000000000ull;  // give up a wait after one second

// Remote stores that complete a transaction count of an mbarrier of the destination CTA.
__device__ __forceinline__ void st_async_v4(uint32_t addr, uint32_t mbar, int a, int b, int c, int d)
{
    asm volatile(
        "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
        "r"(a), "r"(b), "r"(c), "r"(d), "r"(mbar)
        : "memory");
}
__device__ __forceinline__ void st_async_b32(uint32_t addr, uint32_t mbar, int a)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr), "r"(a),
                 "r"(mbar)
                 : "memory");
}
// Bulk copy from this CTA's shared memory to another's; addresses and size are multiples of 16.
__device__ __forceinline__ void bulk_to_cta(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t mbar)
{
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "r"(src), "r"(bytes), "r"(mbar)
                 : "memory");
}
// Makes this thread's writes to shared memory visible to bulk copies issued behind the next barrier.
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_init(uint32_t mbar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t mbar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t mbar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(mbar), "r"(parity)
                 : "memory");
    return ok != 0;
}

__device__ __forceinline__ unsigned long long global_timer_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Waits for the phase with the given parity; false if it has not completed within
// kWaitLimitNs (the clock is read only every 256 unsuccessful polls).
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t mbar, uint32_t parity)
{
    unsigned long long t0 = 0;
    for (unsigned it = 1;; ++it)
    {
        if (mbar_try_wait(mbar, parity)) return true;
        if ((it & 255u) == 0u)
        {
            const unsigned long long now = global_timer_ns();
            if (t0 == 0)
                t0 = now;
            else if (now - t0 > kWaitLimitNs)
                return false;
        }
    }
}


// (false for NaN as well)
__device__ __forceinline__ bool all_finite(float x, float y, float z)
{
    return fabsf(x) <= CUDART_MAX_NORMAL_F && fabsf(y) <= CUDART_MAX_NORMAL_F && fabsf(z) <= CUDART_MAX_NORMAL_F;
}

__device__ __forceinline__ uint32_t bitrev_low(uint32_t v, int bits)
{
    return bits == 0 ? 0u : (__brev(v) >> (32 - bits));
}

// Tie rank of point k: the reference's strided scan + tree keeps, among equal maxima,
// the smallest bit-reversed (k mod bs), then the smallest (k div bs).
__device__ __forceinline__ uint32_t fps_rank(int k, int log2bs)
{
    const uint32_t u = static_cast<uint32_t>(k);
    return (bitrev_low(u & ((1u << log2bs) - 1u), log2bs) << 22) | (u >> log2bs);
}

// Interleaves the low 10 bits of v with two zero bits each (Morton order).
__device__ __forceinline__ uint32_t spread3(uint32_t v)
{
    v &= 0x3FFu;
    v = (v | (v << 16)) & 0x030000FFu;
    v = (v | (v << 8)) & 0x0300F00Fu;
    v = (v | (v << 4)) & 0x030C30C3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

// Position of a cell on the Hilbert curve of a 2^bits-per-axis grid (J. Skilling, "Programming the
// Hilbert curve", 2004: coordinates to transposed index, then the bits interleaved).
__device__ __forceinline__ uint32_t hilbert3(uint32_t x, uint32_t y, uint32_t z, int bits)
{
    const uint32_t m = 1u << (bits - 1);
    for (uint32_t q = m; q > 1u; q >>= 1)
    {
        const uint32_t p = q - 1u;
        if (x & q) x ^= p;
        uint32_t t = (x ^ y) & p;
        if (y & q)
            x ^= p;
        else
        {
            x ^= t;
            y ^= t;
        }
        t = (x ^ z) & p;
        if (z & q)
            x ^= p;
        else
        {
            x ^= t;
            z ^= t;
        }
    }
    y ^= x;
    z ^= y;
    uint32_t t = 0;
    for (uint32_t q = m; q > 1u; q >>= 1)
        if (z & q) t ^= q - 1u;
    return spread3(z ^ t) | (spread3(y ^ t) << 1) | (spread3(x ^ t) << 2);
}

}  // namespace tpk
