// Thin wrappers around the PTX that the tensor-core kernels share: mbarriers with bounded waits, tensor memory, tcgen05.
#pragma once
#include <cstdint>

namespace dg {

constexpr int kWaitLimit = 1 << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int limit = kWaitLimit)      // bounded
{
    for (int i = 0; i < limit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}
// 16 consecutive accumulator columns of this warp's 32 tensor-memory lanes (no wait: pair with tcgen05.wait::ld).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r)
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void umma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// One lane of a converged warp.  A warp that walks through its work together and lets this lane alone issue keeps the addresses of MMAs and
// barriers in uniform registers; with a single lane in the whole loop they had to be moved there for every MMA, 60 to 100 ns each.
__device__ __forceinline__ bool elect_one()
{
    uint32_t one;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(one));
    return one != 0;
}
// ---- CTA pairs: two CTAs of a cluster, on the two SMs of a TPC, that the tensor cores treat as one (cta_group::2) ------------------
// The address of the even CTA's barrier in the cluster's shared memory, given this CTA's own.
__device__ __forceinline__ uint32_t in_leader(uint32_t bar)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(bar), "r"(0));
    return r;
}
// Without a release at cluster scope, which costs some 1,900 clocks: what it reports is what the tensor cores, not another CTA's threads,
// touch next - operands behind fence.proxy.async, or an accumulator whose tcgen05.ld has been waited for.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar)
{
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void umma_commit_pair(uint32_t bar)      // arrives at the barrier of that offset in both CTAs
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void cluster_sync()
{
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// What a role waits for before it leaves the CTA, whether its loop came to its end or gave up: a copy that lands, or an MMA that
// reads, after the CTA is gone would do so in the shared and tensor memory of the next one.
// The loads of stages 0 .. issued - 1 of a ring (one full barrier a stage): the last round of every stage.
__device__ __forceinline__ void await_loads(uint32_t full0, int issued, int stages)
{
    for (int t = issued > stages ? issued - stages : 0; t < issued; ++t) mbar_wait(full0 + 8 * (t % stages), (t / stages) & 1);
}
// All MMAs this thread has issued; `done` is a barrier of its own, with a count of 1.
__device__ __forceinline__ void await_mmas(uint32_t done)
{
    umma_commit(done);
    mbar_wait(done, 0);
}
__device__ __forceinline__ void await_mmas_pair(uint32_t done)      // by the issuing CTA; the other one leaves after it, behind a cluster barrier
{
    umma_commit_pair(done);
    mbar_wait(done, 0);
}

}  // namespace dg
