// sm_100a primitives used by the tensor-core kernels: mbarriers with bounded waits, bulk copies
// (into the issuing CTA alone), TMEM allocation, tcgen05.mma / commit / ld, shared-memory matrix descriptors.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace acb {
namespace tc {

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t globaltimer_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// try_wait with a suspend-time hint: the thread sleeps in hardware until the phase completes or
// the hint (ns) expires, instead of spinning on the issue slots the other warps need.
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity, uint32_t hint_ns = 1000000u)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(hint_ns)
        : "memory");
    return ok != 0;
}

// Wait for the phase with `parity` to complete.  Gives up after `limit_ns` or when another thread
// of the CTA has raised `*abort`; returns false then (the caller records the timeout).  The hardware
// suspend of one try_wait is capped at the limit (and at 1 ms), so a short limit is honoured.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, volatile int *abort, uint64_t limit_ns)
{
    const uint32_t hint = limit_ns < 1000000u ? (uint32_t)limit_ns : 1000000u;
    if (mbar_try_wait(bar, parity, hint)) return true;
    const uint64_t t0 = globaltimer_ns();
    while (true) {
        if (mbar_try_wait(bar, parity, hint)) return true;
        if (*abort) return false;
        if (globaltimer_ns() - t0 > limit_ns) {
            *abort = 1;
            return false;
        }
    }
}

// Wait for asynchronous work this thread issued itself (bulk copies, MMAs) to finish before the CTA
// releases shared memory or tensor memory after an abort.  Such work completes on its own, so the
// abort flag is ignored and the limit is generous; returns false only if even that runs out.
__device__ __forceinline__ bool mbar_drain(uint64_t *bar, uint32_t parity, uint64_t limit_ns)
{
    const uint64_t t0 = globaltimer_ns();
    while (!mbar_try_wait(bar, parity)) {
        if (globaltimer_ns() - t0 > limit_ns) return false;
    }
    return true;
}

// Drain limit for a wait limit: four times the limit, at least 200 ms.
__host__ __device__ constexpr uint64_t drain_limit_ns(uint64_t limit_ns)
{
    return 4 * limit_ns > 200000000ull ? 4 * limit_ns : 200000000ull;
}

// Data between the CTAs of a cluster: asynchronous stores to the same place of another CTA's shared memory, counted on
// that CTA's mbarrier, and bounded waits for them.  One word per CTA, `stop`, ends a cluster early: whoever gives up
// raises it in every CTA, no wait holds on beside it, and the roles leave their loops instead of going on with what they
// have, so that nobody sends more than the step at hand.  cluster_end then tells every CTA alike.
__device__ __forceinline__ uint32_t cluster_addr(const volatile void *p, int rank)
{
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(const_cast<const void *>(p))), "r"(rank));
    return a;
}

__device__ __forceinline__ void cluster_send(int rank, const double *dst, double v, const uint64_t *bar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(
                     cluster_addr(dst, rank)),
                 "d"(v), "r"(cluster_addr(bar, rank))
                 : "memory");
}

__device__ __forceinline__ void cluster_send(int rank, const double2 *dst, double2 v, const uint64_t *bar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(
                     cluster_addr(dst, rank)),
                 "d"(v.x), "d"(v.y), "r"(cluster_addr(bar, rank))
                 : "memory");
}

__device__ __forceinline__ bool cluster_try(uint32_t bar, uint32_t parity, uint32_t hint_ns)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(hint_ns)
        : "memory");
    return ok != 0;
}

// A wait whose first try has failed, or with a limit so short that the first try counts.
static __device__ __noinline__ bool cluster_wait_on(uint32_t bar, uint32_t parity, const volatile int *stop,
                                                    uint64_t limit_ns)
{
    const uint64_t t0 = globaltimer_ns();
    while (true) {
        const bool ok = cluster_try(bar, parity, limit_ns < 100000u ? (uint32_t)limit_ns : 100000u);
        const bool late = globaltimer_ns() - t0 > limit_ns;
        if (ok) return !late;
        if (late || *stop) return false;
    }
}

// Wait for what the other CTAs send.  Gives up after `limit_ns` or where `stop` is raised; returns false then.  The
// hardware suspends a try for some microseconds whatever its hint; what arrives after the limit is too late all the
// same.  The loop is out of line: inline it made a step of the tridiagonalisation 5 % longer.
__device__ __forceinline__ bool cluster_wait(const uint64_t *bar, uint32_t parity, const volatile int *stop,
                                             uint64_t limit_ns)
{
    return (limit_ns >= 100000u && cluster_try(smem_u32(bar), parity, 100000u)) ||
           cluster_wait_on(smem_u32(bar), parity, stop, limit_ns);
}

// Raise `stop` in all `nctas` CTAs of the cluster (each of them is between its first cluster barrier and cluster_end).
__device__ __forceinline__ void cluster_stop(volatile int *stop, int nctas)
{
    for (int r = 0; r < nctas; ++r)
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr(stop, r)), "r"(1) : "memory");
}

// The end of a kernel's roles, by every thread of the cluster: whether it was stopped.  If so, what was still under way
// has a millisecond to land before a CTA may exit.
template <class Cluster>
__device__ __forceinline__ bool cluster_end(Cluster &cluster, const volatile int *stop)
{
    cluster.sync();   // every send has been issued and every flag raised
    if (!*stop) return false;
    const uint64_t t0 = globaltimer_ns();
    for (int i = 0; i < 100000 && globaltimer_ns() - t0 < 1000000; ++i) __nanosleep(1000);
    cluster.sync();
    return true;
}

__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Bulk global -> shared copy completing on an mbarrier (into the issuing CTA alone).
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t *dst_smem, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor, K-major, no swizzle: 8-row x 16-byte core matrices;
// lbo = byte distance between K-adjacent core matrices, sbo = between 8-row groups.
__device__ __forceinline__ uint64_t sdesc_noswizzle(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor: dense, F32 accumulator, A/B K-major, M = 128.
// fmt: 1 = BF16 (kind::f16), 2 = TF32 (kind::tf32).
__host__ __device__ constexpr uint32_t idesc_m128(uint32_t fmt, uint32_t n)
{
    return (1u << 4) | (fmt << 7) | (fmt << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}

// One lane of a converged warp (the same one at every call).
__device__ __forceinline__ bool elect_one()
{
    uint32_t p;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum)
        : "memory");
}

__device__ __forceinline__ void mma_tf32(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread t of the warp receives lane (base lane + t).
// The wait is part of the same asm statement so no use of the registers can move above it.
__device__ __forceinline__ void tmem_ld_x32(uint32_t taddr, float (&v)[32])
{
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Hardware approximations (MUFU): rsqrt ~2^-22 relative; sin/cos ~2^-21 absolute on [-pi, pi].
__device__ __forceinline__ float rsqrt_approx(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ void sincos_approx(float x, float &s, float &c)
{
    asm("sin.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(x));
    asm("cos.approx.ftz.f32 %0, %1;" : "=f"(c) : "f"(x));
}

// Packed FP32 pairs (sm_100a .f32x2 arithmetic): one instruction does the same operation on the
// two halves of a 64-bit register pair, so two mics' steering terms issue as one instruction.
__device__ __forceinline__ uint64_t f2(float lo, float hi)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_split(uint64_t v, float &lo, float &hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t f2_splat(float x) { return f2(x, x); }
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t f2_sub(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

__device__ __forceinline__ void tmem_ld_x8(uint32_t taddr, float (&v)[8])
{
    uint32_t r[8];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_ld_x16(uint32_t taddr, float (&v)[16])
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

}  // namespace tc
}  // namespace acb
