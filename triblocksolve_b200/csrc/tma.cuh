/*
 * tma.cuh -- thin inline-PTX wrappers for the Blackwell (sm_100a) bulk-copy
 * engine and shared-memory mbarriers used by the streaming kernels.
 *
 * Only the untiled bulk form is used (cp.async.bulk global -> shared, each
 * copy into the issuing CTA alone): every copy starts on a 16-byte boundary and moves a multiple
 * of 16 bytes, which the callers guarantee through the even-cell layout.
 * Every wait is bounded by a clock64 budget; on expiry the caller gets
 * `false`, records ST_TIMEOUT and leaves instead of spinning forever.
 */
#ifndef TBS_TMA_CUH
#define TBS_TMA_CUH

#include <cstdint>

namespace tbs {

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
}

/* make initialised barriers visible to the async (bulk-copy) proxy */
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

/* arrival (count 1) on `bar` by the lanes with `on` set, without a branch */
__device__ __forceinline__ void mbar_arrive_if(uint64_t *bar, bool on) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(smem_u32(bar)),
        "r"((unsigned)on)
        : "memory");
}

/* whether phase `parity` of `bar` has completed; does not wait */
__device__ __forceinline__ bool mbar_test(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

/* Wait for phase `parity` of `bar` to complete; false after ~budget cycles. */
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity,
                                          long long budget = (1LL << 31)) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - t0 > budget) return false;
    }
    return true;
}

/* bulk copy global -> this CTA's shared memory, completing on `bar` */
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes,
                                         uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

/* same, with an L2 eviction-priority policy (evict_first for streams that
 * are read once per sweep, so that reused vectors stay resident) */
__device__ __forceinline__ uint64_t policy_evict_first() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}

__device__ __forceinline__ uint64_t policy_evict_last() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}

/* global store / load with an L2 eviction policy */
__device__ __forceinline__ void st_hint(double *p, double v, uint64_t pol) {
    asm volatile("st.global.L2::cache_hint.f64 [%0], %1, %2;" ::"l"(p), "d"(v), "l"(pol) : "memory");
}
__device__ __forceinline__ void st_hint(float *p, float v, uint64_t pol) {
    asm volatile("st.global.L2::cache_hint.f32 [%0], %1, %2;" ::"l"(p), "f"(v), "l"(pol) : "memory");
}
__device__ __forceinline__ double ld_hint(const double *p, uint64_t pol) {
    double v;
    asm volatile("ld.global.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(pol) : "memory");
    return v;
}
__device__ __forceinline__ float ld_hint(const float *p, uint64_t pol) {
    float v;
    asm volatile("ld.global.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol) : "memory");
    return v;
}

__device__ __forceinline__ void bulk_g2s_hint(void *dst, const void *src, uint32_t bytes,
                                              uint64_t *bar, uint64_t pol) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint "
        "[%0], [%1], %2, [%3], %4;" ::"r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(pol)
        : "memory");
}

/* 8-byte asynchronous copies global -> shared memory, in groups of the
 * issuing thread */
__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
/* all but the newest N groups have landed */
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

/* makes this thread's writes to shared memory visible to the bulk copies
 * that are issued after the next barrier */
__device__ __forceinline__ void fence_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

/* bulk copy / bulk FP64 add, this CTA's shared memory -> global (addresses
 * and size multiples of 16 bytes), in the issuing thread's open group */
__device__ __forceinline__ void bulk_s2g(void *dst, const void *src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
                 "r"(smem_u32(src)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_add_s2g(void *dst, const void *src, uint32_t bytes) {
    asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f64 [%0], [%1], %2;" ::"l"(dst),
                 "r"(smem_u32(src)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_s2g_commit() {
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
/* all but the newest N of this thread's committed groups are complete: read,
 * and written */
template <int N>
__device__ __forceinline__ void bulk_s2g_wait_but() {
    asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}
/* this thread's ordinary accesses (and those it has seen) before its bulk
 * copies that follow, and the other way round */
__device__ __forceinline__ void fence_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }
__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
/* the shared memory of this thread's committed groups has been read */
__device__ __forceinline__ void bulk_s2g_wait_read() {
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

}  // namespace tbs

#endif /* TBS_TMA_CUH */
