// async_ptx.h -- inline PTX for the LU-SGS wavefront kernels: mbarriers,
// bulk (TMA) copies into shared memory, and gpu-scope acquire/release flags.
// Every wait built on these helpers is bounded by its caller.
#pragma once

#include <cuda_runtime.h>

namespace scfd {
namespace ptx {

__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_gpu(int* p, int v) {
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// arrive (release, CTA scope) without a transaction count
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.shared.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// the same for the lanes with `pred` set, without a branch
__device__ __forceinline__ void mbar_arrive_if(unsigned long long* bar, bool pred) {
    asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %1, 0;\n @p mbarrier.arrive.shared.b64 _, [%0];\n}\n" ::"r"(
                     smem_u32(bar)),
                 "r"((int)pred)
                 : "memory");
}
// shared-memory store for the lanes with `pred` set, without a branch.  No memory
// clobber: it is ordered with other asm volatile statements only, so loads that do
// not read the location can be scheduled around it.
__device__ __forceinline__ void st_shared_if(double* dst, double v, bool pred) {
    asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %2, 0;\n @p st.shared.f64 [%0], %1;\n}\n" ::"r"(smem_u32(dst)), "d"(v),
                 "r"((int)pred));
}
__device__ __forceinline__ void st_shared_if(float* dst, float v, bool pred) {
    asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %2, 0;\n @p st.shared.f32 [%0], %1;\n}\n" ::"r"(smem_u32(dst)), "f"(v),
                 "r"((int)pred));
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// one bulk copy global -> shared of `bytes` (multiple of 16, both addresses
// 16-byte aligned), completing on `bar`
__device__ __forceinline__ void tma_bulk_g2s(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
// true once the phase with parity `phase` of `bar` has completed (acquire, CTA scope)
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned phase) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(phase)
        : "memory");
    return ok != 0;
}

// non-blocking: true if the phase with parity `phase` of `bar` has completed
__device__ __forceinline__ bool mbar_test_wait(unsigned long long* bar, unsigned phase) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(phase)
        : "memory");
    return ok != 0;
}

// ---- thread-block clusters: rank, distributed shared memory -------------
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// all threads of all CTAs of the cluster (release / acquire at cluster scope)
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
// shared::cluster address of the shared-memory location `p` (of this CTA's
// layout) in the CTA of cluster rank `rank`
__device__ __forceinline__ unsigned mapa(const void* p, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
    return r;
}
// the same without release semantics (no fence): for a consumer telling a
// producer that a buffer may be refilled, where the consumer's reads of it
// have long completed when the producer next writes it
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(unsigned rbar) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(rbar) : "memory");
}
// arrive with an expected transaction count on another CTA's mbarrier, no fence
__device__ __forceinline__ void mbar_arrive_expect_tx_cluster_relaxed(unsigned rbar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.relaxed.cluster.shared::cluster.b64 _, [%0], %1;" ::"r"(rbar), "r"(bytes)
                 : "memory");
}
// bulk copy from this CTA's shared memory into another CTA's (shared::cluster
// address), completing `bytes` of transaction count on the receiver's mbarrier
__device__ __forceinline__ void bulk_s2dsmem(unsigned rdst, const void* src, unsigned bytes, unsigned rbar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     rdst),
                 "r"(smem_u32(src)), "r"(bytes), "r"(rbar)
                 : "memory");
}

// generic-proxy shared-memory writes become visible to later bulk copies
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// generic-proxy global accesses are ordered with later bulk copies
__device__ __forceinline__ void fence_proxy_async_global() {
    asm volatile("fence.proxy.async.global;" ::: "memory");
}

}  // namespace ptx
}  // namespace scfd
