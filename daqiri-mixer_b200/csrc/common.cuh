// common.cuh -- shared helpers of the X-engine kernels: status plumbing and
// hand-written sm_100a PTX wrappers (mbarrier, bulk / tensor TMA, tcgen05).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include "mixer.h"

namespace mixer {

// Host: map a CUDA error to a status, remembering the message for debugging.
int cuda_status(cudaError_t e, const char* what);
#define MIXER_CK(call)                                                     \
    do {                                                                   \
        cudaError_t e_ = (call);                                           \
        if (e_ != cudaSuccess) return ::mixer::cuda_status(e_, #call);     \
    } while (0)

// Upper bound for every in-kernel wait (ns of %globaltimer).  A wait that
// runs out sets MIXER_ETIMEOUT in the caller's error word and the kernel
// winds down instead of spinning forever.
constexpr uint64_t kWaitLimitNs = 2000000000ull;

#if defined(__CUDACC__)

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// ---- dependent launches -----------------------------------------------------
// A kernel launched by launch_dependent may start before the kernel ahead of
// it on the stream has finished; nothing it reads or writes in global memory
// may be touched before pdl_wait.  Nor may its pointers be declared
// __restrict__: what the kernel ahead still writes is not constant for this
// one's life, as read-only loads require, and the compiler could move such
// loads over the wait.  pdl_trigger lets the next such kernel start
// once every CTA has called it (or exited).  What it saves is the launch and
// the set-up between two kernels: 64 elements x 16 channels, K 256 (corner-turn
// and GEMM) 12.3 -> 10.9 us; 256 x 128, K 1024 78.2 -> 73.4; 200 x 128, K 1536
// with flush 119.0 -> 112.3.  The corner-turn does not trigger early: the
// GEMM's CTAs then take their SMs from its last ones (dump of 512 heaps at 256
// x 128 765 -> 774-785 us).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <typename... P, typename... A>
inline cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                                    cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// ---- mbarrier ---------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait for the phase of parity `parity` to complete.  Returns false
// when the limit ran out or *abort became non-zero.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity,
                                          const volatile int* abort = nullptr) {
    if (mbar_test(bar, parity)) return true;
    const uint64_t t0 = globaltimer_ns();
    while (true) {
#pragma unroll 1
        for (int i = 0; i < 32; ++i)
            if (mbar_test(bar, parity)) return true;
        if (abort && *abort) return false;
        if (globaltimer_ns() - t0 > kWaitLimitNs) return false;
    }
}

// ---- TMA --------------------------------------------------------------------
// Untiled bulk copy global -> shared, completion counted on an mbarrier.
// Both addresses 16-byte aligned, size a multiple of 16.
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes,
                                         uint32_t bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            dst),
        "l"(src), "r"(bytes), "r"(bar)
        : "memory");
}
// Tiled 4-D tensor load (no multicast).  x must be 16-byte aligned in bytes.
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar,
                                            int x, int y, int z, int w) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(w)
        : "memory");
}
__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// ---- dynamic work: cluster launch control -----------------------------------
// A running CTA takes over ("cancels") a CTA of its own launch that has not
// started yet: the 16-byte answer lands in shared memory and completes 16
// bytes on an mbarrier.  No further request may follow one that found none.
__device__ __forceinline__ void clc_request(uint32_t dst, uint32_t bar) {
    asm volatile(
        "clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128"
        " [%0], [%1];" ::"r"(dst),
        "r"(bar)
        : "memory");
}
// blockIdx.x of the CTA taken over, or -1 when every CTA has started.  The
// fence orders this read before the next request's write to the same bytes.
__device__ __forceinline__ int64_t clc_answer(uint32_t src) {
    uint32_t x, ok;
    asm volatile(
        "{\n\t.reg .b128 h;\n\t.reg .pred p;\n\t"
        "ld.shared.b128 h, [%2];\n\t"
        "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\t"
        "selp.u32 %1, 1, 0, p;\n\t"
        "mov.u32 %0, 0;\n\t"
        "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %0, h;\n\t"
        "fence.proxy.async.shared::cta;\n\t}"
        : "=r"(x), "=r"(ok)
        : "r"(src)
        : "memory");
    return ok ? (int64_t)x : -1;
}

// ---- tcgen05 ------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Arrive on `bar` once every tcgen05.mma issued so far by this thread is done.
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     bar)
                 : "memory");
}
// D[tmem] (+)= A[smem] * B[smem]^T, int8 x int8 -> int32, one CTA.
__device__ __forceinline__ void mma_i8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                       uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// ---- CTA pairs (cluster of two, tcgen05 cta_group::2) ----------------------
// The pair's leader is cluster rank 0: it issues every pair MMA, which reads
// A rows and half of B from both CTAs' shared memory (same offsets) and writes
// both CTAs' TMEM.  No load here uses cluster multicast.
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// Cluster-window address of the same shared-memory variable in CTA `rank`.
__device__ __forceinline__ uint32_t mapa_shared(uint32_t saddr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}
// Every thread of both CTAs; orders the shared-memory writes before it
// (barrier initialisation, TMEM address) for the peer.
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
                 "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrive on an mbarrier named by its cluster-window address (either CTA).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t caddr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(caddr)
                 : "memory");
}
__device__ __forceinline__ void st_cluster_u32(uint32_t caddr, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(caddr), "r"(v) : "memory");
}
// Tiled 4-D load into this CTA's shared memory whose byte count completes on
// an mbarrier of either CTA of the pair (cluster-window address); no multicast.
__device__ __forceinline__ void tma_load_4d_pair(uint32_t dst, const CUtensorMap* map,
                                                 uint32_t bar_caddr, int x, int y, int z, int w) {
    asm volatile(
        "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_caddr), "r"(x), "r"(y), "r"(z), "r"(w)
        : "memory");
}
// TMEM of a pair: one warp with the same warp index in each CTA, the same
// destination offset in both.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
                 : "memory");
}
// D[tmem of both CTAs] (+)= A[smem, 128 rows per CTA] * B[smem, N/2 rows per CTA]^T.
__device__ __forceinline__ void mma_i8_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                            uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Once every pair MMA issued so far is done, arrive on the mbarrier at
// shared-memory offset `bar` in each CTA of `mask`.
__device__ __forceinline__ void tc_commit_pair(uint32_t bar, uint16_t mask) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64"
        " [%0], %1;" ::"r"(bar),
        "h"(mask)
        : "memory");
}

// Instruction descriptor for kind::i8: D s32, A and B signed int8, both
// K-major, shape M x N.
__host__ __device__ constexpr uint32_t idesc_i8(int M, int N) {
    return (2u << 4)                       // D format: s32
           | (1u << 7)                     // A: signed 8-bit
           | (1u << 10)                    // B: signed 8-bit
           | ((uint32_t)(N >> 3) << 17)    // N / 8
           | ((uint32_t)(M >> 4) << 24);   // M / 16
}
// Shared-memory matrix descriptor of a K-major tile in the 128-byte swizzle
// layout written by TMA: rows of 128 bytes, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t sdesc_sw128(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu)   // start address / 16
           | ((uint64_t)1 << 16)                 // leading byte offset (unused here)
           | ((uint64_t)(1024 >> 4) << 32)       // stride byte offset: 8 rows
           | ((uint64_t)1 << 46)                 // descriptor version (sm_100)
           | ((uint64_t)2 << 61);                // layout: 128-byte swizzle
}

// Same for the 64-byte swizzle: rows of 64 bytes, 8-row groups 512 bytes apart.
__device__ __forceinline__ uint64_t sdesc_sw64(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu)   // start address / 16
           | ((uint64_t)1 << 16)                 // leading byte offset (unused here)
           | ((uint64_t)(512 >> 4) << 32)        // stride byte offset: 8 rows
           | ((uint64_t)1 << 46)                 // descriptor version (sm_100)
           | ((uint64_t)4 << 61);                // layout: 64-byte swizzle
}

#endif  // __CUDACC__

}  // namespace mixer
