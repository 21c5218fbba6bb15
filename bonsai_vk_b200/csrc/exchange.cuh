// exchange.cuh - exchanges between the CTAs of a cluster: stores into another CTA's shared memory that an mbarrier there counts by their
// bytes, and the bounded wait for them. One way across the cluster; a plain store and a cluster barrier wait for the store's
// acknowledgement and make a round trip on top of it, 0.4 us more (attention and the recurrent step, attn_cluster.cu and gdn_step.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace bnk {

// the context's error word after a give-up (bn_sync names the wait)
enum { ERR_ATTN_EXCHANGE = 5, ERR_STEP_EXCHANGE = 6 };

#ifdef __CUDACC__
// the place of `p` in the shared memory of CTA `rank` of the cluster
__device__ __forceinline__ uint32_t remote(const void *p, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(uint32_t(__cvta_generic_to_shared(p))), "r"(rank));
    return r;
}
__device__ __forceinline__ void put(uint32_t addr, float v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr), "r"(__float_as_uint(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ void put2(uint32_t addr, float a, float b, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(addr), "r"(__float_as_uint(a)), "r"(__float_as_uint(b)), "r"(bar) : "memory");
}
// bounded wait for the bytes of a barrier's first phase; on giving up the error word is set to ERR and the caller goes on without waiting
// again (results are then invalid)
template <int ERR>
__device__ __forceinline__ bool arrived(uint32_t bar, int *err, int limit = 1 << 22) {
    for (int it = 0; it < limit; ++it) {
        uint32_t ok;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\nselp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(ok) : "r"(bar) : "memory");
        if (__builtin_expect(ok != 0u, 1)) return true;
    }
    atomicExch(err, ERR);
    return false;
}
// A wait that nothing will ever satisfy, with a short limit: the give-up path of arrived()
template <int ERR>
__global__ void k_wait_selftest_exchange(int *err) {
    __shared__ uint64_t bar;
    const uint32_t b = uint32_t(__cvta_generic_to_shared(&bar));
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\nfence.mbarrier_init.release.cluster;" ::"r"(b) : "memory");
        arrived<ERR>(b, err, 1 << 10);
    }
}
#endif

}  // namespace bnk
