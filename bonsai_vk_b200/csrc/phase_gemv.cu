// phase_gemv.cu - host side of the whole-token kernel's projection phase (phase_body.cuh): which shapes it covers, its shared
// memory, and the self-test of its bounded wait.
#include "phase_body.cuh"

namespace {
using namespace bnk;
using namespace bnk::phase;

// A wait that nothing will ever satisfy, with a short limit: the give-up path of mbar_wait (error word set, kernel
// returns, context stays usable) can be exercised without hanging anything.
__global__ void k_wait_selftest(int *err, int limit) {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0) mbar_wait(&bar, 0, err, nullptr, limit);
}

}  // namespace

namespace bnk {

size_t phase_smem_bytes(int hat_block) { return size_t(phase::smem_bytes(hat_block)); }

bool phase_supported(int M, int K, int hat_block) {
    const int nb = K / 128;
    if (K % 512 || K > phase::MAXK || M < 1) return false;
    if (nb > phase::MAXCH && nb % phase::MAXCH) return false;
    if (hat_block < 16 || hat_block > 4096 || K % hat_block || (hat_block & (hat_block - 1))) return false;
    return true;
}

cudaError_t launch_wait_selftest_ring(cudaStream_t st, int *err) {
    BN_COUNT(1);
    k_wait_selftest<<<1, 32, 0, st>>>(err, 1 << 10);
    return cudaGetLastError();
}

}  // namespace bnk
