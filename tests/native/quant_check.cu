// Exhaustive comparison of the q8_1 quantiser's short forms (rotate_quant.cuh) with the operations that they stand for.
#include "../../bonsai_vk_b200/csrc/rotate_quant.cuh"

namespace {
// every mantissa of one exponent field: div127(x) against the division
__global__ void k_div(unsigned exponent, unsigned long long *bad) {
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < (1u << 23); i += gridDim.x * blockDim.x) {
        const float x = __uint_as_float(exponent << 23 | i);
        if (x > 1e-35f && __float_as_uint(bnk::div127(x)) != __float_as_uint(__fdiv_rn(x, 127.0f))) atomicAdd(bad, 1ull);
    }
}
// bit patterns [first, first + n): code_byte against round half away from zero, clamped
__global__ void k_code(unsigned first, unsigned n, unsigned long long *bad) {
    for (unsigned long long i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float y = __uint_as_float(first + unsigned(i));
        const int want = int(fminf(fmaxf(roundf(y), -127.0f), 127.0f));
        if ((bnk::code_byte(y) & 0xFFu) != (unsigned(want) & 0xFFu)) atomicAdd(bad, 1ull);
    }
}
template <class F> long long count(F launch) {
    unsigned long long *bad = nullptr, n = 0;
    if (cudaMalloc(&bad, 8) != cudaSuccess || cudaMemset(bad, 0, 8) != cudaSuccess) return -1;
    launch(bad);
    const bool ok = cudaMemcpy(&n, bad, 8, cudaMemcpyDeviceToHost) == cudaSuccess;
    cudaFree(bad);
    return ok ? (long long)n : -1;
}
}  // namespace

extern "C" long long check_div127(unsigned exponent) { return count([&](unsigned long long *b) { k_div<<<1024, 256>>>(exponent, b); }); }
extern "C" long long check_code_byte(unsigned first, unsigned n) { return count([&](unsigned long long *b) { k_code<<<2048, 256>>>(first, n, b); }); }
