// act_image.cuh - the activation image of the multi-column projection (q2_gemm.cu): q8_1 codes and scales of up to 32 columns
// (prefill tokens or concurrent sequences).
#pragma once
#include "ops.cuh"

namespace bnk {

constexpr int GEMM_MAX_COLS = 32;
// columns are padded to 8, 16 or 32 (the N of the tensor-core instruction)
inline int gemm_padded_cols(int ncol) { return ncol <= 8 ? 8 : (ncol <= 16 ? 16 : 32); }
// The "activation image" the kernel consumes, per 128 activations (one PTQ1_0 block) of ncp = 8, 16 or 32 columns:
//   codes: column n, sub-block sb (32 activations), k-half kh (16 of them): int8 codes at
//          (n/8) * 1024 + (sb*2 + kh) * 128 + (n%8) * 16   - per group of 8 columns the shared-memory operand layout
//          of the instruction (8 x 16-byte core matrices, K-major, no swizzle), so a stage is one contiguous bulk copy
//   scales: per group of 8 columns 256 bytes at ncp*128 + (n/8)*256: entry (sb, column pair p) at (sb*4 + p) * 16 holds
//           fp32 (d[2p], d[2p+1], -s[2p], -s[2p+1]) - the fp16 values of the q8_1 record, widened, s negated - so that the
//           epilogue's packed two-column arithmetic reads its operands with one 16-byte load
inline size_t gemm_image_block_bytes(int ncp) { return size_t(ncp) * 160; }
inline size_t gemm_image_bytes(int K, int ncol) { return size_t(K / 128) * gemm_image_block_bytes(gemm_padded_cols(ncol)); }

enum PrepMode { PREP_PLAIN = 0, PREP_NORM = 1 };
struct PrepArgs {
    const float *x; size_t x_stride;      // column c reads x + c * x_stride (floats)
    const float *w;                       // PREP_NORM: x <- rms_norm(x) * w over all K values
    const int32_t *signs;                 // K sign values; null = no rotation (quantise x as it is)
    int K, hat_block;
    float eps;
    int ncol;
    uint8_t *image;
    float *inv_out; size_t inv_stride;    // PREP_NORM, optional: the norm factor of column c at inv_out + c * inv_stride
    int mode;
    bool unit_signs;                      // the signs are known to be +-1 (a model's, checked when they are set); else any integers, PREP_PLAIN
};
void prep_cols(cudaStream_t st, const PrepArgs &a);

inline bool gemm_supported(int M, int K, int ncol) { return M >= 1 && K >= 1024 && K % 1024 == 0 && ncol >= 1 && ncol <= GEMM_MAX_COLS; }
// one tiny kernel whose only wait can never complete and gives up after about a thousand tries: sets *err = 2 and returns
cudaError_t launch_wait_selftest_gemm(cudaStream_t st, int *err);

}  // namespace bnk
