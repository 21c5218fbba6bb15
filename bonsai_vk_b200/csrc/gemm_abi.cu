// gemm_abi.cu - C entry points of the multi-column tensor-core projection (declared in include/bonsai_cuda.h).
#include "act_image.cuh"
#include "q2.cuh"
#include "phase_gemv.cuh"

#include <algorithm>

extern "C" {

size_t bn_gemm_image_bytes(int K, int ncol) {
    if (K <= 0 || K % 128 || ncol < 1 || ncol > bnk::GEMM_MAX_COLS) return 0;
    return bnk::gemm_image_bytes(K, ncol);
}

int bn_gemm_act_quant(bn_ctx *ctx, const bn_buf *x, size_t x_off, size_t x_stride, int K, int ncol, const bn_buf *signs,
                      size_t signs_off, int hat_block, bn_buf *image, size_t image_off) {
    BN_REQUIRE(ctx, BN_ERR_ARG, "bn_gemm_act_quant: null context");
    BN_REQUIRE(K > 0 && K % 1024 == 0, BN_ERR_ARG, "bn_gemm_act_quant: K=%d must be a multiple of 1024", K);
    BN_REQUIRE(ncol >= 1 && ncol <= bnk::GEMM_MAX_COLS, BN_ERR_ARG, "bn_gemm_act_quant: %d columns (1..%d)", ncol, bnk::GEMM_MAX_COLS);
    BN_REQUIRE(x_stride >= size_t(K), BN_ERR_ARG, "bn_gemm_act_quant: column stride %zu is shorter than K", x_stride);
    BN_RANGE(x, x_off, (size_t(ncol - 1) * x_stride + K) * 4, 4, "bn_gemm_act_quant x");
    BN_RANGE(image, image_off, bnk::gemm_image_bytes(K, ncol), 128, "bn_gemm_act_quant image");
    if (signs) {
        BN_REQUIRE(hat_block >= 16 && hat_block <= 4096 && (hat_block & (hat_block - 1)) == 0 && K % hat_block == 0, BN_ERR_ARG,
                   "bn_gemm_act_quant: hadamard block %d must be a power of two in [16, 4096] dividing K", hat_block);
        BN_RANGE(signs, signs_off, size_t(K) * 4, 4, "bn_gemm_act_quant signs");
    }
    bnk::PrepArgs a = {};
    a.x = bn_ptr<float>(x, x_off); a.x_stride = x_stride;
    a.signs = signs ? bn_ptr<int32_t>(signs, signs_off) : nullptr;
    a.K = K; a.hat_block = hat_block; a.ncol = ncol; a.image = bn_ptr<uint8_t>(image, image_off); a.mode = bnk::PREP_PLAIN;
    bnk::prep_cols(ctx->stream, a);
    return bn_launch_check(ctx, "k_prep_cols");
}

size_t bn_gemm_tiled_bytes(int M, int K) {
    if (M <= 0 || K <= 0 || K % 1024) return 0;
    return bnk::q2_bytes(M, K);
}

int bn_gemm_repack(bn_ctx *ctx, const bn_buf *w, size_t w_off, int M, int K, bn_buf *tiled, size_t tiled_off) {
    BN_REQUIRE(ctx, BN_ERR_ARG, "bn_gemm_repack: null context");
    BN_REQUIRE(M > 0 && K > 0 && K % 1024 == 0, BN_ERR_ARG, "bn_gemm_repack: bad shape M=%d K=%d (K %% 1024 != 0)", M, K);
    BN_RANGE(w, w_off, size_t(M) * (K / 128) * 28, 4, "bn_gemm_repack W");
    BN_RANGE(tiled, tiled_off, bnk::q2_bytes(M, K), 128, "bn_gemm_repack out");
    bnk::q2_repack(ctx->stream, bn_ptr<uint32_t>(w, w_off), M, K, bn_ptr<uint8_t>(tiled, tiled_off));
    return bn_launch_check(ctx, "k_q2_repack");
}

int bn_gemm_q81(bn_ctx *ctx, const bn_buf *w, size_t w_off, int w_tiled, int M, int K, const bn_buf *image, size_t image_off, int ncol,
                bn_buf *out, size_t out_off, size_t out_stride) {
    BN_REQUIRE(ctx, BN_ERR_ARG, "bn_gemm_q81: null context");
    BN_REQUIRE(bnk::gemm_supported(M, K, ncol), BN_ERR_ARG, "bn_gemm_q81: unsupported shape M=%d K=%d columns=%d (K %% 1024 == 0, 1..%d columns)",
               M, K, ncol, bnk::GEMM_MAX_COLS);
    BN_REQUIRE(out_stride >= size_t(M), BN_ERR_ARG, "bn_gemm_q81: column stride %zu is shorter than M", out_stride);
    if (w_tiled) BN_RANGE(w, w_off, bnk::q2_bytes(M, K), 128, "bn_gemm_q81 W (tiled)");
    else BN_RANGE(w, w_off, size_t(M) * (K / 128) * 28, 16, "bn_gemm_q81 W");
    BN_RANGE(image, image_off, bnk::gemm_image_bytes(K, ncol), 128, "bn_gemm_q81 image");
    BN_RANGE(out, out_off, (size_t(ncol - 1) * out_stride + M) * 4, 4, "bn_gemm_q81 out");
    auto args = [&](const uint8_t *W, int r0, int rows) {
        bnk::Q2GemmArgs q = {};
        q.W = W; q.M = rows; q.K = K; q.image = bn_ptr<uint8_t>(image, image_off); q.ncol = ncol;
        q.out = bn_ptr<float>(out, out_off) + r0; q.out_stride = out_stride; q.err = ctx->err_dev;
        return q;
    };
    // Native rows are unpacked by the warps that use them (one launch less, no tiles through memory) where q2_gemm_in_place says so. The
    // others are unpacked into two-bit tiles first, in chunks of at most 48 MB of scratch, which stay in L2 - unless the call is inside
    // a capture (a graph may outlive the scratch), or there is no memory left for it.
    const int step = int(std::max<size_t>(1, (size_t(48) << 20) / (size_t(K / 512) * bnk::Q2_PIECE))) * 16;
    cudaError_t e = cudaSuccess;
    if (w_tiled) e = bnk::launch_q2_gemm(ctx->stream, ctx->sm_count, args(bn_ptr<uint8_t>(w, w_off), 0, M), bnk::g_pdl);
    else if (bnk::q2_gemm_in_place(ctx->sm_count, M, K, ncol, M <= step) || !bn_scratch_available(ctx, bnk::q2_bytes(std::min(M, step), K)))
        e = bnk::launch_q2_gemm_native(ctx->stream, ctx->sm_count, args(bn_ptr<uint8_t>(w, w_off), 0, M), bnk::g_pdl);
    else {
        uint8_t *tiles = reinterpret_cast<uint8_t *>(ctx->scratch);
        for (int r0 = 0; r0 < M && e == cudaSuccess; r0 += step) {
            const int n = std::min(step, M - r0);
            bnk::q2_repack(ctx->stream, bn_ptr<uint32_t>(w, w_off) + size_t(r0) * (K / 128) * 7, n, K, tiles);
            e = bnk::launch_q2_gemm(ctx->stream, ctx->sm_count, args(tiles, r0, n), bnk::g_pdl);
        }
    }
    if (e != cudaSuccess) return bn_cuda_fail(e, "k_q2_gemm");
    return bn_launch_check(ctx, "k_q2_gemm");
}

int bn_selftest_wait(bn_ctx *ctx, int which) {
    BN_REQUIRE(ctx, BN_ERR_ARG, "bn_selftest_wait: null context");
    BN_REQUIRE(which >= 0 && which <= 3, BN_ERR_ARG, "bn_selftest_wait: which=%d (0 = copy-ring wait, 1 = tensor-core pipeline wait, 2 = attention's exchange, 3 = the recurrent step's)", which);
    auto launch = which == 0 ? bnk::launch_wait_selftest_ring : which == 1 ? bnk::launch_wait_selftest_gemm
                : which == 2 ? bnk::launch_wait_selftest_exchange : bnk::launch_wait_selftest_step;
    cudaError_t e = launch(ctx->stream, ctx->err_dev);
    if (e != cudaSuccess) return bn_cuda_fail(e, "bn_selftest_wait");
    return BN_OK;
}

}  // extern "C"
