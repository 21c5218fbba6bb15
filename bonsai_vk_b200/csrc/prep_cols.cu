// prep_cols.cu - the activation image of the multi-column projection (layout: act_image.cuh): per column [rms norm] -> signs ->
// Hadamard -> q8_1 codes and scales. One CTA of 512 threads per column and span of 4096 values, eight values per thread, on the
// helpers of the single-sequence prologue (rotate_quant.cuh), so the same bits. Bound by that chain's latency (2.5 us for a
// normed 4096-wide input; 5 us with the transform split into shuffles and shared-memory passes of two stages each).
#include "act_image.cuh"
#include "rotate_quant.cuh"

namespace {
using namespace bnk;
constexpr int NT = 512;
constexpr int IMG_COL = 160;                   // image bytes per column and block: 128 int8 codes + 4 x (fp32 d, fp32 -s)

__global__ void __launch_bounds__(NT) k_prep_cols(const PrepArgs a, int log_hb, float hat_inv, float inv_k, int ncp) {
    __shared__ __align__(16) float xs[XS8_SPAN];
    __shared__ float red[256];
    const int c = blockIdx.y, tid = threadIdx.x, lane = tid & 31, at = blockIdx.x * 4096 + tid * 8;
    const bool on = at < a.K;
    // constants first: they depend on no earlier kernel
    f32pair nw[4] = {0, 0, 0, 0};
    if (on && c < a.ncol) {
        if (a.mode == PREP_NORM) load8(a.w + at, nw);
        if (a.signs) {
            int sg[8];
            if ((reinterpret_cast<uintptr_t>(a.signs) & 15) == 0) {
                const int4 s0 = *reinterpret_cast<const int4 *>(a.signs + at), s1 = *reinterpret_cast<const int4 *>(a.signs + at + 4);
                sg[0] = s0.x; sg[1] = s0.y; sg[2] = s0.z; sg[3] = s0.w; sg[4] = s1.x; sg[5] = s1.y; sg[6] = s1.z; sg[7] = s1.w;
            } else {
#pragma unroll
                for (int k = 0; k < 8; ++k) sg[k] = a.signs[at + k];
            }
            if (a.unit_signs) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    nw[k] ^= (unsigned long long)(uint32_t(sg[2 * k]) & 0x80000000u) | (unsigned long long)(uint32_t(sg[2 * k + 1]) & 0x80000000u) << 32;
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) nw[k] = pair_of(float(sg[2 * k]), float(sg[2 * k + 1]));
            }
        }
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // where this thread's eight codes and (every fourth thread) its sub-block's scales go
    unsigned char *blk = a.image + size_t(at >> 7) * size_t(ncp) * IMG_COL;
    const int sb = (at >> 5) & 3, kh = (at >> 4) & 1;
    uint2 *codes = reinterpret_cast<uint2 *>(blk + (c / 8) * 1024 + (sb * 2 + kh) * 128 + (c & 7) * 16 + (at & 15));
    float *scales = reinterpret_cast<float *>(blk + size_t(ncp) * 128 + (c / 8) * 256 + (sb * 4 + ((c & 7) >> 1)) * 16) + (c & 1);
    if (c >= a.ncol) {                         // padding column: zero codes and scales
        if (on) {
            *codes = make_uint2(0u, 0u);
            if (!(tid & 3)) { scales[0] = 0.0f; scales[2] = 0.0f; }
        }
        return;
    }
    const float *x = a.x + size_t(c) * a.x_stride;
    f32pair v[4] = {0, 0, 0, 0};
    if (on) {
        if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) load8(x + at, v);
        else {
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] = pair_of(x[at + 2 * k], x[at + 2 * k + 1]);
        }
    }
    if (a.mode == PREP_NORM) {
        // 256 lanes sum the squares of their run of consecutive values ascending, then the fixed tree (rms_norm.comp order)
        const int per = (a.K + 255) >> 8;
        if (a.K == 4096) {                     // a lane's run is two neighbouring threads' values
            float sq = 0.0f, e[8];
#pragma unroll
            for (int k = 0; k < 4; ++k) split_pair(pair_mul(v[k], v[k]), e[2 * k], e[2 * k + 1]);
#pragma unroll
            for (int k = 0; k < 8; ++k) sq = __fadd_rn(sq, e[k]);
            sq = __shfl_up_sync(0xFFFFFFFFu, sq, 1);
#pragma unroll
            for (int k = 0; k < 8; ++k) sq = __fadd_rn(sq, e[k]);
            if (tid & 1) red[tid >> 1] = sq;
        } else if (tid < 256) {
            float sq = 0.0f;
            for (int i = 0; i < per; ++i) {
                const int d = tid * per + i;
                if (d < a.K) { const float f = x[d]; sq = __fadd_rn(sq, __fmul_rn(f, f)); }
            }
            red[tid] = sq;
        }
        __syncthreads();
        const float ss = norm_tree256(red, lane);
        const float inv = __frcp_rn(__fsqrt_rn(__fadd_rn(inv_k != 0.0f ? __fmul_rn(ss, inv_k) : __fdiv_rn(ss, float(a.K)), a.eps)));
        if (a.inv_out && blockIdx.x == 0 && tid == 0) a.inv_out[size_t(c) * a.inv_stride] = inv;
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = pair_mul(pair_mul(v[k], pair_of(inv, inv)), nw[k]);
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = a.unit_signs || !a.signs ? v[k] ^ nw[k] : pair_mul(v[k], nw[k]);
    }
    if (!on) {
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = 0ull;
    }
    if (a.signs) {
        fwht_pairs8(v, 3);
        span_store8(xs, tid, v);
        fwht_spans(xs, tid, 1, log_hb, [] { __syncthreads(); });
        span_load8(xs, tid, v);
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = pair_mul(v[k], pair_of(hat_inv, hat_inv));
    }
    const Q8x8 q = quant8_pairs(v);
    if (on) {
        *codes = make_uint2(q.w0, q.w1);
        if (!(tid & 3)) {                      // (d, s) rounded to fp16 as the q8_1 record keeps them, stored as fp32 d and -s
            scales[0] = half_bits_to_float(float_to_half_bits(q.d));
            scales[2] = -half_bits_to_float(float_to_half_bits(__fmul_rn(q.d, float(q.sum))));
        }
    }
}

}  // namespace

namespace bnk {

void prep_cols(cudaStream_t st, const PrepArgs &a) {
    const int hb = a.signs ? a.hat_block : 16;
    launch_spread<k_prep_cols>(dim3((a.K + 4095) / 4096, gemm_padded_cols(a.ncol)), dim3(NT), 0, st, a, 31 - __builtin_clz(unsigned(hb)), 1.0f / sqrtf(float(hb)),
           (a.K & (a.K - 1)) == 0 ? 1.0f / float(a.K) : 0.0f, gemm_padded_cols(a.ncol));
}

}  // namespace bnk
