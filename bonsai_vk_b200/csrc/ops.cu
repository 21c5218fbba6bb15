// ops.cu - the non-GEMV kernels of the decode path: Hadamard rotation, norms, elementwise fusions,
// embedding gather, gated-delta-net update, decode attention over the quantised KV cache, argmax.
//
// Floating-point order is part of the contract with the CPU oracle: sums use the fixed trees
// stated next to each kernel, transcendentals are evaluated in double and rounded once, and the
// file is compiled without fused-multiply-add contraction (fmaf is written where one is meant).
#include "ops.cuh"
#include "quant.cuh"
#include "rotate_quant.cuh"

namespace {

// ---- block-wide helpers ------------------------------------------------------------------------
// tree over n = blockDim.x partials in shared memory: p[i] += p[i + s], s = n/2 .. 1
__device__ __forceinline__ float block_tree_sum(float *p, int n) {
    for (int s = n >> 1; s > 0; s >>= 1) {
        __syncthreads();
        if (int(threadIdx.x) < s) p[threadIdx.x] = __fadd_rn(p[threadIdx.x], p[threadIdx.x + s]);
    }
    __syncthreads();
    return p[0];
}

// in-place Sylvester-Walsh-Hadamard butterflies over N floats in shared memory, h ascending
// (reference: runtime_vk/shaders/hat4096.comp:41-60), then the 1/sqrt(N) factor.
// N values = N / hb independent transforms of width hb side by side.
__device__ __forceinline__ void fwht_smem(float *s, int N, int hb, float inv) {
    for (int h = 1; h < hb; h <<= 1) {
        __syncthreads();
        for (int i = threadIdx.x; i < (N >> 1); i += blockDim.x) {
            const int j = ((i & ~(h - 1)) << 1) | (i & (h - 1));
            const float a = s[j], c = s[j + h];
            s[j] = __fadd_rn(a, c);
            s[j + h] = __fsub_rn(a, c);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < N; i += blockDim.x) s[i] = __fmul_rn(s[i], inv);
    __syncthreads();
}

// ---- rotation (+ quantisation) -------------------------------------------------------------------
// one CTA of 512 threads per span (a Hadamard block of `hb` values, or 128 values = one quantiser block when the Hadamard
// block is smaller): y = H(s . x); optional q8_1 pack of the span.
__global__ void __launch_bounds__(512) k_rotate_quant(const float *__restrict__ x, const int32_t *__restrict__ signs,
                                                      int block, int hb, float inv, float *__restrict__ y,
                                                      uint32_t *__restrict__ q81, uint32_t *__restrict__ table) {
    bnk::pdl_sync();
    extern __shared__ float s[];                   // block floats + 4 x 128 bytes
    int8_t *qs = reinterpret_cast<int8_t *>(s + block);
    const size_t base = size_t(blockIdx.x) * block;
    for (int i = threadIdx.x; i < block; i += blockDim.x) s[i] = __fmul_rn(x[base + i], float(signs[base + i]));
    fwht_smem(s, block, hb, inv);
    if (y) for (int i = threadIdx.x; i < block; i += blockDim.x) y[base + i] = s[i];
    if (q81) {
        const int grp = threadIdx.x >> 7, i = threadIdx.x & 127;       // 4 groups of 128 threads
        const bnk::TableSlots slots = bnk::table_slots(i);
        for (int b = grp; b < block / 128; b += 4) {
            const size_t gb = base / 128 + b;
            bnk::quant_block_128(s[b * 128 + i], i, slots, qs + grp * 128, q81 + gb * bnk::Q81_DWORDS,
                                 table + gb * bnk::BF_WORDS, 1 + grp);
        }
    }
}

// ---- embedding gather (reference addressing: runtime_vk/shaders/gather_rows.comp:12-16) and its inverse rotation ----------------
// y = s . H(row): one CTA per span of 4096 values and column, eight values per thread, on the transform of the projections'
// prologue (rotate_quant.cuh). A kernel each, the rotation on one pair of values per thread and stage, took 13 us; this one 3 us.
__global__ void __launch_bounds__(512) k_embed_rotate(const uint32_t *__restrict__ W, int K, const int *__restrict__ tok_ptr, const int32_t *__restrict__ signs,
                                                      int log_hb, float inv, float *__restrict__ y, bnk::Cols cols) {
    __shared__ __align__(16) float xs[bnk::XS8_SPAN];
    const int t = threadIdx.x, at = blockIdx.x * 4096 + t * 8;
    int sg[8] = {};
    if (at < K) {
#pragma unroll
        for (int k = 0; k < 8; ++k) sg[k] = signs[at + k];
    }
    bnk::pdl_sync();
    { const size_t col = blockIdx.z; tok_ptr = bnk::colp(tok_ptr, col * cols.arena); y = bnk::colp(y, col * cols.arena); }
    float e[8] = {};
    if (at < K) {
        const uint32_t *blk = W + (size_t(tok_ptr[0]) * (K / 128) + at / 128) * 7;
        const float d = half_bits_to_float(blk[6] >> 16);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int el = (at & 127) + k;
            int byte, r;
            if (el < 80) { byte = el & 15; r = el >> 4; }
            else if (el < 120) { byte = 16 + ((el - 80) & 7); r = (el - 80) >> 3; }
            else { byte = 24 + ((el - 120) & 1); r = (el - 120) >> 1; }
            uint32_t v = (blk[byte >> 2] >> ((byte & 3) * 8)) & 0xFFu;
            for (int i = 0; i < r; ++i) v = (v * 3u) & 0xFFu;
            e[k] = __fmul_rn(float(int((v * 3u) >> 8)) - 1.0f, d);
        }
    }
    bnk::f32pair v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = bnk::pair_of(e[2 * k], e[2 * k + 1]);
    bnk::fwht_pairs8(v, 3);
    bnk::span_store8(xs, t, v);
    bnk::fwht_spans(xs, t, 1, log_hb, [] { __syncthreads(); });
    bnk::span_load8(xs, t, v);
    if (at < K) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            bnk::split_pair(v[k], e[0], e[1]);
            y[at + 2 * k] = __fmul_rn(__fmul_rn(e[0], inv), float(sg[2 * k]));
            y[at + 2 * k + 1] = __fmul_rn(__fmul_rn(e[1], inv), float(sg[2 * k + 1]));
        }
    }
}

// ---- RMS norm (reference: runtime_vk/shaders/rms_norm.comp:60-103) --------------------------------
// 256 lanes, lane l sums the squares of its `per` consecutive elements ascending, lane partials
// combined by the fixed tree; y = (x * inv) * w.
__global__ void __launch_bounds__(256) k_rms_norm(const float *__restrict__ x, const float *__restrict__ w, int cols,
                                                  float eps, float *__restrict__ y) {
    bnk::pdl_sync();
    __shared__ float part[256];
    const int l = threadIdx.x, per = (cols + 255) / 256;
    const float *xr = x + size_t(blockIdx.x) * cols;
    float s = 0.0f;
    for (int i = 0; i < per; ++i) {
        const int d = l * per + i;
        if (d < cols) { const float v = xr[d]; s = __fadd_rn(s, __fmul_rn(v, v)); }
    }
    part[l] = s;
    const float ss = block_tree_sum(part, 256);
    const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, float(cols)), eps)));
    float *yr = y + size_t(blockIdx.x) * cols;
    for (int i = 0; i < per; ++i) {
        const int d = l * per + i;
        if (d < cols) { const float v = __fmul_rn(xr[d], inv); yr[d] = w ? __fmul_rn(v, w[d]) : v; }
    }
}

__global__ void k_add_inplace(float *__restrict__ res, const float *__restrict__ d, int n) {
    bnk::pdl_sync();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) res[i] = __fadd_rn(d[i], res[i]);
}

__global__ void k_swiglu(const float *__restrict__ a, const float *__restrict__ b, int n, float *__restrict__ y, bnk::Cols cols) {
    bnk::pdl_sync();
    { const size_t col = blockIdx.z; a = bnk::colp(a, col * cols.arena); b = bnk::colp(b, col * cols.arena); y = bnk::colp(y, col * cols.arena); }
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = __fmul_rn(silu_f(a[i]), b[i]);
}

// small fp32 projection: one warp per row; lane l takes float4 groups l, l+32, ... with one fmaf per
// element, then a 32-lane xor tree (reference: runtime_vk/shaders/gemv_f32.comp).
__global__ void k_gemv_f32_small(const float *__restrict__ W, int M, int K, const float *__restrict__ x,
                                 float *__restrict__ out) {
    bnk::pdl_sync();
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= M) return;
    const float4 *wr = reinterpret_cast<const float4 *>(W + size_t(row) * K);
    const float4 *xv = reinterpret_cast<const float4 *>(x);
    float a = 0.0f;
    for (int i = lane; i < K / 4; i += 32) {
        const float4 w = wr[i], v = xv[i];
        a = fmaf(w.x, v.x, a); a = fmaf(w.y, v.y, a); a = fmaf(w.z, v.z, a); a = fmaf(w.w, v.w, a);
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) a = __fadd_rn(a, __shfl_xor_sync(0xFFFFFFFFu, a, s));
    if (lane == 0) out[row] = a;
}

// ---- gated delta net ------------------------------------------------------------------------------
// gate = ssm_a * softplus(alpha + dt_bias), beta = sigmoid(beta_raw)   (bonsai_forward.h:528-535)
__global__ void k_gdn_gates(const float *alpha, const float *beta_raw, const float *dt_bias, const float *ssm_a, int n,
                            float *gate, float *beta) {
    bnk::pdl_sync();
    const int i = threadIdx.x;
    if (i >= n) return;
    const float a = __fadd_rn(alpha[i], dt_bias[i]);
    const float sp = a > 20.0f ? a : log_f(__fadd_rn(1.0f, exp_f(a)));
    gate[i] = __fmul_rn(sp, ssm_a[i]);
    beta[i] = sigmoid_f(beta_raw[i]);
}

// 4-tap causal depthwise conv + silu + history shift (runtime_vk/shaders/conv_silu.comp:35-49)
__global__ void k_conv_silu(const float *__restrict__ x, const float *__restrict__ w, float *__restrict__ hist,
                            int channels, float *__restrict__ y) {
    bnk::pdl_sync();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= channels) return;
    float *s = hist + 3 * size_t(c);
    const float *wc = w + 4 * size_t(c);
    const float s0 = s[0], s1 = s[1], s2 = s[2], xn = x[c];
    float acc = __fmul_rn(wc[0], s0);
    acc = __fadd_rn(acc, __fmul_rn(wc[1], s1));
    acc = __fadd_rn(acc, __fmul_rn(wc[2], s2));
    acc = __fadd_rn(acc, __fmul_rn(wc[3], xn));
    y[c] = silu_f(acc);
    s[0] = s1; s[1] = s2; s[2] = xn;
}

// L2 norm of 128-wide rows, mode 1 (runtime_vk/shaders/l2_norm.comp:59-78); one warp per row
__global__ void k_l2_norm_rows(const float *__restrict__ x, int rows, float eps, float *__restrict__ y) {
    bnk::pdl_sync();
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), l = threadIdx.x & 31;
    if (row >= rows) return;
    const float *xr = x + size_t(row) * 128;
    const float a = xr[l], b = xr[l + 32], c = xr[l + 64], d = xr[l + 96];
    const float ss = bnk::warp_tree128(__fmul_rn(a, a), __fmul_rn(b, b), __fmul_rn(c, c), __fmul_rn(d, d));
    const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(ss, eps)));
    float *yr = y + size_t(row) * 128;
    yr[l] = __fmul_rn(a, inv); yr[l + 32] = __fmul_rn(b, inv); yr[l + 64] = __fmul_rn(c, inv); yr[l + 96] = __fmul_rn(d, inv);
}

// delta rule (runtime_vk/shaders/gdn_delta.comp:78-102), one warp per (v-head h, state row j):
// S *= exp(g); pred = sum_i S_i k_i; u = beta (v_j - pred); S_i = fma(k_i, u, S_i); o_j = (sum_i S_i q_i) / sqrt(dim)
__global__ void __launch_bounds__(256) k_gdn_delta(int heads, int qk_heads, const float *__restrict__ q,
                                                   const float *__restrict__ k, const float *__restrict__ v,
                                                   const float *__restrict__ gate, const float *__restrict__ beta,
                                                   float *__restrict__ state, float *__restrict__ o, float scale) {
    bnk::pdl_sync();
    const int h = blockIdx.y, j = blockIdx.x * 8 + (threadIdx.x >> 5), l = threadIdx.x & 31;
    const int hq = h % qk_heads;
    const float eg = exp_f(gate[h]), bt = beta[h];
    const float *kr = k + hq * 128, *qr = q + hq * 128;
    float *S = state + (size_t(h) * 128 + j) * 128;
    float s[4], kk[4], qq[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) { s[e] = __fmul_rn(S[l + 32 * e], eg); kk[e] = kr[l + 32 * e]; qq[e] = qr[l + 32 * e]; }
    const float pred = bnk::warp_tree128(__fmul_rn(s[0], kk[0]), __fmul_rn(s[1], kk[1]), __fmul_rn(s[2], kk[2]), __fmul_rn(s[3], kk[3]));
    const float u = __fmul_rn(bt, __fsub_rn(v[h * 128 + j], pred));
#pragma unroll
    for (int e = 0; e < 4; ++e) { s[e] = fmaf(kk[e], u, s[e]); S[l + 32 * e] = s[e]; }
    const float ov = bnk::warp_tree128(__fmul_rn(s[0], qq[0]), __fmul_rn(s[1], qq[1]), __fmul_rn(s[2], qq[2]), __fmul_rn(s[3], qq[3]));
    if (l == 0) o[h * 128 + j] = __fmul_rn(ov, scale);
}

// Fused gated-delta-net mixer of one layer, one CTA of 512 threads per v-head: the two small fp32 projections
// of the normed residual and their gate functions (bonsai_forward.h:523-535), conv + silu of the head's q, k
// and v channels, L2 norms, the delta rule on the head's 128 state rows, then the per-head RMS, ssm_norm,
// swiglu(z, .) and the v-grouped permutation (bonsai_forward.h:559-567) straight into the next projection's
// input. The conv history is double-buffered by position parity: the two v-heads that share a q/k head both
// read its taps while one of them writes the shifted taps into the other buffer.
// Arithmetic and its order are those of the stand-alone kernels above.
// MINB = CTAs per SM the register budget is set for: 1 for a single sequence (32 CTAs in all; the loads hoisted above
// the dependency wait keep ~90 registers live, measured 4 % of a token faster than the 64-register build), 2 when many
// sequences fill the GPU with CTAs (measured 3 % of a 32-sequence pass faster than one CTA per SM). With several sequences the
// projection in front is the several-column one, which releases its dependents behind its own dependency wait, so the residual and its norm
// factor, which the kernel in front of that one wrote, may be read before the wait here: the two dot products, their gate functions and
// the row's loads pass while the projection's last CTAs run. With the outputs' gate off the tail (it was one warp's, behind everything)
// a step of 8 sequences takes 1.995 instead of 2.012 ms, a recurrent block of 2 / 8 / 32 sequences 65.3 / 67.9 / 161.5 -> 63.6 / 65.8 / 158.2 us.
template <int MINB>
__global__ void __launch_bounds__(512, MINB) k_gdn_core(int heads, int qk_heads, int hidden, const float *__restrict__ qkv,
                                                  const float *__restrict__ conv_w, float *__restrict__ hist0,
                                                  float *__restrict__ hist1, const int *__restrict__ pos_ptr,
                                                  const float *__restrict__ x, const float *__restrict__ inv_ptr,
                                                  const float *__restrict__ norm_w, const float *__restrict__ alpha_w,
                                                  const float *__restrict__ beta_w, const float *__restrict__ dt_bias,
                                                  const float *__restrict__ ssm_a, float *__restrict__ state,
                                                  const float *__restrict__ z, const float *__restrict__ ssm_norm, float eps,
                                                  float *__restrict__ y, float scale, bnk::Cols cols) {
    { const size_t col = blockIdx.z; qkv = bnk::colp(qkv, col * cols.arena); hist0 = bnk::colp(hist0, col * cols.conv); hist1 = bnk::colp(hist1, col * cols.conv); pos_ptr = bnk::colp(pos_ptr, col * cols.arena); x = bnk::colp(x, col * cols.arena); inv_ptr = bnk::colp(inv_ptr, col * cols.arena); state = bnk::colp(state, col * cols.gdn); z = bnk::colp(z, col * cols.arena); y = bnk::colp(y, col * cols.arena); }
    constexpr bool PRE = MINB == 2;
    __shared__ float sq[128], sk[128], sv[128], so[128], sz[128], sgb[2];
    __shared__ int place;
    extern __shared__ float4 dyn[];                // [3][hidden/4]: normed residual, row h of ssm_alpha, row h of ssm_beta
    const int h = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int hq = h % qk_heads, n4 = hidden / 4;
    // ---- before the dependency wait: everything that the preceding kernel (the qkv / gate projection) does not write.
    // Constants, this layer's recurrent state and conv taps (last written one token ago) and the position (set before
    // the pass) are requested while the projection's last CTAs are still running; nothing else may be, older kernels of
    // the pass may be unfinished too (the rule at bnk::launch).
    const bool odd = pos_ptr[0] & 1;               // a token at position p reads taps from buffer p & 1, writes the other
    const float *hist_rd = odd ? hist1 : hist0;
    float *hist_wr = odd ? hist0 : hist1;
    float S[8][4];                                 // state rows of this warp (8 of the head's 128)
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const float *Sr = state + (size_t(h) * 128 + warp * 8 + r) * 128;
#pragma unroll
        for (int e = 0; e < 4; ++e) S[r][e] = Sr[lane + 32 * e];
    }
    const int cch = tid < 128 ? hq * 128 + tid : (tid < 256 ? qk_heads * 128 + hq * 128 + (tid - 128) : 2 * qk_heads * 128 + h * 128 + (tid - 256));
    float tap0 = 0.0f, tap1 = 0.0f, tap2 = 0.0f, cw0 = 0.0f, cw1 = 0.0f, cw2 = 0.0f, cw3 = 0.0f;
    if (tid < 384) {
        const float *sr = hist_rd + 3 * size_t(cch);
        const float *wc = conv_w + 4 * size_t(cch);
        tap0 = sr[0]; tap1 = sr[1]; tap2 = sr[2];
        cw0 = wc[0]; cw1 = wc[1]; cw2 = wc[2]; cw3 = wc[3];
    }
    {
        const float4 *ra = reinterpret_cast<const float4 *>(alpha_w + size_t(h) * hidden), *rb = reinterpret_cast<const float4 *>(beta_w + size_t(h) * hidden);
        for (int i = tid; i < n4; i += 512) { dyn[n4 + i] = ra[i]; dyn[2 * n4 + i] = rb[i]; }
    }
    if (tid == 0) place = heads / qk_heads * hq + h / qk_heads;              // the head's place in the v-grouped permutation
    const float nwz = tid >= 384 ? ssm_norm[tid - 384] : 0.0f;
    auto residual = [&] {   // the normed residual goes to shared memory for the two dependent dot-product chains
        const float inv = __ldcg(inv_ptr);
        const float4 *xv = reinterpret_cast<const float4 *>(x), *nw = reinterpret_cast<const float4 *>(norm_w);
        for (int i = tid; i < n4; i += 512) {
            const float4 a4 = __ldcg(xv + i), w4 = nw[i];
            dyn[i] = make_float4(__fmul_rn(__fmul_rn(a4.x, inv), w4.x), __fmul_rn(__fmul_rn(a4.y, inv), w4.y),
                                 __fmul_rn(__fmul_rn(a4.z, inv), w4.z), __fmul_rn(__fmul_rn(a4.w, inv), w4.w));
        }
    };
    auto gates = [&] {
        if (warp < 14) return;
        // row h of ssm_alpha (warp 14) or ssm_beta (warp 15) times the normed residual: lane l takes float4 groups
        // l, l+32, ... with one fmaf per element, then a 32-lane xor tree (k_gemv_f32_small)
        const float4 *wr = dyn + (warp == 14 ? n4 : 2 * n4);
        float acc = 0.0f;
#pragma unroll 4
        for (int i = lane; i < n4; i += 32) {
            const float4 w4 = wr[i], a4 = dyn[i];
            acc = fmaf(w4.x, a4.x, acc); acc = fmaf(w4.y, a4.y, acc); acc = fmaf(w4.z, a4.z, acc); acc = fmaf(w4.w, a4.w, acc);
        }
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(0xFFFFFFFFu, acc, s));
        if (lane == 0) {
            if (warp == 14) {
                const float al = __fadd_rn(acc, dt_bias[h]);
                const float sp = al > 20.0f ? al : log_f(__fadd_rn(1.0f, exp_f(al)));
                sgb[0] = exp_f(__fmul_rn(sp, ssm_a[h]));
            } else sgb[1] = sigmoid_f(acc);
        }
    };
    if (PRE) {
        residual();
        __syncthreads();
        gates();
    }
    bnk::pdl_sync();
    if (!PRE) residual();
    const bool own_qk = h < qk_heads;              // the first of the v-heads sharing q/k head hq writes its taps
    if (tid < 384) {
        const float xn = qkv[cch];
        float acc = __fmul_rn(cw0, tap0);
        acc = __fadd_rn(acc, __fmul_rn(cw1, tap1));
        acc = __fadd_rn(acc, __fmul_rn(cw2, tap2));
        acc = __fadd_rn(acc, __fmul_rn(cw3, xn));
        if (tid >= 256 || own_qk) { float *sw = hist_wr + 3 * size_t(cch); sw[0] = tap1; sw[1] = tap2; sw[2] = xn; }
        const float cv = silu_f(acc);
        if (tid < 128) sq[tid] = cv; else if (tid < 256) sk[tid - 128] = cv; else sv[tid - 256] = cv;
    } else sz[tid - 384] = silu_f(z[h * 128 + tid - 384]);                   // (the gate of the outputs, off the tail)
    __syncthreads();
    if (!PRE) gates();
    float qq[4], kk[4];
    {
        const float a0 = sq[lane], a1 = sq[lane + 32], a2 = sq[lane + 64], a3 = sq[lane + 96];
        const float iq = __frcp_rn(__fsqrt_rn(__fadd_rn(bnk::warp_tree128(__fmul_rn(a0, a0), __fmul_rn(a1, a1), __fmul_rn(a2, a2), __fmul_rn(a3, a3)), 1e-12f)));
        qq[0] = __fmul_rn(a0, iq); qq[1] = __fmul_rn(a1, iq); qq[2] = __fmul_rn(a2, iq); qq[3] = __fmul_rn(a3, iq);
        const float b0 = sk[lane], b1 = sk[lane + 32], b2 = sk[lane + 64], b3 = sk[lane + 96];
        const float ik = __frcp_rn(__fsqrt_rn(__fadd_rn(bnk::warp_tree128(__fmul_rn(b0, b0), __fmul_rn(b1, b1), __fmul_rn(b2, b2), __fmul_rn(b3, b3)), 1e-12f)));
        kk[0] = __fmul_rn(b0, ik); kk[1] = __fmul_rn(b1, ik); kk[2] = __fmul_rn(b2, ik); kk[3] = __fmul_rn(b3, ik);
    }
    __syncthreads();
    const float eg = sgb[0], bt = sgb[1];
    // four rows at a time; their trees share six shuffles (a level's two values change hands between the lanes that go on with
    // one and those that go on with the other), as the shuffles' throughput bounds this part
    const bool b4 = lane & 16, b3 = lane & 8;
    auto trees4 = [&](const float (&v)[4]) {           // lane l: the sum of row (l >> 4) + 2 * (l >> 3 & 1)
        const float x = __fadd_rn(b4 ? v[1] : v[0], __shfl_xor_sync(0xFFFFFFFFu, b4 ? v[0] : v[1], 16));
        const float y = __fadd_rn(b4 ? v[3] : v[2], __shfl_xor_sync(0xFFFFFFFFu, b4 ? v[2] : v[3], 16));
        float s = __fadd_rn(b3 ? y : x, __shfl_xor_sync(0xFFFFFFFFu, b3 ? x : y, 8));
#pragma unroll
        for (int d = 4; d > 0; d >>= 1) s = __fadd_rn(s, __shfl_xor_sync(0xFFFFFFFFu, s, d));
        return s;
    };
#pragma unroll
    for (int r0 = 0; r0 < 8; r0 += 4) {
        float p[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            float (&s)[4] = S[r0 + r];
#pragma unroll
            for (int e = 0; e < 4; ++e) s[e] = __fmul_rn(s[e], eg);
            p[r] = __fadd_rn(__fadd_rn(__fmul_rn(s[0], kk[0]), __fmul_rn(s[2], kk[2])), __fadd_rn(__fmul_rn(s[1], kk[1]), __fmul_rn(s[3], kk[3])));
        }
        const float pred = trees4(p);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int j = warp * 8 + r0 + r;
            float *Sr = state + (size_t(h) * 128 + j) * 128;
            float (&s)[4] = S[r0 + r];
            const float u = __fmul_rn(bt, __fsub_rn(sv[j], __shfl_sync(0xFFFFFFFFu, pred, (r & 1) * 16 + (r >> 1) * 8)));
#pragma unroll
            for (int e = 0; e < 4; ++e) { s[e] = fmaf(kk[e], u, s[e]); Sr[lane + 32 * e] = s[e]; }
            p[r] = __fadd_rn(__fadd_rn(__fmul_rn(s[0], qq[0]), __fmul_rn(s[2], qq[2])), __fadd_rn(__fmul_rn(s[1], qq[1]), __fmul_rn(s[3], qq[3])));
        }
        const float ov = trees4(p);
        if (!(lane & 7)) so[warp * 8 + r0 + (lane >> 4) + ((lane >> 3) & 1) * 2] = __fmul_rn(ov, scale);
    }
    __syncthreads();
    if (tid >= 384) {
        // per-head RMS (no weight), * ssm_norm, swiglu(z, .), destination head of the v-grouped permutation
        float e[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) e[i] = so[lane + 32 * i];
        const float ss = bnk::warp_tree128(__fmul_rn(e[0], e[0]), __fmul_rn(e[1], e[1]), __fmul_rn(e[2], e[2]), __fmul_rn(e[3], e[3]));
        const float inv = __frcp_rn(__fsqrt_rn(__fadd_rn(__fmul_rn(ss, 1.0f / 128.0f), eps)));
        const int d = tid - 384;
        y[place * 128 + d] = __fmul_rn(sz[d], __fmul_rn(__fmul_rn(so[d], inv), nwz));
    }
}

// per-head RMS (no weight; 128 squares, tree), * ssm_norm, swiglu(z, .), v-grouped permutation
// (bonsai_forward.h:559-567, permute_vg.comp:32-42). One warp per SOURCE head.
__global__ void k_gdn_out(int heads, int qk_heads, const float *__restrict__ o, const float *__restrict__ z,
                          const float *__restrict__ ssm_norm, float eps, float *__restrict__ y) {
    bnk::pdl_sync();
    const int hs = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), l = threadIdx.x & 31;
    if (hs >= heads) return;
    const float *orow = o + hs * 128;
    float e[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) e[i] = orow[l + 32 * i];
    const float ss = bnk::warp_tree128(__fmul_rn(e[0], e[0]), __fmul_rn(e[1], e[1]), __fmul_rn(e[2], e[2]), __fmul_rn(e[3], e[3]));
    const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, 128.0f), eps)));
    // destination head hd reads source head hd/sub + nq*(hd%sub)  =>  source hs feeds hd = sub*(hs%nq) + hs/nq
    const int sub = heads / qk_heads;
    const int hd = sub * (hs % qk_heads) + hs / qk_heads;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int d = l + 32 * i;
        const float n = __fmul_rn(__fmul_rn(e[i], inv), ssm_norm[d]);
        y[hd * 128 + d] = __fmul_rn(silu_f(z[hs * 128 + d]), n);
    }
}

// ---- greedy pick: first maximum (Sampler::pick, runtime_vk/bonsai_forward.h:2568-2570) ----------
// the warp's largest value, of equal ones the smallest index (any order of comparisons gives the same)
__device__ __forceinline__ void better_of_warp(float &v, int &i) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        const float w = __shfl_xor_sync(0xFFFFFFFFu, v, s);
        const int k = __shfl_xor_sync(0xFFFFFFFFu, i, s);
        if (w > v || (w == v && k < i)) { v = w; i = k; }
    }
}
__global__ void __launch_bounds__(1024) k_argmax_part(const float *__restrict__ x, int n, float *__restrict__ bv,
                                                      int *__restrict__ bi, bnk::Cols cols) {
    bnk::pdl_sync();
    { const size_t col = blockIdx.z; x = bnk::colp(x, col * cols.arena); bv = bnk::colp(bv, col * cols.arena); bi = bnk::colp(bi, col * cols.arena); }
    __shared__ float sv[32];
    __shared__ int si[32];
    const int t = threadIdx.x;
    float best = -INFINITY; int idx = 0x7FFFFFFF;
    const int step = gridDim.x * 1024;
    for (int i = blockIdx.x * 1024 + t; i < n; i += 4 * step) {        // four loads at a time
        float v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = i + k * step < n ? x[i + k * step] : -INFINITY;
#pragma unroll
        for (int k = 0; k < 4; ++k) if (i + k * step < n && (v[k] > best || (v[k] == best && i + k * step < idx))) { best = v[k]; idx = i + k * step; }
    }
    better_of_warp(best, idx);
    if (!(t & 31)) { sv[t >> 5] = best; si[t >> 5] = idx; }
    __syncthreads();
    if (t < 32) {
        best = sv[t]; idx = si[t];
        better_of_warp(best, idx);
        if (t == 0) { bv[blockIdx.x] = best; bi[blockIdx.x] = idx; }
    }
}
// cand != null (the rows are one shard of the output head, starting at row0): the column's candidate (value, global
// row or 0x7FFFFFFF when no row qualified) also goes to cand[2 * column], for the pick over all shards
__global__ void k_argmax_final(const float *__restrict__ bv, const int *__restrict__ bi, int nparts, int *out, bnk::Cols cols,
                               float *__restrict__ cand, int row0) {
    bnk::pdl_sync();
    { const size_t col = blockIdx.z; bv = bnk::colp(bv, col * cols.arena); bi = bnk::colp(bi, col * cols.arena); out = bnk::colp(out, col * cols.arena); }
    float best = -INFINITY; int idx = 0x7FFFFFFF;
    for (int p = threadIdx.x; p < nparts; p += 32) {
        const float v = bv[p];
        const int k = bi[p];
        if (v > best || (v == best && k < idx)) { best = v; idx = k; }
    }
    better_of_warp(best, idx);
    if (threadIdx.x != 0) return;
    // a row of NaN or -inf never satisfies v > best: fall back to index 0 as the scalar loop does
    out[0] = idx == 0x7FFFFFFF ? 0 : idx;
    if (cand) {
        cand[2 * blockIdx.z] = best;
        reinterpret_cast<int *>(cand)[2 * blockIdx.z + 1] = idx == 0x7FFFFFFF ? idx : idx + row0;
    }
}
// the pick over the shards' candidates: first maximum, shards in ascending row order. One thread per column.
__global__ void k_pick_shards(const float *__restrict__ cands, int n_shards, int ncol, int *__restrict__ out) {
    bnk::pdl_sync();
    const int c = threadIdx.x;
    if (c >= ncol) return;
    float best = -INFINITY; int idx = 0x7FFFFFFF;
    for (int s = 0; s < n_shards; ++s) {
        const float v = cands[(size_t(s) * ncol + c) * 2];
        const int i = reinterpret_cast<const int *>(cands)[(size_t(s) * ncol + c) * 2 + 1];
        if (v > best || (v == best && i < idx)) { best = v; idx = i; }
    }
    out[c] = idx == 0x7FFFFFFF ? 0 : idx;
}

}  // namespace

namespace bnk {

bool g_pdl = true;

void rotate_quant(cudaStream_t st, const float *x, const int32_t *signs, int n, int block, float *y, uint32_t *pack) {
    const float inv = 1.0f / sqrtf(float(block));
    uint32_t *q81 = pack, *table = pack ? pack + size_t(n / 128) * Q81_DWORDS : nullptr;
    const int span = block < 128 ? 128 : block;
    launch(k_rotate_quant, dim3(n / span), dim3(512), size_t(span) * 4 + 512, st, x, signs, span, block, inv, y, q81, table);
}
void embed_rotate(cudaStream_t st, const uint32_t *W, int K, const int *tok_ptr, const int32_t *signs, int block, float *y, Cols cols) {
    launch_spread<k_embed_rotate>(dim3((K + 4095) / 4096, 1, cols.z()), dim3(512), 0, st, W, K, tok_ptr, signs, 31 - __builtin_clz(unsigned(block)), 1.0f / sqrtf(float(block)), y, cols);
}
void rms_norm(cudaStream_t st, const float *x, const float *w, int rows, int cols, float eps, float *y) {
    launch(k_rms_norm, dim3(rows), dim3(256), 0, st, x, w, cols, eps, y); 
}
void add_inplace(cudaStream_t st, float *res, const float *d, int n) { launch(k_add_inplace, dim3((n + 255) / 256), dim3(256), 0, st, res, d, n);  }
void swiglu(cudaStream_t st, const float *a, const float *b, int n, float *y, Cols cols) {
    launch(k_swiglu, dim3((n + 255) / 256, 1, cols.z()), dim3(256), 0, st, a, b, n, y, cols);
}
void gemv_f32_small(cudaStream_t st, const float *W, int M, int K, const float *x, float *out) {
    launch(k_gemv_f32_small, dim3((M + 7) / 8), dim3(256), 0, st, W, M, K, x, out); 
}
void gdn_gates(cudaStream_t st, const float *alpha, const float *beta_raw, const float *dt_bias, const float *ssm_a, int n,
               float *gate, float *beta) {
    launch(k_gdn_gates, dim3(1), dim3(64), 0, st, alpha, beta_raw, dt_bias, ssm_a, n, gate, beta); 
}
void conv_silu(cudaStream_t st, const float *x, const float *w, float *hist, int channels, float *y) {
    launch(k_conv_silu, dim3((channels + 255) / 256), dim3(256), 0, st, x, w, hist, channels, y); 
}
void l2_norm_rows(cudaStream_t st, const float *x, int rows, float eps, float *y) {
    launch(k_l2_norm_rows, dim3((rows + 7) / 8), dim3(256), 0, st, x, rows, eps, y); 
}
void gdn_delta(cudaStream_t st, GdnDims d, const float *q, const float *k, const float *v, const float *gate,
               const float *beta, float *state, float *o) {
    launch(k_gdn_delta, dim3(dim3(d.dim / 8, d.heads)), dim3(256), 0, st, d.heads, d.qk_heads, q, k, v, gate, beta, state, o,
                                                          1.0f / sqrtf(float(d.dim))); 
}
void gdn_core_fused(cudaStream_t st, GdnDims d, int hidden, const float *qkv, const float *conv_w, float *hist0,
                    float *hist1, const int *pos_ptr, const float *x, const float *inv_ptr, const float *norm_w, const float *alpha_w,
                    const float *beta_w, const float *dt_bias, const float *ssm_a, float *state, const float *z,
                    const float *ssm_norm, float eps, float *y, Cols cols, bool alone) {
    static bool attr = false;
    if (!attr) {
        cudaFuncSetAttribute(k_gdn_core<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 3 * 16384 * 4);
        cudaFuncSetAttribute(k_gdn_core<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 3 * 16384 * 4);
        attr = true;
    }
    if (cols.z() > 1) launch_as(g_pdl && !alone, k_gdn_core<2>, dim3(d.heads, 1, cols.z()), dim3(512), size_t(hidden) * 12, st, d.heads, d.qk_heads, hidden, qkv, conv_w, hist0, hist1, pos_ptr, x, inv_ptr,
                                                         norm_w, alpha_w, beta_w, dt_bias, ssm_a, state, z, ssm_norm, eps, y,
                                                         1.0f / sqrtf(float(d.dim)), cols);
    else launch_as(g_pdl && !alone, k_gdn_core<1>, dim3(d.heads, 1, cols.z()), dim3(512), size_t(hidden) * 12, st, d.heads, d.qk_heads, hidden, qkv, conv_w, hist0, hist1, pos_ptr, x, inv_ptr,
                                                         norm_w, alpha_w, beta_w, dt_bias, ssm_a, state, z, ssm_norm, eps, y,
                                                         1.0f / sqrtf(float(d.dim)), cols); 
}
void gdn_out(cudaStream_t st, GdnDims d, const float *o, const float *z, const float *ssm_norm, float eps, float *y) {
    launch(k_gdn_out, dim3((d.heads + 7) / 8), dim3(256), 0, st, d.heads, d.qk_heads, o, z, ssm_norm, eps, y); 
}
void argmax_first(cudaStream_t st, const float *x, int n, int *out_idx, float *scratch_val, int *scratch_idx, Cols cols, float *cand, int row0) {
    const int parts = 64;
    launch(k_argmax_part, dim3(parts, 1, cols.z()), dim3(1024), 0, st, x, n, scratch_val, scratch_idx, cols); 
    launch(k_argmax_final, dim3(1, 1, cols.z()), dim3(32), 0, st, scratch_val, scratch_idx, parts, out_idx, cols, cand, row0);
}
void pick_shards(cudaStream_t st, const float *cands, int n_shards, int ncol, int *out) {
    launch(k_pick_shards, dim3(1), dim3(32), 0, st, cands, n_shards, ncol, out);
}

}  // namespace bnk
