// gdn_seq.cu - the gated-delta-net mixer of one layer for several consecutive positions of ONE sequence (batched prefill).
// Only the delta rule itself is sequential in time. Everything in front of it (alpha / beta projections and gates, conv + silu,
// L2 norms) and behind it (head norm, ssm_norm, swiglu(z, .), permutation) is done for all positions side by side, and the
// delta rule walks the positions inside one kernel with its state rows in registers. Before, the fused single-position core
// was launched once per position, about 12 us each: more than half of the 43 ms of a 100-token prompt, which now takes 14 ms.
// Arithmetic and its order are those of k_gdn_core (ops.cu).
#include "ops.cuh"
#include "rotate_quant.cuh"

namespace {

// grid (2 x heads, positions / 4), 256 threads. Even CTAs: conv + silu + L2 norms of four positions of one value head (and of q / k
// head h, where h is one). Odd CTAs: alpha and beta of one value head for the same positions, one warp per dot: as a second task of
// the even CTAs' warps the dots took 18 us with the rest; side by side, 4 us.
constexpr int PP = 4;
__global__ void __launch_bounds__(256) k_gdn_seq_pre(bnk::GdnSeq a, int n) {
    __shared__ float sq[PP][256];                  // q and k channels of the positions
    const int h = blockIdx.x >> 1, c0 = blockIdx.y * PP, np = min(PP, n - c0), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool own_qk = h < a.qk_heads;
    if (blockIdx.x & 1) {
        const int p = warp >> 1, beta = warp & 1, n4 = a.hidden / 4;
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (p >= np) return;
        const float inv = bnk::colp(a.inv, (c0 + p) * a.stride)[0];
        const float4 *xv = reinterpret_cast<const float4 *>(bnk::colp(a.x, (c0 + p) * a.stride)), *nw = reinterpret_cast<const float4 *>(a.norm_w);
        const float4 *wr = reinterpret_cast<const float4 *>((beta ? a.beta_w : a.alpha_w) + size_t(h) * a.hidden);
        float acc = 0.0f;
#pragma unroll 8
        for (int i = lane; i < n4; i += 32) {
            const float4 x4 = xv[i], w4 = nw[i], r4 = wr[i];
            acc = fmaf(r4.x, __fmul_rn(__fmul_rn(x4.x, inv), w4.x), acc); acc = fmaf(r4.y, __fmul_rn(__fmul_rn(x4.y, inv), w4.y), acc);
            acc = fmaf(r4.z, __fmul_rn(__fmul_rn(x4.z, inv), w4.z), acc); acc = fmaf(r4.w, __fmul_rn(__fmul_rn(x4.w, inv), w4.w), acc);
        }
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(0xFFFFFFFFu, acc, s));
        if (lane == 0) {
            if (beta) bnk::colp(a.bt, (c0 + p) * a.stride)[h] = sigmoid_f(acc);
            else {
                const float al = __fadd_rn(acc, a.dt_bias[h]);
                const float sp = al > 20.0f ? al : log_f(__fadd_rn(1.0f, exp_f(al)));
                bnk::colp(a.eg, (c0 + p) * a.stride)[h] = exp_f(__fmul_rn(sp, a.ssm_a[h]));
            }
        }
        return;
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const float *hist = (a.pos[0] & 1) ? a.hist1 : a.hist0;
    // input of channel ch at position c of the block; positions before it are the history taps
    auto in = [&](int ch, int c) { return c < 0 ? hist[3 * size_t(ch) + 3 + c] : bnk::colp(a.qkv, c * a.stride)[ch]; };
    auto conv = [&](int ch, int c) {
        const float *wc = a.conv_w + 4 * size_t(ch);
        float acc = __fmul_rn(wc[0], in(ch, c - 3));
        acc = __fadd_rn(acc, __fmul_rn(wc[1], in(ch, c - 2)));
        acc = __fadd_rn(acc, __fmul_rn(wc[2], in(ch, c - 1)));
        acc = __fadd_rn(acc, __fmul_rn(wc[3], in(ch, c)));
        return silu_f(acc);
    };
    for (int i = tid; i < 128 * np; i += 256) {
        const int p = i >> 7, d = i & 127;
        bnk::colp(a.v, (c0 + p) * a.stride)[h * 128 + d] = conv(2 * a.qk_heads * 128 + h * 128 + d, c0 + p);
    }
    if (own_qk)
#pragma unroll 4
        for (int p = 0; p < np; ++p) sq[p][tid] = conv((tid < 128 ? 0 : a.qk_heads * 128) + h * 128 + (tid & 127), c0 + p);
    __syncthreads();
    if (own_qk && warp < 2 * np) {                 // L2 norms: warp = (position, q / k)
        const int p = warp >> 1, k = warp & 1;
        const float *s = sq[p] + k * 128;
        const float e0 = s[lane], e1 = s[lane + 32], e2 = s[lane + 64], e3 = s[lane + 96];
        const float i = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(bnk::warp_tree128(__fmul_rn(e0, e0), __fmul_rn(e1, e1), __fmul_rn(e2, e2), __fmul_rn(e3, e3)), 1e-12f)));
        float *y = bnk::colp(a.qk, (c0 + p) * a.stride) + (k * a.qk_heads + h) * 128;
        y[lane] = __fmul_rn(e0, i); y[lane + 32] = __fmul_rn(e1, i); y[lane + 64] = __fmul_rn(e2, i); y[lane + 96] = __fmul_rn(e3, i);
    }
}

// grid heads x 4: 32 state rows of a head, four per warp, in registers for all positions. The head's q and k of every position
// are staged in shared memory first. Per position a row's chain is two 128-value trees (prediction, output) with the update
// between; the output trees of one position run beside the prediction trees of the next, eight trees on nine shuffles: a level's
// two values change hands between the lanes that go on with one and those that go on with the other (the shuffles' throughput
// bounds the loop: with five per tree and two rows per warp 1000 cycles a position, now 400).
// One CTA per SM (launch_spread): launched early, beside the CTAs of the kernel in front, several landed on one SM while
// others stayed idle (37 against 19 us in the 9B shape's schedule of 32 positions).
__device__ __forceinline__ float fold(float a, float b, int s, bool up) {    // lanes with bit s clear: a + a', set: b + b' (a', b' of lane ^ s)
    return __fadd_rn(up ? b : a, __shfl_xor_sync(0xFFFFFFFFu, up ? a : b, s));
}
__global__ void __launch_bounds__(256) k_gdn_seq(bnk::GdnSeq a, int n) {
    extern __shared__ float dyn[];                 // [n][256]: q then k; [n][32] v; [n][2] gates
    float *sv = dyn + n * 256, *sg = sv + n * 32;
    const int h = blockIdx.x >> 2, q4 = blockIdx.x & 3, hq = h % a.qk_heads, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    float S[4][4];                                 // (the kernel in front writes no state)
    float *Sr = a.state + (size_t(h) * 128 + q4 * 32 + warp * 4) * 128 + lane;
    asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[r][e] = Sr[r * 128 + 32 * e];
    for (int i = tid; i < n * 64; i += 256) {
        const int c = i >> 6, d = (i & 63) * 4;
        const float *src = bnk::colp(a.qk, c * a.stride) + ((d < 128 ? 0 : a.qk_heads) + hq) * 128 + (d & 127);
        *reinterpret_cast<float4 *>(dyn + c * 256 + d) = *reinterpret_cast<const float4 *>(src);
    }
    for (int i = tid; i < n * 32; i += 256) sv[i] = bnk::colp(a.v, (i >> 5) * a.stride)[h * 128 + q4 * 32 + (i & 31)];
    if (tid < n) { sg[2 * tid] = bnk::colp(a.eg, tid * a.stride)[h]; sg[2 * tid + 1] = bnk::colp(a.bt, tid * a.stride)[h]; }
    __syncthreads();
    float ov[4] = {0.0f, 0.0f, 0.0f, 0.0f};        // this lane's part of the previous position's outputs
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
    for (int c = 0; c <= n; ++c) {
        float k[4], q[4], pr[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (c < n) {
            const float *qk = dyn + c * 256 + lane;
            const float eg = sg[2 * c];
#pragma unroll
            for (int e = 0; e < 4; ++e) { q[e] = qk[32 * e]; k[e] = qk[128 + 32 * e]; }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
#pragma unroll
                for (int e = 0; e < 4; ++e) S[r][e] = __fmul_rn(S[r][e], eg);
                pr[r] = __fadd_rn(__fadd_rn(__fmul_rn(S[r][0], k[0]), __fmul_rn(S[r][2], k[2])), __fadd_rn(__fmul_rn(S[r][1], k[1]), __fmul_rn(S[r][3], k[3])));
            }
        }
        // lanes 0..15: predictions, 16..31: outputs; within them bit 3 and bit 2 name the row
        float x[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) x[r] = fold(pr[r], ov[r], 16, b4);
        float t = fold(fold(x[0], x[1], 8, b3), fold(x[2], x[3], 8, b3), 4, b2);
        t = __fadd_rn(t, __shfl_xor_sync(0xFFFFFFFFu, t, 2));
        t = __fadd_rn(t, __shfl_xor_sync(0xFFFFFFFFu, t, 1));
        if (c && (lane & 19) == 16) bnk::colp(a.o, (c - 1) * a.stride)[h * 128 + q4 * 32 + warp * 4 + ((lane >> 3) & 1) + ((lane >> 1) & 2)] = __fmul_rn(t, a.scale);
        if (c < n) {
            const float bt = sg[2 * c + 1];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float u = __fmul_rn(bt, __fsub_rn(sv[c * 32 + warp * 4 + r], __shfl_sync(0xFFFFFFFFu, t, (r & 1) * 8 + (r >> 1) * 4)));
#pragma unroll
                for (int e = 0; e < 4; ++e) S[r][e] = fmaf(k[e], u, S[r][e]);
                ov[r] = __fadd_rn(__fadd_rn(__fmul_rn(S[r][0], q[0]), __fmul_rn(S[r][2], q[2])), __fadd_rn(__fmul_rn(S[r][1], q[1]), __fmul_rn(S[r][3], q[3])));
            }
        }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int e = 0; e < 4; ++e) Sr[r * 128 + 32 * e] = S[r][e];
}

// Both tap buffers end as position after position leaves them: the last three inputs of every channel in the buffer of the next
// position's parity, the three in front of the last position in the other one (which a single position does not touch). Any pass
// over one of these positions again reads what a token-serial prompt would have left it. All reads of a channel come before its
// stores: with an odd n the second buffer is the one being read.
__device__ __forceinline__ void seq_taps(const bnk::GdnSeq &a, int n, int ch) {
    const int p0 = a.pos[0];
    const float *rd = ((p0 & 1) ? a.hist1 : a.hist0) + 3 * size_t(ch);
    float *wr = (((p0 + n) & 1) ? a.hist1 : a.hist0) + 3 * size_t(ch), *wr2 = (((p0 + n) & 1) ? a.hist0 : a.hist1) + 3 * size_t(ch);
    float t[4];                                    // inputs n - 4 .. n - 1 (the first one only for n > 1)
#pragma unroll
    for (int i = 0; i < 4; ++i) { const int c = n - 4 + i; t[i] = c < -3 ? 0.0f : (c < 0 ? rd[3 + c] : bnk::colp(a.qkv, c * a.stride)[ch]); }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        wr[i] = t[i + 1];
        if (n > 1) wr2[i] = t[i];
    }
}
// one warp per (source head, position): per-head RMS, * ssm_norm, swiglu(z, .), v-grouped permutation (k_gdn_out, ops.cu). The CTAs
// behind those of the heads bring the conv taps up to date, a channel per thread (in k_gdn_seq, whose chain is the longer one, the
// second buffer's stores cost 0.6 us a launch, 0.4 % of a 100-token prompt; here nothing).
__global__ void __launch_bounds__(256) k_gdn_seq_post(bnk::GdnSeq a, const float *__restrict__ z, const float *__restrict__ ssm_norm, float eps, float *__restrict__ y) {
    const int hs = blockIdx.x * 8 + (threadIdx.x >> 5), l = threadIdx.x & 31;
    const size_t off = blockIdx.y * a.stride;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int own = (a.heads + 7) / 8;
    if (int(blockIdx.x) >= own) {
        const int ch = ((blockIdx.x - own) * gridDim.y + blockIdx.y) * 256 + threadIdx.x;
        if (ch < (2 * a.qk_heads + a.heads) * 128) seq_taps(a, gridDim.y, ch);
        return;
    }
    if (hs >= a.heads) return;
    const float *o = bnk::colp(a.o, off) + hs * 128;
    float e[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) e[i] = o[l + 32 * i];
    const float ss = bnk::warp_tree128(__fmul_rn(e[0], e[0]), __fmul_rn(e[1], e[1]), __fmul_rn(e[2], e[2]), __fmul_rn(e[3], e[3]));
    const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, 128.0f), eps)));
    const int sub = a.heads / a.qk_heads, hd = sub * (hs % a.qk_heads) + hs / a.qk_heads;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int d = l + 32 * i;
        bnk::colp(y, off)[hd * 128 + d] = __fmul_rn(silu_f(bnk::colp(z, off)[hs * 128 + d]), __fmul_rn(__fmul_rn(e[i], inv), ssm_norm[d]));
    }
}

}  // namespace

namespace bnk {

void gdn_sequence(cudaStream_t st, const GdnSeq &a, int n, const float *z, const float *ssm_norm, float eps, float *y) {
    launch_spread<k_gdn_seq_pre>(dim3(a.heads * 2, (n + PP - 1) / PP), dim3(256), 0, st, a, n);
    launch_spread<k_gdn_seq>(dim3(a.heads * 4), dim3(256), size_t(n) * 290 * 4, st, a, n);       // at most 32 positions: 37 KB
    const int taps = ((2 * a.qk_heads + a.heads + 1) / 2 + n - 1) / n;     // CTAs of 256 channels, over n rows
    launch_spread<k_gdn_seq_post>(dim3((a.heads + 7) / 8 + taps, n), dim3(256), 0, st, a, z, ssm_norm, eps, y);
}

}  // namespace bnk
