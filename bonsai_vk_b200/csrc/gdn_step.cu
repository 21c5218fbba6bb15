// gdn_step.cu - the gated-delta-net mixer of one layer for one token of one sequence, heads x 4 CTAs in clusters of 4.
//
// What bounds it is the latency between the two projections around it, so everything that does not need the first one's result
// is done while that one is still running: 256 threads of 48 registers and 34 KB leave room for a CTA beside a (lean) projection
// CTA on every SM. The earlier kernel, 512 threads of 126 registers, had to wait for the SM to empty and started its 5 us then.
// The projection releases this grid behind its own dependency wait, so the residual it reads is complete when a CTA starts here:
//     before the wait  state rows into registers, conv taps, the norm of the residual, the two small projections (alpha, beta)
//                      and their gate functions
//     after it         conv + silu, L2 norms, delta rule, head norm over the cluster, ssm_norm, swiglu(z, .), permutation
// From the end of the projection in front to the end of the one behind (9B shape): 12.7 us before, 8.7 us then, of which 0.9 us
// go back in the first projection, which shares its SMs; another 0.7 us went with the cluster barrier behind the outputs (counted
// stores now: a barrier waits for the stores' acknowledgement, then makes a round trip), the divisions of the head's place and two
// divisions by square roots: 48 greedy tokens 51.0 -> 50.2 ms. Arithmetic and its order are those of k_gdn_core (ops.cu).
#include "exchange.cuh"
#include "ops.cuh"
#include "rotate_quant.cuh"

namespace {
using namespace bnk;

constexpr int T = 256, ERR = ERR_STEP_EXCHANGE;

__device__ __forceinline__ void cp16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(uint32_t(__cvta_generic_to_shared(dst))), "l"(src) : "memory");
}
// v to the place of `p` in the shared memory of CTA `cta` of the cluster
__device__ __forceinline__ void push(float *p, int cta, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote(p, cta)), "f"(v) : "memory");
}

__global__ void __cluster_dims__(4, 1, 1) __launch_bounds__(T, 5) k_gdn_step(const GdnStep a) {
    extern __shared__ float4 dyn[];                // [2][hidden / 4]: normed residual, row h of alpha or beta
    __shared__ float red[256], sq[128], sk[128], sv[32], so[128], sgb[2];     // so: the head's 128 outputs, every quarter pushed here by its CTA
    const int h = blockIdx.x >> 2, q4 = blockIdx.x & 3, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int hq = h % a.qk_heads, n4 = a.hidden >> 2;
    __shared__ uint64_t outs;                      // counts the bytes of so[]
    if (tid == 0) {
        const uint32_t b = uint32_t(__cvta_generic_to_shared(&outs));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\nfence.mbarrier_init.release.cluster;" ::"r"(b) : "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], 512;" ::"r"(b) : "memory");
    }
    // "I am running": the matching wait sits in front of the first store into a neighbour's shared memory
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (q4 < 2) {                                  // the first quarter computes the head's alpha, the second its beta
        const float4 *row = reinterpret_cast<const float4 *>((q4 ? a.beta_w : a.alpha_w) + size_t(h) * a.hidden);
        for (int i = tid; i < n4; i += T) cp16(dyn + n4 + i, row + i);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    // state rows (written a token ago, read through L2)
    float *Sr = a.state + (size_t(h) * 128 + q4 * 32 + warp * 4) * 128 + lane;
    float S[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[r][e] = __ldcg(Sr + r * 128 + 32 * e);
    // conv taps: thread t holds q or k channel t, the first warp a v channel too; the three products of the past are added here
    const bool odd = __ldcg(a.pos) & 1;            // a token at position p reads taps from buffer p & 1, writes the other
    const float *hist_rd = odd ? a.hist1 : a.hist0;
    float *hist_wr = odd ? a.hist0 : a.hist1;
    struct Chan { int c; float acc, w3, t1, t2; };
    auto past = [&](int c) {
        const float *s = hist_rd + 3 * size_t(c);
        const float4 w = *reinterpret_cast<const float4 *>(a.conv_w + 4 * size_t(c));
        Chan r;
        r.c = c; r.t1 = __ldcg(s + 1); r.t2 = __ldcg(s + 2); r.w3 = w.w;
        r.acc = __fadd_rn(__fadd_rn(__fmul_rn(w.x, __ldcg(s)), __fmul_rn(w.y, r.t1)), __fmul_rn(w.z, r.t2));
        return r;
    };
    const Chan qk = past((tid < 128 ? 0 : a.qk_heads * 128) + hq * 128 + (tid & 127));
    Chan vc = {};
    if (tid < 32) vc = past(2 * a.qk_heads * 128 + h * 128 + q4 * 32 + tid);
    // norm of the residual (rms_norm.comp order: 256 runs of consecutive values, then the fixed tree)
    if (q4 < 2) {
        const int per = (a.hidden + 255) >> 8;
        float s = 0.0f;
        if (per == 16) {
            const float4 *xv = reinterpret_cast<const float4 *>(a.x + tid * 16);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 v = __ldcg(xv + i);
                s = __fadd_rn(s, __fmul_rn(v.x, v.x)); s = __fadd_rn(s, __fmul_rn(v.y, v.y)); s = __fadd_rn(s, __fmul_rn(v.z, v.z)); s = __fadd_rn(s, __fmul_rn(v.w, v.w));
            }
        } else
            for (int i = 0; i < per; ++i) {
                const int d = tid * per + i;
                if (d < a.hidden) { const float v = __ldcg(a.x + d); s = __fadd_rn(s, __fmul_rn(v, v)); }
            }
        red[tid] = s;
    }
    if (q4 < 2) {
        __syncthreads();
        const float inv = __frcp_rn(__fsqrt_rn(__fadd_rn(mean_of(norm_tree256(red, lane), a.hidden), a.eps)));
        const float4 *xv = reinterpret_cast<const float4 *>(a.x), *nw = reinterpret_cast<const float4 *>(a.norm_w);
        for (int i = tid; i < n4; i += T) {
            const float4 x = __ldcg(xv + i), w = nw[i];
            dyn[i] = make_float4(__fmul_rn(__fmul_rn(x.x, inv), w.x), __fmul_rn(__fmul_rn(x.y, inv), w.y), __fmul_rn(__fmul_rn(x.z, inv), w.z), __fmul_rn(__fmul_rn(x.w, inv), w.w));
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
    }
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");      // all four CTAs of the head are running
    if (q4 < 2 && warp == 7) {
        // lane l takes float4 groups l, l + 32, ... with one fmaf per element, then the xor tree
        float acc = 0.0f;
#pragma unroll 4
        for (int i = lane; i < n4; i += 32) {
            const float4 w4 = dyn[n4 + i], x4 = dyn[i];
            acc = fmaf(w4.x, x4.x, acc); acc = fmaf(w4.y, x4.y, acc); acc = fmaf(w4.z, x4.z, acc); acc = fmaf(w4.w, x4.w, acc);
        }
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(0xFFFFFFFFu, acc, s));
        if (lane < 4) {                            // the gate's factor, from lane c into CTA c
            float r;
            if (q4 == 0) {
                const float al = __fadd_rn(acc, a.dt_bias[h]);
                const float sp = al > 20.0f ? al : log_f(__fadd_rn(1.0f, exp_f(al)));
                r = exp_f(__fmul_rn(sp, a.ssm_a[h]));
            } else r = sigmoid_f(acc);
            push(sgb + q4, lane, r);
        }
        __syncwarp();
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    const float xn = a.qkv[qk.c], zz = warp == 1 ? a.z[h * 128 + q4 * 32 + lane] : 0.0f;
    float xv = 0.0f;
    if (tid < 32) xv = a.qkv[vc.c];
    {
        const float cv = silu_f(__fadd_rn(qk.acc, __fmul_rn(qk.w3, xn)));
        if (tid < 128) sq[tid] = cv; else sk[tid - 128] = cv;
        // one writer per channel: q and k by the first quarter of the first of the value heads that share them
        if (h < a.qk_heads && q4 == 0) { float *w = hist_wr + 3 * size_t(qk.c); w[0] = qk.t1; w[1] = qk.t2; w[2] = xn; }
        if (tid < 32) {
            sv[tid] = silu_f(__fadd_rn(vc.acc, __fmul_rn(vc.w3, xv)));
            float *w = hist_wr + 3 * size_t(vc.c);
            w[0] = vc.t1; w[1] = vc.t2; w[2] = xv;
        }
    }
    __syncthreads();
    float qq[4], kk[4];
    {
#pragma unroll
        for (int e = 0; e < 4; ++e) { qq[e] = sq[lane + 32 * e]; kk[e] = sk[lane + 32 * e]; }
        const float iq = __frcp_rn(__fsqrt_rn(__fadd_rn(warp_tree128(__fmul_rn(qq[0], qq[0]), __fmul_rn(qq[1], qq[1]), __fmul_rn(qq[2], qq[2]), __fmul_rn(qq[3], qq[3])), 1e-12f)));
        const float ik = __frcp_rn(__fsqrt_rn(__fadd_rn(warp_tree128(__fmul_rn(kk[0], kk[0]), __fmul_rn(kk[1], kk[1]), __fmul_rn(kk[2], kk[2]), __fmul_rn(kk[3], kk[3])), 1e-12f)));
#pragma unroll
        for (int e = 0; e < 4; ++e) { qq[e] = __fmul_rn(qq[e], iq); kk[e] = __fmul_rn(kk[e], ik); }
    }
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");      // the head's two factors are in every CTA's sgb[]
    const float eg = sgb[0], bt = sgb[1];
    float pr[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
#pragma unroll
        for (int e = 0; e < 4; ++e) S[r][e] = __fmul_rn(S[r][e], eg);
        pr[r] = __fadd_rn(__fadd_rn(__fmul_rn(S[r][0], kk[0]), __fmul_rn(S[r][2], kk[2])), __fadd_rn(__fmul_rn(S[r][1], kk[1]), __fmul_rn(S[r][3], kk[3])));
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1)               // four trees side by side
#pragma unroll
        for (int r = 0; r < 4; ++r) pr[r] = __fadd_rn(pr[r], __shfl_xor_sync(0xFFFFFFFFu, pr[r], s));
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const float u = __fmul_rn(bt, __fsub_rn(sv[warp * 4 + r], pr[r]));
#pragma unroll
        for (int e = 0; e < 4; ++e) S[r][e] = fmaf(kk[e], u, S[r][e]);
        pr[r] = __fadd_rn(__fadd_rn(__fmul_rn(S[r][0], qq[0]), __fmul_rn(S[r][2], qq[2])), __fadd_rn(__fmul_rn(S[r][1], qq[1]), __fmul_rn(S[r][3], qq[3])));
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1)
#pragma unroll
        for (int r = 0; r < 4; ++r) pr[r] = __fadd_rn(pr[r], __shfl_xor_sync(0xFFFFFFFFu, pr[r], s));
    if (lane < 16) {                               // lane = (CTA, row): push this warp's four outputs into all four so[]
        const int row = lane & 3;
        const float o = __fmul_rn(row == 0 ? pr[0] : (row == 1 ? pr[1] : (row == 2 ? pr[2] : pr[3])), a.scale);
        put(remote(so + q4 * 32 + warp * 4 + row, lane >> 2), o, remote(&outs, lane >> 2));
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int e = 0; e < 4; ++e) Sr[r * 128 + 32 * e] = S[r][e];
    float gz = 0.0f, nw = 0.0f;                    // this CTA's share of the gate, and its place, off the tail (a double-precision exp; divisions)
    int hd = 0;
    if (warp == 1) { gz = silu_f(zz); nw = a.ssm_norm[q4 * 32 + lane]; hd = a.heads / a.qk_heads * hq + h / a.qk_heads; }
    // the head's 128 outputs are in every CTA's so[] (counted stores: a cluster barrier waits for their acknowledgement first)
    if (!arrived<ERR>(uint32_t(__cvta_generic_to_shared(&outs)), a.err))
        asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");      // (given up: the others end first)
    if (warp == 1) {
        float e[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) e[i] = so[i * 32 + lane];
        const float ss = warp_tree128(__fmul_rn(e[0], e[0]), __fmul_rn(e[1], e[1]), __fmul_rn(e[2], e[2]), __fmul_rn(e[3], e[3]));
        const float inv = __frcp_rn(__fsqrt_rn(__fadd_rn(__fmul_rn(ss, 1.0f / 128.0f), a.eps)));
        const int d = q4 * 32 + lane;
        a.y[hd * 128 + d] = __fmul_rn(gz, __fmul_rn(__fmul_rn(so[d], inv), nw));
    }
}

}  // namespace

namespace bnk {

cudaError_t launch_wait_selftest_step(cudaStream_t st, int *err) {
    BN_COUNT(1);
    k_wait_selftest_exchange<ERR><<<1, 32, 0, st>>>(err);
    return cudaGetLastError();
}

void gdn_step(cudaStream_t st, const GdnStep &a, bool alone) {
    static bool attr = false;
    if (!attr) {
        cudaFuncSetAttribute(k_gdn_step, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * 16384 * 4);
        cudaFuncSetAttribute(k_gdn_step, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        attr = true;
    }
    launch_as(g_pdl && !alone, k_gdn_step, dim3(a.heads * 4), dim3(T), size_t(a.hidden) * 8, st, a);
}

}  // namespace bnk
