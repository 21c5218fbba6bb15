// attn.cu - decode attention over the quantised KV cache: prep (head norm, rope, cache insert), scores, softmax numerators,
// PV over splits of the keys, combine. The order of every floating-point sum is part of the contract with the CPU oracle (the
// file is compiled without fused-multiply-add contraction; fmaf is written where one is meant).
//
// One query token reads every key and value once: 71 MB at 32 768 keys, 11 us of memory. What bounds the kernels is CUDA-core
// work, because the contract fixes one fused multiply-add per (key, head, dim) for the scores and a rounded product and a
// rounded sum per (key, head, dim), keys ascending, for PV; and below a few thousand keys the five launches' latency.
#include "attn_octet.cuh"

namespace {
using namespace bnk;

__device__ __forceinline__ void pdl_early() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// q8_0 of one 32-element block held one value per lane (recipe: attn_norm_rope2.comp:39-49,184-217). Division and rounding are
// those of the projections' quantiser (rotate_quant.cuh); the largest magnitude of the warp is one instruction, which leaves NaNs out
// as fmaxf does.
__device__ __forceinline__ void q80_store(float v, int lane, int8_t *codes, uint16_t *scale) {
    float amax;
    asm("redux.sync.max.abs.f32 %0, %1, 0xffffffff;" : "=f"(amax) : "f"(v));
    const bool some = amax > 1e-35f;
    const float d = some ? div127(amax) : 0.0f, id = some ? __frcp_rn(d) : 0.0f;
    codes[lane] = int8_t(code_byte(__fmul_rn(v, id)));
    if (lane == 0) *scale = (uint16_t)float_to_half_bits(d);
}

// one CTA per head row (n_head query rows, then n_kv key rows) and column or token; a thread per dim (head_dim = 256), and a ninth warp
// for the serial sum, beside which the others deal with the row that needs no norm (gate, or quantised V).
// Query rows: RMS norm * weight, NeoX rope on the first n_rot dims, fp16 rounding, gate split; the row's softmax maximum is
// cleared. Key rows: the same norm / rope, then cache insert (fp16 or q8_0) of K and of the raw V row.
// Columns (cols.n > 0) are sequences; tokens (the op-level insert) are consecutive positions whose rows follow each other, and
// only the last one's query is kept. The rope factors need the position only (set before the pass: the rule at bnk::launch)
// and are worked out before the wait: a double-precision power, sine and cosine are most of this kernel's chain.
// What bounds it is that chain (256 dependent additions, 0.7 us) and the quantiser behind it. With V quantised last, by divisions and five
// shuffles, a key row's CTA took 1.5 us from the dependency wait on; an insert and an attention over 64 keys 9.72 -> 9.53 us, 500 keys
// 10.18 -> 9.93.
constexpr int PREP_T = 288;
__global__ void __launch_bounds__(PREP_T) k_attn_prep(AttnDims a, AttnPos where, const float *__restrict__ qg, const float *__restrict__ kin,
                                                   const float *__restrict__ vin, const float *__restrict__ qn_w, const float *__restrict__ kn_w,
                                                   KvLayer kv, float *__restrict__ q16f, float *__restrict__ gate, unsigned *__restrict__ mx, Cols cols) {
    const int tok = cols.n > 0 ? 0 : blockIdx.z;
    if (cols.n > 0) { const size_t col = blockIdx.z; qg = colp(qg, col * cols.arena); kin = colp(kin, col * cols.arena); vin = colp(vin, col * cols.arena); where.ptr = colp(where.ptr, col * cols.arena); kv.k_data = colp(kv.k_data, col * cols.kv); kv.k_scale = colp(kv.k_scale, col * cols.kv); kv.v_data = colp(kv.v_data, col * cols.kv); kv.v_scale = colp(kv.v_scale, col * cols.kv); q16f = colp(q16f, col * cols.arena); gate = colp(gate, col * cols.arena); mx = colp(mx, col * cols.arena); }
    __shared__ __align__(16) float part[256];
    __shared__ float sx[256];
    __shared__ float ssum;
    const int d = threadIdx.x, hd = a.head_dim, w = blockIdx.x;
    const bool is_q = w < a.n_head, elem = d < 256;
    const int h = is_q ? w : w - a.n_head;
    if (is_q && tok + 1 < int(gridDim.z) && cols.n == 0) return;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int pos = where.get() + tok;
    const float *nwp = is_q ? qn_w : kn_w;
    const int half = a.n_rot >> 1, p = d < half ? d : d - half, pd = d < half ? d + half : d - half;
    const float nw = elem ? nwp[d] : 0.0f, inv_hd = 1.0f / float(hd);      // (a power of two: the product with it is the quotient)
    float c = 1.0f, s = 0.0f, nwr = 0.0f;
    if (d < a.n_rot) {                             // (the ninth warp has no dims: n_rot <= 256)
        const float ex = __fdiv_rn(__fmul_rn(-2.0f, float(p)), float(a.n_rot));
        const float th = float(pow(double(a.rope_base), double(ex)));
        const float ang = __fmul_rn(float(pos), th);
        c = float(cos(double(ang))); s = float(sin(double(ang)));
        nwr = nwp[pd];
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const float *src = is_q ? qg + size_t(h) * 2 * hd : kin + (size_t(tok) * a.n_kv + h) * hd;
    const size_t row = (size_t(pos) * a.n_kv + h) * hd;
    const int lane = d & 31, blk = d >> 5;
    float x = 0.0f, vr = 0.0f;
    if (elem) {
        x = src[d];
        vr = is_q ? src[hd + d] : vin[(size_t(tok) * a.n_kv + h) * hd + d];
        sx[d] = x;
        part[d] = __fmul_rn(x, x);
    }
    __syncthreads();
    if (elem) {
        if (is_q) {
            gate[size_t(h) * hd + d] = vr;
            if (d == 0) mx[h] = 0u;
        } else if (a.v_mode == 1) reinterpret_cast<__half *>(kv.v_data)[row + d] = __float2half_rn(vr);
        else q80_store(vr, lane, reinterpret_cast<int8_t *>(kv.v_data) + row + blk * 32, kv.v_scale + row / 32 + blk);
    } else if (lane == 0) {
        // the 256 squares are added serially in ascending order, as the reference's CPU mirror adds them
        // (attn_vk.h:102-108), so that the fp16 operands below are the mirror's bit for bit
        float acc = 0.0f;
        const float4 *p4 = reinterpret_cast<const float4 *>(part);
        float4 v[8], n[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = p4[i];
#pragma unroll
        for (int b = 0; b < 8; ++b) {              // (the next eight loads in front of these additions)
#pragma unroll
            for (int i = 0; i < 8; ++i) n[i] = p4[min(b + 1, 7) * 8 + i];
#pragma unroll
            for (int i = 0; i < 8; ++i) { acc = __fadd_rn(acc, v[i].x); acc = __fadd_rn(acc, v[i].y); acc = __fadd_rn(acc, v[i].z); acc = __fadd_rn(acc, v[i].w); }
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = n[i];
        }
        ssum = acc;
    }
    __syncthreads();
    if (!elem) return;
    const float inv = __frcp_rn(__fsqrt_rn(__fadd_rn(__fmul_rn(ssum, inv_hd), a.eps)));
    float y = __fmul_rn(__fmul_rn(x, inv), nw);
    if (d < a.n_rot) {
        const float xp = __fmul_rn(__fmul_rn(sx[pd], inv), nwr);
        y = d < half ? __fsub_rn(__fmul_rn(y, c), __fmul_rn(xp, s)) : __fadd_rn(__fmul_rn(y, c), __fmul_rn(xp, s));
    }
    if (is_q) {
        q16f[size_t(h) * hd + d] = __half2float(__float2half_rn(y));
        return;
    }
    if (a.k_mode == 1) reinterpret_cast<__half *>(kv.k_data)[row + d] = __float2half_rn(y);
    else q80_store(y, lane, reinterpret_cast<int8_t *>(kv.k_data) + row + blk * 32, kv.k_scale + row / 32 + blk);
}

// Scores: a warp takes octets of consecutive keys of one kv head (attn_octet.cuh), the next octet's rows in flight while it works
// on one; the gqa query heads of the kv head share every K row (merge idea: attn_qk_softmax_gqa.glslh:15-24). The maximum of the
// scaled scores of each head goes to mx with one atomic per CTA (a maximum has no order).
// Measured at 32 768 keys: 21 us with one octet per warp (its query loads and latency were most of it), 18 us so.
template <int KMODE>
__global__ void __launch_bounds__(256, 2) k_attn_scores4(AttnDims a, AttnPos where, const float *__restrict__ q16f, KvLayer kv,
                                                         float *__restrict__ score, float scale, unsigned *__restrict__ mx, Cols cols) {
    { const size_t col = blockIdx.z; q16f = colp(q16f, col * cols.arena); where.ptr = colp(where.ptr, col * cols.arena); kv.k_data = colp(kv.k_data, col * cols.kv); kv.k_scale = colp(kv.k_scale, col * cols.kv); score = colp(score, col * cols.arena); mx = colp(mx, col * cols.arena); }
    __shared__ unsigned smx[4];
    if (threadIdx.x < 4) smx[threadIdx.x] = 0u;
    const int kvh = blockIdx.y, lane = threadIdx.x & 31, hd = a.head_dim;
    pdl_early();
    const int nfill = where.get() + 1, step = gridDim.x * 64;
    int jb = (blockIdx.x * 8 + (threadIdx.x >> 5)) * 8;
    if (blockIdx.x * 64 >= nfill) return;          // (the whole CTA)
    KeyOctet<KMODE> keys;
    if (jb < nfill) keys.fetch(kv, a.n_kv, kvh, hd, lane, jb, nfill - 1);
    f32pair qd[4][8];
    load_queries<4>(q16f, kvh * 4, hd, lane, qd);
    const f32pair magic2 = pair_of(CODE_MAGIC, CODE_MAGIC);
    float best = -INFINITY;                        // of head lane & 3
    for (; jb < nfill; jb += step) {
        float v[32];                               // v[4u + g]: (key jb + u, head g)
        octet_parts<4>(keys, qd, magic2, v);
        if (jb + step < nfill) keys.fetch(kv, a.n_kv, kvh, hd, lane, jb + step, nfill - 1);
        octet_totals<32>(v, lane);                 // lane l: value l
        const int j = jb + (lane >> 2);
        if (j < nfill) {
            score[size_t(kvh * 4 + (lane & 3)) * a.cap + j] = v[0];
            best = fmaxf(best, __fmul_rn(v[0], scale));
        }
    }
#pragma unroll
    for (int s = 4; s < 32; s <<= 1) best = fmaxf(best, __shfl_xor_sync(0xFFFFFFFFu, best, s));
    __syncthreads();                               // smx is cleared
    if (lane < 4) atomicMax(smx + lane, ord(best));
    __syncthreads();
    if (threadIdx.x < 4) atomicMax(mx + kvh * 4 + threadIdx.x, smx[threadIdx.x]);
}

// The same scores for any number of query heads per kv head: a warp takes 8 consecutive keys of one kv head and walks the query
// heads one after the other - per (key, head) the same fmaf chain over the lane's 8 dims and the same xor-butterfly tree.
template <int KMODE>
__global__ void __launch_bounds__(256) k_attn_scores_any(AttnDims a, int gqa, AttnPos where, const float *__restrict__ q16f, KvLayer kv,
                                                         float *__restrict__ score, float scale, unsigned *__restrict__ mx, Cols cols) {
    { const size_t col = blockIdx.z; q16f = colp(q16f, col * cols.arena); where.ptr = colp(where.ptr, col * cols.arena); kv.k_data = colp(kv.k_data, col * cols.kv); kv.k_scale = colp(kv.k_scale, col * cols.kv); score = colp(score, col * cols.arena); mx = colp(mx, col * cols.arena); }
    pdl_early();
    const int kvh = blockIdx.y, lane = threadIdx.x & 31, hd = a.head_dim;
    const int nfill = where.get() + 1;
    const int jb = (blockIdx.x * 8 + (threadIdx.x >> 5)) * 8;
    if (jb >= nfill) return;
    float kf[8][8];                              // this lane's 8 dims of the 8 keys
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        const int j = min(jb + u, nfill - 1);
        const size_t row = (size_t(j) * a.n_kv + kvh) * hd;
        if (KMODE == 1) {
            const uint4 raw = *reinterpret_cast<const uint4 *>(reinterpret_cast<const __half *>(kv.k_data) + row + lane * 8);
            const __half2 *h2 = reinterpret_cast<const __half2 *>(&raw);
#pragma unroll
            for (int e = 0; e < 4; ++e) { const float2 f = __half22float2(h2[e]); kf[u][2 * e] = f.x; kf[u][2 * e + 1] = f.y; }
        } else {
            const uint2 raw = *reinterpret_cast<const uint2 *>(reinterpret_cast<const int8_t *>(kv.k_data) + row + lane * 8);
            const float sc = half_bits_to_float(kv.k_scale[row / 32 + (lane >> 2)]);
            const int8_t *c8 = reinterpret_cast<const int8_t *>(&raw);
#pragma unroll
            for (int e = 0; e < 8; ++e) kf[u][e] = __fmul_rn(sc, float(int(c8[e])));
        }
    }
    for (int g = 0; g < gqa; ++g) {
        const float4 *qv = reinterpret_cast<const float4 *>(q16f + size_t(kvh * gqa + g) * hd + lane * 8);
        const float4 q0 = qv[0], q1 = qv[1];
        const float qe[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
        float best = -INFINITY;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            float acc = 0.0f;
#pragma unroll
            for (int e = 0; e < 8; ++e) acc = fmaf(qe[e], kf[u][e], acc);
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(0xFFFFFFFFu, acc, off));
            if (jb + u < nfill) {
                if (lane == u) score[size_t(kvh * gqa + g) * a.cap + jb + u] = acc;
                best = fmaxf(best, __fmul_rn(acc, scale));
            }
        }
        if (lane == 0) atomicMax(mx + kvh * gqa + g, ord(best));
    }
}

// Softmax numerators and their sums, spread over 8 CTAs per head with the summation order of one 1024-thread CTA: "virtual
// thread" vt adds the keys vt, vt+1024, ... ascending, and the 1024 partial sums are combined by the fixed tree p[i] += p[i + s],
// s = 512 .. 1. A CTA owns 16 residues modulo 128 and all eight virtual threads of each, so the tree's first three steps stay
// inside it; the last seven, over 128 sums per head, are evaluated by every warp that needs the total (k_attn_pv): no barrier
// between CTAs (a cluster barrier or an arrival counter here cost 1.5 us). The exponentials of a virtual thread's next eight
// keys are evaluated by eight real threads and added in order from shared memory.
// With several columns one CTA per head and column is enough to fill the GPU, and a virtual thread is a real one (PARTS = 1):
// 32 columns of a short cache are 512 CTAs then instead of 4096 with a few keys each (21 -> 6 us).
constexpr int EXPSUM_PARTS = 8;
template <int PARTS>
__global__ void __launch_bounds__(1024) k_attn_expsum(AttnDims a, AttnPos where, const float *__restrict__ score, float scale, float *__restrict__ pe,
                                                      float *__restrict__ partial, const unsigned *__restrict__ mxp, Cols cols) {
    { const size_t col = blockIdx.z; where.ptr = colp(where.ptr, col * cols.arena); score = colp(score, col * cols.arena); pe = colp(pe, col * cols.arena); partial = colp(partial, col * cols.arena); mxp = colp(mxp, col * cols.arena); }
    if (PARTS == 1) {
        __shared__ float all[1024];
        const int h = blockIdx.x, t = threadIdx.x;
        pdl_early();
        const int nfill = where.get() + 1;
        const float mx = unord(mxp[h]);
        const float *sr = score + size_t(h) * a.cap;
        float *pr = pe + size_t(h) * a.cap;
        float sum = 0.0f;
#pragma unroll 2
        for (int j = t; j < nfill; j += 1024) {
            const float e = exp_f(__fsub_rn(__fmul_rn(sr[j], scale), mx));
            pr[j] = e;
            sum = __fadd_rn(sum, e);
        }
        all[t] = sum;
        __syncthreads();
        if (t < 128) {
            float v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = all[128 * k + t];
            partial[size_t(h) * 128 + t] = __fadd_rn(__fadd_rn(__fadd_rn(v[0], v[4]), __fadd_rn(v[2], v[6])), __fadd_rn(__fadd_rn(v[1], v[5]), __fadd_rn(v[3], v[7])));
        }
        return;
    }
    __shared__ float ex[2][1024];
    __shared__ float sums[128];
    const int h = blockIdx.x, t = threadIdx.x, i = t & 127, vt = (i >> 4) * 128 + blockIdx.y * 16 + (i & 15), sub = t >> 7;
    pdl_early();
    const int nfill = where.get() + 1;
    const float mx = unord(mxp[h]);
    const float *sr = score + size_t(h) * a.cap;
    float *pr = pe + size_t(h) * a.cap;
    float sum = 0.0f;
    int buf = 0;
    for (int j0 = 0; j0 < nfill; j0 += 8192, buf ^= 1) {
        const int j = j0 + vt + 1024 * sub;
        float e = 0.0f;
        if (j < nfill) { e = exp_f(__fsub_rn(__fmul_rn(sr[j], scale), mx)); pr[j] = e; }
        ex[buf][t] = e;
        __syncthreads();
        if (sub == 0) {
#pragma unroll
            for (int s = 0; s < 8; ++s) if (j0 + vt + 1024 * s < nfill) sum = __fadd_rn(sum, ex[buf][128 * s + t]);
        }
    }
    if (sub == 0) sums[t] = sum;
    __syncthreads();
    if (t < 16) {
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = sums[16 * k + t];
        partial[size_t(h) * 128 + blockIdx.y * 16 + t] = __fadd_rn(__fadd_rn(__fadd_rn(v[0], v[4]), __fadd_rn(v[2], v[6])), __fadd_rn(__fadd_rn(v[1], v[5]), __fadd_rn(v[3], v[7])));
    }
}

// PV: grid (n_kv, splits, columns); a thread owns DPT output dims of all GQA heads of the kv head and walks the split's keys
// ascending: acc = acc + p*v with p = fp16(e / total), product and sum rounded (attn_pv_q8v.comp:85-112). V comes through a
// ring of two 32-key tiles in shared memory (cp.async; small enough that the 1024 CTAs of a long context are all resident),
// probabilities are staged as one [key][head] row, so a key costs a thread three shared-memory loads whatever the number of
// dims. The rounded products of two dims are one fma.f32x2 with -0 (x * y - 0 is the rounded product; the -0 is an
// argument `nz`, because the assembler contracts a packed multiply, or one with a constant -0, with the packed add behind it). DPT: two or four
// where splits and columns fill the GPU (pv_any), else 1 (short caches: the keys' serial chain is what takes the time).
constexpr int PV_TILE = 32;
template <int GQA, int DPT, int VMODE>
__global__ void __launch_bounds__(256 / DPT) k_attn_pv(AttnDims a, AttnPos where, const float *__restrict__ pe, const float *__restrict__ partial,
                                                       KvLayer kv, int splits, float *__restrict__ part, float nz, Cols cols) {
    constexpr int T = 256 / DPT, ROW = VMODE == 0 ? 256 : 512, VB = PV_TILE * ROW, TILE_BYTES = VB + (VMODE == 0 ? PV_TILE * 16 : 0);
    extern __shared__ __align__(16) unsigned char dyn[];
    { const size_t col = blockIdx.z; pe = colp(pe, col * cols.arena); partial = colp(partial, col * cols.arena); where.ptr = colp(where.ptr, col * cols.arena); kv.v_data = colp(kv.v_data, col * cols.kv); kv.v_scale = colp(kv.v_scale, col * cols.kv); part = colp(part, col * cols.arena); }
    float *ps = reinterpret_cast<float *>(dyn + 2 * TILE_BYTES);           // [key][GQA]
    const int kvh = blockIdx.x, sp = blockIdx.y, tid = threadIdx.x, hd = a.head_dim;
    pdl_early();
    const int nfill = where.get() + 1, per = (nfill + splits - 1) / splits, j0 = sp * per, n = max(0, min(nfill, j0 + per) - j0);
    if (n == 0) return;                            // k_attn_combine leaves empty splits out (the first is never empty)
    auto fetch = [&](int jb, int buf) {            // a tile of keys from jb of the split on
        const uint32_t dst = uint32_t(__cvta_generic_to_shared(dyn)) + buf * TILE_BYTES;
        const int m = min(PV_TILE, n - jb);
        const unsigned char *vd = reinterpret_cast<const unsigned char *>(kv.v_data) + (size_t(j0 + jb) * a.n_kv + kvh) * ROW;
        for (int i = tid; i < m * (ROW / 16); i += T) {
            const int k = i / (ROW / 16), b = (i % (ROW / 16)) * 16;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + k * ROW + b), "l"(vd + size_t(k) * a.n_kv * ROW + b) : "memory");
        }
        if (VMODE == 0)
            for (int k = tid; k < m; k += T)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + VB + k * 16), "l"(kv.v_scale + (size_t(j0 + jb + k) * a.n_kv + kvh) * (hd / 32)) : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0, 0);
    if (n > PV_TILE) fetch(PV_TILE, 1);
    float tot[GQA], pt[GQA][4];
#pragma unroll
    for (int g = 0; g < GQA; ++g)
#pragma unroll
        for (int k = 0; k < 4; ++k) pt[g][k] = partial[size_t(kvh * GQA + g) * 128 + (tid & 31) + 32 * k];
#pragma unroll
    for (int g = 0; g < GQA; ++g) tot[g] = warp_tree128(pt[g][0], pt[g][1], pt[g][2], pt[g][3]);
    for (int k = tid; k < n; k += T) {
        const float *e = pe + size_t(kvh * GQA) * a.cap + j0 + k;
        float x[GQA];
#pragma unroll
        for (int g = 0; g < GQA; ++g) x[g] = e[size_t(g) * a.cap];
#pragma unroll
        for (int g = 0; g < GQA; ++g) ps[k * GQA + g] = __half2float(__float2half_rn(__fdiv_rn(x[g], tot[g])));
    }
    f32pair acc2[GQA][2];
    float acc[GQA];
#pragma unroll
    for (int g = 0; g < GQA; ++g) { acc2[g][0] = acc2[g][1] = 0ull; acc[g] = 0.0f; }
    const f32pair nzero = pair_of(nz, nz);
    const f32pair magic2 = pair_of(CODE_MAGIC, CODE_MAGIC);
    int buf = 0;
    for (int jb = 0; jb < n; jb += PV_TILE, buf ^= 1) {
        if (jb + PV_TILE < n) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        const unsigned char *tile = dyn + buf * TILE_BYTES;
        const int lim = min(PV_TILE, n - jb);
        const float *pk = ps + jb * GQA;
#pragma unroll 4
        for (int k = 0; k < lim; ++k) {
            float p[GQA];
            if (GQA % 4 == 0) {
#pragma unroll
                for (int g = 0; g < GQA / 4; ++g) {
                    const float4 f = *reinterpret_cast<const float4 *>(pk + k * GQA + 4 * g);
                    p[(4 * g) % GQA] = f.x; p[(4 * g + 1) % GQA] = f.y; p[(4 * g + 2) % GQA] = f.z; p[(4 * g + 3) % GQA] = f.w;
                }
            } else {
#pragma unroll
                for (int g = 0; g < GQA; ++g) p[g] = pk[k * GQA + g];
            }
            if (DPT == 4) {
                f32pair v01, v23;
                if (VMODE == 0) {
                    const float s = half_bits_to_float(*reinterpret_cast<const uint16_t *>(tile + VB + k * 16 + (tid >> 3) * 2));
                    const uint32_t c = *reinterpret_cast<const uint32_t *>(tile + k * 256 + tid * 4) ^ 0x80808080u;
                    v01 = pair_mul(pair_of(s, s), pair_sub(pair_of(code_f<0>(c), code_f<1>(c)), magic2));
                    v23 = pair_mul(pair_of(s, s), pair_sub(pair_of(code_f<2>(c), code_f<3>(c)), magic2));
                } else {
                    const uint2 c = *reinterpret_cast<const uint2 *>(tile + k * 512 + tid * 8);
                    v01 = pair_of(half_bits_to_float(c.x), half_bits_to_float(c.x >> 16));
                    v23 = pair_of(half_bits_to_float(c.y), half_bits_to_float(c.y >> 16));
                }
#pragma unroll
                for (int g = 0; g < GQA; ++g) {
                    const f32pair pp = pair_of(p[g], p[g]);
                    acc2[g][0] = pair_add(acc2[g][0], pair_fma(pp, v01, nzero));
                    acc2[g][1] = pair_add(acc2[g][1], pair_fma(pp, v23, nzero));
                }
            } else if (DPT == 2) {
                f32pair v;
                if (VMODE == 0) {
                    const float s = half_bits_to_float(*reinterpret_cast<const uint16_t *>(tile + VB + k * 16 + (tid >> 4) * 2));
                    const uint32_t c = uint32_t(*reinterpret_cast<const uint16_t *>(tile + k * 256 + tid * 2)) ^ 0x8080u;
                    v = pair_mul(pair_of(s, s), pair_sub(pair_of(code_f<0>(c), code_f<1>(c)), magic2));
                } else {
                    const uint32_t c = *reinterpret_cast<const uint32_t *>(tile + k * 512 + tid * 4);
                    v = pair_of(half_bits_to_float(c), half_bits_to_float(c >> 16));
                }
#pragma unroll
                for (int g = 0; g < GQA; ++g) acc2[g][0] = pair_add(acc2[g][0], pair_fma(pair_of(p[g], p[g]), v, nzero));
            } else {
                float v;
                if (VMODE == 0) {
                    const float s = half_bits_to_float(*reinterpret_cast<const uint16_t *>(tile + VB + k * 16 + (tid >> 5) * 2));
                    v = __fmul_rn(s, __fsub_rn(__uint_as_float(0x4B000000u | (uint32_t(tile[k * 256 + tid]) ^ 0x80u)), CODE_MAGIC));
                } else v = half_bits_to_float(*reinterpret_cast<const uint16_t *>(tile + k * 512 + tid * 2));
#pragma unroll
                for (int g = 0; g < GQA; ++g) acc[g] = __fadd_rn(acc[g], __fmul_rn(p[g], v));
            }
        }
        if (jb + 2 * PV_TILE < n) { __syncthreads(); fetch(jb + 2 * PV_TILE, buf); }
    }
#pragma unroll
    for (int g = 0; g < GQA; ++g) {
        float *o = part + (size_t(sp) * a.n_head + kvh * GQA + g) * hd + tid * DPT;
        if (DPT == 4) *reinterpret_cast<ulonglong2 *>(o) = make_ulonglong2(acc2[g][0], acc2[g][1]);
        else if (DPT == 2) *reinterpret_cast<f32pair *>(o) = acc2[g][0];
        else o[0] = acc[g];
    }
}

constexpr int COMBINE_FEW = 8;
// combine the splits ascending, then the sigmoid gate: 32 outputs per CTA, whose partials come in with all threads at once and
// are added in order from shared memory (16 CTAs walking them in batches of 64 loads took 9 us for 64 splits, 24 us for 256).
// Clears the row maxima again: the kept query may attend once more, over other positions.
__global__ void __launch_bounds__(256) k_attn_combine(AttnDims a, AttnPos where, const float *__restrict__ part, int splits,
                                                      const float *__restrict__ gate, float *__restrict__ pregate, float *__restrict__ gated,
                                                      unsigned *__restrict__ mx, Cols cols) {
    { const size_t col = blockIdx.z; part = colp(part, col * cols.arena); where.ptr = colp(where.ptr, col * cols.arena); gate = colp(gate, col * cols.arena); pregate = colp(pregate, col * cols.arena); gated = colp(gated, col * cols.arena); mx = colp(mx, col * cols.arena); }
    __shared__ float sp[256][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, i = blockIdx.x * 32 + lane, n = a.n_head * a.head_dim;
    pdl_early();
    const int nfill = where.get() + 1, per = (nfill + splits - 1) / splits, used = (nfill + per - 1) / per;      // splits with keys
    for (int s = warp; s < used; s += 8) sp[s][lane] = part[size_t(s) * n + i];
    float gt = 0.0f;
    if (warp == 0) gt = __fdiv_rn(1.0f, __fadd_rn(1.0f, exp_f(-gate[i])));
    __syncthreads();
    if (warp) return;
    float acc = sp[0][lane];
    int s = 1;
    for (; s + 8 <= used; s += 8) {
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = sp[s + u][lane];
#pragma unroll
        for (int u = 0; u < 8; ++u) acc = __fadd_rn(acc, v[u]);
    }
    for (; s < used; ++s) acc = __fadd_rn(acc, sp[s][lane]);
    if (pregate) pregate[i] = acc;
    gated[i] = __fmul_rn(acc, gt);
    if (i % a.head_dim == 0) mx[i / a.head_dim] = 0u;
}

// the same for few splits and several columns: a thread per output (32 columns x 8 splits: 512 CTAs instead of 4096, 8 -> 4 us)
__global__ void __launch_bounds__(256) k_attn_combine_few(AttnDims a, AttnPos where, const float *__restrict__ part, int splits,
                                                          const float *__restrict__ gate, float *__restrict__ pregate, float *__restrict__ gated,
                                                          unsigned *__restrict__ mx, Cols cols) {
    { const size_t col = blockIdx.z; part = colp(part, col * cols.arena); where.ptr = colp(where.ptr, col * cols.arena); gate = colp(gate, col * cols.arena); pregate = colp(pregate, col * cols.arena); gated = colp(gated, col * cols.arena); mx = colp(mx, col * cols.arena); }
    const int i = blockIdx.x * 256 + threadIdx.x, n = a.n_head * a.head_dim;
    pdl_early();
    if (i >= n) return;
    const int nfill = where.get() + 1, per = (nfill + splits - 1) / splits, used = (nfill + per - 1) / per;      // splits with keys
    const float gt = __fdiv_rn(1.0f, __fadd_rn(1.0f, exp_f(-gate[i])));
    float v[COMBINE_FEW];
#pragma unroll
    for (int s = 0; s < COMBINE_FEW; ++s) v[s] = s < used ? part[size_t(s) * n + i] : 0.0f;
    float acc = v[0];
#pragma unroll
    for (int s = 1; s < COMBINE_FEW; ++s) if (s < used) acc = __fadd_rn(acc, v[s]);
    if (pregate) pregate[i] = acc;
    gated[i] = __fmul_rn(acc, gt);
    if (i % a.head_dim == 0) mx[i / a.head_dim] = 0u;
}

template <int GQA, int DPT, int VMODE>
void pv(cudaStream_t st, AttnDims a, AttnPos where, const float *pe, const float *partial, KvLayer kv, int splits, float *part, Cols cols) {
    constexpr int TILE_BYTES = PV_TILE * (VMODE == 0 ? 256 + 16 : 512);
    const size_t smem = 2 * TILE_BYTES + size_t(GQA) * ((a.cap + splits - 1) / splits) * 4;
    // (1024 CTAs at 32 768 positions: seven per SM everywhere instead of up to eleven; of two warps, four dims a thread, 57 -> 49 us a layer)
    launch_spread<k_attn_pv<GQA, DPT, VMODE>, 8>(dim3(a.n_kv, splits, cols.z()), dim3(256 / DPT), smem, st, a, where, pe, partial, kv, splits, part, -0.0f, cols);
}
template <int GQA>
void pv_any(cudaStream_t st, AttnDims a, AttnPos where, const float *pe, const float *partial, KvLayer kv, int splits, float *part, Cols cols) {
    // Several dims per thread from three CTAs per two SMs on (8 columns x 8 splits x 4 heads: 28 -> 22 us). Two dims is twice the warps
    // for an eighth more instructions. Four heads a value gain by it up to 4096 CTAs (32 000 keys, four dims and two: 44.0 and 42.1 us with
    // four kv heads, 23.7 and 22.1 with one; 8 columns at 2048 positions 85.6 and 83.1 us a block; 16 columns at 8192, 4096 CTAs, the same,
    // 32 columns 356 and 362) - unless one column's CTAs are more than four an SM and leave a tenth of the last round empty, which
    // the fewer warps hide (three kv heads, 768 CTAs: 12 000 of 16 384 keys 21.8 and 22.3). Eight heads a value issue enough with four
    // dims: two up to three CTAs an SM (256 CTAs, 32 000 keys 48.8 and 48.0; 384, three sequences at 8192 253.5 and 251.6 us a stage; 512,
    // 768, 2048, 32 000 keys 73.6 and 75.1, 103.0 and 105.4, 245 and 252). Fewer heads have too little work per value (two heads: 50.6
    // and 51.4).
    const size_t ctas = size_t(a.n_kv) * splits * cols.z(), per = (ctas + 147) / 148;
    const bool uneven = cols.z() == 1 && per > 4 && ctas * 10 < per * 148 * 9;
    const int dims = ctas < 200 ? 1 : ((GQA == 4 && ctas <= 4096 && !uneven) || (GQA == 8 && per <= 3) ? 2 : 4);
    constexpr int TWO = GQA >= 4 ? 2 : 4;
    if (a.v_mode == 0) {
        if (dims == 1) pv<GQA, 1, 0>(st, a, where, pe, partial, kv, splits, part, cols);
        else if (dims == 2) pv<GQA, TWO, 0>(st, a, where, pe, partial, kv, splits, part, cols);
        else pv<GQA, 4, 0>(st, a, where, pe, partial, kv, splits, part, cols);
    } else if (dims == 1) pv<GQA, 1, 1>(st, a, where, pe, partial, kv, splits, part, cols);
    else if (dims == 2) pv<GQA, TWO, 1>(st, a, where, pe, partial, kv, splits, part, cols);
    else pv<GQA, 4, 1>(st, a, where, pe, partial, kv, splits, part, cols);
}

}  // namespace

namespace bnk {

void attn_prep(cudaStream_t st, AttnDims a, const float *qg, const float *kin, const float *vin, const float *qn_w,
               const float *kn_w, AttnPos where, KvLayer kv, float *q16f, float *gate, float *esum, Cols cols, int tokens) {
    unsigned *mx = reinterpret_cast<unsigned *>(esum + size_t(a.n_head) * 128);
    const dim3 grid(a.n_head + a.n_kv, 1, cols.n > 0 ? cols.z() : tokens);
    // (one token's few CTAs run beside the projection in front of them)
    if (grid.z == 1) launch(k_attn_prep, grid, dim3(PREP_T), 0, st, a, where, qg, kin, vin, qn_w, kn_w, kv, q16f, gate, mx, cols);
    else launch_spread<k_attn_prep>(grid, dim3(PREP_T), 0, st, a, where, qg, kin, vin, qn_w, kn_w, kv, q16f, gate, mx, cols);
}
void attn_decode(cudaStream_t st, AttnDims a, const float *q16f, const float *gate, AttnPos where, KvLayer kv,
                 float *score, float *p16f, float *esum, float *pv_part, int splits, float *pregate, float *gated, int *err, Cols cols) {
    // one query token: one launch up to 8192 positions. With several columns (serving, prefill) the chain of kernels below
    // fills the GPU better than 64 large CTAs per column (8 columns at 2048 positions: 2.46 against 2.62 ms a pass).
    if (cols.z() == 1 && attn_cluster(st, a, q16f, gate, where, kv, splits, pregate, gated, cols, err)) return;
    // grids are sized for the cache capacity; CTAs beyond the filled prefix return at once.
    // esum: [n_head][128] partial softmax sums, then n_head row maxima (cleared by attn_prep and again by the combine kernel)
    unsigned *mx = reinterpret_cast<unsigned *>(esum + size_t(a.n_head) * 128);
    const float scale = 1.0f / sqrtf(float(a.head_dim));
    const int gqa = a.n_head / a.n_kv;            // 1, 2, 4 or 8 (checked where the dimensions enter: bn_model_create, the attention ABI)
    if (gqa == 4) {
        // octets per warp: as many as leave two CTAs per SM, at most 8
        const size_t ctas = size_t((a.cap + 63) / 64) * a.n_kv * cols.z();
        int rounds = int((ctas + 295) / 296);
        rounds = rounds < 1 ? 1 : (rounds > 8 ? 8 : rounds);
        const dim3 sg(((a.cap + 63) / 64 + rounds - 1) / rounds, a.n_kv, cols.z());
        if (a.k_mode == 1) launch_spread<k_attn_scores4<1>>(sg, dim3(256), 0, st, a, where, q16f, kv, score, scale, mx, cols);
        else launch_spread<k_attn_scores4<0>>(sg, dim3(256), 0, st, a, where, q16f, kv, score, scale, mx, cols);
    } else {
        const dim3 sg((a.cap + 63) / 64, a.n_kv, cols.z());
        if (a.k_mode == 1) launch_spread<k_attn_scores_any<1>>(sg, dim3(256), 0, st, a, gqa, where, q16f, kv, score, scale, mx, cols);
        else launch_spread<k_attn_scores_any<0>>(sg, dim3(256), 0, st, a, gqa, where, q16f, kv, score, scale, mx, cols);
    }
    // eight CTAs per head while all of them are resident at once (two per SM)
    if (a.n_head * EXPSUM_PARTS * cols.z() <= 296) launch_spread<k_attn_expsum<EXPSUM_PARTS>>(dim3(a.n_head, EXPSUM_PARTS, cols.z()), dim3(1024), 0, st, a, where, score, scale, p16f, esum, mx, cols);
    else launch_spread<k_attn_expsum<1>>(dim3(a.n_head, 1, cols.z()), dim3(1024), 0, st, a, where, score, scale, p16f, esum, mx, cols);
    if (gqa == 4) pv_any<4>(st, a, where, p16f, esum, kv, splits, pv_part, cols);
    else if (gqa == 1) pv_any<1>(st, a, where, p16f, esum, kv, splits, pv_part, cols);
    else if (gqa == 2) pv_any<2>(st, a, where, p16f, esum, kv, splits, pv_part, cols);
    else pv_any<8>(st, a, where, p16f, esum, kv, splits, pv_part, cols);
    if (splits <= COMBINE_FEW && cols.z() > 1)
        launch_spread<k_attn_combine_few>(dim3((a.n_head * a.head_dim + 255) / 256, 1, cols.z()), dim3(256), 0, st, a, where, pv_part, splits, gate, pregate, gated, mx, cols);
    else
        launch_spread<k_attn_combine>(dim3(a.n_head * a.head_dim / 32, 1, cols.z()), dim3(256), 0, st, a, where, pv_part, splits, gate, pregate, gated, mx, cols);
}

}  // namespace bnk
