// attn_cluster.cu - decode attention of one query token in ONE launch, for caches of up to 8192 positions: a thread-block cluster
// of 16 CTAs per kv head (or several, for parts of its query heads) keeps scores, numerators, probabilities and partial outputs in distributed shared memory. The chain of
// four kernels in attn.cu costs about 3.5 us of latency per kernel on the device and 2.2 us each on the host, whatever the
// length; here the CTAs exchange four times (maxima, numerators, sums, partial outputs) by stores into each other's shared memory that
// an mbarrier over there counts, so an exchange costs one way across the cluster. As plain stores and a cluster barrier it cost the
// stores' acknowledgement and the barrier's round trip as well, some 0.4 us each: with the insert in front 1501 keys (8192 positions)
// 11.5 -> 9.9 us, 4096 keys 17.4 -> 15.3, 64 keys 9.5 -> 7.9 (the scales of V by asynchronous copies, 0.4 us of it, included).
// What bounds it: latency below 1000 keys, then instruction issue of scores and values on its 64 SMs.
//
// Arithmetic and the order of every sum are those of attn.cu (and of the CPU oracle): scores by an fmaf chain over 8 dims per
// lane and the xor tree; 1024 "virtual threads" of ascending partial softmax sums combined by the tree 512 .. 1; probabilities
// rounded to fp16; PV per split of the keys, ascending, product and sum rounded; splits added ascending; sigmoid gate.
//
// Split of the work. The number of splits is fixed by the capacity (1, 8 or 64), so the 16 CTAs share them as
//     64 splits: 4 per CTA, all 256 dims        8 splits: one per two CTAs, 128 dims each        1 split: 16 dims per CTA
// A CTA scores the keys of its splits (its share of them where CTAs share a split) and brings their V slice into shared memory
// with cp.async meanwhile. Numerators go to the CTAs that share the split and to the CTA that sums their residue modulo 128.
#include "attn_octet.cuh"
#include "exchange.cuh"

#include <cstdlib>

namespace {
using namespace bnk;

constexpr int CL = 16, T = 512, RL = 128 / CL, HD = 256, SMEM_MAX = 227 << 10;

struct Shape { int nsl, spc, D, rcap; };       // CTAs per split, splits per CTA, dims per CTA, keys of a CTA's splits at most
__host__ __device__ __forceinline__ Shape shape_of(int splits, int cap) {
    Shape s;
    s.nsl = splits >= CL ? 1 : CL / splits;
    s.spc = splits >= CL ? splits / CL : 1;
    s.D = HD / s.nsl;
    s.rcap = s.spc * ((cap + splits - 1) / splits);
    return s;
}
struct Lay { int v, vsc, eg, eb, sums, mx, part, red, bars, total; };
template <int GQA, int VMODE> __host__ __device__ __forceinline__ Lay layout(const Shape &s, int splits, int cap) {
    Lay l;
    int o = 0;
    l.v = o; o += s.rcap * s.D * (VMODE ? 2 : 1);
    o = (o + 15) & ~15;
    l.vsc = o; if (!VMODE) o += s.rcap * (s.D >= 32 ? s.D / 32 : 1) * 2;
    o = (o + 15) & ~15;
    l.eg = o; o += s.rcap * GQA * 4;
    o = (o + 15) & ~15;
    l.eb = o; o += GQA * ((cap + 127) / 128) * RL * 4;
    l.sums = o; o += GQA * 128 * 4;
    l.mx = o; o += CL * GQA * 4;
    o = (o + 15) & ~15;
    l.part = o; o += splits * (GQA * HD / CL) * 4;
    l.red = o; o += 2 * GQA * 4;
    l.bars = o = (o + 7) & ~7; o += 4 * 8;
    l.total = o;
    return l;
}

constexpr int ERR = ERR_ATTN_EXCHANGE;

struct Args {
    AttnDims a;
    AttnPos where;
    const float *q16f, *gate;
    KvLayer kv;
    int splits;
    int log_parts;                             // clusters per kv head, GQA of its query heads each
    float scale, nz;                           // nz = -0: see k_attn_pv in attn.cu
    float *pregate, *gated;
    Cols cols;
    int *err;
};

template <int GQA, int KMODE, int VMODE>
__global__ void __launch_bounds__(T, 1) k_attn_cluster(const Args g) {
    constexpr int G = GQA < 4 ? GQA : 4, NV = 8 * G, GSH = G == 4 ? 0 : (G == 2 ? 1 : 2), OPC = GQA * HD / CL;
    extern __shared__ __align__(16) unsigned char smem[];
    const size_t col = blockIdx.z;
    const AttnDims &a = g.a;
    const float *q16f = colp(g.q16f, col * g.cols.arena), *gate = colp(g.gate, col * g.cols.arena);
    const KvLayer kv = {colp(static_cast<char *>(g.kv.k_data), col * g.cols.kv), colp(g.kv.k_scale, col * g.cols.kv),
                        colp(static_cast<char *>(g.kv.v_data), col * g.cols.kv), colp(g.kv.v_scale, col * g.cols.kv)};
    const AttnPos where = {colp(g.where.ptr, col * g.cols.arena), g.where.imm};
    const Shape sh = shape_of(g.splits, a.cap);
    const Lay L = layout<GQA, VMODE>(sh, g.splits, a.cap);
    unsigned char *vs = smem + L.v;
    uint16_t *vsc = reinterpret_cast<uint16_t *>(smem + L.vsc);
    float *eg = reinterpret_cast<float *>(smem + L.eg), *eb = reinterpret_cast<float *>(smem + L.eb), *sums = reinterpret_cast<float *>(smem + L.sums);
    float *mxs = reinterpret_cast<float *>(smem + L.mx), *part = reinterpret_cast<float *>(smem + L.part);
    unsigned *red = reinterpret_cast<unsigned *>(smem + L.red);
    float *tot = reinterpret_cast<float *>(red + GQA);
    const int rank = blockIdx.x, kvh = blockIdx.y >> g.log_parts, head0 = blockIdx.y * GQA, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // (the position was set before the pass: the rule at bnk::launch)
    const int nfill = where.get() + 1, splits = g.splits, per = (nfill + splits - 1) / splits, used = (nfill + per - 1) / per;
    const int grp = rank / sh.nsl, sl = rank - grp * sh.nsl;             // which splits, which dims of them
    const int r0 = min(nfill, grp * sh.spc * per), n = min(nfill, (grp + 1) * sh.spc * per) - r0;
    const int o0 = r0 + n * sl / sh.nsl, o1 = r0 + n * (sl + 1) / sh.nsl; // keys this CTA scores
    // the four exchanges and the bytes that come with each: maxima; numerators (of this CTA's residues, and of a split that it shares);
    // sums; partial outputs
    const uint32_t bars = uint32_t(__cvta_generic_to_shared(smem + L.bars));
    if (tid == 0) {
        const int own = (nfill >> 7) * RL + max(0, min(RL, (nfill & 127) - rank * RL));
        const int bytes[4] = {CL * GQA * 4, (own + (sh.nsl > 1 ? n : 0)) * GQA * 4, GQA * 128 * 4, used * OPC * 4};
#pragma unroll
        for (int i = 0; i < 4; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bars + i * 8));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 4; ++i) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bars + i * 8), "r"(bytes[i]) : "memory");
    }
    if (tid < GQA) red[tid] = 0u;
    // "I am running, my barriers count": waited for before the first store into a neighbour
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    bool alive = true;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    // ---- K octets of the first round and the V slice on their way ------------------------------------------------------
    // (KeyOctet::fetch and, below, load_queries in place: called, they make the fp16 kernel up to 2 % slower, 11.7 against 11.4 us at
    // 1501 keys with the insert)
    KeyOctet<KMODE> keys;
    auto fetch = [&](int jo) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const size_t row = (size_t(min(jo + u, o1 - 1)) * a.n_kv + kvh) * HD;
            if (KMODE == 1) keys.raw16[u] = *reinterpret_cast<const uint4 *>(reinterpret_cast<const __half *>(kv.k_data) + row + lane * 8);
            else {
                keys.raw8[u] = *reinterpret_cast<const uint2 *>(reinterpret_cast<const int8_t *>(kv.k_data) + row + lane * 8);
                keys.sc[u] = kv.k_scale[row / 32 + (lane >> 2)];
            }
        }
    };
    int jb = o0 + warp * 8;
    if (jb < o1) fetch(jb);
    {
        const int rb = sh.D * (VMODE ? 2 : 1), ch = rb / 16;              // bytes and 16-byte pieces of a key's slice
        const unsigned char *src = static_cast<const unsigned char *>(kv.v_data) + ((size_t(r0) * a.n_kv + kvh) * HD + sl * sh.D) * (VMODE ? 2 : 1);
        const size_t stride = size_t(a.n_kv) * HD * (VMODE ? 2 : 1);
        const uint32_t dst = uint32_t(__cvta_generic_to_shared(vs));
        const int csh = 31 - __clz(ch);
        for (int i = tid; i < n << csh; i += T) {
            const int k = i >> csh, b = (i & (ch - 1)) * 16;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + k * rb + b), "l"(src + k * stride + b) : "memory");
        }
    }
    // its scales: eight, four (with the copies) or one per key (through a register, stored behind the scores)
    const int nsc = sh.D >= 32 ? sh.D / 32 : 1, ssh = 31 - __clz(nsc);
    const uint16_t *vsrc = kv.v_scale + (size_t(r0) * a.n_kv + kvh) * (HD / 32) + sl * sh.D / 32;
    uint16_t vs0 = 0;
    if (VMODE == 0) {
        const uint32_t dst = uint32_t(__cvta_generic_to_shared(vsc));
        if (nsc == 1) { if (tid < n) vs0 = vsrc[size_t(tid) * a.n_kv * (HD / 32)]; }
        else
            for (int i = tid; i < n; i += T) {
                const uint16_t *s = vsrc + size_t(i) * a.n_kv * (HD / 32);
                if (nsc == 8) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * 16), "l"(s) : "memory");
                else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + i * 8), "l"(s) : "memory");
            }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");

    // ---- scores ------------------------------------------------------------------------------------------------------------
    const f32pair magic2 = pair_of(CODE_MAGIC, CODE_MAGIC);
#pragma unroll 1
    for (int hp = 0; hp < GQA / G; ++hp) {
        if (hp && o0 + warp * 8 < o1) { jb = o0 + warp * 8; fetch(jb); }
        f32pair qd[G][8];
#pragma unroll
        for (int h = 0; h < G; ++h) {
            const float4 *qv = reinterpret_cast<const float4 *>(q16f + size_t(head0 + hp * G + h) * HD + lane * 8);
            const float4 q0 = qv[0], q1 = qv[1];
            qd[h][0] = pair_of(q0.x, q0.x); qd[h][1] = pair_of(q0.y, q0.y); qd[h][2] = pair_of(q0.z, q0.z); qd[h][3] = pair_of(q0.w, q0.w);
            qd[h][4] = pair_of(q1.x, q1.x); qd[h][5] = pair_of(q1.y, q1.y); qd[h][6] = pair_of(q1.z, q1.z); qd[h][7] = pair_of(q1.w, q1.w);
        }
        float best = -INFINITY;                // of head hp * G + ((lane & 3) >> GSH)
        for (jb = o0 + warp * 8; jb < o1; jb += T / 4) {
            float v[NV];                       // v[G u + h]: this lane's part of (key jb + u, head h)
            octet_parts<G>(keys, qd, magic2, v);
            if (jb + T / 4 < o1) fetch(jb + T / 4);
            octet_totals<NV>(v, lane);
            const int j = jb + (lane >> 2);
            if (j < o1) {
                eg[(j - r0) * GQA + hp * G + ((lane & 3) >> GSH)] = v[0];
                best = fmaxf(best, __fmul_rn(v[0], g.scale));
            }
        }
#pragma unroll
        for (int s = 4; s < 32; s <<= 1) best = fmaxf(best, __shfl_xor_sync(0xFFFFFFFFu, best, s));
        if (hp == 0) __syncthreads();          // red is cleared
        if (lane < 4) atomicMax(red + hp * G + (lane >> GSH), ord(best));
    }
    if (VMODE == 0 && nsc == 1)
        for (int i = tid; i < n; i += T) vsc[i] = i == tid ? vs0 : vsrc[size_t(i) * a.n_kv * (HD / 32)];
    __syncthreads();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // every CTA is running
    for (int i = tid; i < CL * GQA; i += T) put(remote(mxs + rank * GQA + i % GQA, i / GQA), unord(red[i % GQA]), remote(smem + L.bars, i / GQA));
    // (the gate of the outputs that this CTA finishes, off the tail)
    const int orow = head0 * HD + rank * OPC + tid;
    float gt = 0.0f;
    if (tid < OPC) gt = __fdiv_rn(1.0f, __fadd_rn(1.0f, exp_f(-gate[orow])));
    alive = arrived<ERR>(bars, g.err);

    // ---- numerators: to the CTAs that share the split and to the one that sums the residue ------------------------------------
    {
        float mx = -INFINITY;
        const int h = tid % GQA;               // (T is a multiple of GQA: a thread stays with one head)
#pragma unroll
        for (int r = 0; r < CL; ++r) mx = fmaxf(mx, mxs[r * GQA + h]);
        for (int i = (o0 - r0) * GQA + tid; i < (o1 - r0) * GQA; i += T) {
            // (o0 - r0) * GQA is a multiple of GQA, so i % GQA == h
            const int j = r0 + i / GQA, res = j & 127;
            const float e = exp_f(__fsub_rn(__fmul_rn(eg[i], g.scale), mx));
            put(remote(eb + (h * ((a.cap + 127) >> 7) + (j >> 7)) * RL + res % RL, res / RL), e, remote(smem + L.bars + 8, res / RL));
            if (sh.nsl == 1) eg[i] = e;
            else for (int p = 0; p < sh.nsl; ++p) put(remote(eg + i, grp * sh.nsl + p), e, remote(smem + L.bars + 8, grp * sh.nsl + p));
        }
    }
    if (alive) alive = arrived<ERR>(bars + 8, g.err);
    // ---- softmax sums: thread (head, residue, a) adds the keys of virtual thread 128 a + residue ascending ---------------------
    if (tid < GQA * RL * 8) {
        const int av = tid & 7, rl = (tid >> 3) % RL, h = (tid >> 3) / RL, res = rank * RL + rl;
        const float *p = eb + h * ((a.cap + 127) >> 7) * RL + rl;
        float s = 0.0f;
        for (int m = av; m * 128 + res < nfill; m += 8) s = __fadd_rn(s, p[m * RL]);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) s = __fadd_rn(s, __shfl_xor_sync(0xFFFFFFFFu, s, o));      // tree steps 512, 256, 128
        put(remote(sums + h * 128 + res, av), s, remote(smem + L.bars + 16, av));
        put(remote(sums + h * 128 + res, av + 8), s, remote(smem + L.bars + 16, av + 8));
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (alive) alive = arrived<ERR>(bars + 16, g.err);
    if (warp < GQA) {
        const float *p = sums + warp * 128 + lane;
        float s = __fadd_rn(__fadd_rn(p[0], p[64]), __fadd_rn(p[32], p[96]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s = __fadd_rn(s, __shfl_xor_sync(0xFFFFFFFFu, s, o));
        if (lane == 0) tot[warp] = s;
    }
    __syncthreads();
    for (int i = tid; i < n * GQA; i += T) eg[i] = __half2float(__float2half_rn(__fdiv_rn(eg[i], tot[i % GQA])));
    __syncthreads();

    // ---- PV ----------------------------------------------------------------------------------------------------------------------
    auto probs = [&](int k, float (&p)[GQA]) {
        if (GQA % 4 == 0) {
#pragma unroll
            for (int i = 0; i < GQA / 4; ++i) {
                const float4 f = *reinterpret_cast<const float4 *>(eg + k * GQA + 4 * i);
                p[(4 * i) % GQA] = f.x; p[(4 * i + 1) % GQA] = f.y; p[(4 * i + 2) % GQA] = f.z; p[(4 * i + 3) % GQA] = f.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < GQA; ++i) p[i] = eg[k * GQA + i];
        }
    };
    auto value = [&](int k, int d) {           // dim d of the CTA's slice
        if (VMODE) return half_bits_to_float(reinterpret_cast<const uint16_t *>(vs)[k * sh.D + d]);
        const float s = half_bits_to_float(vsc[(k << ssh) + (d >> 5)]);
        return __fmul_rn(s, __fsub_rn(__uint_as_float(0x4B000000u | (uint32_t(vs[k * sh.D + d]) ^ 0x80u)), CODE_MAGIC));
    };
    if (sh.nsl == 1) {                         // a thread: two dims, all heads, one of four splits
        const int s = tid >> 7, d = (tid & 127) * 2, k0 = s * per, k1 = min(n, k0 + per);
        const f32pair nzero = pair_of(g.nz, g.nz);
        f32pair acc[GQA];
#pragma unroll
        for (int h = 0; h < GQA; ++h) acc[h] = 0ull;
#pragma unroll 4
        for (int k = k0; k < k1; ++k) {
            float p[GQA];
            probs(k, p);
            f32pair v;
            if (VMODE) {
                const uint32_t c = *reinterpret_cast<const uint32_t *>(vs + (k * HD + d) * 2);
                v = pair_of(half_bits_to_float(c), half_bits_to_float(c >> 16));
            } else {
                const float sv = half_bits_to_float(vsc[k * 8 + (d >> 5)]);
                const uint32_t c = uint32_t(*reinterpret_cast<const uint16_t *>(vs + k * HD + d)) ^ 0x8080u;
                v = pair_mul(pair_of(sv, sv), pair_sub(pair_of(code_f<0>(c), code_f<1>(c)), magic2));
            }
#pragma unroll
            for (int h = 0; h < GQA; ++h) acc[h] = pair_add(acc[h], pair_fma(pair_of(p[h], p[h]), v, nzero));
        }
        if (k0 < n) {
#pragma unroll
            for (int h = 0; h < GQA; ++h) {
                float x, y;
                split_pair(acc[h], x, y);
                const int o = h * HD + d;
                put2(remote(part + (grp * 4 + s) * OPC + o % OPC, o / OPC), x, y, remote(smem + L.bars + 24, o / OPC));
            }
        }
    } else if (sh.nsl == 2) {                  // 128 threads (one warp per scheduler): one dim, all heads
        if (tid < 128 && n > 0) {
            float acc[GQA];
#pragma unroll
            for (int h = 0; h < GQA; ++h) acc[h] = 0.0f;
#pragma unroll 4
            for (int k = 0; k < n; ++k) {
                float p[GQA];
                probs(k, p);
                const float v = value(k, tid);
#pragma unroll
                for (int h = 0; h < GQA; ++h) acc[h] = __fadd_rn(acc[h], __fmul_rn(p[h], v));
            }
#pragma unroll
            for (int h = 0; h < GQA; ++h) {
                const int o = h * HD + sl * 128 + tid;
                put(remote(part + grp * OPC + o % OPC, o / OPC), acc[h], remote(smem + L.bars + 24, o / OPC));
            }
        }
    } else if (tid < 16 * GQA) {               // one split: a thread owns one dim of one head
        const int d = tid & 15, h = tid >> 4;
        float acc = 0.0f;
#pragma unroll 8
        for (int k = 0; k < n; ++k) acc = __fadd_rn(acc, __fmul_rn(eg[k * GQA + h], value(k, d)));
        const int o = h * HD + sl * 16 + d;
        put(remote(part + o % OPC, o / OPC), acc, remote(smem + L.bars + 24, o / OPC));
    }
    // a CTA that has its part of every exchange has all that is stored into it; one that gave up waits for the others to end
    if (alive) alive = arrived<ERR>(bars + 24, g.err);
    if (!alive) asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
    // ---- splits ascending, gate ----------------------------------------------------------------------------------------------------
    if (tid < OPC) {
        float s = part[tid];
        int i = 1;
        for (; i + 8 <= used; i += 8) {
            float x[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) x[u] = part[(i + u) * OPC + tid];
#pragma unroll
            for (int u = 0; u < 8; ++u) s = __fadd_rn(s, x[u]);
        }
        for (; i < used; ++i) s = __fadd_rn(s, part[i * OPC + tid]);
        if (g.pregate) colp(g.pregate, col * g.cols.arena)[orow] = s;
        colp(g.gated, col * g.cols.arena)[orow] = __fmul_rn(s, gt);
    }
}

// clusters of the largest CTAs that run at once (0: none); asked once, before the first launch: 16 CTAs are beyond the portable
// cluster size, and a launch that does not fit would leave an error behind, or an invalid capture
template <int GQA, int KMODE, int VMODE>
int clusters_at_once() {
    static const int n = [] {
        auto kernel = k_attn_cluster<GQA, KMODE, VMODE>;
        cudaLaunchConfig_t most = {};
        most.gridDim = dim3(CL, 64); most.blockDim = dim3(T); most.dynamicSmemBytes = SMEM_MAX;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = CL; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
        most.attrs = at; most.numAttrs = 1;
        int clusters = 0;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX) == cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&clusters, kernel, &most) == cudaSuccess && clusters > 0) return clusters;
        cudaGetLastError();                    // (a refusal is an answer, not a failed call)
        return 0;
    }();
    return n;
}
template <int GQA, int KMODE, int VMODE>
bool launch_c(cudaStream_t st, const Args &g, size_t smem) {
    auto kernel = k_attn_cluster<GQA, KMODE, VMODE>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CL, g.a.n_kv << g.log_parts, g.cols.z()); cfg.blockDim = dim3(T); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CL; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = g_pdl ? 2 : 1;
    BN_COUNT(1);
    cudaLaunchKernelEx(&cfg, kernel, g);       // (a failure now is one of the caller's, who asks for the last error)
    return true;
}
template <int GQA>
int clusters_of(const Args &g) {
    if (g.a.k_mode) return g.a.v_mode ? clusters_at_once<GQA, 1, 1>() : clusters_at_once<GQA, 1, 0>();
    return g.a.v_mode ? clusters_at_once<GQA, 0, 1>() : clusters_at_once<GQA, 0, 0>();
}
template <int GQA>
bool launch_g(cudaStream_t st, Args g) {
    if constexpr (GQA > 1) {
        // Two clusters with half the heads each where they run at once (K and V are read twice, from L2): few kv heads leave the GPU idle.
        // One kv head of eight heads, with the insert: 64 keys 9.5 -> 7.7 us, 1501 13.9 -> 8.8, 4096 23.1 -> 12.8. 4000 keys (one cluster
        // a kv head -> several): two kv heads of eight 22.2 -> 14.7, of four 14.5 -> 12.2, of two 12.0 -> 11.0; three of eight 22.3 -> 14.7,
        // of four 14.7 -> 12.2, of two 12.1 -> 11.0. Of 80 shapes of one to three kv heads two lose by it, 300 keys at 8 splits (10.1 ->
        // 10.3). (Four kv heads would need eight clusters; fewer fit.)
        if ((g.a.n_kv << (g.log_parts + 1)) * int(g.cols.z()) <= clusters_of<GQA / 2>(g)) {
            Args half = g;
            ++half.log_parts;
            if (launch_g<GQA / 2>(st, half)) return true;
        }
    }
    if (!clusters_of<GQA>(g)) return false;
    const Shape sh = shape_of(g.splits, g.a.cap);
    const size_t smem = size_t((g.a.v_mode ? layout<GQA, 1>(sh, g.splits, g.a.cap) : layout<GQA, 0>(sh, g.splits, g.a.cap)).total);
    if (smem > SMEM_MAX) return false;
    if (g.a.k_mode) return g.a.v_mode ? launch_c<GQA, 1, 1>(st, g, smem) : launch_c<GQA, 1, 0>(st, g, smem);
    return g.a.v_mode ? launch_c<GQA, 0, 1>(st, g, smem) : launch_c<GQA, 0, 0>(st, g, smem);
}

}  // namespace

namespace bnk {

cudaError_t launch_wait_selftest_exchange(cudaStream_t st, int *err) {
    BN_COUNT(1);
    k_wait_selftest_exchange<ERR><<<1, 32, 0, st>>>(err);
    return cudaGetLastError();
}

bool attn_cluster(cudaStream_t st, AttnDims a, const float *q16f, const float *gate, AttnPos where, KvLayer kv, int splits, float *pregate, float *gated, Cols cols, int *err) {
    if (a.cap > 8192 || (splits != 1 && splits != 8 && splits != 64)) return false;
    if (getenv("BONSAI_ATTN_CHAIN")) return false;                         // the answer "does not fit", for comparisons
    const Args g = {a, where, q16f, gate, kv, splits, 0, 1.0f / sqrtf(float(a.head_dim)), -0.0f, pregate, gated, cols, err};
    switch (a.n_head / a.n_kv) {
        case 1: return launch_g<1>(st, g);
        case 2: return launch_g<2>(st, g);
        case 4: return launch_g<4>(st, g);
        case 8: return launch_g<8>(st, g);
    }
    return false;
}

}  // namespace bnk
