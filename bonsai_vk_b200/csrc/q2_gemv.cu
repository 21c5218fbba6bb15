// q2_gemv.cu - the projection of one activation vector over the two-bit weight tiles (q2.cuh), with the preparation of its
// input in front: [rms norm] -> signs -> Hadamard -> q8_1, then int8 tensor-core dots, then the fp32 combination of the
// contract (t_sb = fma(d, I, -s); v = d_w ((t0 + t1) + (t2 + t3)); p_g = (v0 + v1) + (v2 + v3); out = p_0 + p_1 + ...).
//
// What bounds it: memory when it streams (two-bit tiles read 34 bytes per 128 weights), a latency chain of about 1 us in the
// preparation otherwise. Per 16 x 512 piece a warp issues 64 ANDs, 16 mma, 5 loads and about 40 instructions of epilogue -
// 2 warp instructions per 128-weight row-block against 9.1 of the kernel that unpacks base-3 bytes in the loop.
//
// Work split. A CTA of 16 warps owns a run of 16-row tiles over all of K; the pieces (tile, group of four blocks) of that run
// are dealt to the warps in memory order, so with K = 4096 (8 groups) a warp keeps one group. A piece's group sums p_g go to
// shared memory, and after a barrier one thread per row adds them in ascending order: no atomics, no sums that leave the CTA.
// Data movement. A CTA's share of the matrix is one contiguous range; a 17th warp brings it into shared memory with a few bulk
// copies (one piece per warp each), and every projection asks for the NEXT one's weights to be fetched into L2 at its own
// start. Measured beside it: pieces loaded straight into registers (one or two ahead, 8 % slower on the output head, where the
// ring runs at the DRAM's rate), one bulk copy per piece and warp (the issue sits on each warp's chain: 66 against 44 us for the
// head), 16-byte cp.async (1.5 us of load/store-unit time before the first wait), products of one piece interleaved with the
// sums of the one before (spills). One CTA per SM: with two resident (the next projection's beside this one's) the block
// scheduler puts two CTAs of one projection on the same SM and leaves others idle (1.71 against 1.42 ms per token).
#include "q2.cuh"
#include "rotate_quant.cuh"
#include "phase_gemv.cuh"

#include <algorithm>
#include <array>

namespace {
using namespace bnk;

constexpr int NT = 512, NW = NT / 32;          // compute threads; a 17th warp issues the copies
constexpr int CHUNK = NW * Q2_PIECE;           // one piece per warp, contiguous in memory: one bulk copy
constexpr int EARLY = 1, MAX_SLOTS = 6, SMEM_MAX = 227 << 10;
struct Lay {                                    // dynamic shared memory, bytes
    int bars, codes, ds, red, xs, fin, ring;
};
// fin: bytes of group sums that come from a cluster's CTAs
__host__ __device__ constexpr Lay layout(int K, int fin = 0) {
    Lay l{};
    l.bars = 0;
    l.codes = 128;
    l.ds = l.codes + K;
    l.red = l.ds + (K / 32) * 4;
    l.xs = l.red + 256 * 4;
    l.fin = l.xs + (K + 4095) / 4096 * XS8_SPAN * 4;
    l.ring = (l.fin + fin + 127) & ~127;
    return l;
}
constexpr int PBUF = XS8_SPAN;                 // floats of the transform's buffer that hold group sums afterwards

__device__ __forceinline__ unsigned long long gtime() { unsigned long long t; asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t)); return t; }
#define Q2_STAMP(i) do { if (a.stamps && blockIdx.x == 0 && threadIdx.x == 0) a.stamps[i] = gtime(); } while (0)

// barrier over the 16 compute warps (the copy warp never joins it)
__device__ __forceinline__ void csync() { asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory"); }
// bounded wait: on giving up the error word is set and the caller goes on to its end without waiting again (results are then
// invalid)
__device__ __forceinline__ bool slot_wait(uint32_t bar, uint32_t parity, int *err) {
    for (int it = 0; it < (1 << 22); ++it) {
        uint32_t ok;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (__builtin_expect(ok != 0u, 1)) return true;
    }
    atomicExch(err, 1);
    return false;
}
// sign bits 2k and 2k + 1 of a byte as a pair of sign masks
__device__ __forceinline__ f32pair sign_pair(uint32_t sg, int k) {
    return (unsigned long long)((sg << (31 - 2 * k)) & 0x80000000u) | (unsigned long long)((sg << (30 - 2 * k)) & 0x80000000u) << 32;
}

// a CTA's rank in its cluster, its cluster's number
template <int WHICH> __device__ __forceinline__ int special() {
    int v;
    if (WHICH == 0) asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(v));
    else asm("mov.u32 %0, %%clusterid.x;" : "=r"(v));
    return v;
}
// to the other CTAs of the cluster: this one is running. Nothing is published with it: as a release it waits for the accesses before
// it, 0.3 us of every launch (48 tokens 52.8 ms, relaxed 52.4).
__device__ __forceinline__ void running() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
// SPANS: spans of 4096 values whose inputs a thread holds at once (1: K <= 4096; 4: up to 16384)
// LEAN: 80 registers instead of 94, so that beside the 17 warps (five of them on one of the SM's four schedulers, each with
// 16 384 registers) the CTA of a latency-bound mixer kernel fits, and a shared-memory carve-out that leaves room for it: the
// kernel behind the projections of a layer's input. It costs 0.6 us here (12 288 x 4096: 3.0 -> 3.6 us in the loop) and takes
// 3.5 us off what follows.
// SPLIT: K is a whole number of spans and a cluster's CTAs share it, one span each: a CTA prepares its own 4096 values only (three
// spans in every CTA took 4.5 us of the FFN's down projection, one takes 2) and takes its groups of the cluster's row tiles, as many
// pieces as before. A tile's group sums go through distributed shared memory to the CTA that adds them, rank (tile mod CTAs);
// one cluster barrier. Down projection of the 9B shape in its chain: 9.5 -> 7.0 us from the last CTA in front to its own last one.
template <int SPANS, bool LEAN, bool SPLIT>
__global__ void __launch_bounds__(LEAN ? 768 : NT + 32, 1) k_q2_gemv(const Q2Args a) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int parts = SPLIT ? a.K >> 12 : 1, K = SPLIT ? 4096 : a.K, rank = SPLIT ? special<0>() : 0;
    const Lay L = layout(K, SPLIT ? a.fin : 0);
    unsigned char *codes = smem + L.codes;
    uint32_t *dsw = reinterpret_cast<uint32_t *>(smem + L.ds);
    float *red = reinterpret_cast<float *>(smem + L.red), *xs = reinterpret_cast<float *>(smem + L.xs);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tig = lane & 3;
    Q2_STAMP(0);

    // ---- this CTA's tiles ------------------------------------------------------------------------------------------
    const int ng = K >> 9, cta = SPLIT ? special<1>() : blockIdx.x, slots = a.slots;
    const int t0 = cta * a.share.q + min(cta, a.share.r), nt = a.share.q + (cta < a.share.r);
    const int npieces = nt * ng, nchunks = (npieces + NW - 1) / NW;
    const uint32_t full = uint32_t(__cvta_generic_to_shared(smem + L.bars)), empty = full + MAX_SLOTS * 8;

    if (SPLIT) running();
    if (warp == NW) {
        // ---- copy warp. Before the previous kernel is done: one chunk of weights into the ring (more would hold up the input
        // vector, which follows it through the same queue, by up to a microsecond) and the NEXT projection's weights (a
        // share of this grid) towards L2; the other slots once the input vector is in registers; refills.
        const uint8_t *W = a.W + (SPLIT ? size_t(t0) * parts + rank : size_t(t0)) * ng * Q2_PIECE;
        auto request = [&](int i, int s) {
            const uint32_t bytes = uint32_t(min(NW, npieces - i * NW)) * Q2_PIECE;
            if (SPLIT) {                           // (a chunk is two tiles' groups of this span)
                constexpr uint32_t half = CHUNK / 2;
                const uint32_t dst = uint32_t(__cvta_generic_to_shared(smem + L.ring)) + s * CHUNK;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full + s * 8), "r"(bytes) : "memory");
                for (uint32_t o = 0; o < bytes; o += half)
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                 ::"r"(dst + o), "l"(W + size_t(i * 2 + (o ? 1 : 0)) * parts * half), "r"(half), "r"(full + s * 8) : "memory");
                return;
            }
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full + s * 8), "r"(bytes) : "memory");
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         ::"r"(uint32_t(__cvta_generic_to_shared(smem + L.ring)) + s * CHUNK), "l"(W + size_t(i) * CHUNK), "r"(bytes), "r"(full + s * 8) : "memory");
        };
        if (lane == 0) {
            for (int s = 0; s < slots; ++s) {
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full + s * 8));
                asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(empty + s * 8), "n"(NW));
            }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            for (int i = 0; i < min(EARLY, slots); ++i) request(i, i);
            q2_prefetch_next(a.next, blockIdx.x, 0, 1);
        }
        __syncwarp();
        asm volatile("bar.arrive 2, %0;" ::"n"(NT + 32) : "memory");
        if (!a.late) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        asm volatile("bar.sync 3, %0;" ::"n"(NT + 32) : "memory");
        if (lane == 0) for (int i = EARLY; i < min(slots, nchunks); ++i) request(i, i);
        for (int i = slots, s = 0, ph = 0; i < nchunks; ++i) {
            if (!slot_wait(empty + s * 8, ph, a.err)) break;
            if (lane == 0) request(i, s);
            if (++s == slots) { s = 0; ph ^= 1; }
        }
        if (SPLIT) {                               // (both cluster barriers with the other warps)
            __syncwarp();
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        }
        return;
    }

    // constants of the preparation depend on no earlier kernel: norm weights with the signs applied to them (the sign of the
    // product is the product of the signs), or the signs as masks
    const int base = tid * 8, nspan = SPANS == 1 ? 1 : (K + 4095) >> 12;
    const uint8_t *signs = a.sgn + rank * 512;
    const float *x0 = a.x0 + rank * 4096;
    f32pair nw[4] = {0, 0, 0, 0};
    uint32_t sg[SPANS];
#pragma unroll
    for (int s = 0; s < SPANS; ++s) sg[s] = base + s * 4096 < K ? signs[(base >> 3) + s * 512] : 0u;
    if (SPANS == 1 && a.pro == Q2_NORM && base < K) load8(a.w + base, nw);
    Q2_STAMP(1);
    // The next kernel may start now: before its own wait it reads constants and words set before the pass (the rule at bnk::launch).
    if (!a.late) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (SPANS == 1) {
#pragma unroll
        for (int k = 0; k < 4; ++k) nw[k] ^= sign_pair(sg[0], k);
    }
    asm volatile("bar.sync 2, %0;" ::"n"(NT + 32) : "memory");          // the ring's barriers are initialised
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (a.late) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    Q2_STAMP(2);

    // ---- input preparation -------------------------------------------------------------------------------------------
    f32pair v[SPANS][4];
#pragma unroll
    for (int s = 0; s < SPANS; ++s)
        if (base + s * 4096 < K) load8(x0 + base + s * 4096, v[s]);
        else {
#pragma unroll
            for (int k = 0; k < 4; ++k) v[s][k] = 0ull;
        }
    // the residual of the row this thread finishes first
    float resid = 0.0f;
    const int row0 = SPLIT ? (t0 + (tid >> 4) * parts + rank) * 16 + (tid & 15) : t0 * 16 + tid;
    if (a.resid_out && row0 < min((t0 + nt) * 16, a.M)) resid = a.resid_in[row0];
    f32pair inv2 = pair_of(1.0f, 1.0f);
    if (a.pro == Q2_NORM) {
        // rms_norm.comp order: 256 lanes sum the squares of their run of `per` consecutive values ascending, then the tree
        const int per = (K + 255) >> 8;
        if (SPANS == 1 && per == 16) {             // K = 4096: a lane's run is two neighbouring threads' values
            float sq = 0.0f, e[8];
#pragma unroll
            for (int k = 0; k < 4; ++k) split_pair(pair_mul(v[0][k], v[0][k]), e[2 * k], e[2 * k + 1]);
#pragma unroll
            for (int k = 0; k < 8; ++k) sq = __fadd_rn(sq, e[k]);
            sq = __shfl_up_sync(0xFFFFFFFFu, sq, 1);         // (an odd thread goes on from its even neighbour's sum)
#pragma unroll
            for (int k = 0; k < 8; ++k) sq = __fadd_rn(sq, e[k]);
            if (tid & 1) red[tid >> 1] = sq;
        } else if (tid < 256) {
            float sq = 0.0f;
            for (int i = 0; i < per; ++i) {
                const int d = tid * per + i;
                if (d < K) { const float x = x0[d]; sq = __fadd_rn(sq, __fmul_rn(x, x)); }
            }
            red[tid] = sq;
        }
        csync();
        const float ss = norm_tree256(red, lane);
        const float inv = __frcp_rn(__fsqrt_rn(__fadd_rn(a.inv_k != 0.0f ? __fmul_rn(ss, a.inv_k) : __fdiv_rn(ss, float(K)), a.eps)));
        if (a.inv_out && blockIdx.x == 0 && tid == 0) a.inv_out[0] = inv;
        inv2 = pair_of(inv, inv);
    }
    Q2_STAMP(3);
#pragma unroll
    for (int s = 0; s < SPANS; ++s) {
        if (s < nspan) {
            if (SPANS > 1) {
                if (a.pro == Q2_NORM && base + s * 4096 < K) {
                    load8(a.w + base + s * 4096, nw);
#pragma unroll
                    for (int k = 0; k < 4; ++k) v[s][k] = pair_mul(pair_mul(v[s][k], inv2), nw[k]);
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) v[s][k] ^= sign_pair(sg[s], k);
            } else if (a.pro == Q2_NORM) {
#pragma unroll
                for (int k = 0; k < 4; ++k) v[s][k] = pair_mul(pair_mul(v[s][k], inv2), nw[k]);
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) v[s][k] ^= nw[k];
            }
            fwht_pairs8(v[s], 3);                  // the stages h = 1, 2, 4
            span_store8(xs + s * XS8_SPAN, tid, v[s]);
        }
    }
    asm volatile("bar.arrive 3, %0;" ::"n"(NT + 32) : "memory");          // to the copy warp: the input is here
    fwht_spans(xs, tid, nspan, a.log_hat, [] { csync(); });
    Q2_STAMP(4);
#pragma unroll 1
    for (int s = 0; s < nspan; ++s) {
        f32pair y[4];
        span_load8(xs + s * XS8_SPAN, tid, y);
#pragma unroll
        for (int k = 0; k < 4; ++k) y[k] = pair_mul(y[k], pair_of(a.hat_inv, a.hat_inv));
        const Q8x8 q = quant8_pairs(y);
        const int at = base + s * 4096;
        if (at < K) {
            // codes of (block, sub-block b, elements 8t .. 8t + 7) at block * 128 + (b & 1) * 64 + t * 16 + (b >> 1) * 8
            const int b = (at >> 5) & 3, e8 = (at >> 3) & 3;
            *reinterpret_cast<uint2 *>(codes + (at & ~127) + (b & 1) * 64 + e8 * 16 + (b >> 1) * 8) = make_uint2(q.w0, q.w1);
            if (e8 == 0) dsw[at >> 5] = float_to_half_bits(q.d) | (float_to_half_bits(__fmul_rn(q.d, float(q.sum))) << 16);
        }
    }
    csync();
    Q2_STAMP(5);

    // ---- pieces ------------------------------------------------------------------------------------------------------
    uint2 B[4][4];                                 // operand B of [block][sub-block]: the codes in the lanes of column 2j + (s & 1), zero in the others
    f32pair d01 = 0, d23 = 0, n01 = 0, n23 = 0;    // block tig: (d0, d1/4), (d2/16, d3/64), (-s0, -s1), (-s2, -s3)
    int group = -1;
    auto set_group = [&](int gr) {
        const uint4 own = *reinterpret_cast<const uint4 *>(codes + (gr * 4 + (g >> 1)) * 128 + (g & 1) * 64 + tig * 16);   // sub-blocks (g & 1) and (g & 1) + 2
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            B[c >> 1][c & 1] = g == c ? make_uint2(own.x, own.y) : make_uint2(0u, 0u);
            B[c >> 1][(c & 1) + 2] = g == c ? make_uint2(own.z, own.w) : make_uint2(0u, 0u);
        }
        const uint4 ds = *reinterpret_cast<const uint4 *>(dsw + (gr * 4 + tig) * 4);
        d01 = pair_of(half_bits_to_float(ds.x), half_bits_to_float(ds.y) * 0.25f);
        d23 = pair_of(half_bits_to_float(ds.z) * 0.0625f, half_bits_to_float(ds.w) * 0.015625f);
        n01 = pair_of(-half_bits_to_float(ds.x >> 16), -half_bits_to_float(ds.y >> 16));
        n23 = pair_of(-half_bits_to_float(ds.z >> 16), -half_bits_to_float(ds.w >> 16));
        group = gr;
    };
    const f32pair magic2 = pair_of(__int_as_float(Q2_MAGIC), __int_as_float(Q2_MAGIC));
    // tiles per run of group sums: what the transform's buffer holds
    const int run = a.run, gstep = a.gstep;
    int u = warp, gr = warp, slot = 0;
    while (gr >= ng) gr -= ng;                     // (eight groups at K = 4096: one step at most)
    uint32_t phase = 0;
    bool alive = true;
    // one piece: its group sums p_g of 16 rows go to `dst` (SPLIT: to the CTA that adds them)
    const int per_part = parts == 2 ? 128 : (parts == 3 ? 86 : 64);      // tile / parts = tile * per_part >> 8 for the few tiles of a cluster
    float *fin = reinterpret_cast<float *>(smem + L.fin);                 // [tile of this CTA][group of all K][16]
    auto piece = [&](float *dst) {
        if (gr != group) set_group(gr);
        gr += gstep; if (gr >= ng) gr -= ng;
        if (alive) alive = slot_wait(full + slot * 8, phase, a.err);
        const unsigned char *src = smem + L.ring + slot * CHUNK + warp * Q2_PIECE;
        uint4 c[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) c[q] = *reinterpret_cast<const uint4 *>(src + lane * 16 + q * 512);
        const uint32_t dw = *reinterpret_cast<const uint32_t *>(src + Q2_SCALES + lane * 4);
        if (u - warp + slots * NW < npieces) {     // the slot is refilled: this warp's part of it is in registers
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty + slot * 8) : "memory");
        }
        if (++slot == slots) { slot = 0; phase ^= 1; }
        int e[4], f[4];                            // sub-blocks (0, 1) and (2, 3) of block tig, rows g and g + 8
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint4 &lo = c[j >> 1], &hi = c[2 + (j >> 1)];
            const uint32_t l0 = (j & 1) ? lo.z : lo.x, l1 = (j & 1) ? lo.w : lo.y, h0 = (j & 1) ? hi.z : hi.x, h1 = (j & 1) ? hi.w : hi.y;
            constexpr uint32_t m0 = 0x03030303u, m1 = m0 << 2, m2 = m0 << 4, m3 = m0 << 6;
            if (j == 0) {
                q2_mma_first(e, l0 & m0, h0 & m0, l1 & m0, h1 & m0, B[j][0].x, B[j][0].y);
                q2_mma_first(f, l0 & m2, h0 & m2, l1 & m2, h1 & m2, B[j][2].x, B[j][2].y);
            } else {
                q2_mma(e, l0 & m0, h0 & m0, l1 & m0, h1 & m0, B[j][0].x, B[j][0].y);
                q2_mma(f, l0 & m2, h0 & m2, l1 & m2, h1 & m2, B[j][2].x, B[j][2].y);
            }
            q2_mma(e, l0 & m1, h0 & m1, l1 & m1, h1 & m1, B[j][1].x, B[j][1].y);
            q2_mma(f, l0 & m3, h0 & m3, l1 & m3, h1 & m3, B[j][3].x, B[j][3].y);
        }
        auto block_sum = [&](int e0, int e1, int f0, int f1, uint32_t w) {
            float x0, x1, x2, x3;
            split_pair(pair_fma(d01, pair_sub(pair_of(__int_as_float(e0), __int_as_float(e1)), magic2), n01), x0, x1);
            split_pair(pair_fma(d23, pair_sub(pair_of(__int_as_float(f0), __int_as_float(f1)), magic2), n23), x2, x3);
            return __fmul_rn(half_bits_to_float(w), __fadd_rn(__fadd_rn(x0, x1), __fadd_rn(x2, x3)));
        };
        float va = block_sum(e[0], e[1], f[0], f[1], dw), vb = block_sum(e[2], e[3], f[2], f[3], dw >> 16);
        va = __fadd_rn(va, __shfl_xor_sync(0xFFFFFFFFu, va, 1)); vb = __fadd_rn(vb, __shfl_xor_sync(0xFFFFFFFFu, vb, 1));
        va = __fadd_rn(va, __shfl_xor_sync(0xFFFFFFFFu, va, 2)); vb = __fadd_rn(vb, __shfl_xor_sync(0xFFFFFFFFu, vb, 2));
        if (SPLIT) {
            const int tile = u / 8, round = tile * per_part >> 8, to = tile - round * parts;
            uint32_t at;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(uint32_t(__cvta_generic_to_shared(fin + ((round * parts + rank) * 8 + (u & 7)) * 16 + g + 8 * tig))), "r"(to));
            if (tig < 2) asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(tig ? vb : va) : "memory");
        } else if (tig < 2) dst[g + 8 * tig] = tig ? vb : va;
    };
    Q2_STAMP(6);
    if (SPLIT) {
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");              // every CTA is running
        for (; u < npieces; u += NW) piece(nullptr);
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        const int n = parts * 8;
        if (row0 < min((t0 + nt) * 16, a.M)) {
            const float *own = fin + (tid >> 4) * n * 16 + (tid & 15);
            float s = own[0];
            for (int k = 1; k < n; k += 8) {       // (loads first, then the adds in ascending order)
                float x[8];
#pragma unroll
                for (int b = 0; b < 8; ++b) x[b] = own[min(k + b, n - 1) * 16];
#pragma unroll
                for (int b = 0; b < 8; ++b) if (b < 7 || k + 7 < n) s = __fadd_rn(s, x[b]);
            }
            if (a.out) a.out[row0] = s;
            if (a.resid_out) a.resid_out[row0] = __fadd_rn(s, resid);
        }
        Q2_STAMP(7);
        return;
    }
    for (int c0 = 0; c0 < nt; c0 += run) {
        const int c1 = min(nt, c0 + run), uend = c1 * ng, rows = (c1 - c0) * 16;
        // what the sums below need, worked out ahead of the barrier
        const float *own = xs + (tid >> 4) * ng * 16 + (tid & 15);
        const int row = (t0 + c0) * 16 + tid;
        for (; u < uend; u += NW) piece(xs + (u - c0 * ng) * 16);
        csync();
        for (int i0 = 0; i0 < rows; i0 += NT, own += (NT / 16) * ng * 16) {
            const bool on = i0 + tid < rows;
            float s = 0.0f;
            if (on) {
                if (ng == 8) {                     // (loads first, then the adds in ascending order)
                    float x[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) x[k] = own[k * 16];
                    s = x[0];
#pragma unroll
                    for (int k = 1; k < 8; ++k) s = __fadd_rn(s, x[k]);
                } else {
                    s = own[0];
                    int k = 1;
                    for (; k + 8 <= ng; k += 8) {
                        float x[8];
#pragma unroll
                        for (int b = 0; b < 8; ++b) x[b] = own[(k + b) * 16];
#pragma unroll
                        for (int b = 0; b < 8; ++b) s = __fadd_rn(s, x[b]);
                    }
#pragma unroll 4
                    for (; k < ng; ++k) s = __fadd_rn(s, own[k * 16]);
                }
                if (!a.swiglu && row + i0 < a.M) {
                    if (a.out) a.out[row + i0] = s;
                    if (a.resid_out) a.resid_out[row + i0] = __fadd_rn(s, row + i0 == row0 ? resid : a.resid_in[row + i0]);
                }
            }
            if (a.swiglu) {                        // rows r and r + 8 of a tile: gate and up of one FFN row
                const float up = __shfl_down_sync(0xFFFFFFFFu, s, 8);
                if (on && !(tid & 8)) a.out[((row + i0) >> 4) * 8 + (tid & 7)] = __fmul_rn(silu_f(s), up);
            }
        }
        if (c1 < nt) csync();
    }
    Q2_STAMP(7);
}

// A warp per piece: lane (row, block) unpacks 28 bytes into shared memory, eight rows at a time, and the finished piece leaves
// as 16-byte stores (stored straight from the lanes, 8 bytes of every 16, it ran at a third of the rate). Rows 0..7 of a tile
// come from Wa and 8..15 from Wb, `half` rows apart in each (Wb = Wa + 8 rows and half = 16 for a single matrix).
__global__ void __launch_bounds__(256) k_q2_repack(const uint32_t *__restrict__ Wa, const uint32_t *__restrict__ Wb, int half, int Ma, int Mb, int nb,
                                                   size_t pieces, uint8_t *__restrict__ out) {
    __shared__ __align__(16) uint8_t stage[8][Q2_PIECE];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ng = nb >> 2, r = lane >> 2, j = lane & 3;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    uint8_t *piece = stage[warp];
    for (size_t p = size_t(blockIdx.x) * 8 + warp; p < pieces; p += size_t(gridDim.x) * 8) {
        const int tile = int(p / ng), gr = int(p - size_t(tile) * ng), row = tile * half + r;
        uint32_t w[2][7];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t *src = (h ? Wb : Wa) + (size_t(row) * nb + gr * 4 + j) * 7;
            const bool on = row < (h ? Mb : Ma);
#pragma unroll
            for (int k = 0; k < 7; ++k) w[h][k] = on ? src[k] : 0u;
        }
        __syncwarp();                          // the previous piece has left
#pragma unroll
        for (int h = 0; h < 2; ++h) q2_unpack_block(w[h], piece, h, r, j);
        __syncwarp();
        uint4 *d = reinterpret_cast<uint4 *>(out + p * Q2_PIECE);
        const uint4 *s = reinterpret_cast<const uint4 *>(piece);
#pragma unroll
        for (int i = 0; i < 4; ++i) d[i * 32 + lane] = s[i * 32 + lane];
        if (lane < 8) d[128 + lane] = s[128 + lane];
    }
}
__global__ void k_sign_bits(const int32_t *__restrict__ signs, int nwords, uint8_t *__restrict__ bits) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nwords) return;
    uint32_t b = 0;
    for (int k = 0; k < 8; ++k) b |= (signs[i * 8 + k] < 0 ? 1u : 0u) << k;
    bits[i] = uint8_t(b);
}

template <int SPANS, bool LEAN, bool SPLIT = false>
cudaError_t launch_spans(cudaStream_t st, int sm_count, Q2Args a, bool pdl, int clusters = 0) {
    // as many chunks of weights as fit beside the rest, and at least half of an SM's shared memory in all, so that two CTAs of a
    // launch never share an SM (see above)
    const int parts = SPLIT ? a.K / 4096 : 1, K = SPLIT ? 4096 : a.K, units = SPLIT ? clusters : sm_count;
    const int ng = K / 512, tiles = (a.M + 15) / 16, split = tiles < units ? tiles : units, grid = split * parts;
    a.share = {tiles / split, tiles % split};
    const int most = a.share.q + (a.share.r > 0), chunks = (most * ng + NW - 1) / NW;
    a.fin = SPLIT ? (most + parts - 1) / parts * (a.K / 512) * 64 : 0;
    a.slots = std::min({chunks, MAX_SLOTS, (SMEM_MAX - layout(K, a.fin).ring) / CHUNK});
    const int smem = std::max(layout(K, a.fin).ring + a.slots * CHUNK, 116 << 10);
    // once, to the largest value, whatever this launch needs: with a limit that grows from call to call a second thread could lower
    // it again under the first (an SM changes its carve-out only when it is empty, so every projection asks for the largest one)
    static const cudaError_t limits = [] {
        cudaError_t e = cudaFuncSetAttribute(k_q2_gemv<SPANS, LEAN, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX);
        return e != cudaSuccess ? e : cudaFuncSetAttribute(k_q2_gemv<SPANS, LEAN, SPLIT>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    }();
    if (limits != cudaSuccess) return limits;
    a.inv_k = (a.K & (a.K - 1)) == 0 ? 1.0f / float(a.K) : 0.0f;
    a.log_hat = 31 - __builtin_clz(unsigned(a.hat_block));
    a.run = std::max(1, PBUF / (16 * ng)); a.gstep = NW % ng;
    if (a.next.W) a.next.share = {a.next.units / grid, a.next.units % grid};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(NT + 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    int n = 0;
    if (pdl) { at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[n++].val.programmaticStreamSerializationAllowed = 1; }
    if (SPLIT) { at[n].id = cudaLaunchAttributeClusterDimension; at[n].val.clusterDim.x = parts; at[n].val.clusterDim.y = 1; at[n++].val.clusterDim.z = 1; }
    cfg.attrs = at;
    cfg.numAttrs = n;
    BN_COUNT(1);
    return cudaLaunchKernelEx(&cfg, k_q2_gemv<SPANS, LEAN, SPLIT>, a);
}

// Clusters of `parts` CTAs, one CTA per SM, that start together behind a kernel whose CTAs end one by one: an eighth fewer than the
// occupancy query finds room for. Counted over 330 down projections in a chain of the 9B shape's, with 3 CTAs and room for 45: 45
// clusters had one held up until another ended in 262 of them (11.0 us on average), 43 in 28 (7.3 us), 40 in none (6.96 us), and
// 34 take 7.24 us.
int split_clusters(int parts) {
    static const std::array<int, 9> most = [] {
        std::array<int, 9> m{};
        cudaError_t e = cudaFuncSetAttribute(k_q2_gemv<1, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX);
        for (int p = 2; p <= 4 && e == cudaSuccess; ++p) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(p * 64); cfg.blockDim = dim3(NT + 32); cfg.dynamicSmemBytes = SMEM_MAX;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension; at[0].val.clusterDim.x = p; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
            cfg.attrs = at; cfg.numAttrs = 1;
            if ((e = cudaOccupancyMaxActiveClusters(&m[p], k_q2_gemv<1, false, true>, &cfg)) != cudaSuccess) m[p] = 0;
        }
        if (e != cudaSuccess) cudaGetLastError();  // (a refusal is an answer, not a failed call)
        return m;
    }();
    return most[parts] - most[parts] / 8;
}

}  // namespace

namespace bnk {

bool q2_gemv_supported(int K, int hat_block) {
    return K >= 512 && K % 512 == 0 && K <= 16384 && hat_block >= 16 && hat_block <= 4096 && (hat_block & (hat_block - 1)) == 0 && K % hat_block == 0;
}

void q2_gemv_prepare() { split_clusters(2); }

// A span per CTA of a cluster where that costs no CTA more than one further piece per warp: 0.8 us against 2.4 us of preparation per
// span saved. A layer's down projection in four-layer models, us saved for 1024 / 4096 / 5120 / 7168 rows: K = 8192 2.0 / 1.7 / 1.1 / 0 to
// 0.9 (65 clusters), 12 288 3.7 / 2.9 / 2.9 / 2.2 (40), 16 384 4.7 / 3.7 / 3.7 / not shared: 16 tiles (29).
Q2Split q2_gemv_split(int sm_count, int M, int K) {
    if (K <= 4096 || K % 4096 || K > 16384) return {};
    const int n = split_clusters(K / 4096), tiles = (M + 15) / 16, most = n ? (tiles + n - 1) / n : 0;
    return n && most <= 12 && most * 8 <= (tiles + sm_count - 1) / sm_count * (K / 512) + NW ? Q2Split{n, most} : Q2Split{};
}

cudaError_t launch_q2_gemv(cudaStream_t st, int sm_count, const Q2Args &a, bool pdl) {
    const Q2Split split = a.pro == Q2_PLAIN && !a.swiglu ? q2_gemv_split(sm_count, a.M, a.K) : Q2Split{};
    if (split.clusters) return launch_spans<1, false, true>(st, sm_count, a, pdl, split.clusters);
    if (a.K > 4096) return launch_spans<4, false>(st, sm_count, a, pdl);
    return a.lean ? launch_spans<1, true>(st, sm_count, a, pdl) : launch_spans<1, false>(st, sm_count, a, pdl);
}

static void repack(cudaStream_t st, const uint32_t *Wa, const uint32_t *Wb, int half, int Ma, int Mb, int tiles, int K, uint8_t *out) {
    const size_t pieces = size_t(tiles) * (K / 512);
    launch(k_q2_repack, dim3(unsigned(std::min<size_t>((pieces + 7) / 8, 148 * 8))), dim3(256), 0, st, Wa, Wb, half, Ma, Mb, K / 128, pieces, out);
}
void q2_repack(cudaStream_t st, const uint32_t *W, int M, int K, uint8_t *out) {
    repack(st, W, W + size_t(8) * (K / 128) * 7, 16, M, M - 8, (M + 15) / 16, K, out);
}
void q2_repack_pair(cudaStream_t st, const uint32_t *Wa, const uint32_t *Wb, int M, int K, uint8_t *out) { repack(st, Wa, Wb, 8, M, M, M / 8, K, out); }
void pack_sign_bits(cudaStream_t st, const int32_t *signs, int n, uint8_t *bits) {
    BN_COUNT(1);
    k_sign_bits<<<(n / 8 + 255) / 256, 256, 0, st>>>(signs, n / 8, bits);
}

}  // namespace bnk
