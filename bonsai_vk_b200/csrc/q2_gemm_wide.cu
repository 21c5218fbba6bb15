// q2_gemm_wide.cu - the projection of 17 to 32 activation columns over the two-bit weight tiles (q2.cuh): the arithmetic of
// q2_gemm.cu, with the data brought in by a producer warp.
//
// What bounds it: the instruction rate. Blackwell's integer and fp32 instructions share their lanes, and a packed fp32 instruction
// takes two turns, so the work of (16 rows, 8 columns, 128 weights) - 4 mma, 8 ANDs, 16 conversions, 22 packed fp32 operations,
// 4 multiplications - costs a scheduler about 90 cycles with two or three warps at it, and removing every shared-memory read from
// the loop changes nothing. That is 19 us for 24 576 x 4096 x 32; the kernel takes 27 us with weights from DRAM, back
// to back and without the preparation of the columns (under ncu with cold caches 32.5, where the wave-by-wave kernel of q2_gemm.cu,
// which loses to its barriers and to weights loaded on demand, took 45.4); 4096 x 12 288: 20.2 us.
//
// Work split. 12 compute warps of 160 registers: a warp has two row tiles, 16 of the columns and a segment of K, and walks the
// segment group by group with everything in registers (two tiles x 16 columns share the operands: half the ANDs and half the
// operand reads of one tile x 8). Segments: as many as there are warps without row tiles of their own. The first segment's warp
// adds its group sums p_g as they come, the others leave theirs in shared memory, and the first adds them in ascending order at
// the end, so no sum leaves the CTA. Data: image steps of 256 values and groups of weights in two rings, filled by one thread
// (measured beside it: each warp fetching its own weights with bulk copies or cp.async, 27 and 31 us: the issue takes a quarter of
// the loop). The four warps of the producer's warpgroup give their registers to the others.
#include "q2.cuh"
#include "rotate_quant.cuh"

#include <algorithm>

namespace {
using namespace bnk;

constexpr int NW = 12, NT = (NW + 4) * 32;             // compute warps, and the producer's warpgroup
constexpr int MT = 2, CG = 2;                          // a warp's row tiles and groups of 8 columns
constexpr int NCP = 32, H = NCP / (CG * 8), NG = NCP / 8;
constexpr int SMEM_MAX = 227 << 10, HEAD = 128;        // HEAD: where the sums begin, behind the barriers
constexpr int MAX_SLOTS = 4, MAX_WSLOTS = 3;
constexpr int IMG_COL = 160;                           // image bytes per column and block (act_image.cuh)

struct Split {                                         // see the launch
    int segs, gs;                                      // segments of K, groups of a segment
    int tiles;                                         // row tiles per pass
    int slots, wslots, imgs, wts;                      // image steps and groups of weights held; their shared memory offsets
};

__device__ __forceinline__ void bulk(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mma(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}

__global__ void __launch_bounds__(NT, 1) k_q2_gemm_wide(const Q2GemmArgs a, const Split sp) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tig = lane & 3;
    const int ng = a.K >> 9, S = sp.segs, gs = sp.gs;
    const int t0 = blockIdx.x * a.share.q + min(int(blockIdx.x), a.share.r), nt = a.share.q + (int(blockIdx.x) < a.share.r);
    const int npass = (nt + sp.tiles - 1) / sp.tiles, groups = npass * gs, slots = sp.slots;
    const int half = warp % H, seg = warp / H % S, row = warp / (H * S) * MT;        // a warp's 16 columns, segment, first row tile of a pass
    const uint32_t full = uint32_t(__cvta_generic_to_shared(smem)), empty = full + MAX_SLOTS * 8, wfull = empty + MAX_SLOTS * 8, wempty = wfull + MAX_WSLOTS * 8;
    float *sums = reinterpret_cast<float *>(smem + HEAD);
    const int step = NCP * IMG_COL * 2, wgroup = sp.tiles * Q2_PIECE;  // bytes of a segment: image of a step, weights of a group
    if (tid == 0) {
        for (int s = 0; s < slots; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full + s * 8));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(empty + s * 8), "n"(NW));
        }
        for (int s = 0; s < sp.wslots; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(wfull + s * 8));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(wempty + s * 8), "n"(NW));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    bool alive = true;

    if (warp >= NW) {
        // ---- copies: one thread (a bulk copy costs it 70 cycles; on a compute warp's path that was a quarter of the loop) ----------
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        if (warp == NW + 1) {
            // this CTA's weights (as far as the previous projection has not fetched them) and the next projection's towards L2
            const uint8_t *own = a.W + size_t(t0) * ng * Q2_PIECE;
            const int bytes = min(nt * ng * Q2_PIECE, Q2_NEXT_BYTES);
            for (int o = lane * 16384; o < bytes; o += 32 * 16384) q2_prefetch(own + o, min(16384, bytes - o));
            if (lane == 0) q2_prefetch_next(a.next, blockIdx.x, 0, 1);
        }
        if (warp != NW || lane) return;
        int w_u = 0, w_i = 0, w_pass = 0, w_slot = 0, w_phase = 1;        // the next group of weights
        auto weights = [&]() {
            if (alive && w_u >= sp.wslots) alive = q2_wait(wempty + w_slot * 8, w_phase, a.err);
            if (!alive) return;
            const int tb = w_pass * sp.tiles, n = min(sp.tiles, nt - tb), ns = S > 1 ? (ng - w_i + gs - 1) / gs : 1;      // ns: segments that have a group i
            const uint8_t *src = a.W + (size_t(t0 + tb) * ng + w_i) * Q2_PIECE;
            const uint32_t dst = full + sp.wts + w_slot * S * wgroup, bar = wfull + w_slot * 8;
            expect(bar, ns * n * Q2_PIECE);
            for (int s = 0; s < ns; ++s)
                for (int m = 0; m < n; ++m) bulk(dst + s * wgroup + m * Q2_PIECE, src + (size_t(m) * ng + s * gs) * Q2_PIECE, Q2_PIECE, bar);
            ++w_u;
            if (++w_slot == sp.wslots) { w_slot = 0; w_phase ^= 1; }
            if (++w_i == gs) { w_i = 0; ++w_pass; }
        };
        // weights that no kernel still running writes are asked for ahead of the dependency wait (100-token prefill 13.76 -> 13.70 ms; the
        // same in k_q2_gemm, whose units load theirs into registers, changed nothing)
        if (!a.warm) asm volatile("griddepcontrol.wait;" ::: "memory");
        int slot = 0, phase = 1;
        for (int u = 0, i = 0; u < groups; ++u) {
            if (w_u <= u) weights();
            if (u == 0 && a.warm) asm volatile("griddepcontrol.wait;" ::: "memory");
            const int ns = S > 1 ? (ng - i + gs - 1) / gs : 1;
            for (int jp = 0; jp < 2; ++jp) {
                if (alive && 2 * u + jp >= slots) alive = q2_wait(empty + slot * 8, phase, a.err);
                if (!alive) return;
                expect(full + slot * 8, ns * step);
                for (int s = 0; s < ns; ++s) bulk(full + sp.imgs + (slot * S + s) * step, a.image + size_t((s * gs + i) * 2 + jp) * step, step, full + slot * 8);
                if (++slot == slots) { slot = 0; phase ^= 1; }
            }
            if (w_u < groups) weights();
            if (++i == gs) i = 0;
        }
        return;
    }

    // ---- sums ----------------------------------------------------------------------------------------------------------------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 160;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");        // (behind the wait: see k_q2_gemm; the copies' warps end without it)
    f32pair acc[MT][CG][2];
    int slot = 0, phase = 0, wslot = 0, wphase = 0;                      // slots of the step and the group, and the parity of their use
    for (int pass = 0; pass < npass; ++pass) {
        const int tb = pass * sp.tiles, n = min(sp.tiles, nt - tb);
        const bool on = row < n;
        for (int i = 0; i < gs; ++i) {
            f32pair us[MT][CG][2];                 // v0 + v1 of rows g, g + 8
#pragma unroll
            for (int jp = 0; jp < 2; ++jp) {
                if (jp == 0 && alive) alive = q2_wait(wfull + wslot * 8, wphase, a.err);
                if (alive) alive = q2_wait(full + slot * 8, phase, a.err);
                if (on && seg * gs + i < ng) {
                    const unsigned char *img = smem + sp.imgs + (slot * S + seg) * step + half * (CG * 1024) + (tig >> 1) * 128 + g * 16 + (tig & 1) * 8;
                    const unsigned char *scl = smem + sp.imgs + (slot * S + seg) * step + NCP * 128 + half * (CG * 256) + tig * 16;
                    const unsigned char *wp = smem + sp.wts + (wslot * S + seg) * wgroup + row * Q2_PIECE;
                    uint4 lo[MT], hi[MT];
                    uint2 dw[MT];
#pragma unroll
                    for (int m = 0; m < MT; ++m) {
                        lo[m] = *reinterpret_cast<const uint4 *>(wp + m * Q2_PIECE + jp * 512 + lane * 16);
                        hi[m] = *reinterpret_cast<const uint4 *>(wp + m * Q2_PIECE + 1024 + jp * 512 + lane * 16);
                        dw[m] = *reinterpret_cast<const uint2 *>(wp + m * Q2_PIECE + 2048 + g * 16 + jp * 8);
                    }
                    f32pair ve[MT][CG][2];
#pragma unroll
                    for (int jj = 0; jj < 2; ++jj) {
                        const int bo = jj * NCP * IMG_COL;
                        uint2 B[CG][4];
                        f32pair sd[CG][4], sn[CG][4];
#pragma unroll
                        for (int cg = 0; cg < CG; ++cg)
#pragma unroll
                            for (int s = 0; s < 4; ++s) {
                                B[cg][s] = *reinterpret_cast<const uint2 *>(img + bo + cg * 1024 + s * 256);
                                const ulonglong2 sc = *reinterpret_cast<const ulonglong2 *>(scl + bo + cg * 256 + s * 64);
                                // the dot of sub-block s comes as 4^s I
                                const float sh = s == 0 ? 1.0f : (s == 1 ? 0.25f : (s == 2 ? 0.0625f : 0.015625f));
                                sd[cg][s] = s ? pair_mul(sc.x, pair_of(sh, sh)) : sc.x;
                                sn[cg][s] = sc.y;
                            }
#pragma unroll
                        for (int m = 0; m < MT; ++m) {
                            const uint32_t l0 = jj ? lo[m].z : lo[m].x, l1 = jj ? lo[m].w : lo[m].y, h0 = jj ? hi[m].z : hi[m].x, h1 = jj ? hi[m].w : hi[m].y;
                            const uint32_t dwj = jj ? dw[m].y : dw[m].x;
                            const float dlo = half_bits_to_float(dwj), dhi = half_bits_to_float(dwj >> 16);
                            f32pair tl[CG][4], th[CG][4];
#pragma unroll
                            for (int s = 0; s < 4; ++s) {
                                const uint32_t mask = 0x03030303u << (2 * s), a0 = l0 & mask, a1 = h0 & mask, a2 = l1 & mask, a3 = h1 & mask;
#pragma unroll
                                for (int cg = 0; cg < CG; ++cg) {
                                    int d[4];
                                    mma(d, a0, a1, a2, a3, B[cg][s].x, B[cg][s].y);
                                    tl[cg][s] = pair_fma(sd[cg][s], pair_of(__int2float_rn(d[0]), __int2float_rn(d[1])), sn[cg][s]);
                                    th[cg][s] = pair_fma(sd[cg][s], pair_of(__int2float_rn(d[2]), __int2float_rn(d[3])), sn[cg][s]);
                                }
                            }
#pragma unroll
                            for (int cg = 0; cg < CG; ++cg) {
                                float x, y;
                                split_pair(pair_add(pair_add(tl[cg][0], tl[cg][1]), pair_add(tl[cg][2], tl[cg][3])), x, y);
                                const f32pair vl = pair_of(__fmul_rn(dlo, x), __fmul_rn(dlo, y));
                                split_pair(pair_add(pair_add(th[cg][0], th[cg][1]), pair_add(th[cg][2], th[cg][3])), x, y);
                                const f32pair vh = pair_of(__fmul_rn(dhi, x), __fmul_rn(dhi, y));
                                if (jj == 0) { ve[m][cg][0] = vl; ve[m][cg][1] = vh; }
                                else { ve[m][cg][0] = pair_add(ve[m][cg][0], vl); ve[m][cg][1] = pair_add(ve[m][cg][1], vh); }
                            }
                        }
                    }
#pragma unroll
                    for (int m = 0; m < MT; ++m)
#pragma unroll
                        for (int cg = 0; cg < CG; ++cg)
#pragma unroll
                            for (int e = 0; e < 2; ++e) us[m][cg][e] = jp == 0 ? ve[m][cg][e] : pair_add(us[m][cg][e], ve[m][cg][e]);
                }
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty + slot * 8) : "memory");
                if (++slot == slots) { slot = 0; phase ^= 1; }
            }
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(wempty + wslot * 8) : "memory");
            if (++wslot == sp.wslots) { wslot = 0; wphase ^= 1; }
            if (on && seg * gs + i < ng) {
                if (seg == 0) {                    // us = p_i; the first segment's groups are added as they come
#pragma unroll
                    for (int m = 0; m < MT; ++m)
#pragma unroll
                        for (int cg = 0; cg < CG; ++cg)
#pragma unroll
                            for (int e = 0; e < 2; ++e) acc[m][cg][e] = i == 0 ? us[m][cg][e] : pair_add(acc[m][cg][e], us[m][cg][e]);
                } else {                           // the others' wait in shared memory: [group][tile][column group][16 rows][8 columns]
#pragma unroll
                    for (int m = 0; m < MT; ++m)
                        if (row + m < n) {
                            float *dst = sums + ((size_t((seg - 1) * gs + i) * sp.tiles + row + m) * NG + half * CG) * 128 + g * 8 + 2 * tig;
#pragma unroll
                            for (int cg = 0; cg < CG; ++cg) {
                                *reinterpret_cast<f32pair *>(dst + cg * 128) = us[m][cg][0];
                                *reinterpret_cast<f32pair *>(dst + cg * 128 + 64) = us[m][cg][1];
                            }
                        }
                }
            }
        }
        if (S > 1) asm volatile("bar.sync 1, %0;" ::"n"(NW * 32) : "memory");     // the other segments' group sums are there
        if (on && seg == 0) {
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                if (row + m >= n) break;
                const int tile = t0 + tb + row + m;
#pragma unroll
                for (int cg = 0; cg < CG; ++cg) {
                    const int col = half * 16 + cg * 8 + 2 * tig;
                    const float *p = sums + (size_t(row + m) * NG + half * CG + cg) * 128 + g * 8 + 2 * tig;
                    for (int gi = 0; gi < ng - gs; ++gi, p += sp.tiles * NG * 128) {
                        acc[m][cg][0] = pair_add(acc[m][cg][0], *reinterpret_cast<const f32pair *>(p));
                        acc[m][cg][1] = pair_add(acc[m][cg][1], *reinterpret_cast<const f32pair *>(p + 64));
                    }
                    float v[4];                    // (row g, columns col, col + 1), (row g + 8, ...)
                    split_pair(acc[m][cg][0], v[0], v[1]);
                    split_pair(acc[m][cg][1], v[2], v[3]);
                    if (a.swiglu) {                // rows r and r + 8 of a tile: gate and up of one FFN row
#pragma unroll
                        for (int e = 0; e < 2; ++e)
                            if (col + e < a.ncol) a.out[size_t(col + e) * a.out_stride + tile * 8 + g] = __fmul_rn(silu_f(v[e]), v[2 + e]);
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int rw = tile * 16 + g + (e >> 1) * 8, c = col + (e & 1);
                            if (rw < a.M && c < a.ncol) {
                                float r = v[e];
                                if (a.resid) r = __fadd_rn(r, a.resid[size_t(c) * a.resid_stride + rw]);
                                a.out[size_t(c) * a.out_stride + rw] = r;
                            }
                        }
                    }
                }
            }
        }
        if (S > 1 && pass + 1 < npass) asm volatile("bar.sync 1, %0;" ::"n"(NW * 32) : "memory");
    }
}

}  // namespace

namespace bnk {

cudaError_t launch_q2_gemm_wide(cudaStream_t st, int sm_count, Q2GemmArgs a, bool pdl) {
    static bool attr_set = false;
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(k_q2_gemm_wide, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX);
        if (e != cudaSuccess) return e;
        attr_set = true;
    }
    const int ng = a.K / 512, tiles = (a.M + 15) / 16, grid = std::min(tiles, sm_count);
    a.share = {tiles / grid, tiles % grid};
    const int nt = a.share.q + (a.share.r > 0);
    // segments: the warps over, as far as the sums and three image steps fit
    Split sp;
    int smem = 0;
    for (sp.segs = std::max(1, std::min(ng, NW / (H * ((nt + MT - 1) / MT))));; --sp.segs) {
        sp.gs = (ng + sp.segs - 1) / sp.segs;
        sp.segs = (ng + sp.gs - 1) / sp.gs;
        const int room = NW / (H * sp.segs) * MT, npass = (nt + room - 1) / room, groups = npass * sp.gs;
        sp.tiles = std::min(room, ((nt + npass - 1) / npass + MT - 1) / MT * MT);
        const int step = sp.segs * NCP * IMG_COL * 2, group = sp.segs * sp.tiles * Q2_PIECE;
        sp.imgs = HEAD + (ng - sp.gs) * sp.tiles * NCP * 64;
        sp.slots = std::min({MAX_SLOTS, 2 * groups, (SMEM_MAX - sp.imgs - 2 * group) / step});
        if (sp.segs > 1 && sp.slots < std::min(3, 2 * groups)) continue;
        sp.wts = sp.imgs + sp.slots * step;
        sp.wslots = std::min({MAX_WSLOTS, groups, (SMEM_MAX - sp.wts) / group});
        smem = sp.wts + sp.wslots * group;
        break;
    }
    if (a.next.W) a.next.share = {a.next.units / grid, a.next.units % grid};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = std::max(smem, 116 << 10);                      // one CTA per SM, as in q2_gemv.cu
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    BN_COUNT(1);
    return cudaLaunchKernelEx(&cfg, k_q2_gemm_wide, a, sp);
}

}  // namespace bnk
