// q2_gemm.cu - the projection of several activation columns (prefill tokens, concurrent sequences) over the two-bit weight
// tiles of q2.cuh: integer tensor-core dots per (row, column, sub-block), combined in fp32 in the single-column kernel's order,
//     t_sb = fma(d, I, -s); v = d_w ((t0 + t1) + (t2 + t3)); p_g = (v0 + v1) + (v2 + v3); out = p_0 + p_1 + ...
// so a column is bit-identical to the single-column projection of its vector.
//
// What bounds it: memory at 8 columns; beyond, the fp32 combination, which the contract fixes at 26 packed operations per
// (16 rows, 8 columns, 128 weights) - 13 cycles of the SM's FMA pipes - against 4 mma (8 cycles of the tensor cores) and 16
// ANDs per 16 rows. The accumulators of mma.sync are registers, in the layout the combination wants; tcgen05 would bring them
// through tensor memory and hand-offs between warps: the kernel that did so, with the operand decoded into tensor memory, took
// 28 / 33 us for 24 576 x 4096 at 8 / 16 columns (a tcgen05.mma of 128 rows costs 190 cycles whatever its column count, and the
// tensor pipe is idle either way). Here, weights from DRAM, back to back, without the preparation of the columns: 11.1 / 15.4 us;
// 4096 x 12 288: 7.2 / 11.5 us.
//
// Work split. A CTA of 12 or 16 warps owns a run of row tiles over all of K. K is walked in waves of `kc` groups (512 weights each);
// a wave's piece of the activation image is double-buffered in shared memory. A wave's units (MT row tiles, one group, up to 16
// columns) are dealt to the warps; a unit keeps everything in registers and leaves its group sums p_g in shared memory, where
// after a barrier every thread adds its own (row, column)s' in ascending order. MT = 2 or 3 (1 for native rows, and where a CTA has few) row tiles share a group's operands and
// scales: with one, shared-memory reads (24 wavefronts per 16 rows x 8 columns x 128 weights) would bound the loop.
#include "q2.cuh"
#include "rotate_quant.cuh"

#include <algorithm>

namespace {
using namespace bnk;

constexpr int SMEM_MAX = 227 << 10;
constexpr int IMG_COL = 160;                   // image bytes per column and block (act_image.cuh)
constexpr int MAX_TILES = 12;                  // row tiles per pass over K (a thread keeps their running sums in registers)

// FIRST: the load stays where it stands, in front of a wait
template <bool FIRST> __device__ __forceinline__ uint4 weights16(const uint8_t *p) {
    if (!FIRST) return __ldg(reinterpret_cast<const uint4 *>(p));
    uint4 v;
    asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
// NATIVE: W holds the file's rows; a warp unpacks each of its pieces in a corner of shared memory of its own first. Bound by that
// unpacking, 250 instructions a piece: 16 warps also for 8 columns (128 x 12 288: 10.2 -> 9.1 us, 4096 rows and more the same).
// 12 warps (168 registers a thread), or units of one tile, have room for a unit's weights to be on their way while the image is: LATE.
// EARLY: the dependent launch is released ahead of this kernel's own dependency wait. Late is what k_gdn_core needs, and costs nothing
// but in the build of 16 columns and two tiles on 12 warps, alone with its preparation (12 288 x 4096 11.60 us early, 11.75 late;
// 10 000 x 6144 14.53 and 14.70). A model's passes run the late build throughout: with both in turn four blocks of 12 sequences take
// 330.5 us, with the late one 328.7.
template <int NCP, int MT, int NT, bool NATIVE, bool EARLY>
__global__ void __launch_bounds__(NT, 1) k_q2_gemm(const Q2GemmArgs a) {
    constexpr int NW = NT / 32;
    constexpr bool LATE = NATIVE || MT == 1 || (NT == 384 && MT == 2);
    constexpr int NG = NCP / 8, NGW = NG >= 2 ? 2 : 1, H = NG / NGW;      // column groups: all, per unit; units across the columns
    // A unit's group by a division, or by a multiplier that waits in shared memory (in a register it spills 16 columns' units). The
    // division is up to a tenth of a unit: 12 288 x 4096 x 8 8.84 -> 8.67 us, native 3000 x 5120 x 4 8.76 -> 8.35, 16 columns native
    // 4096 x 12 288 20.8 -> 20.4. Two builds are faster with it: three tiles (20 000 x 12 288 x 8 26.6 us, 28.6 without) and 16 columns
    // on 12 warps (9000 x 2048 7.01, 7.18).
    constexpr bool DIVIDE = MT == 3 || (NCP == 16 && MT == 2 && NT == 384);
    constexpr int ITEMS = (MAX_TILES * 16 * NCP + NT - 1) / NT;
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tig = lane & 3, cta = blockIdx.x;
    const int ng = a.K >> 9, kc = a.kc, nw = (ng + kc - 1) / kc;
    const int t0 = cta * a.share.q + min(cta, a.share.r), nt = a.share.q + (cta < a.share.r);
    const int npass = (nt + a.tiles - 1) / a.tiles, nchunks = nw == 1 ? 1 : npass * nw;
    const uint32_t gbytes = 4 * NCP * IMG_COL;                            // image bytes of a group
    const uint32_t bars = uint32_t(__cvta_generic_to_shared(smem));
    unsigned char *img = smem + 128;
    float *sums = reinterpret_cast<float *>(img + (nchunks > 1 ? 2 : 1) * kc * gbytes);
    unsigned char *stage = reinterpret_cast<unsigned char *>(sums + size_t(kc) * a.tiles * 16 * NCP) + warp * Q2_PIECE;       // NATIVE only
    const size_t rowbytes = size_t(a.K >> 7) * 28;
    auto request = [&](int q, int w) {                                     // image piece of chunk q (its wave w) into buffer q & 1
        const int g0 = w * kc, n = min(kc, ng - g0);
        const uint32_t bytes = uint32_t(n) * gbytes, bar = bars + (q & 1) * 8;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(uint32_t(__cvta_generic_to_shared(img)) + (q & 1) * kc * gbytes), "l"(a.image + size_t(g0) * gbytes), "r"(bytes), "r"(bar) : "memory");
    };
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bars));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bars + 8));
        if (!DIVIDE) {
            // i / nur = i * per >> 16 for the few hundred units of a wave (nur <= 12); the last pass may have fewer tiles
            auto per = [&](int n) { return 65536 / ((n + MT - 1) / MT) + 1; };
            asm volatile("st.shared.v2.s32 [%0], {%1, %2};" ::"r"(bars + 16), "r"(per(min(a.tiles, nt))), "r"(per(nt - (npass - 1) * a.tiles)) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (lane == 0) {
        // this CTA's weights (as far as the previous projection has not fetched them) and the next projection's towards L2
        const uint8_t *own = a.W + (NATIVE ? size_t(t0) * 16 * rowbytes : size_t(t0) * ng * Q2_PIECE);
        const int bytes = int(min(NATIVE ? size_t(min(nt * 16, a.M - t0 * 16)) * rowbytes : size_t(nt) * ng * Q2_PIECE, size_t(Q2_NEXT_BYTES)));
        for (int o = warp * 16384; o < bytes; o += NW * 16384) q2_prefetch(own + o, min(16384, bytes - o));
        q2_prefetch_next(a.next, cta, warp, NW);
    }
    if (EARLY) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // Released here, the kernel behind this one may read ahead of its own wait what was complete before this one's (k_gdn_core does).
    // Where this grid has a CTA on every SM the dependents have no room before one ends anyway.
    if (!EARLY) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (tid == 0) for (int q = 0; q < min(2, nchunks); ++q) request(q, q < nw ? q : 0);

    const f32pair magic2 = pair_of(__int_as_float(Q2_MAGIC), __int_as_float(Q2_MAGIC));
    bool alive = true;
    int q = 0;
    for (int pass = 0; pass < npass; ++pass) {
        const int tb = pass * a.tiles, n = min(a.tiles, nt - tb), nur = (n + MT - 1) / MT;      // this pass's tiles, units of rows
        const uint8_t *W = a.W + size_t(t0 + tb) * ng * Q2_PIECE;
        const uint32_t per_at = bars + (pass + 1 == npass ? 20 : 16);
        float acc[ITEMS];
        for (int w = 0; w < nw; ++w) {
            const int g0 = w * kc, gn = min(kc, ng - g0);
            const int buf = nchunks > 1 ? q & 1 : 0;
            // the wave's image piece, LATE: behind the loads (or the unpacking) of the first unit's weights
            bool here = nchunks == 1 && pass > 0;
            auto await_image = [&] { if (!here) { here = true; if (alive) alive = q2_wait(bars + buf * 8, (q >> 1) & 1, a.err); } };
            if (!LATE) await_image();
            const unsigned char *chunk = img + buf * kc * gbytes;
            for (int u = warp; u < gn * nur * H; u += NW) {
                int gl;
                if (DIVIDE) gl = u / (H * nur);
                else {
                    asm volatile("ld.shared.s32 %0, [%1];" : "=r"(gl) : "r"(per_at));
                    gl = u / H * gl >> 16;
                }
                const int h = u % H, ur = DIVIDE ? (u / H) % nur : u / H - gl * nur;
                const uint8_t *src = W + (size_t(ur * MT) * ng + g0 + gl) * Q2_PIECE;
                uint4 c[MT][4], dw[MT];
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const uint8_t *p = src + size_t(min(m, n - 1 - ur * MT)) * ng * Q2_PIECE;
                    if (NATIVE) {                  // lane (row g or g + 8, block tig); rows beyond M are zero
                        const int r0 = (t0 + tb + ur * MT + min(m, n - 1 - ur * MT)) * 16 + g;
#pragma unroll
                        for (int hf = 0; hf < 2; ++hf) {
                            const int r = r0 + 8 * hf;
                            const uint32_t *wp = reinterpret_cast<const uint32_t *>(a.W + size_t(r) * rowbytes) + ((g0 + gl) * 4 + tig) * 7;
                            uint32_t w[7];
#pragma unroll
                            for (int k = 0; k < 7; ++k) w[k] = r < a.M ? wp[k] : 0u;
                            q2_unpack_block(w, stage, hf, g, tig);
                        }
                        __syncwarp();
                        p = stage;
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) c[m][k] = NATIVE ? *reinterpret_cast<const uint4 *>(p + k * 512 + lane * 16) : weights16<LATE>(p + k * 512 + lane * 16);
                    dw[m] = NATIVE ? *reinterpret_cast<const uint4 *>(p + Q2_SCALES + g * 16) : weights16<LATE>(p + Q2_SCALES + g * 16);
                    if (NATIVE) __syncwarp();      // every lane has its part before the next piece is unpacked
                }
                if (LATE) await_image();
                f32pair us[MT][NGW][2], ve[MT][NGW][2];                   // v0 + v1; v0 or v2 (rows g, g + 8)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const unsigned char *blk = chunk + (gl * 4 + j) * (NCP * IMG_COL);
                    uint2 B[NGW][4];
                    f32pair sd[NGW][4], sn[NGW][4];
#pragma unroll
                    for (int cg = 0; cg < NGW; ++cg) {
                        const int c8 = h * NGW + cg;
#pragma unroll
                        for (int s = 0; s < 4; ++s) {
                            B[cg][s] = *reinterpret_cast<const uint2 *>(blk + c8 * 1024 + s * 256 + (tig >> 1) * 128 + g * 16 + (tig & 1) * 8);
                            const ulonglong2 sc = *reinterpret_cast<const ulonglong2 *>(blk + NCP * 128 + c8 * 256 + (s * 4 + tig) * 16);
                            // the dot of sub-block s comes as 4^s I
                            const float sh = s == 0 ? 1.0f : (s == 1 ? 0.25f : (s == 2 ? 0.0625f : 0.015625f));
                            sd[cg][s] = s ? pair_mul(sc.x, pair_of(sh, sh)) : sc.x;
                            sn[cg][s] = sc.y;
                        }
                    }
#pragma unroll
                    for (int m = 0; m < MT; ++m) {
                        const uint4 &lo = c[m][j >> 1], &hi = c[m][2 + (j >> 1)];
                        const uint32_t l0 = (j & 1) ? lo.z : lo.x, l1 = (j & 1) ? lo.w : lo.y, h0 = (j & 1) ? hi.z : hi.x, h1 = (j & 1) ? hi.w : hi.y;
                        const uint32_t dwj = j == 0 ? dw[m].x : (j == 1 ? dw[m].y : (j == 2 ? dw[m].z : dw[m].w));
                        const float dlo = half_bits_to_float(dwj), dhi = half_bits_to_float(dwj >> 16);
                        uint32_t A[4][4];
#pragma unroll
                        for (int s = 0; s < 4; ++s) {
                            const uint32_t mask = 0x03030303u << (2 * s);
                            A[s][0] = l0 & mask; A[s][1] = h0 & mask; A[s][2] = l1 & mask; A[s][3] = h1 & mask;
                        }
#pragma unroll
                        for (int cg = 0; cg < NGW; ++cg) {
                            f32pair tl[4], th[4];
#pragma unroll
                            for (int s = 0; s < 4; ++s) {
                                int d[4];
                                q2_mma_first(d, A[s][0], A[s][1], A[s][2], A[s][3], B[cg][s].x, B[cg][s].y);
                                tl[s] = pair_fma(sd[cg][s], pair_sub(pair_of(__int_as_float(d[0]), __int_as_float(d[1])), magic2), sn[cg][s]);
                                th[s] = pair_fma(sd[cg][s], pair_sub(pair_of(__int_as_float(d[2]), __int_as_float(d[3])), magic2), sn[cg][s]);
                            }
                            float x, y;
                            split_pair(pair_add(pair_add(tl[0], tl[1]), pair_add(tl[2], tl[3])), x, y);
                            const f32pair vl = pair_of(__fmul_rn(dlo, x), __fmul_rn(dlo, y));
                            split_pair(pair_add(pair_add(th[0], th[1]), pair_add(th[2], th[3])), x, y);
                            const f32pair vh = pair_of(__fmul_rn(dhi, x), __fmul_rn(dhi, y));
                            if (j == 0 || j == 2) { ve[m][cg][0] = vl; ve[m][cg][1] = vh; }
                            else if (j == 1) { us[m][cg][0] = pair_add(ve[m][cg][0], vl); us[m][cg][1] = pair_add(ve[m][cg][1], vh); }
                            else {
                                const f32pair pl = pair_add(us[m][cg][0], pair_add(ve[m][cg][0], vl)), ph = pair_add(us[m][cg][1], pair_add(ve[m][cg][1], vh));
                                if (ur * MT + m < n) {                    // [group][tile][column group][16 rows][8 columns]
                                    float *dst = sums + (size_t(gl * n + ur * MT + m) * NG + h * NGW + cg) * 128 + g * 8 + 2 * tig;
                                    *reinterpret_cast<f32pair *>(dst) = pl;
                                    *reinterpret_cast<f32pair *>(dst + 64) = ph;
                                }
                            }
                        }
                    }
                }
            }
            __syncthreads();                       // the wave's group sums are there, its image piece is no longer read
            if (nchunks > 1) {
                if (tid == 0 && q + 2 < nchunks) request(q + 2, (q + 2) % nw);
                ++q;
            }
            const int items = n * NG * 128;
#pragma unroll
            for (int k = 0; k < ITEMS; ++k) {
                const int i = tid + k * NT;
                if (i < items) {
                    const float *p = sums + i;
                    float s = w == 0 ? p[0] : __fadd_rn(acc[k], p[0]);
                    for (int gi = 1; gi < gn; ++gi) s = __fadd_rn(s, p[gi * items]);
                    acc[k] = s;
                }
            }
            if (w + 1 < nw) __syncthreads();
        }
        const int items = n * NG * 128;
        if (a.swiglu) {                            // rows r and r + 8 of a tile: gate and up of one FFN row
            __syncthreads();
#pragma unroll
            for (int k = 0; k < ITEMS; ++k) if (tid + k * NT < items) sums[tid + k * NT] = acc[k];
            __syncthreads();
            for (int i = tid; i < items / 2; i += NT) {
                const int tc = i >> 6, r = (i >> 3) & 7, col = (tc % NG) * 8 + (i & 7);
                if (col < a.ncol)
                    a.out[size_t(col) * a.out_stride + (t0 + tb + tc / NG) * 8 + r] = __fmul_rn(silu_f(sums[tc * 128 + r * 8 + (i & 7)]), sums[tc * 128 + 64 + r * 8 + (i & 7)]);
            }
        } else {
#pragma unroll
            for (int k = 0; k < ITEMS; ++k) {
                const int i = tid + k * NT, tc = i >> 7, row = (t0 + tb + tc / NG) * 16 + ((i >> 3) & 15), col = (tc % NG) * 8 + (i & 7);
                if (i < items && row < a.M && col < a.ncol) {
                    float r = acc[k];
                    if (a.resid) r = __fadd_rn(r, a.resid[size_t(col) * a.resid_stride + row]);
                    a.out[size_t(col) * a.out_stride + row] = r;
                }
            }
        }
        if (pass + 1 < npass) __syncthreads();
    }
}

// A wait that nothing will ever satisfy, with a short limit: the give-up path of q2_wait (error word = 2, kernel returns)
__global__ void k_wait_selftest_gemm(int *err) {
    __shared__ uint64_t bar;
    const uint32_t b = uint32_t(__cvta_generic_to_shared(&bar));
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\nfence.mbarrier_init.release.cluster;" ::"r"(b) : "memory");
        q2_wait(b, 0, err, 1 << 10);
    }
}

// Groups per wave: all of K where its image piece fits beside its group sums (one wave: no barrier in between, and the units spread over
// more warps), else as many as fit with the image piece twice. tiles: row tiles per pass, stages: bytes in which warps unpack.
int wave_bytes(int ng, int kc, int tiles, int ncp, int stages) {
    return 128 + kc * ((kc >= ng ? 1 : 2) * 4 * ncp * IMG_COL + tiles * 16 * ncp * 4) + stages;
}
int wave_groups(int ng, int tiles, int ncp, int stages) {
    int kc = ng;
    if (wave_bytes(ng, kc, tiles, ncp, stages) > SMEM_MAX) for (kc = std::min(ng - 1, 8); kc > 1 && wave_bytes(ng, kc, tiles, ncp, stages) > SMEM_MAX;) kc = (kc + 1) / 2;
    return kc;
}
// units one behind the other in a warp, over all waves of one pass
int unit_rounds(int ng, int tiles, int ncp, int mt, int warps) {
    const int kc = wave_groups(ng, tiles, ncp, 0);
    auto rounds = [&](int groups) { return ((tiles + mt - 1) / mt * groups + warps - 1) / warps; };
    return ng / kc * rounds(kc) + (ng % kc ? rounds(ng % kc) : 0);
}
constexpr int NATIVE_NT = 512;
template <int NCP, int MT, int NT, bool NATIVE = false, bool EARLY = false>
cudaError_t launch_t(cudaStream_t st, int sm_count, Q2GemmArgs a, bool pdl) {
    static bool attr_set = false;
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(k_q2_gemm<NCP, MT, NT, NATIVE, EARLY>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX);
        if (e != cudaSuccess) return e;
        attr_set = true;
    }
    const int ng = a.K / 512, tiles = (a.M + 15) / 16, grid = std::min(tiles, sm_count);
    a.share = {tiles / grid, tiles % grid};
    a.tiles = std::min(a.share.q + (a.share.r > 0), MAX_TILES);
    const int stages = NATIVE ? NT / 32 * Q2_PIECE : 0;
    a.kc = wave_groups(ng, a.tiles, NCP, stages);
    if (a.next.W) a.next.share = {a.next.units / grid, a.next.units % grid};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = std::max(wave_bytes(ng, a.kc, a.tiles, NCP, stages), 116 << 10);             // one CTA per SM, as in q2_gemv.cu
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    BN_COUNT(1);
    return cudaLaunchKernelEx(&cfg, k_q2_gemm<NCP, MT, NT, NATIVE, EARLY>, a);
}

}  // namespace

namespace bnk {

cudaError_t launch_q2_gemm(cudaStream_t st, int sm_count, const Q2GemmArgs &a, bool pdl, bool late) {
    const int ncp = a.ncol <= 8 ? 8 : (a.ncol <= 16 ? 16 : 32), tiles = (a.M + 15) / 16;
    // Units of several row tiles share operand reads, units of one spread over more warps. Times with the preparation of the columns.
    // One tile, 16 warps: a CTA with one tile (a second one in a unit is the first again: 1024 x 4096 x 8 5.3 us with units of two, 4.9
    // with one, 1024 x 8192 x 16 9.0 and 7.5), or so few units that most warps have none (3000 x 1024 x 8 4.4 and 4.0).
    // 8 columns, 12 warps: two or three tiles by the rounds of a warp times what a unit costs, its tiles and about one more for its
    // operands: 5500 x 4096 6.8 us with two, 6.3 with three; 8192 x 4096 7.1 and 8.4; 20 000 x 4096 from L2 11.0 and 9.6. Where that
    // is even (24 576 x 4096 from L2, say, where they are equal in a serving step): three if they divide the tiles. Three also for many
    // tiles that come from DRAM (the output head 82.6 us with three, 88 with two) and for several passes.
    // 16 columns, two tiles: the number of warps that leaves fewer of them without a unit in the last round, 16 on a tie (24 576 x 4096
    // 18.8 against 19.0 us; 4096 x 4096 6.8 with 12, 7.6 with 16).
    const int nt = (tiles + sm_count - 1) / sm_count, ng = a.K / 512, n = std::min(nt, MAX_TILES);
    const bool single = nt == 1 || nt * ng <= 4;
    if (ncp == 8) {
        if (single) return launch_t<8, 1, 512>(st, sm_count, a, pdl);
        const int two = unit_rounds(ng, n, 8, 2, 12) * 3, three = unit_rounds(ng, n, 8, 3, 12) * 4;
        const bool by_three = nt > (a.warm ? MAX_TILES : 6) || three < two || (three == two && nt % 3 == 0);
        return by_three ? launch_t<8, 3, 384>(st, sm_count, a, pdl) : launch_t<8, 2, 384>(st, sm_count, a, pdl);
    }
    if (ncp == 16) {
        if (single) return launch_t<16, 1, 512>(st, sm_count, a, pdl);
        if (unit_rounds(ng, n, 16, 2, 16) * 16 <= unit_rounds(ng, n, 16, 2, 12) * 12) return launch_t<16, 2, 512>(st, sm_count, a, pdl);
        return late ? launch_t<16, 2, 384>(st, sm_count, a, pdl) : launch_t<16, 2, 384, false, true>(st, sm_count, a, pdl);
    }
    // 32 columns: a wave of all of K fits only the smallest matrices, where this kernel's units fill more warps (4096 x 4096, with the
    // preparation of the columns: 12.6 against 13.6 us); beyond, q2_gemm_wide.cu
    return tiles <= 2 * sm_count && a.K <= 4096 ? launch_t<32, 2, 512>(st, sm_count, a, pdl) : launch_q2_gemm_wide(st, sm_count, a, pdl);
}

// Against unpacking into tiles first, with the preparation of the columns, rows from DRAM (us, tiles -> in place):
//   up to 8 columns   always: 1500 x 4096 10.3 -> 5.9, 3000 x 5120 9.6 -> 8.0, 24 576 x 4096 25.5 -> 22.8, 8192 x 12 288 26.5 -> 24.2
//                     (four row tiles a CTA and K from 14 336 on, where K goes in waves: between 0.94 and 1.09 of the other way)
//   9 to 16 columns   while K goes in one wave (20 000 x 5120 30.3 -> 27.9, 24 576 x 4096 31.0 -> 30.0), a CTA has up to three row tiles
//                     (7000 x 12 288 31.2 -> 28.9) or the tiles would take several chunks (24 576 x 12 288 95.5 -> 89.4). Otherwise every
//                     wave ends in a barrier behind one or two units a warp, and unpacking is the part that waits: 16 384 x 6144
//                     30.1 -> 32.5, 14 000 x 7168 28.3 -> 32.3, 8192 x 12 288 32.9 -> 34.9; of 226 such shapes the worst loses 4 %
//   17 and more       every piece is unpacked twice (a unit has 16 columns), which pays while a CTA has few pieces (row tiles x groups of
//                     512 weights): 1500 x 4096 x 24 17.9 -> 9.8 with 8 of them, 512 x 5120 14.9 -> 13.7 with 10, but 3000 x 5120
//                     17.6 -> 18.4 with 20 and 24 576 x 4096 41.8 -> 61.9
bool q2_gemm_in_place(int sm_count, int M, int K, int ncol, bool one_chunk) {
    const int ng = K / 512, tiles = ((M + 15) / 16 + sm_count - 1) / sm_count;
    if (ncol > 16) return tiles * ng <= 12;
    return ncol <= 8 || tiles <= 3 || !one_chunk || wave_groups(ng, std::min(tiles, MAX_TILES), 16, NATIVE_NT / 32 * Q2_PIECE) == ng;
}
cudaError_t launch_q2_gemm_native(cudaStream_t st, int sm_count, const Q2GemmArgs &a, bool pdl) {
    if (a.ncol <= 8) return launch_t<8, 1, NATIVE_NT, true>(st, sm_count, a, pdl);
    if (a.ncol <= 16) return launch_t<16, 1, NATIVE_NT, true>(st, sm_count, a, pdl);
    return launch_t<32, 1, NATIVE_NT, true>(st, sm_count, a, pdl);
}

cudaError_t launch_wait_selftest_gemm(cudaStream_t st, int *err) {
    BN_COUNT(1);
    k_wait_selftest_gemm<<<1, 32, 0, st>>>(err);
    return cudaGetLastError();
}

}  // namespace bnk
