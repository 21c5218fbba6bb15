// ptq_stream.cu - PTQ1_0 x q8_1 matrix-vector product straight from the file's native rows (bn_gemv_q81), any K that is a
// whole number of 128-weight blocks and any 4-byte aligned matrix.
//
// The arithmetic and the way the trits reach the tensor cores are those of ptq_gemv.cu: one multiply by 3^(t+1) turns two weight
// bytes into an int8 operand register [r, T, r', T'] and the operand table of the activation pack (two columns per sub-block)
// does the rest. What bounds it is instruction issue and, nearly as much, memory: per 16 x 128 weights 32 products (two cycles of a
// scheduler each, as shift-and-adds one), 8 byte permutes, 8 tensor-core steps, 7 loads and a quarter of the epilogue, 80 warp
// instructions in all, against 145 in the kernel this replaces (two blocks per warp, sums across the warps of the CTA inside the loop,
// 16 bulk copies of 896 bytes per 16 rows): 248 320 x 4096 in 116 us before. The tensor cores need 27 us of it (half of every operand
// is residue bytes). A line of DRAM holds parts of two pieces of a row, which are taken at different times: 445 MB are read for this
// matrix of 222 (131 072 x 4096: 232 MB for 117), 68 us at the copy rate. Measured beside it: pieces of a tile taken side by side, so
// that no line comes in twice: with the warps' operands reloaded 96 us, from a table in shared memory and 16 warps 80 us.
//
// Work split. A CTA of 12 warps (16 of 128 registers each were slower: 16.1 against 13.9 us at 24 576 x 4096) owns a run of 16-row tiles
// over all of K. The pieces (16 rows x 4 blocks, the unit p_g of the summation order) of a run are dealt to the warps group-major, so a
// warp stays with one group's operand table - 64 registers - for most of its pieces; group sums meet in shared memory, where one thread
// per row adds them in ascending order.
// Data movement. A piece is 16 rows of 112 bytes, brought by cp.async into a ring of its warp's own: 16 or 8 bytes at a time where the
// rows' alignment allows, else the up to eight 16-byte granules that hold a row's bytes (ALIGN 0, granules.cuh), from which a lane reads
// at its row's place. Four bytes at a time, 14 copies a piece instead of four, took the issue slots: 30 000 x 4736 22.6 -> 18.1 us, 50 000
// x 6528 43.1 -> 32.0, 100 000 x 2176 34.8 -> 26.7. Rows of more alignment lose by it (1000 x 8192 6.9 against 7.5, 20 000 x 12 288 26.5
// against 27.7; 60 000 x 1280 13.8 against 13.5). The pitch of 112 bytes is free of bank conflicts for every load of the loop: eight rows
// start four banks apart and the four lanes of a row read words 0, 2, 3, 5 (one in each residue modulo 4). So is that of 144, but the rows
// of an odd number of blocks lie at different places in their granules, which makes most loads conflicts of two.
#include "granules.cuh"
#include "ops.cuh"
#include "q2.cuh"
#include "rotate_quant.cuh"

#include <algorithm>

namespace {
using namespace bnk;

constexpr int NT = 384, NW = NT / 32, MAX_PIECES = 1536, MAGIC = 0x4B400000;   // bits of 12582912.0f

template <int ALIGN> struct Ring { static constexpr int STAGES = ALIGN ? 5 : 4, PITCH = ALIGN ? 112 : 144, PIECE = 16 * PITCH, BYTES = NW * STAGES * PIECE; };

struct StreamArgs {
    const unsigned char *W;
    int M, nb;
    const uint32_t *q81;                       // q8_1 records, 36 dwords per block
    const uint2 *bf;                           // operand table, [block][8][32 lanes]
    float *out;
    int q, r, run;                             // CTA c owns q tiles, the first r CTAs one more; tiles per run
};

__device__ __forceinline__ void mma(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint2 b) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b.x), "r"(b.y));
}
// the first step of a chain takes its accumulators from constants: the dot that is read directly starts at MAGIC
__device__ __forceinline__ void mma_first(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint2 b) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%10,%11};\n"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b.x), "r"(b.y), "r"(MAGIC), "r"(0));
}
template <int ALIGN> __device__ __forceinline__ void cp_async(uint32_t dst, const void *src) {
    if (ALIGN == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(ALIGN) : "memory");
}

struct Bytes { uint32_t h0, h1, h2, hq; };
__device__ __forceinline__ Bytes split(uint32_t f, uint32_t s, uint32_t w6, uint32_t sel2) {
    return {__byte_perm(f, 0u, 0x4240u), __byte_perm(f, 0u, 0x4341u), __byte_perm(s, 0u, sel2), __byte_perm(w6, 0u, 0x4140u)};
}
// two blocks of the same 16 rows: two chains of eight dependent tensor-core steps side by side (products v * 3^(t+1), written out: as the
// loop below 1 % slower)
__device__ __forceinline__ void block_dots2(int (&c)[4], int (&e)[4], const uint32_t *r0, const uint32_t *r1, int first, int second, uint32_t sel2, uint32_t cq,
                                            const uint2 (&B)[8], const uint2 (&E)[8]) {
    const Bytes a = split(r0[first], r0[second], r0[6], sel2), b = split(r1[first], r1[second], r1[6], sel2);
    const Bytes f = split(r0[7 + first], r0[7 + second], r0[13], sel2), g = split(r1[7 + first], r1[7 + second], r1[13], sel2);
    mma_first(c, a.h0 * 3u, b.h0 * 3u, a.h0 * 9u, b.h0 * 9u, B[0]);
    mma_first(e, f.h0 * 3u, g.h0 * 3u, f.h0 * 9u, g.h0 * 9u, E[0]);
    mma(c, a.h0 * 27u, b.h0 * 27u, a.h0 * 81u, b.h0 * 81u, B[1]);
    mma(e, f.h0 * 27u, g.h0 * 27u, f.h0 * 81u, g.h0 * 81u, E[1]);
    mma(c, a.h0 * 243u, b.h0 * 243u, a.h1 * 3u, b.h1 * 3u, B[2]);
    mma(e, f.h0 * 243u, g.h0 * 243u, f.h1 * 3u, g.h1 * 3u, E[2]);
    mma(c, a.h1 * 9u, b.h1 * 9u, a.h1 * 27u, b.h1 * 27u, B[3]);
    mma(e, f.h1 * 9u, g.h1 * 9u, f.h1 * 27u, g.h1 * 27u, E[3]);
    mma(c, a.h1 * 81u, b.h1 * 81u, a.h1 * 243u, b.h1 * 243u, B[4]);
    mma(e, f.h1 * 81u, g.h1 * 81u, f.h1 * 243u, g.h1 * 243u, E[4]);
    mma(c, a.h2 * 3u, b.h2 * 3u, a.h2 * 9u, b.h2 * 9u, B[5]);
    mma(e, f.h2 * 3u, g.h2 * 3u, f.h2 * 9u, g.h2 * 9u, E[5]);
    mma(c, a.h2 * 27u, b.h2 * 27u, a.h2 * 81u, b.h2 * 81u, B[6]);
    mma(e, f.h2 * 27u, g.h2 * 27u, f.h2 * 81u, g.h2 * 81u, E[6]);
    mma(c, a.h2 * 243u, b.h2 * 243u, a.hq * cq, b.hq * cq, B[7]);
    mma(e, f.h2 * 243u, g.h2 * 243u, f.hq * cq, g.hq * cq, E[7]);
}
// the same with each product from the one before, as a shift-and-add; operand register r is the byte pairs r / 5 times 3^(r % 5 + 1), the
// sixteenth the last two bytes at a level of the lane's own
__device__ __forceinline__ void block_dots2_chained(int (&c)[4], int (&e)[4], const uint32_t *r0, const uint32_t *r1, int first, int second, uint32_t sel2, uint32_t cq,
                                            const uint2 (&B)[8], const uint2 (&E)[8]) {
    const Bytes v[4] = {split(r0[first], r0[second], r0[6], sel2), split(r1[first], r1[second], r1[6], sel2),
                        split(r0[7 + first], r0[7 + second], r0[13], sel2), split(r1[7 + first], r1[7 + second], r1[13], sel2)};
    uint32_t h[3][4];
#pragma unroll
    for (int k = 0; k < 4; ++k) { h[0][k] = v[k].h0; h[1][k] = v[k].h1; h[2][k] = v[k].h2; }
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        uint32_t x[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int r = 2 * m + i;
                x[i][k] = r == 15 ? v[k].hq * cq : times3(h[r / 5 % 3][k]);
                if (r < 15) h[r / 5 % 3][k] = x[i][k];
            }
        if (m == 0) { mma_first(c, x[0][0], x[0][1], x[1][0], x[1][1], B[0]); mma_first(e, x[0][2], x[0][3], x[1][2], x[1][3], E[0]); }
        else { mma(c, x[0][0], x[0][1], x[1][0], x[1][1], B[m]); mma(e, x[0][2], x[0][3], x[1][2], x[1][3], E[m]); }
    }
}
// x[b]: this lane's sub-block (lane & 3) of block b -> the sum (t0 + t1) + (t2 + t3) of block lane & 3
__device__ __forceinline__ float quad_transpose_sum(const float (&x)[4], bool odd, bool hi) {
    const float ya = __fadd_rn(odd ? x[1] : x[0], __shfl_xor_sync(0xFFFFFFFFu, odd ? x[0] : x[1], 1));
    const float yb = __fadd_rn(odd ? x[3] : x[2], __shfl_xor_sync(0xFFFFFFFFu, odd ? x[2] : x[3], 1));
    return __fadd_rn(hi ? yb : ya, __shfl_xor_sync(0xFFFFFFFFu, hi ? ya : yb, 2));
}

template <int ALIGN, bool MANY>
__global__ void __launch_bounds__(NT, 1) k_ptq_stream(const StreamArgs a) {
    constexpr int ST = Ring<ALIGN>::STAGES, PITCH = Ring<ALIGN>::PITCH, PIECE = Ring<ALIGN>::PIECE;
    extern __shared__ __align__(16) unsigned char smem[];
    uint4 *offs = reinterpret_cast<uint4 *>(smem + Ring<ALIGN>::BYTES);    // where a lane's four 16-byte copies of a piece start
    float *sums = reinterpret_cast<float *>(smem + Ring<ALIGN>::BYTES + 512); // [group][tile of the run][16]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tig = lane & 3, cta = blockIdx.x;
    const int nb = a.nb, ng = (nb + 3) >> 2;
    const int t0 = cta * a.q + min(cta, a.r), nt = a.q + (cta < a.r);
    const size_t rowbytes = size_t(nb) * 28;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (ALIGN == 16 && warp == 1) {
        uint32_t o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) { const int c = min(i * 32 + lane, 111); o[i] = uint32_t(c / 7) * uint32_t(rowbytes) + (c % 7) * 16; }
        offs[lane] = make_uint4(o[0], o[1], o[2], o[3]);
    }
    __syncthreads();
    if (tid == 0) {                            // the first part of this CTA's rows starts towards L2 (the matrix may not be read before the wait)
        const uintptr_t p = (reinterpret_cast<uintptr_t>(a.W + size_t(t0) * 16 * rowbytes) + 15) & ~uintptr_t(15);
        const uintptr_t e = reinterpret_cast<uintptr_t>(a.W + size_t(min((t0 + nt) * 16, a.M)) * rowbytes) & ~uintptr_t(15);
        const long bytes = min(long(e) - long(p), 131072l);
        for (long o = 0; o < bytes; o += 16384) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p + o), "r"(int(min(16384l, bytes - o))) : "memory");
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");

    const int first = (tig == 0) ? 0 : (tig == 1) ? 2 : (tig == 2) ? 3 : 5, second = tig < 2 ? 1 : 4;
    const uint32_t cq = (tig == 0) ? 3u : (tig == 1) ? 9u : (tig == 2) ? 27u : 81u, sel2 = (tig & 1) ? 0x4341u : 0x4240u;
    const bool odd = tig & 1, hi = tig & 2;
    const unsigned char *ring = smem + warp * ST * PIECE;
    const uint32_t ring_s = uint32_t(__cvta_generic_to_shared(ring));
    // `at`: where this lane finds its words of row g (and, eight pitches on, of row g + 8). ALIGN 0, nfull and nlast: whether the granule
    // that this lane copies holds any of a full group's blocks, of the last group's. (Worked out per piece, a CTA's first piece came 0.1 us
    // later. With all eight granules of a short last group, and the matrix's first and last tiles through a rolled loop: 333 x 384 2.61 us,
    // 2.50 so and 2.58 with 4-byte copies; 200 000 x 640 20.4, 18.4, 25.0; 20 000 x 5760 12.9, 13.2, 16.4.)
    const uintptr_t w0 = reinterpret_cast<uintptr_t>(a.W);
    const Granules gran = {w0, w0 + size_t(a.M) * rowbytes, rowbytes, a.M, nb};
    const int place = gran.place(lane >> 3);
    const bool nfull = gran.holds(place, 0, lane & 7), nlast = gran.holds(place, ng - 1, lane & 7);
    const int at = g * PITCH + (ALIGN ? 0 : gran.place(g));
    uint2 B[4][8];
    float d[4], ns[4];
    int group = -1;
    bool live = true;                          // block 4 * group + tig exists
    auto set_group = [&](int gr) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int b = gr * 4 + j;
            const bool on = b < nb;
#pragma unroll
            for (int m = 0; m < 8; ++m) B[j][m] = on ? a.bf[(size_t(b) * 8 + m) * 32 + lane] : make_uint2(0u, 0u);
            const uint32_t ds = on ? a.q81[size_t(b) * Q81_DWORDS + tig] : 0u;
            d[j] = half_bits_to_float(ds); ns[j] = -half_bits_to_float(ds >> 16);
        }
        live = gr * 4 + tig < nb;
        group = gr;
    };
    for (int c0 = 0; c0 < nt; c0 += a.run) {
        const int n = min(a.run, nt - c0), total = n * ng;
        const int p0 = int((long long)warp * total / NW), p1 = int((long long)(warp + 1) * total / NW);
        int fg = p0 / n, ft = p0 - fg * n, fs = 0, fp = p0;       // next piece to request: group, tile, slot
        auto request = [&] {
            if (fp < p1) {
                constexpr int W = ALIGN ? ALIGN : 4, CH = 112 / W; // copies per row
                const unsigned char *src = a.W + size_t(t0 + c0 + ft) * 16 * rowbytes + size_t(fg) * 112;
                const int rmax = a.M - 1 - (t0 + c0 + ft) * 16, have = ALIGN == 16 ? CH : min(4, nb - fg * 4) * 28 / W;
                const uint32_t dst = ring_s + fs * PIECE;
                if (ALIGN == 0) {
                    const uint32_t to = dst + (lane >> 3) * PITCH + (lane & 7) * 16;
                    gran.copies((t0 + c0 + ft) * 16, fg, lane, fg + 1 < ng ? nfull : nlast,
                                [&](int i, uintptr_t s) { cp_async<16>(to + i * 4 * PITCH, reinterpret_cast<const void *>(s)); },
                                [&](int i, int k, uintptr_t s) { cp_async<4>(to + i * 4 * PITCH + k, reinterpret_cast<const void *>(s)); });
                } else if (ALIGN == 16 && rmax >= 15) {
                    const uint4 o = offs[lane];
                    cp_async<16>(dst + lane * 16, src + o.x); cp_async<16>(dst + lane * 16 + 512, src + o.y); cp_async<16>(dst + lane * 16 + 1024, src + o.z);
                    if (lane < 16) cp_async<16>(dst + lane * 16 + 1536, src + o.w);
                } else
#pragma unroll
                for (int i = 0; i < (16 * CH + 31) / 32; ++i) {
                    const int c = i * 32 + lane, row = c / CH, k = c - row * CH;
                    if (c < 16 * CH && (ALIGN == 16 || k < have)) cp_async<W>(dst + c * W, src + size_t(min(row, rmax)) * rowbytes + k * W);
                }
                ++fp; if (++ft == n) { ft = 0; ++fg; }
                if (++fs == ST) fs = 0;
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        for (int i = 0; i < ST - 1; ++i) request();
        int gr = fg, slot = 0;
        gr = p0 / n;
        int tl = p0 - gr * n;
        for (int p = p0; p < p1; ++p) {
            if (gr != group) set_group(gr);
            asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
            __syncwarp();                      // every lane's copies are there, and every lane is done with the slot requested next
            request();
            const uint32_t *r0 = reinterpret_cast<const uint32_t *>(ring + slot * PIECE + at), *r1 = r0 + 8 * PITCH / 4;
            int c[4][4];
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
                if (MANY) block_dots2_chained(c[j], c[j + 1], r0 + 7 * j, r1 + 7 * j, first, second, sel2, cq, B[j], B[j + 1]);
                else block_dots2(c[j], c[j + 1], r0 + 7 * j, r1 + 7 * j, first, second, sel2, cq, B[j], B[j + 1]);
            }
            const uint32_t da = r0[7 * tig + 6], db = r1[7 * tig + 6];
            float xa[4], xb[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                xa[j] = fmaf(d[j], __fsub_rn(__int_as_float(c[j][0] - 3 * c[j][1]), 12582912.0f), ns[j]);
                xb[j] = fmaf(d[j], __fsub_rn(__int_as_float(c[j][2] - 3 * c[j][3]), 12582912.0f), ns[j]);
            }
            float va = __fmul_rn(half_bits_to_float(da >> 16), quad_transpose_sum(xa, odd, hi));
            float vb = __fmul_rn(half_bits_to_float(db >> 16), quad_transpose_sum(xb, odd, hi));
            if (ALIGN != 16 && !live) va = vb = 0.0f;
            va = __fadd_rn(va, __shfl_xor_sync(0xFFFFFFFFu, va, 1)); vb = __fadd_rn(vb, __shfl_xor_sync(0xFFFFFFFFu, vb, 1));
            va = __fadd_rn(va, __shfl_xor_sync(0xFFFFFFFFu, va, 2)); vb = __fadd_rn(vb, __shfl_xor_sync(0xFFFFFFFFu, vb, 2));
            if (tig < 2) sums[p * 16 + g + 8 * tig] = tig ? vb : va;
            if (++tl == n) { tl = 0; ++gr; }
            if (++slot == ST) slot = 0;
        }
        __syncthreads();
        for (int i = tid; i < n * 16; i += NT) {
            const int row = (t0 + c0) * 16 + i;
            if (row >= a.M) break;
            const float *p = sums + i;
            float s = p[0];
            int k = 1;
            for (; k + 7 <= ng; k += 7) {      // seven loads, then their adds in ascending order
                float x[7];
#pragma unroll
                for (int u = 0; u < 7; ++u) x[u] = p[(k + u) * n * 16];
#pragma unroll
                for (int u = 0; u < 7; ++u) s = __fadd_rn(s, x[u]);
            }
            for (; k < ng; ++k) s = __fadd_rn(s, p[k * n * 16]);
            a.out[row] = s;
        }
        if (c0 + n < nt) __syncthreads();
    }
}

template <int ALIGN, bool MANY = false>
cudaError_t launch_a(cudaStream_t st, int grid, const StreamArgs &a) {
    const size_t smem = size_t(Ring<ALIGN>::BYTES) + 512 + size_t(a.run) * ((a.nb + 3) / 4) * 64;
    static bool set = false;
    if (!set) {
        cudaError_t e = cudaFuncSetAttribute(k_ptq_stream<ALIGN, MANY>, cudaFuncAttributeMaxDynamicSharedMemorySize, Ring<ALIGN>::BYTES + 512 + MAX_PIECES * 64);
        if (e != cudaSuccess) return e;
        set = true;
    }
    launch(k_ptq_stream<ALIGN, MANY>, dim3(grid), dim3(NT), smem, st, a);
    return cudaGetLastError();
}

}  // namespace

namespace bnk {

bool ptq_stream_supported(int K) { return (K / 128 + 3) / 4 <= MAX_PIECES; }

cudaError_t ptq_stream(cudaStream_t st, int sm_count, const void *W, int M, int K, const uint32_t *pack, float *out) {
    StreamArgs a = {};
    a.W = static_cast<const unsigned char *>(W); a.M = M; a.nb = K / 128;
    a.q81 = pack; a.bf = reinterpret_cast<const uint2 *>(pack + size_t(a.nb) * Q81_DWORDS); a.out = out;
    const int tiles = (M + 15) / 16, grid = std::min(tiles, sm_count), ng = (a.nb + 3) / 4;
    a.q = tiles / grid; a.r = tiles % grid;
    const int most = a.q + (a.r > 0);
    a.run = std::min(most, MAX_PIECES / ng);
    // the widest copy that every row of every piece starts on (4 bytes: granules)
    const uintptr_t align = reinterpret_cast<uintptr_t>(W) | uintptr_t(a.nb * 28);
    // A chain of shift-and-adds per half-word pair where a CTA has many pieces (248 320 x 4096: 81.6 -> 77.5 us in a loop over the matrix,
    // 87.1 -> 84.3 with two matrices in turn, 88.9 -> 87.2 with the quantiser in front; 30 000 x 8192 23.9 -> 23.4 in the loop),
    // products side by side where the first piece's latency counts (1024 x 4096 3.2 against 3.4 us, 7000 x 3584 5.4 against
    // 5.5) and where copies of 8 bytes take the issue slots.
    const bool many = most * ng >= 10 * NW;
    if (align % 16 == 0) return many ? launch_a<16, true>(st, grid, a) : launch_a<16>(st, grid, a);
    if (align % 8 == 0) return launch_a<8>(st, grid, a);
    return many ? launch_a<0, true>(st, grid, a) : launch_a<0>(st, grid, a);
}

}  // namespace bnk
