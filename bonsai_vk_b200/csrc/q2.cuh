// q2.cuh - the load-time weight layout of the projections ("two-bit tiles") and the kernels' common pieces.
//
// A PTQ1_0 block packs five trits into a byte, and unpacking them is what bounds a projection that reads it directly: two
// integer operations per trit against 0.22 bytes of memory traffic. The model therefore keeps its projection weights a
// second time with two bits per trit (34 bytes per 128 weights instead of 28), arranged so that ONE bitwise AND turns
// four packed trits into a ready int8 tensor-core operand register:
//   * the four two-bit fields of a byte belong to the four 32-weight sub-blocks of its block, so the field that is masked
//     out selects the sub-block, and the value in place is 4^s * code (code = trit + 1 in {0, 1, 2}, at most 128: a u8);
//   * the factor 4^s stays in the exact int32 dot and is taken out through the activation scale: fma(d / 4^s, 4^s * I, -s)
//     is the same float as fma(d, I, -s), because scaling by a power of two is exact (d is an fp16 value, far from the
//     fp32 underflow range; 4^s * I < 2^22).
// A piece = 16 rows x 4 blocks (512 weights of K) = 2176 bytes, contiguous: 4 x 512 bytes of codes, then 128 bytes of fp16
// block scales. Within the codes lane (g = lane / 4, t = lane % 4) of a warp finds at [quarter q = 2R + m][lane] 16 bytes:
// row 8R + g, blocks 2m and 2m + 1, packed dwords 2t and 2t + 1 of each. Packed dword d, byte b, field s holds element
// 32s + 4d + b of the block. Scales: word [g][block] = (row g | row g + 8 << 16). Pieces follow each other group (of four
// blocks) by group, then row tile by row tile. Rows beyond M are zero.
// That is the m16n8k32 A-fragment order for "all 32 k-slots from one sub-block": the single-sequence kernel gives the eight
// columns of the instruction to (block, sub-block parity), the multi-column kernel to eight activation vectors.
#pragma once
#include "ops.cuh"

namespace bnk {

constexpr int Q2_PIECE = 2176, Q2_SCALES = 2048;

inline size_t q2_bytes(int M, int K) { return size_t((M + 15) / 16) * size_t(K / 512) * Q2_PIECE; }
// native row-major PTQ1_0 -> two-bit tiles; the pair: rows 0..7 of a tile from the first matrix, 8..15 from the second (gate and
// up of an FFN; M rows each, M % 8 == 0). K % 512 == 0.
void q2_repack(cudaStream_t st, const uint32_t *W, int M, int K, uint8_t *out);
void q2_repack_pair(cudaStream_t st, const uint32_t *Wa, const uint32_t *Wb, int M, int K, uint8_t *out);
// sign values -> one bit per value (set = -1), 8 values per byte
void pack_sign_bits(cudaStream_t st, const int32_t *signs, int n, uint8_t *bits);

enum Q2Prologue { Q2_PLAIN = 0, Q2_NORM = 1 };
// what follows this projection in the schedule: its weights (and norm weights) are prefetched into L2 from here
struct Q2Share { int q, r; };             // CTA c takes q units, the first r CTAs one more
// per CTA: 38 MB in all (31 from a split projection's 120), more than any projection of a block; the whole output head would push
// everything else out of L2
constexpr int Q2_NEXT_BYTES = 256 << 10;
struct Q2Next {
    const uint8_t *W = nullptr;
    int units = 0, unit_bytes = 0;        // row tiles and their bytes
    int max_bytes = Q2_NEXT_BYTES;        // per CTA
    const float *w = nullptr;
    int w_bytes = 0;
    Q2Share share = {0, 0};               // filled in by the launch: the units dealt to THIS launch's CTAs
    // recurrent state that the mixer behind this projection reads: `cols` pieces, any CTA any part of them
    const float *state = nullptr;
    int cols = 0, col_bytes = 0;
    size_t col_stride = 0;                // bytes
    // and the rows of that mixer's small projections: two matrices of `rows_bytes`
    const float *rows[2] = {nullptr, nullptr};
    int rows_bytes = 0;
};
struct Q2Args {
    const uint8_t *W;            // two-bit tiles
    int M, K;                    // valid rows; K % 512 == 0, K <= 16384
    int swiglu;                  // a pair of matrices: out[r] = silu(first_r) * second_r, M = rows of both together
    float *out;                  // optional
    const float *resid_in;       // with resid_out: resid_out = sum + resid_in
    float *resid_out;
    int pro;
    const float *x0, *w;         // input; Q2_NORM: x = rms_norm(x0) * w
    const uint8_t *sgn;          // sign bits of the K values
    int hat_block;
    float hat_inv, eps;
    float inv_k;                 // filled in by the launch: 1 / K when K is a power of two, else 0 (divide);
    int log_hat;                 // log2(hat_block);
    Q2Share share;               // the CTAs' shares of the row tiles;
    int slots, fin;              // ring slots; bytes of group sums from a cluster's CTAs
    int run, gstep;              // row tiles per run of group sums; warps modulo groups (divisions that would sit in front of the first piece)
    float *inv_out;              // Q2_NORM, optional: 1/sqrt(mean(x0^2) + eps)
    int late;                    // release the dependent launch behind this kernel's own dependency wait (see GdnStep)
    int lean;                    // leave room for the next kernel's CTA on the SM (a mixer follows)
    Q2Next next;
    int *err;                    // device error word (bounded waits)
    unsigned long long *stamps;  // optional, 8 device time stamps of CTA 0 (see PhaseArgs)
};
bool q2_gemv_supported(int K, int hat_block);
// asks what launches depend on (how many clusters fit): once, ahead of any capture
void q2_gemv_prepare();
// how a projection of a plain input shares K among the CTAs of clusters: how many clusters (0: it does not), most row tiles of one
struct Q2Split { int clusters = 0, tiles = 0; };
Q2Split q2_gemv_split(int sm_count, int M, int K);
cudaError_t launch_q2_gemv(cudaStream_t st, int sm_count, const Q2Args &a, bool pdl);

struct Q2GemmArgs {
    const uint8_t *W;            // two-bit tiles
    int M, K;                    // valid rows; K % 512 == 0
    int swiglu;                  // as in Q2Args
    const uint8_t *image;        // activation image (act_image.cuh), ncol columns padded to 8, 16 or 32
    int ncol;
    float *out; size_t out_stride;                 // column c at out + c * out_stride
    const float *resid; size_t resid_stride;       // optional: out = sum + resid (may alias out)
    Q2Next next;
    int *err;
    int warm;                                      // the projection in front fetches W towards L2 (Q2Next), and no kernel that may still be running writes it
    int kc, tiles;                                 // filled in by the launch;
    Q2Share share;                                 // filled in by the launch: the CTAs' shares of the row tiles
};
// late: the dependent launch is released behind this kernel's own dependency wait in every build, so that the kernel behind may read ahead
// of its wait what was complete before this one's (k_gdn_core). All of a model's projections are: see k_q2_gemm.
cudaError_t launch_q2_gemm(cudaStream_t st, int sm_count, const Q2GemmArgs &a, bool pdl, bool late = false);
// the same with W in the file's native rows (16-byte aligned, K % 1024 == 0): each warp unpacks its pieces itself, no scratch
// whether that is the faster way: `one_chunk`, the matrix unpacked into tiles beforehand would fit the scratch at once
bool q2_gemm_in_place(int sm_count, int M, int K, int ncol, bool one_chunk);
cudaError_t launch_q2_gemm_native(cudaStream_t st, int sm_count, const Q2GemmArgs &a, bool pdl);
cudaError_t launch_q2_gemm_wide(cudaStream_t st, int sm_count, Q2GemmArgs a, bool pdl);      // 17 to 32 columns (q2_gemm_wide.cu)

#ifdef __CUDACC__
__device__ __forceinline__ void q2_prefetch(const uint8_t *p, int bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
// thread `part` of `parts`: CTA `cta`'s share of the next projection's weights, and its norm weights, and this CTA's part of the state,
// towards L2 (several threads, because a prefetch costs the one that asks for it some 70 cycles). Shares are this grid's: below
// Q2_NEXT_BYTES all weights are asked for, whatever the shares. The output head's are 1.8 MB, so behind the split down projection (120
// CTAs, the head has 148) their first 256 KB are not what the head's CTAs read first. Shares of the head's grid, the 28 beyond this one's
// dealt out in pieces, made every token slower, since each projection runs that code ahead of its dependency wait: 48 tokens 52.5 ->
// 52.8 ms, 100-token prefill 13.66 -> 13.75 ms.
__device__ __forceinline__ void q2_prefetch_next(const Q2Next &n, int cta, int part, int parts) {
    for (int k = cta + part * int(gridDim.x), per = (n.col_bytes + 16383) >> 14; k < n.cols * per; k += parts * int(gridDim.x)) {
        const int o = k % per * 16384;
        q2_prefetch(reinterpret_cast<const uint8_t *>(n.state) + size_t(k / per) * n.col_stride + o, min(16384, n.col_bytes - o));
    }
    for (int o = (cta + part * int(gridDim.x)) * 4096; o < n.rows_bytes; o += parts * int(gridDim.x) * 4096) {
        q2_prefetch(reinterpret_cast<const uint8_t *>(n.rows[0]) + o, min(4096, n.rows_bytes - o));
        q2_prefetch(reinterpret_cast<const uint8_t *>(n.rows[1]) + o, min(4096, n.rows_bytes - o));
    }
    if (!n.W) return;
    const uint8_t *src = n.W + size_t(cta * n.share.q + min(cta, n.share.r)) * n.unit_bytes;
    const int bytes = min((n.share.q + (cta < n.share.r)) * n.unit_bytes, n.max_bytes);
    for (int o = part * 16384; o < bytes; o += parts * 16384) q2_prefetch(src + o, min(16384, bytes - o));
    if (cta == 0 && n.w) for (int o = part * 16384; o < n.w_bytes; o += parts * 16384) q2_prefetch(reinterpret_cast<const uint8_t *>(n.w) + o, min(16384, n.w_bytes - o));
}
constexpr int Q2_MAGIC = 0x4B400000;           // bits of 12582912.0f: adding an int |i| < 2^22 gives the bits of 12582912 + i

// bounded wait of the multi-column kernels: on giving up the error word is set and the caller goes on to its end without waiting
// again (results are then invalid)
__device__ __forceinline__ bool q2_wait(uint32_t bar, uint32_t parity, int *err, int limit = 1 << 22) {
    for (int it = 0; it < limit; ++it) {
        uint32_t ok;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (__builtin_expect(ok != 0u, 1)) return true;
    }
    atomicExch(err, 2);
    return false;
}

// D = A (u8) x B (s8) + C; the first instruction of a chain takes its C from constants
__device__ __forceinline__ void q2_mma_first(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(Q2_MAGIC));
}
__device__ __forceinline__ void q2_mma(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// x * 3 as a shift-and-add, which runs at twice the rate of a multiplication (left to itself the compiler makes it one again)
__device__ __forceinline__ uint32_t times3(uint32_t x) {
    uint32_t y;
    asm("{\n.reg .u32 t;\nshl.b32 t, %1, 1;\nadd.u32 %0, t, %1;\n}\n" : "=r"(y) : "r"(x));
    return y;
}
// four packed bytes: five base-3 digits per byte, each in a byte of its own word (T_t = (b * 3^(t+1)) >> 8 is the base-3 prefix of
// byte b, digit t = T_t - 3 T_(t-1))
__device__ __forceinline__ void q2_unpack4(uint32_t w, uint32_t *o, int stride) {
    uint32_t e = __byte_perm(w, 0u, 0x4240u), d = __byte_perm(w, 0u, 0x4341u), prev = 0u;
#pragma unroll
    for (int t = 0; t < 5; ++t) {
        e = times3(e); d = times3(d);
        const uint32_t T = __byte_perm(e, d, 0x7351u);
        o[t * stride] = T - 3u * prev;
        prev = T;
    }
}
// one native block (row 8 * h + r, block j of a piece) into its places in the piece
__device__ __forceinline__ void q2_unpack_block(const uint32_t (&w)[7], uint8_t *piece, int h, int r, int j) {
    uint32_t o[32];
#pragma unroll
    for (int k = 0; k < 4; ++k) q2_unpack4(w[k], o + k, 4);
    q2_unpack4(w[4], o + 20, 2);
    q2_unpack4(w[5], o + 21, 2);
    const uint32_t v = __byte_perm(w[6], 0u, 0x4140u);
    const uint32_t ta = __byte_perm(v * 3u, v * 9u, 0x7531u), tb = __byte_perm(v * 27u, v * 81u, 0x7531u);
    o[30] = ta - 3u * (ta << 16);
    o[31] = tb - 3u * __byte_perm(ta, tb, 0x5432u);
    uint8_t *dst = piece + (h * 2 + (j >> 1)) * 512 + r * 64 + (j & 1) * 8;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        uint2 q;
        q.x = o[2 * t] | o[8 + 2 * t] << 2 | o[16 + 2 * t] << 4 | o[24 + 2 * t] << 6;
        q.y = o[2 * t + 1] | o[9 + 2 * t] << 2 | o[17 + 2 * t] << 4 | o[25 + 2 * t] << 6;
        *reinterpret_cast<uint2 *>(dst + t * 16) = q;
    }
    *reinterpret_cast<uint16_t *>(piece + Q2_SCALES + (r * 4 + j) * 4 + h * 2) = uint16_t(w[6] >> 16);
}
#endif

}  // namespace bnk
