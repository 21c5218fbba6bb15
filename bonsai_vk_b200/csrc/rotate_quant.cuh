// rotate_quant.cuh - the pieces of "rotate, then quantise" that the projection kernels' input preparation (q2_gemv.cu), the
// multi-column activation image (prep_cols.cu) and the whole-token kernel (phase_body.cuh) share, so that all of them produce
// the same bits: the mean of a power-of-two count, the sign flip, the butterflies of the Sylvester-Walsh-Hadamard transform
// (reference network: runtime_vk/shaders/hat4096.comp:41-60) and the q8_1 quantiser (recipe:
// runtime_vk/shaders/attn_norm_rope2.comp:39-49).
#pragma once
#include "common.cuh"

namespace bnk {

// t / K rounded to nearest: for a power of two the product with 1/K is the same float (an exact scaling, rounded once
// when the result is subnormal, as the quotient is) and skips the division sequence. 1 / x below is __frcp_rn, the
// correctly rounded reciprocal, which is what the division 1.0f / x returns.
__device__ __forceinline__ float mean_of(float t, int K) {
    return (K & (K - 1)) == 0 ? __fmul_rn(t, __frcp_rn(float(K))) : __fdiv_rn(t, float(K));
}
// x * sign for sign = +1 / -1 (bn_model_set_signs refuses anything else): flipping the sign bit is the same float as the
// product, zeros and NaNs included, and needs no int -> float conversion
__device__ __forceinline__ float apply_sign(float x, int sg) { return __uint_as_float(__float_as_uint(x) ^ (uint32_t(sg) & 0x80000000u)); }
// butterflies h = 1, 2, 4 inside a thread's 8 consecutive elements, h = 8..128 across the lanes of a warp
__device__ __forceinline__ void fwht_regs_lanes(float (&v)[8], int lane) {
#pragma unroll
    for (int h = 1; h < 8; h <<= 1)
#pragma unroll
        for (int r = 0; r < 8; ++r)
            if (!(r & h)) { const float x = v[r], y = v[r + h]; v[r] = __fadd_rn(x, y); v[r + h] = __fsub_rn(x, y); }
    // the upper lane of a pair takes partner - own, the lower one own + partner: one fused multiply-add with +-1 (the
    // product is exact, so the result is the rounded difference / sum, bit for bit what fsub / fadd give)
#pragma unroll
    for (int m2 = 1; m2 < 32; m2 <<= 1) {
        const float sgn = (lane & m2) ? -1.0f : 1.0f;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const float pr = __shfl_xor_sync(0xFFFFFFFFu, v[r], m2);
            v[r] = __fmaf_rn(v[r], sgn, pr);
        }
    }
}
// butterflies h = 256, 512, 1024 inside a thread (elements 256 apart), h = 2048 between lanes l and l^16, then the scale;
// each thread rewrites only what it read
__device__ __forceinline__ void fwht_4096_tail(float *xs, int warp, int lane, float hat_inv) {
    const int i0 = (lane & 15) + 16 * warp + 2048 * (lane >> 4);
    float u[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) u[r] = xs[i0 + 256 * r];
#pragma unroll
    for (int h = 1; h < 8; h <<= 1)
#pragma unroll
        for (int r = 0; r < 8; ++r)
            if (!(r & h)) { const float x = u[r], y = u[r + h]; u[r] = __fadd_rn(x, y); u[r + h] = __fsub_rn(x, y); }
    const float sgn = (lane & 16) ? -1.0f : 1.0f;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const float pr = __shfl_xor_sync(0xFFFFFFFFu, u[r], 16);
        u[r] = __fmaf_rn(u[r], sgn, pr);
        xs[i0 + 256 * r] = __fmul_rn(u[r], hat_inv);
    }
}
// q8_1 of a 32-value sub-block held by four neighbouring lanes (4k .. 4k+3), eight consecutive values each; all 32 lanes
// of the warp call it (lanes without a sub-block pass zeros). d = amax / 127 (0 below 1e-35), codes = round half away of
// x / d clamped to +-127, sum = the sub-block's code sum. The low byte of (code + 1.5 * 2^23) read as an integer is the
// code in two's complement (no float -> int conversion); four bytes are gathered with byte permutes and the sum of the
// eight codes is two byte dot products with ones.
struct Q8x8 { uint32_t w0, w1; float d; int sum; };
__device__ __forceinline__ Q8x8 quant8_of32(const float (&e)[8]) {
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(e[i]));
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));
    Q8x8 r;
    r.d = amax > 1e-35f ? __fdiv_rn(amax, 127.0f) : 0.0f;
    const float id = r.d != 0.0f ? __frcp_rn(r.d) : 0.0f;
    uint32_t q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float c = roundf(__fmul_rn(e[i], id));
        c = fminf(fmaxf(c, -127.0f), 127.0f);
        q[i] = __float_as_uint(__fadd_rn(c, 12582912.0f));
    }
    r.w0 = __byte_perm(__byte_perm(q[0], q[1], 0x0040u), __byte_perm(q[2], q[3], 0x0040u), 0x5410u);
    r.w1 = __byte_perm(__byte_perm(q[4], q[5], 0x0040u), __byte_perm(q[6], q[7], 0x0040u), 0x5410u);
    int sum = __dp4a(int(r.w0), 0x01010101, __dp4a(int(r.w1), 0x01010101, 0));
    sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 1);
    sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 2);
    r.sum = sum;
    return r;
}

// ---- the same transform over spans of 4096 values by 512 threads, through shared memory ------------------------------------
// 4096 = 8^4: four passes of three butterfly stages over 8 registers (h = 1..4, 8..32, 64..256, 512..2048), each reading and
// writing the span in place; the first exchange stays inside a warp. What bounds it is instruction fetch and latency, not
// throughput: a projection kernel runs this code once, so every instruction of it is a first fetch (about 4 cycles each were
// measured with two warps per scheduler), and the form with the fewest instructions per thread that still fills the SM wins.
// Measured for one projection's prologue: eight values per thread with the stages 8..128 done by 40 shuffles 1.3 us, 256
// threads with 16 values 0.85 us. Same pairs (a + c, a - c), h ascending, so the same floats.
// Element e lies at xs8(e): 8 floats of padding per 64 and the two 16-byte halves of every 8 exchanged by bit 5, which frees
// all five access patterns from bank conflicts.
constexpr int XS8_SPAN = 4608;                 // floats per span
__device__ __forceinline__ int xs8(int e) { return (e ^ ((e >> 3) & 4)) + ((e >> 6) << 3); }
// packed fp32 pairs: two IEEE single operations per instruction, each half rounded as the scalar instruction
typedef unsigned long long f32pair;
__device__ __forceinline__ f32pair pair_of(float a, float b) { f32pair r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void split_pair(f32pair v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32pair pair_fma(f32pair a, f32pair b, f32pair c) { f32pair d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ f32pair pair_add(f32pair a, f32pair b) { f32pair d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f32pair pair_sub(f32pair a, f32pair b) { f32pair d; asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f32pair pair_mul(f32pair a, f32pair b) { f32pair d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }

// the first `stages` (1..3) of the butterflies h = 1, 2, 4 over 8 values held as pairs (2i, 2i + 1)
__device__ __forceinline__ void fwht_pairs8(f32pair (&v)[4], int stages) {
#pragma unroll
    for (int i = 0; i < 4; ++i) { float a, b; split_pair(v[i], a, b); v[i] = pair_of(__fadd_rn(a, b), __fsub_rn(a, b)); }
#pragma unroll
    for (int h = 1; h < 4; h <<= 1) {
        if (stages > h) {                      // h = 1: second stage, h = 2: third
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (!(r & h)) { const f32pair x = v[r], y = v[r + h]; v[r] = pair_add(x, y); v[r + h] = pair_sub(x, y); }
        }
    }
}
// one pass over a span: 8 values e0 + k << SHIFT, where thread t owns the e0 whose bits SHIFT .. SHIFT + 2 are zero
template <int SHIFT>
__device__ __forceinline__ void fwht_pass(float *xs, int t, int stages) {
    float *p = xs + xs8(((t >> SHIFT) << (SHIFT + 3)) | (t & ((1 << SHIFT) - 1)));
    // stepping e by 1 << SHIFT moves the address by a constant, except that stepping through bit 5 (SHIFT = 3) flips bit 2
    constexpr int STEP = SHIFT >= 6 ? (1 << SHIFT) + ((1 << SHIFT) >> 3) : (1 << SHIFT);
    const int flip = SHIFT == 3 ? ((t & 4) ? -4 : 4) : 0;
    f32pair v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = pair_of(p[2 * k * STEP + (k >= 2 ? flip : 0)], p[(2 * k + 1) * STEP + (k >= 2 ? flip : 0)]);
    fwht_pairs8(v, stages);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float a, b;
        split_pair(v[k], a, b);
        p[2 * k * STEP + (k >= 2 ? flip : 0)] = a;
        p[(2 * k + 1) * STEP + (k >= 2 ? flip : 0)] = b;
    }
}
// this thread's eight consecutive values 8t .. 8t + 7 of a span, in and out
__device__ __forceinline__ void span_store8(float *xs, int t, const f32pair (&v)[4]) {
    ulonglong2 *p = reinterpret_cast<ulonglong2 *>(xs + t * 8 + ((t >> 3) << 3));
    const int s = (t >> 2) & 1;
    p[s] = make_ulonglong2(v[0], v[1]);
    p[s ^ 1] = make_ulonglong2(v[2], v[3]);
}
__device__ __forceinline__ void span_load8(const float *xs, int t, f32pair (&v)[4]) {
    const ulonglong2 *p = reinterpret_cast<const ulonglong2 *>(xs + t * 8 + ((t >> 3) << 3));
    const int s = (t >> 2) & 1;
    const ulonglong2 a = p[s], b = p[s ^ 1];
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
// the whole transform of `spans` spans that lie side by side in shared memory (width hb = 2^log_hb, 16 .. 4096); v: the
// first span's values of this thread after its own first pass are stored by the caller (span_store8). On return the spans
// hold the transformed values (not scaled yet); every thread may read them.
template <class Bar>
__device__ __forceinline__ void fwht_spans(float *xs, int t, int spans, int log_hb, Bar bar) {
    __syncwarp();
#pragma unroll 1
    for (int s = 0; s < spans; ++s) fwht_pass<3>(xs + s * XS8_SPAN, t, log_hb - 3);
    bar();
    if (log_hb > 6) {
#pragma unroll 1
        for (int s = 0; s < spans; ++s) fwht_pass<6>(xs + s * XS8_SPAN, t, log_hb - 6);
        bar();
    }
    if (log_hb > 9) {
#pragma unroll 1
        for (int s = 0; s < spans; ++s) fwht_pass<9>(xs + s * XS8_SPAN, t, log_hb - 9);
        bar();
    }
}
// amax / 127 rounded to nearest in three operations: quotient by the rounded reciprocal, its exact remainder by a fused
// multiply-add, one correction - division by a constant known in advance (Brisebarre, Muller, Raina: Accelerating correctly
// rounded floating-point division when the divisor is known in advance, IEEE Trans. Computers 53, 2004). amax above 1e-35 keeps
// the remainder exact. tests/test_gpu_quantiser.py compares every mantissa with the division, and every code below.
__device__ __forceinline__ float div127(float amax) {
    const float q = __fmul_rn(amax, 1.0f / 127.0f);
    const float d = fmaf(fmaf(-127.0f, q, amax), 1.0f / 127.0f, q);
    return q == INFINITY ? q : d;
}
// code of y as the low byte of a word: round half away of y, clamped to +-127 (|y| < 127.5 but for a NaN, which becomes -127 as
// fminf(fmaxf(.)) has it). y + h rounded down and then floored, h = 1/2 for y >= 0 and the float below 1/2 for y < 0: a tie at
// -k - 1/2 goes to -k - 1, everything else where it belongs (rounding down cannot cross the integer below). No float -> int
// conversion: those run at a sixteenth of the rate and were a third of the quantiser's time.
__device__ __forceinline__ uint32_t code_byte(float y) {
    const float c = fmaxf(y, -127.0f), h = __uint_as_float(0x3F000000u - (__float_as_uint(c) >> 31));
    return __float_as_uint(__fadd_rd(__fadd_rd(c, h), 12582912.0f));
}
// quant8_of32 in fewer instructions (same codes, d and sum)
__device__ __forceinline__ Q8x8 quant8_pairs(const f32pair (&v)[4]) {
    float e[8];
#pragma unroll
    for (int k = 0; k < 4; ++k) split_pair(v[k], e[2 * k], e[2 * k + 1]);
    float m0 = 0.0f, m1 = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i += 2) { m0 = fmaxf(m0, fabsf(e[i])); m1 = fmaxf(m1, fabsf(e[i + 1])); }
    float amax = fmaxf(m0, m1);
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));
    Q8x8 r;
    const bool some = amax > 1e-35f;
    r.d = some ? div127(amax) : 0.0f;
    const float id = some ? __frcp_rn(r.d) : 0.0f;
    uint32_t q[8];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float a, b;
        split_pair(pair_mul(v[k], pair_of(id, id)), a, b);
        q[2 * k] = code_byte(a); q[2 * k + 1] = code_byte(b);
    }
    r.w0 = __byte_perm(__byte_perm(q[0], q[1], 0x0040u), __byte_perm(q[2], q[3], 0x0040u), 0x5410u);
    r.w1 = __byte_perm(__byte_perm(q[4], q[5], 0x0040u), __byte_perm(q[6], q[7], 0x0040u), 0x5410u);
    int sum = __dp4a(int(r.w0), 0x01010101, __dp4a(int(r.w1), 0x01010101, 0));
    sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 1);
    sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 2);
    r.sum = sum;
    return r;
}
// sum over 256 lane partials p[0..255] (each the ascending sum of one lane's run of squares) by the norm's fixed tree
// p[i] += p[i + s], s = 128 .. 1, run by every warp on its own: the same adds in the same order in every warp
__device__ __forceinline__ float norm_tree256(const float *p, int lane) {
    float v[8];
#pragma unroll
    for (int w = 0; w < 8; ++w) v[w] = p[32 * w + lane];
    float t = __fadd_rn(__fadd_rn(__fadd_rn(v[0], v[4]), __fadd_rn(v[2], v[6])), __fadd_rn(__fadd_rn(v[1], v[5]), __fadd_rn(v[3], v[7])));
#pragma unroll
    for (int s2 = 16; s2 > 0; s2 >>= 1) t = __fadd_rn(t, __shfl_xor_sync(0xFFFFFFFFu, t, s2));
    return t;
}

// sum over 128 values held as 4 per lane (elements l, l + 32, l + 64, l + 96) in the order of the reference's shared-memory tree
// sh[l] += sh[l + s], s = 64 .. 1 (gdn_delta.comp tree_reduce)
__device__ __forceinline__ float warp_tree128(float e0, float e1, float e2, float e3) {
    float a = __fadd_rn(__fadd_rn(e0, e2), __fadd_rn(e1, e3));
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) a = __fadd_rn(a, __shfl_xor_sync(0xFFFFFFFFu, a, s));
    return a;
}
// eight consecutive values from a 16-byte aligned place
__device__ __forceinline__ void load8(const float *p, f32pair (&v)[4]) {
    const ulonglong2 *q = reinterpret_cast<const ulonglong2 *>(p);
    const ulonglong2 a = q[0], b = q[1];
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

}  // namespace bnk
