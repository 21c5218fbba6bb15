// attn_octet.cuh - scores of eight consecutive keys of one kv head by a warp, for the chain of kernels (attn.cu) and the one-launch
// kernel (attn_cluster.cu), and the small pieces that both use. Per key and query head: lane l covers dims 8l .. 8l+7 with an
// fmaf chain, then the 32 lane sums meet in the xor-butterfly tree (16, 8, 4, 2, 1). Two keys travel in the halves of packed
// registers.
#pragma once
#include "ops.cuh"
#include "rotate_quant.cuh"

namespace bnk {

// order-preserving image of a float, for atomicMax (0 = below every float)
__device__ __forceinline__ unsigned ord(float f) { const unsigned b = __float_as_uint(f); return (b & 0x80000000u) ? ~b : b | 0x80000000u; }
__device__ __forceinline__ float unord(unsigned k) { return __uint_as_float((k & 0x80000000u) ? k & 0x7FFFFFFFu : ~k); }

// int8 code -> float without the conversion unit: the word's bytes are biased by 128 (one xor for four codes), a byte
// is dropped into the mantissa of 2^23 and 2^23 + 128 is subtracted: exact for every code
constexpr float CODE_MAGIC = 8388736.0f;       // 2^23 + 128
template <int BYTE> __device__ __forceinline__ float code_f(uint32_t biased_word) {
    return __uint_as_float(__byte_perm(biased_word, 0x4B000000u, 0x7440u + BYTE));   // 2^23 + (code + 128), magic still to subtract
}

// this lane's part of eight keys' rows, as they lie in the cache
template <int KMODE> struct KeyOctet {
    uint4 raw16[KMODE == 1 ? 8 : 1];
    uint2 raw8[KMODE == 1 ? 1 : 8];
    uint16_t sc[8];
    // keys j .. j + 7 (those beyond `last` read `last`)
    __device__ __forceinline__ void fetch(const KvLayer &kv, int n_kv, int kvh, int hd, int lane, int j, int last) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const size_t row = (size_t(min(j + u, last)) * n_kv + kvh) * hd;
            if (KMODE == 1) raw16[u] = *reinterpret_cast<const uint4 *>(reinterpret_cast<const __half *>(kv.k_data) + row + lane * 8);
            else {
                raw8[u] = *reinterpret_cast<const uint2 *>(reinterpret_cast<const int8_t *>(kv.k_data) + row + lane * 8);
                sc[u] = kv.k_scale[row / 32 + (lane >> 2)];
            }
        }
    }
    // keys 2 up and 2 up + 1, widened: dim e of both in kf[e]
    __device__ __forceinline__ void widen(int up, f32pair magic2, f32pair (&kf)[8]) const {
        if (KMODE == 1) {
            const __half2 *ha = reinterpret_cast<const __half2 *>(&raw16[2 * up]), *hb = reinterpret_cast<const __half2 *>(&raw16[2 * up + 1]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 fa = __half22float2(ha[e]), fb = __half22float2(hb[e]);
                kf[2 * e] = pair_of(fa.x, fb.x); kf[2 * e + 1] = pair_of(fa.y, fb.y);
            }
        } else {
            const uint32_t a0 = raw8[2 * up].x ^ 0x80808080u, a1 = raw8[2 * up].y ^ 0x80808080u;
            const uint32_t b0 = raw8[2 * up + 1].x ^ 0x80808080u, b1 = raw8[2 * up + 1].y ^ 0x80808080u;
            const f32pair sc2 = pair_of(half_bits_to_float(sc[2 * up]), half_bits_to_float(sc[2 * up + 1]));
            kf[0] = pair_mul(sc2, pair_sub(pair_of(code_f<0>(a0), code_f<0>(b0)), magic2)); kf[1] = pair_mul(sc2, pair_sub(pair_of(code_f<1>(a0), code_f<1>(b0)), magic2));
            kf[2] = pair_mul(sc2, pair_sub(pair_of(code_f<2>(a0), code_f<2>(b0)), magic2)); kf[3] = pair_mul(sc2, pair_sub(pair_of(code_f<3>(a0), code_f<3>(b0)), magic2));
            kf[4] = pair_mul(sc2, pair_sub(pair_of(code_f<0>(a1), code_f<0>(b1)), magic2)); kf[5] = pair_mul(sc2, pair_sub(pair_of(code_f<1>(a1), code_f<1>(b1)), magic2));
            kf[6] = pair_mul(sc2, pair_sub(pair_of(code_f<2>(a1), code_f<2>(b1)), magic2)); kf[7] = pair_mul(sc2, pair_sub(pair_of(code_f<3>(a1), code_f<3>(b1)), magic2));
        }
    }
};
// this lane's eight dims of G query heads from `first` on: (q, q), as both keys of a pair meet the same query value
template <int G> __device__ __forceinline__ void load_queries(const float *q16f, int first, int hd, int lane, f32pair (&qd)[G][8]) {
#pragma unroll
    for (int h = 0; h < G; ++h) {
        const float4 *qv = reinterpret_cast<const float4 *>(q16f + size_t(first + h) * hd + lane * 8);
        const float4 q0 = qv[0], q1 = qv[1];
        qd[h][0] = pair_of(q0.x, q0.x); qd[h][1] = pair_of(q0.y, q0.y); qd[h][2] = pair_of(q0.z, q0.z); qd[h][3] = pair_of(q0.w, q0.w);
        qd[h][4] = pair_of(q1.x, q1.x); qd[h][5] = pair_of(q1.y, q1.y); qd[h][6] = pair_of(q1.z, q1.z); qd[h][7] = pair_of(q1.w, q1.w);
    }
}
// v[G u + h]: this lane's part of (key u of the octet, head h)
template <int G, int KMODE> __device__ __forceinline__ void octet_parts(const KeyOctet<KMODE> &k, const f32pair (&qd)[G][8], f32pair magic2, float (&v)[8 * G]) {
#pragma unroll
    for (int up = 0; up < 4; ++up) {
        f32pair kf[8];
        k.widen(up, magic2, kf);
#pragma unroll
        for (int h = 0; h < G; ++h) {
            f32pair acc = 0ull;
#pragma unroll
            for (int e = 0; e < 8; ++e) acc = pair_fma(qd[h][e], kf[e], acc);
            split_pair(acc, v[2 * up * G + h], v[(2 * up + 1) * G + h]);
        }
    }
}
// all NV = 8 G trees as one transposed butterfly: at distance `off` a lane keeps the half of its values that its bit selects and
// adds the partner's copy of the same values, the same pair sums in the same order; lane l ends with the total of value
// l >> log2(32 / NV) (with fewer than 32 values the last steps are plain)
template <int NV> __device__ __forceinline__ void octet_totals(float (&v)[NV], int lane) {
#pragma unroll
    for (int step = 0; step < 5; ++step) {
        const int off = 16 >> step, m = NV >> step;
        if (m > 1) {
            const bool upper = lane & off;
#pragma unroll
            for (int i = 0; i < m / 2; ++i) {
                const float send = upper ? v[i] : v[i + m / 2], keep = upper ? v[i + m / 2] : v[i];
                v[i] = __fadd_rn(keep, __shfl_xor_sync(0xFFFFFFFFu, send, off));
            }
        } else v[0] = __fadd_rn(v[0], __shfl_xor_sync(0xFFFFFFFFu, v[0], off));
    }
}

}  // namespace bnk
