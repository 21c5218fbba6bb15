// granules.cuh - the 16-byte granules that hold a piece of native rows on 4-byte boundaries (16 rows, up to four blocks of 28 bytes), and
// which of them may be read whole. Plain arithmetic: the kernel's (k_ptq_stream), and a check's on the host.
#pragma once
#include <cstddef>
#include <cstdint>

#ifdef __CUDACC__
#define BN_DEVICE __device__ __forceinline__
#else
#define BN_DEVICE inline
#endif

namespace bnk {

struct Granules {
    uintptr_t w0, w1;                          // the matrix: [w0, w1)
    size_t rowbytes;
    int M, nb;                                 // rows, blocks per row

    // a row's place in its first granule: the same for every group of blocks, and for rows four apart (4 * 28 bytes per block)
    BN_DEVICE int place(size_t row) const { return int((w0 + row * rowbytes) & 15); }
    // whether granule i of a row at `place` holds any of the blocks of a group
    BN_DEVICE bool holds(int place, int group, int i) const { return i * 16 < place + (nb - 4 * group < 4 ? nb - 4 * group : 4) * 28; }
    // A tile of 16 rows from row0 on whose granules all lie in the matrix: the first reaches at most 12 bytes in front of its row, the last
    // as many behind it, less than a row (28 bytes and more).
    BN_DEVICE bool whole(int row0) const { return row0 > 0 && row0 + 16 < M; }
    BN_DEVICE bool inside(uintptr_t s, int bytes) const { return s >= w0 && s + bytes <= w1; }

    // One lane's copies of a piece, where it needs any: granule lane % 8 of rows lane / 8 + 4 i. granule(i, s): 16 bytes at s; word(i, k, s):
    // four bytes at s, k bytes into the granule - the matrix's first and last rows, where a granule reaches out of it.
    template <class Granule, class Word>
    BN_DEVICE void copies(int row0, int group, int lane, bool need, Granule granule, Word word) const {
        const int row = row0 + (lane >> 3);
        uintptr_t s = ((w0 + size_t(row) * rowbytes + uint32_t(group) * 112u) & ~uintptr_t(15)) + uintptr_t(lane & 7) * 16;
        if (whole(row0)) {
#pragma unroll
            for (int i = 0; i < 4; ++i, s += 4 * rowbytes) if (need) granule(i, s);
        } else
#pragma unroll
            for (int i = 0; i < 4; ++i, s += 4 * rowbytes) {
                if (!need || row + 4 * i >= M) continue;
                if (inside(s, 16)) granule(i, s);
                else
#pragma unroll 1
                    for (int k = 0; k < 16; k += 4) if (inside(s + k, 4)) word(i, k, s + k);
            }
    }
};

}  // namespace bnk
