// The copies that k_ptq_stream asks for, of every piece of a matrix, by the kernel's own arithmetic (granules.cuh): bytes read outside of the
// matrix, into the wrong place of a row's slot or beyond it, plus bytes of the rows that are missing there.
#include "../../bonsai_vk_b200/csrc/granules.cuh"

#include <vector>

extern "C" long long check_granules(unsigned long long w0, int M, int nb) {
    const bnk::Granules g = {uintptr_t(w0), uintptr_t(w0) + size_t(M) * nb * 28, size_t(nb) * 28, M, nb};
    long long bad = 0;
    for (int row0 = 0; row0 < M; row0 += 16)
        for (int group = 0; group < (nb + 3) / 4; ++group) {
            std::vector<uintptr_t> slot(16 * 144, 0);                      // the address that each byte of the piece's slot comes from
            for (int lane = 0; lane < 32; ++lane) {
                auto put = [&](int row, int k, uintptr_t s, int bytes) {
                    if (s % bytes || s < g.w0 || s + bytes > g.w1) ++bad;
                    for (int b = 0; b < bytes; ++b)
                        if ((lane & 7) * 16 + k + b < 144) slot[row * 144 + (lane & 7) * 16 + k + b] = s + b; else ++bad;
                };
                g.copies(row0, group, lane, g.holds(g.place(lane >> 3), group, lane & 7), [&](int i, uintptr_t s) { put((lane >> 3) + 4 * i, 0, s, 16); },
                         [&](int i, int k, uintptr_t s) { put((lane >> 3) + 4 * i, k, s, 4); });
            }
            const int bytes = (nb - 4 * group < 4 ? nb - 4 * group : 4) * 28;
            for (int r = 0; r < 16 && row0 + r < M; ++r)
                for (int b = 0; b < bytes; ++b)                           // where a lane of the kernel looks for it: rows r and r + 8 at the place of row r % 8
                    if (slot[r * 144 + g.place(r & 7) + b] != g.w0 + size_t(row0 + r) * g.rowbytes + size_t(group) * 112 + b) ++bad;
        }
    return bad;
}
