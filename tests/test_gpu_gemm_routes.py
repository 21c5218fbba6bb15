"""The several-column projection on both sides of each line of its dispatch: every column equals the single-column projection of its
vector bit for bit (the same sums in the same order), whichever kernel took the call."""
import numpy as np
import pytest

from bonsai_vk_b200 import Context, ptq

pytestmark = pytest.mark.gpu


# launches: 1 where native rows are unpacked in place, 2 where they are unpacked into tiles first
@pytest.mark.parametrize("M,K,ncol,launches", [
    (7104, 7168, 16, 1), (7105, 7168, 16, 2),                    # three and four row tiles per CTA of 148, K in waves
    (21312, 5120, 9, 1), (21313, 5120, 9, 2),                    # nine and ten: K in one wave, in two
    (15408, 12288, 12, 2), (15409, 12288, 12, 1),                # tiles of one chunk of scratch, of two
    (7105, 14336, 8, 1), (2368, 6144, 17, 1), (2369, 6144, 17, 2),
])
def test_native_rows_take_the_faster_way(M, K, ncol, launches):
    test_columns_equal_single_projections(M, K, ncol, False, launches)


@pytest.mark.parametrize("M,K,ncol,tiled", [
    (1, 1024, 1, False), (100, 1024, 16, False), (100, 1024, 17, False),
    (2368, 6144, 17, False), (2369, 6144, 17, False),            # 12 and 24 pieces per CTA of 148
    (2368, 7168, 32, False),                                     # 14
    (4737, 2048, 8, False), (700, 12288, 9, False),
    (14208, 1024, 8, True), (14209, 1024, 8, True),              # 6 and 7 row tiles per CTA
    (28417, 1024, 5, True),                                      # 13: more than one pass
    (4096, 2048, 16, True), (12288, 1024, 11, True),             # units for 12 warps, for 16
    (17, 12288, 16, True), (2367, 12288, 8, True),               # K in waves
    (2368, 8192, 16, True), (2369, 8192, 16, True),              # one and two tiles: units of one, of two
    (2368, 4096, 3, True), (2369, 4096, 3, True), (4736, 1024, 8, True), (4737, 1024, 8, True), (4736, 1024, 9, True),
    (7104, 3072, 8, True), (7104, 4096, 8, True), (11841, 8192, 8, True), (14208, 8192, 2, True),      # units of two and three by rounds
    (11841, 8192, 12, True), (4737, 16384, 8, True), (4736, 14336, 16, True),        # K in waves
])
def test_columns_equal_single_projections(M, K, ncol, tiled, launches=None):
    rng = np.random.default_rng(M + K + ncol)
    rows = min(M, 1024)
    W = np.ascontiguousarray(np.concatenate([ptq.synth_matrix(rng, rows, K)] * (-(-M // rows)), axis=0)[:M])
    X = rng.standard_normal((ncol, K)).astype(np.float32)
    ctx = Context(0)
    wb, xb, image, out = ctx.from_numpy(W), ctx.from_numpy(X), ctx.alloc(ctx.gemm_image_bytes(K, ncol)), ctx.alloc(ncol * M * 4)
    pack, one = ctx.alloc(ctx.act_pack_bytes(K)), ctx.alloc(M * 4)
    wt = ctx.gemm_repack(wb, M, K) if tiled else wb
    ctx.gemm_act_quant(xb, K, ncol, image)
    before = ctx.launches
    ctx.gemm_q81(wt, M, K, image, ncol, out, tiled=tiled)
    ctx.sync()
    taken = ctx.launches - before
    got = out.download(np.uint32, ncol * M).reshape(ncol, M)
    for c in sorted({0, ncol // 2, ncol - 1}):
        ctx.act_quant_q81(xb, K, pack, x_off=c * K * 4)
        ctx.gemv_q81(wb, M, K, pack, one)
        ctx.sync()
        assert np.array_equal(got[c], one.download(np.uint32, M)), f"column {c}"
    assert launches is None or taken == launches
    ctx.close()
