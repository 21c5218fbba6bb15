"""The projection of 17 to 32 columns at the sizes where its split of the work ends: one row tile and as many segments of K as
there are groups, segments of unequal length, a last tile of two rows, tile pairs with one tile only, and more row tiles per CTA
than one pass holds. Bit for bit the oracle's floats, column by column (every sum's order is fixed)."""
import os

import numpy as np
import pytest

from bonsai_vk_b200 import ptq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiled", [False, True])
@pytest.mark.parametrize("M,K,ncol", [(16, 5120, 17), (130, 13312, 32), (4754, 1024, 25), (7105, 3072, 32), (30900, 1024, 18)])
def test_wide_projection_edges(ctx, oracle, M, K, ncol, tiled):
    rng = np.random.default_rng(M + K + ncol)
    rows = min(M, 4096)                       # a large matrix is a chunk of rows repeated
    W = ptq.synth_matrix(rng, rows, K)
    W.reshape(rows, -1, 28)[0, -1, 26:] = (0x00, 0xFC)      # -inf scale in the last block of row 0
    full = np.ascontiguousarray(np.concatenate([W] * (-(-M // rows)), axis=0)[:M])
    X = rng.standard_normal((ncol, K)).astype(np.float32)
    xb, wb, image, out = ctx.from_numpy(X), ctx.from_numpy(full), ctx.alloc(ctx.gemm_image_bytes(K, ncol)), ctx.alloc(ncol * M * 4)
    ctx.gemm_act_quant(xb, K, ncol, image)
    wt = ctx.gemm_repack(wb, M, K) if tiled else wb
    ctx.gemm_q81(wt, M, K, image, ncol, out, tiled=tiled)
    ctx.sync()
    got = out.download(np.float32, ncol * M).reshape(ncol, M)
    for c in sorted({0, 7, 8, 15, 16, ncol - 1}):
        want, _, _ = oracle.gemv_q81(W, rows, K, oracle.quantize_q8_1(X[c]), threads=os.cpu_count() or 1)
        want = np.concatenate([want] * (-(-M // rows)))[:M]
        assert np.array_equal(np.isnan(got[c]), np.isnan(want)), f"column {c}"
        assert np.array_equal(got[c][~np.isnan(want)].view(np.uint32), want[~np.isnan(want)].view(np.uint32)), f"column {c}"
    for b in {id(b): b for b in (xb, wb, image, out, wt)}.values():
        b.free()
