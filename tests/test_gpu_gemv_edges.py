"""The projection streamed from native rows at the sizes where its split of the work ends: one row and one block, groups of four
blocks that are not full (1, 2, 3 blocks left: 4-, 8- and 4-byte copies), a last tile of one row, one tile more than there are
SMs, and a run of tiles whose group sums do not fit at once. Bit for bit the oracle's floats (every sum's order is fixed)."""
import os

import numpy as np
import pytest

from bonsai_vk_b200 import ptq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K", [(1, 128), (17, 384), (33, 768), (2369, 512), (2368, 640), (500, 8960), (153925, 12288)])
def test_streamed_projection_edges(ctx, oracle, M, K):
    rng = np.random.default_rng(M + K)
    rows = min(M, 8192)                       # a large matrix is a chunk of rows repeated
    W = ptq.synth_matrix(rng, rows, K)
    W.reshape(rows, -1, 28)[0, -1, 26:] = (0x00, 0xFC)      # -inf scale in the last block of row 0
    x = rng.standard_normal(K).astype(np.float32)
    full = np.concatenate([W] * (-(-M // rows)), axis=0)[:M]
    wb, xb, pack, out = ctx.from_numpy(full), ctx.from_numpy(x), ctx.alloc(ctx.act_pack_bytes(K)), ctx.alloc(M * 4)
    ctx.act_quant_q81(xb, K, pack)
    ctx.gemv_q81(wb, M, K, pack, out)
    ctx.sync()
    got = out.download(np.float32, M)
    want, _, _ = oracle.gemv_q81(W, rows, K, oracle.quantize_q8_1(x), threads=os.cpu_count() or 1)
    want = np.concatenate([want] * (-(-M // rows)))[:M]
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(got[~np.isnan(want)].view(np.uint32), want[~np.isnan(want)].view(np.uint32))
    for b in (wb, xb, pack, out):
        b.free()
