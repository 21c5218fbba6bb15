"""The single-column projection from native rows on both sides of the line from which a CTA's products are shift-and-adds (120 pieces a
CTA of 148: 15 row tiles at K = 4096), with every trit byte in the matrix, against the oracle bit for bit."""
import numpy as np
import pytest

from bonsai_vk_b200 import ptq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K", [(14 * 16 * 148, 4096), (14 * 16 * 148 + 1, 4096), (120 * 16 * 148 - 15, 512), (35001, 7168)])
def test_many_pieces_per_cta(ctx, oracle, M, K):
    rng = np.random.default_rng(M + K)
    rows = min(M, 2048)
    base = ptq.synth_matrix(rng, rows, K)
    base.reshape(rows, -1, 28)[:256, 0, :26] = np.arange(256, dtype=np.uint8)[:, None]      # all 256 patterns in every position of a block
    W = np.ascontiguousarray(np.concatenate([base] * (-(-M // rows)), axis=0)[:M])
    x = rng.standard_normal(K).astype(np.float32)
    want, _, _ = oracle.gemv_q81(base, rows, K, oracle.quantize_q8_1(x))
    want = np.concatenate([want] * (-(-M // rows)))[:M]
    xb, wb, pack, out = ctx.from_numpy(x), ctx.from_numpy(W), ctx.alloc(ctx.act_pack_bytes(K)), ctx.alloc(M * 4)
    ctx.act_quant_q81(xb, K, pack)
    ctx.gemv_q81(wb, M, K, pack, out)
    ctx.sync()
    assert np.array_equal(out.download(np.uint32, M), want.view(np.uint32))
    for b in (xb, wb, pack, out):
        b.free()
