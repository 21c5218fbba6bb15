"""Single projection from native rows that start on 4-byte boundaries only: they are copied as the 16-byte granules that hold them, those of
the matrix's first and last rows that reach out of it word by word. Heights around a row tile, odd block counts around a group, one piece
and many per CTA, every place of the matrix in a granule, other bytes on both sides of it: the oracle's bits. (They say nothing of what is
read beyond the rows, since no output depends on it: test_granules.py checks the addresses.)"""
import numpy as np
import pytest

from bonsai_vk_b200 import ptq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,w_off", [(1, 128, 4), (33, 128, 4), (36, 128, 0), (33, 256, 4), (15, 384, 12), (16, 128, 0), (17, 640, 0), (33, 896, 4), (512, 4096, 12), (130, 1152, 8),
                                       (2369, 1152, 0), (40000, 640, 0), (9000, 4736, 4)])
def test_rows_of_4_byte_alignment(ctx, oracle, M, K, w_off):
    rng = np.random.default_rng(M + K)
    W = ptq.synth_matrix(rng, M, K)
    x = rng.standard_normal(K).astype(np.float32)
    raw = np.full(W.size + w_off + 16, 0xFF, dtype=np.uint8)
    raw[w_off:w_off + W.size] = W.reshape(-1)
    wb, xb = ctx.from_numpy(raw), ctx.from_numpy(x)
    pack, out = ctx.alloc(ctx.act_pack_bytes(K)), ctx.alloc(M * 4)
    ctx.act_quant_q81(xb, K, pack)
    for _ in range(2):
        ctx.gemv_q81(wb, M, K, pack, out, w_off=w_off)
    ctx.sync()
    ref, _, _ = oracle.gemv_q81(W, M, K, oracle.quantize_q8_1(x))
    assert np.array_equal(out.download(np.uint32, M), ref.view(np.uint32))
    for b in (wb, xb, pack, out):
        b.free()
