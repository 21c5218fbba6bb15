"""A model whose FFN is wider than the fused projection kernels take (16 384): it decodes through the stand-alone kernels, with
columns or without, its sharded output head works, and only the multi-sequence pass itself is refused, when it is prepared."""
import numpy as np
import pytest

from bonsai_vk_b200 import BonsaiError, Model, synth
from tests._oracle import OracleModel

pytestmark = pytest.mark.gpu


def test_wide_ffn_with_columns(ctx):
    hp = synth.tiny(n_layer=2, attn_interval=2, ffn=17408, batch_cols=4, n_streams=4, vocab=640)
    tensors, signs = synth.make_model(hp, seed=7)
    gm, om = Model(ctx, hp, tensors, signs), OracleModel(hp, tensors, signs)
    for pos, t in enumerate((5, 630, 77)):
        gt = gm.token(t, pos)
        ol, ores = om.token(t, pos)
        assert gt == om.argmax(ol) and np.array_equal(gm.logits().view(np.uint32), ol.view(np.uint32)), f"position {pos}"
    with pytest.raises(BonsaiError, match="fused"):
        gm.stage_prepare(0, 4)
    with pytest.raises(BonsaiError, match="fused"):
        gm.prefill([1, 2], 3)
    # the residual of the last token through two shards of the head: the same pick
    hid, cands, out = ctx.from_numpy(np.tile(ores, (3, 1)).astype(np.float32)), ctx.alloc(2 * 3 * 8), ctx.alloc(3 * 4)
    for i, rows in enumerate(((0, 384), (384, 640))):
        m = Model(ctx, hp, tensors, signs, head_rows=rows)
        m.head_batch(3, hid, cands, out_off=i * 3 * 8)
        ctx.sync()
        m.close()
    gm.pick_batch(3, 2, cands, out)
    ctx.sync()
    assert list(out.download(np.int32, 3)) == [gt] * 3
    gm.close(); om.close()
    for b in (hid, cands, out):
        b.free()
