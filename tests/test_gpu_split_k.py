"""The down projection whose K is shared by the CTAs of a cluster: widths of two, three and four spans of 4096, one to several row tiles
per cluster in uneven shares, against the oracle bit for bit."""
import numpy as np
import pytest

from bonsai_vk_b200 import Model, synth
from tests._oracle import OracleModel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ffn,hat_block,hidden", [(8192, 1024, 1024), (12288, 256, 1024), (16384, 1024, 1024), (12288, 2048, 2048)])
def test_split_down_projection(ctx, ffn, hat_block, hidden):
    hp = synth.tiny(n_layer=2, attn_interval=2, hidden=hidden, n_head=hidden // 256, n_kv=hidden // 1024, gdn_heads=hidden // 128, gdn_qk_heads=hidden // 256,
                    ffn=ffn, hat_block=hat_block, vocab=640)
    tensors, signs = synth.make_model(hp, seed=3)
    gm, om = Model(ctx, hp, tensors, signs), OracleModel(hp, tensors, signs)
    for pos, t in enumerate((5, 630, 77)):
        gt = gm.token(t, pos)
        ol, ores = om.token(t, pos)
        assert gt == om.argmax(ol) and np.array_equal(gm.logits().view(np.uint32), ol.view(np.uint32)), f"position {pos}"
        assert np.array_equal(gm.residual().view(np.uint32), ores.view(np.uint32)), f"position {pos}"
    gm.close(); om.close()
