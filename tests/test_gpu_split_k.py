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
    assert ctx.projection_split(hidden, ffn)[0] > 0        # otherwise the general kernel gives the same floats
    tensors, signs = synth.make_model(hp, seed=3)
    gm, om = Model(ctx, hp, tensors, signs), OracleModel(hp, tensors, signs)
    for pos, t in enumerate((5, 630, 77)):
        gt = gm.token(t, pos)
        ol, ores = om.token(t, pos)
        assert gt == om.argmax(ol) and np.array_equal(gm.logits().view(np.uint32), ol.view(np.uint32)), f"position {pos}"
        assert np.array_equal(gm.residual().view(np.uint32), ores.view(np.uint32)), f"position {pos}"
    gm.close(); om.close()


@pytest.mark.parametrize("hidden,ffn", [(7168, 12288), (5120, 16384)])
def test_more_chunks_than_ring_slots(ctx, hidden, ffn):
    """11 or 12 row tiles per cluster: six chunks of weights in five slots."""
    assert ctx.projection_split(hidden, ffn)[1] in (11, 12)
    hp = synth.tiny(n_layer=1, attn_interval=2, hidden=hidden, n_head=hidden // 256, n_kv=hidden // 1024, gdn_heads=hidden // 128, gdn_qk_heads=hidden // 256,
                    ffn=ffn, hat_block=1024, vocab=640)
    tensors, signs = synth.make_model(hp, seed=4)
    gm, om = Model(ctx, hp, tensors, signs), OracleModel(hp, tensors, signs)
    for pos, t in enumerate((5, 630)):
        gt = gm.token(t, pos)
        ol, ores = om.token(t, pos)
        assert gt == om.argmax(ol) and np.array_equal(gm.logits().view(np.uint32), ol.view(np.uint32)), f"position {pos}"
        assert np.array_equal(gm.residual().view(np.uint32), ores.view(np.uint32)), f"position {pos}"
    gm.close(); om.close()


def test_which_projections_share_k(ctx):
    """The rule on both sides: widths that are whole spans, shares of up to twelve tiles, one further piece per warp at most."""
    assert ctx.projection_split(4096, 4096) == ctx.projection_split(4096, 10240) == ctx.projection_split(4096, 20480) == (0, 0)
    for M, K in ((4096, 12288), (7168, 12288), (5120, 16384), (8192, 8192)):
        n, tiles = ctx.projection_split(M, K)
        assert 0 < n * (K // 4096) <= ctx.info()["sm_count"] and tiles == -(-M // 16 // n)
    for M, K in ((8192, 12288), (6144, 16384), (248320, 8192)):
        assert ctx.projection_split(M, K) == (0, 0)
