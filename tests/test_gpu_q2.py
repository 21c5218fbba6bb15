"""The model's projections over the two-bit weight tiles, at the sizes where tiles, groups, spans and the ring end: the
narrowest and widest inputs, widths that are no multiple of 4096, a vocabulary that is no multiple of the 16-row tile, fewer
tiles than SMs. Logits must be the oracle's bit for bit (every sum's order is fixed, so the tolerance is zero)."""
import numpy as np
import pytest

from bonsai_vk_b200 import Model, synth
from tests._oracle import OracleModel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_layer,hidden,ffn,vocab,hat", [
    (2, 512, 512, 130, 512),         # one group of four blocks per row, one partial tile more than full ones
    (2, 2048, 5120, 333, 1024),      # the down projection's input ends inside its second span
    (1, 1024, 8192, 16, 256),        # two whole spans; a head of a single tile
    (1, 4096, 16384, 2100, 4096),    # the widest input: four spans, rings of three chunks
])
def test_two_bit_projections_match_the_oracle(ctx, n_layer, hidden, ffn, vocab, hat):
    hp = synth.HParams(n_layer=n_layer, hidden=hidden, ffn=ffn, vocab=vocab, n_head=hidden // 256, n_kv=max(1, hidden // 1024),
                       gdn_heads=hidden // 128, gdn_qk_heads=max(1, hidden // 256), hat_block=hat, cap=16, attn_interval=2)
    tensors, signs = synth.make_model(hp, seed=hidden + ffn)
    gm, om = Model(ctx, hp, tensors, signs), OracleModel(hp, tensors, signs)
    for pos, t in enumerate(np.random.default_rng(ffn).integers(0, vocab, size=3)):
        gm.token(int(t), pos)
        ol, _ = om.token(int(t), pos)
        assert np.array_equal(gm.logits().view(np.uint32), ol.view(np.uint32)), f"logits differ at position {pos}"
    gm.close(); om.close()
