"""The sweep that times the recurrent cores advances the state exactly as many cores one after the other do: on a model with one
recurrent layer, where every core of the sweep works on the state that the core in front writes, the state afterwards is the one
that a sweep with plain launches leaves."""
import os

import numpy as np
import pytest

from bonsai_vk_b200 import Model, synth
from bonsai_vk_b200 import lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("one_cta", [False, True])
def test_sweep_advances_the_state_in_order(ctx, monkeypatch, one_cta):
    hp = synth.tiny(n_layer=2, attn_interval=2, gdn_heads=8)
    tensors, signs = synth.make_model(hp, seed=4)
    if one_cta:
        monkeypatch.setenv("BONSAI_GDN_ONE_CTA_PER_HEAD", "1")
    states = []
    for plain in (False, True):
        if plain:
            os.environ["BONSAI_NO_PDL"] = "1"
        try:
            m = Model(ctx, hp, tensors, signs)
        finally:
            os.environ.pop("BONSAI_NO_PDL", None)
        for p, t in enumerate((3, 99, 1024)):
            m.token(t, p)
        for _ in range(4):
            m.mixer_sweep_us(reps=50)
        states.append(m.read(L.READ_GDN_STATE, np.uint32, hp.gdn_heads * hp.gdn_dim ** 2))
        m.close()
    Model(ctx, hp, tensors, signs).close()        # (programmatic launches on again for whoever comes next)
    assert np.array_equal(*states)
