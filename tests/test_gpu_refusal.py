"""A projection launch that the runtime refuses (host side; nothing faults) while a schedule is captured or enqueued: the call reports it,
no graph without that projection is kept, and the calls behind it give the oracle's floats."""
import numpy as np
import pytest

from bonsai_vk_b200 import BonsaiError, Context, Model, synth
from tests._oracle import OracleModel

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", ["token", "decode", "stage", "prefill", "sweep"])
def test_refused_launch_is_reported(path):
    hp = synth.tiny(n_layer=2, attn_interval=2, batch_cols=4)
    tensors, signs = synth.make_model(hp, seed=5)
    ctx, st = Context(0), torch.cuda.Stream()
    ctx.use_stream(st.cuda_stream)
    m, om = Model(ctx, hp, tensors, signs), OracleModel(hp, tensors, signs)
    out = ctx.alloc(16)
    calls = {"token": lambda: m.token(5, 0), "decode": lambda: m.decode(5, 0, 1)[0], "prefill": lambda: m.prefill([5], 0)}

    def stage():
        m.stage_prepare(0)
        m.stage(0, 5, 0, None, out)
        ctx.sync()
        return int(out.download(np.int32, 1)[0])
    call = stage if path == "stage" else calls.get(path, calls["token"])
    ctx.selftest_refusal()
    with pytest.raises(BonsaiError):
        m.gemv_sweep_ms(1) if path == "sweep" else call()
    m.reset()
    want, _ = om.token(5, 0)
    assert call() == om.argmax(want)
    assert np.array_equal(m.logits().view(np.uint32), want.view(np.uint32))
    m.close(); om.close(); ctx.close()
