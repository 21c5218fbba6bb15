"""Two threads, each with a context and a model of its own width, decode at the same time: kernel limits are process-wide, so what
one thread's launches need must hold whatever the other launches. The streams are those of the same models decoded one at a time."""
import threading

import numpy as np
import pytest

from bonsai_vk_b200 import Context, Model, synth

pytestmark = pytest.mark.gpu


def _decode(ctx, hp, tensors, signs, rounds):
    out = []
    for _ in range(rounds):
        m = Model(ctx, hp, tensors, signs)
        nxt = m.prefill([3, 7, 11], 0)
        out.append([nxt] + m.decode(nxt, 3, 6) + [m.token(5, 9)])
        out.append(m.logits().view(np.uint32).copy())
        m.close()
    return out


def test_two_contexts_on_two_threads():
    shapes = [synth.tiny(n_layer=2, attn_interval=2, batch_cols=3, ffn=f) for f in (1024, 12288)]
    models = [(hp, *synth.make_model(hp, seed=hp.ffn)) for hp in shapes]
    ctxs = [Context(0) for _ in models]
    got = [None] * len(models)

    def work(i):
        try:
            got[i] = _decode(ctxs[i], *models[i], 6)
        except Exception as e:                # noqa: BLE001 - handed to the main thread
            got[i] = e

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(models))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i, (g, m) in enumerate(zip(got, models)):
        assert not isinstance(g, Exception), g
        want = _decode(ctxs[i], *m, 1)
        for r in range(6):
            assert g[2 * r] == want[0] and np.array_equal(g[2 * r + 1], want[1]), f"thread {i}, round {r}"
    for c in ctxs:
        c.close()
