"""Batched prefill leaves the model where a token-serial prompt leaves it - both conv-tap buffers, recurrent state, cache rows and
logits, bit for bit - so that not only the straight continuation but any later pass gives the serial model's floats: the last
position once more, and the whole prompt again from its first position, without a reset. Blocks of 1 to 32 tokens (with up to
three the taps come partly from the history), odd and even, from odd and even positions."""
import numpy as np
import pytest

from bonsai_vk_b200 import Model, synth
from bonsai_vk_b200 import lib as L

pytestmark = pytest.mark.gpu


def _same(a, b, what):
    assert np.array_equal(a.logits().view(np.uint32), b.logits().view(np.uint32)), f"{what}: logits differ"
    hp = a.hp
    gdn = [i for i in range(hp.n_layer) if not hp.is_attn(i)]
    for gi in range(len(gdn)):
        for sel, n in ((L.READ_GDN_STATE, hp.gdn_heads * hp.gdn_dim ** 2), (L.READ_CONV_HIST, hp.qkv_dim * 3)):
            x, y = a.read(sel, np.uint32, n, gi), b.read(sel, np.uint32, n, gi)
            assert np.array_equal(x, y), f"{what}: read {sel} of recurrent layer {gi} differs"
    n = hp.cap * hp.n_kv * hp.head_dim
    for li in range(hp.n_layer - len(gdn)):
        for sel, dt, k in ((L.READ_K_DATA, np.int8, n), (L.READ_K_SCALE, np.uint16, n // 32), (L.READ_V_DATA, np.int8, n), (L.READ_V_SCALE, np.uint16, n // 32)):
            assert np.array_equal(a.read(sel, dt, k, li), b.read(sel, dt, k, li)), f"{what}: read {sel} of attention layer {li} differs"


def _run(serial, blocked, vocab, start, blocks, seed):
    rng = np.random.default_rng(seed)
    lead = [int(t) for t in rng.integers(0, vocab, size=start)]
    prompt = [int(t) for t in rng.integers(0, vocab, size=sum(blocks))]
    for m in (serial, blocked):
        m.reset()
        for p, t in enumerate(lead):
            m.token(t, p, want_next=False)

    def feed(what):
        at = 0
        for n in blocks:
            nb = blocked.prefill(prompt[at:at + n], start + at)
            for i in range(at, at + n):
                ns = serial.token(prompt[i], start + i)
            assert nb == ns, f"{what}: pick after position {start + at + n - 1}"
            at += n
        _same(serial, blocked, what)
        return ns

    feed("prompt")
    end = start + len(prompt)
    for m in (serial, blocked):
        m.token(prompt[-1], end - 1, want_next=False)
    _same(serial, blocked, "last position once more")
    nxt = feed("prompt again")
    assert serial.decode(nxt, end, 3) == blocked.decode(nxt, end, 3)
    _same(serial, blocked, "continuation")


@pytest.fixture(scope="module")
def tiny_pair(ctx):
    tensors, signs = synth.make_model(synth.tiny(), seed=21)
    serial, blocked = Model(ctx, synth.tiny(), tensors, signs), Model(ctx, synth.tiny(batch_cols=32), tensors, signs)
    yield serial, blocked
    serial.close(); blocked.close()


@pytest.mark.parametrize("start,blocks", [
    (0, [1]), (1, [1, 1]), (0, [2]), (3, [2, 2]), (0, [3]), (5, [3, 3]), (10, [5]), (0, [17]), (7, [17]), (2, [32]), (9, [32]),
    (0, [16, 5]), (4, [8, 8, 1]), (1, [32, 2])])
def test_blocks_leave_the_serial_state(tiny_pair, start, blocks):
    _run(*tiny_pair, synth.tiny().vocab, start, blocks, seed=start + 100 * sum(blocks))


def test_odd_prompt_in_blocks_of_8_at_the_9b_shape(ctx):
    hp = synth.HParams(n_layer=4, vocab=2048, cap=64)
    tensors, signs = synth.make_model_repeated(hp, seed=2)
    serial = Model(ctx, hp, tensors, signs)
    blocked = Model(ctx, synth.HParams(n_layer=4, vocab=2048, cap=64, batch_cols=8), tensors, signs)
    for start in (0, 3):
        _run(serial, blocked, hp.vocab, start, [8, 8, 5], seed=start)
    serial.close(); blocked.close()
