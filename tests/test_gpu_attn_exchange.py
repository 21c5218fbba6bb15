"""The exchanges of the one-launch attention: every CTA waits for exactly the bytes that its neighbours store into it, which depends on
the filled prefix modulo 128 (residues of eight keys per CTA) and on how many splits have keys. A prefix on each side of those
lines, in caches of one, eight and 64 splits: the bits of the chain of kernels; and the wait gives up when nothing comes."""
import numpy as np
import pytest

from bonsai_vk_b200 import lib as L
from bonsai_vk_b200.lib import BonsaiError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap,heads,v_mode", [(256, (16, 4), 0), (510, (8, 1), 1), (1024, (16, 4), 1), (2048, (4, 4), 0), (4096, (8, 4), 1), (8192, (16, 4), 0)])
def test_prefixes_around_the_residues(ctx, monkeypatch, cap, heads, v_mode):
    n_head, n_kv = heads
    hd, rng = 256, np.random.default_rng(cap)
    keys = min(cap, 1100)
    k, v = (rng.standard_normal((keys, n_kv * hd)).astype(np.float32) for _ in range(2))
    qg, nw = rng.standard_normal((n_head, 2 * hd)).astype(np.float32), (1 + 0.1 * rng.standard_normal(hd)).astype(np.float32)
    dims = L.AttnDimsC(n_head=n_head, n_kv=n_kv, head_dim=hd, n_rot=64, cap=cap, k_mode=0, v_mode=v_mode, rms_eps=1e-6, rope_base=1e7)
    kvb, scb = ctx.attn_sizes(dims)
    kv, scr, bk, bv, bq, bn = ctx.alloc(kvb), ctx.alloc(scb), *(ctx.from_numpy(x) for x in (k, v, qg, nw))
    pre, out = ctx.alloc(n_head * hd * 4), ctx.alloc(n_head * hd * 4)
    ctx.attn_insert(dims, kv, bk, bv, keys, 0, bq, bn, bn, scr)
    for n in (1, 2, 7, 8, 9, 63, 64, 65, 120, 121, 127, 128, 129, 136, 137, 255, 256, 511, 513, 1023, 1024, 1025, 1100):
        if n > keys:
            break
        got = []
        for chain in (False, True):
            monkeypatch.setenv("BONSAI_ATTN_CHAIN", "1") if chain else monkeypatch.delenv("BONSAI_ATTN_CHAIN", raising=False)
            before = ctx.launches
            ctx.attn_attend(dims, kv, n - 1, scr, pre, out)
            ctx.sync()
            assert (ctx.launches - before > 1) == chain
            got.append((pre.download(np.uint32, n_head * hd), out.download(np.uint32, n_head * hd)))
        assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1]), f"{n} keys"
    for b in (kv, scr, bk, bv, bq, bn, pre, out):
        b.free()


def test_the_wait_gives_up(ctx):
    ctx.sync()
    ctx.selftest_wait(2)
    with pytest.raises(BonsaiError, match="exchange of the attention clusters"):
        ctx.sync()
    ctx.sync()
