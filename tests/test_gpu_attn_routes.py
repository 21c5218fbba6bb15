"""Decode attention of one query token through the chain of kernels instead of the one cluster launch (what a device without room
for 16-CTA clusters gets): accepted without an error, and the same bits, over the capacities, head ratios and cache kinds of both."""
import numpy as np
import pytest

from bonsai_vk_b200 import lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap,keys", [(64, 63), (510, 510), (512, 200), (2048, 2047), (4096, 1), (8192, 8100)])
@pytest.mark.parametrize("heads", [(4, 4), (8, 4), (16, 4), (8, 1)])
def test_chain_gives_the_cluster_kernels_bits(ctx, monkeypatch, cap, keys, heads):
    n_head, n_kv = heads
    k_mode, v_mode = [(0, 0), (1, 0), (1, 1), (0, 1)][(n_head // 4 + n_kv + cap) % 4]
    v_mode = 0 if cap == 8192 else v_mode          # (fp16 values of 8192 positions do not fit a cluster)
    hd, rng = 256, np.random.default_rng(cap + keys)
    k, v = (rng.standard_normal((keys, n_kv * hd)).astype(np.float32) for _ in range(2))
    qg, nw = rng.standard_normal((n_head, 2 * hd)).astype(np.float32), (1 + 0.1 * rng.standard_normal(hd)).astype(np.float32)
    dims = L.AttnDimsC(n_head=n_head, n_kv=n_kv, head_dim=hd, n_rot=64, cap=cap, k_mode=k_mode, v_mode=v_mode, rms_eps=1e-6, rope_base=1e7)
    kvb, scb = ctx.attn_sizes(dims)
    kv, scr, bk, bv, bq, bn = ctx.alloc(kvb), ctx.alloc(scb), *(ctx.from_numpy(x) for x in (k, v, qg, nw))
    pre, out = ctx.alloc(n_head * hd * 4), ctx.alloc(n_head * hd * 4)
    ctx.attn_insert(dims, kv, bk, bv, keys, 0, bq, bn, bn, scr)
    got = []
    for chain in (False, True):
        monkeypatch.setenv("BONSAI_ATTN_CHAIN", "1") if chain else monkeypatch.delenv("BONSAI_ATTN_CHAIN", raising=False)
        before = ctx.launches
        ctx.attn_attend(dims, kv, keys - 1, scr, pre, out)
        ctx.sync()
        assert (ctx.launches - before > 1) == chain, "not the route that this comparison is about"
        got.append((pre.download(np.uint32, n_head * hd), out.download(np.uint32, n_head * hd)))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    for b in (kv, scr, bk, bv, bq, bn, pre, out):
        b.free()
