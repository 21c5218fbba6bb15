"""Decode attention at the lengths where its kernels' work splits end: one key, the last key of an octet and the first of the
next, a cache of one split, the 32-key tiles of PV, the 8192 keys of one round of exponentials; the kept query attending twice.
Every sum's order is fixed, so the outputs must be the oracle's bit for bit (tolerance zero)."""
import ctypes as C

import numpy as np
import pytest

from bonsai_vk_b200 import lib as L
from bonsai_vk_b200 import synth
from tests._oracle import OracleModel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("keys,cap,k_mode,v_mode,heads", [
    (1, 64, 0, 0, (16, 4)), (8, 64, 0, 0, (4, 1)), (9, 510, 1, 0, (4, 1)), (63, 512, 0, 1, (16, 4)), (64, 4096, 0, 0, (16, 4)),
    (65, 4096, 1, 1, (8, 4)), (513, 514, 0, 0, (8, 1)), (4097, 8192, 0, 0, (16, 4)), (8193, 16384, 0, 0, (4, 4)),
    (12289, 16384, 1, 1, (16, 4))])
def test_attention_edges(ctx, keys, cap, k_mode, v_mode, heads):
    n_head, n_kv = heads
    hd, rng = 256, np.random.default_rng(keys)
    k, v = (rng.standard_normal((keys, n_kv * hd)).astype(np.float32) for _ in range(2))
    qg = rng.standard_normal((n_head, 2 * hd)).astype(np.float32)
    qn, kn = ((1 + 0.1 * rng.standard_normal(hd)).astype(np.float32) for _ in range(2))
    dims = L.AttnDimsC(n_head=n_head, n_kv=n_kv, head_dim=hd, n_rot=64, cap=cap, k_mode=k_mode, v_mode=v_mode, rms_eps=1e-6, rope_base=1e7)
    kvb, scb = ctx.attn_sizes(dims)
    kv, scr, bk, bv, bq, bqn, bkn = ctx.alloc(kvb), ctx.alloc(scb), *(ctx.from_numpy(x) for x in (k, v, qg, qn, kn))
    pre, out = ctx.alloc(n_head * hd * 4), ctx.alloc(n_head * hd * 4)
    ctx.attn_insert(dims, kv, bk, bv, keys, 0, bq, bqn, bkn, scr)
    hp = synth.HParams(n_layer=4, hidden=n_head * hd, n_head=n_head, n_kv=n_kv, cap=cap, vocab=128, k_mode=k_mode, v_mode=v_mode)
    om = OracleModel(hp, {"blk.3.attn_q_norm.weight": qn, "blk.3.attn_k_norm.weight": kn}, np.ones(4, dtype=np.int32))
    want_pre, want = (np.empty(n_head * hd, dtype=np.float32) for _ in range(2))
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    om.o.lib.bo_attn_fill_and_attend(om.m, 3, 0, keys, p(qg), p(k), p(v), p(want_pre), p(want))
    om.close()
    if keys > 2:                              # over a prefix first: its maximum must not stay behind
        ctx.attn_attend(dims, kv, keys // 2, scr, None, out)
    for _ in range(2):
        ctx.attn_attend(dims, kv, keys - 1, scr, pre, out)
        ctx.sync()
        assert np.array_equal(pre.download(np.uint32, n_head * hd), want_pre.view(np.uint32))
        assert np.array_equal(out.download(np.uint32, n_head * hd), want.view(np.uint32))
    for b in (kv, scr, bk, bv, bq, bqn, bkn, pre, out):
        b.free()
