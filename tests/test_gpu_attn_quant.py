"""The cache insert's q8_0 codes and scales of raw V rows at the values where its quantiser could go wrong: zeros, magnitudes
below the cut-off, exact ties, the largest magnitudes, infinities and NaNs beside ordinary values. Whole numbers and fp16 bits: equal."""
import numpy as np
import pytest

from bonsai_vk_b200 import lib as L

pytestmark = pytest.mark.gpu


def _q8_0(block):
    """d = amax / 127 (NaNs left out, 0 up to 1e-35), codes = round half away of v * (1 / d), clamped; a NaN becomes -127"""
    f = np.float32
    amax = f(np.max(np.where(np.isnan(block), f(0), np.abs(block))))
    with np.errstate(all="ignore"):
        d = amax / f(127) if amax > f(1e-35) else f(0)
        y = block * (f(1) / d if d != 0 else f(0))
        r = np.where(np.isnan(y), f(-127), np.clip(np.trunc(np.abs(y).astype(np.float64) + 0.5) * np.sign(y), -127, 127))
        return r.astype(np.int8), np.float16(d).view(np.uint16)


@pytest.mark.parametrize("tokens", [1, 3])
def test_inserted_values_at_the_edges(ctx, tokens):
    n_kv, hd, rng = 4, 256, np.random.default_rng(tokens)
    v = rng.standard_normal((tokens, n_kv * hd)).astype(np.float32)
    b = v.reshape(-1, 32)
    b[0] = 0
    b[1] = 1e-36
    b[2, :6] = [127.0, 0.5, -0.5, 1.5, -2.5, 126.5]
    b[2, 6:] = np.arange(26) - 12.5
    b[3] *= np.float32(3e38)
    b[4, 7], b[5, 3], b[6, 0], b[7, :] = np.inf, -np.inf, np.nan, np.nan
    b[8, 1:] = 0
    b[9] = -1e-35
    b[10] *= np.float32(1e-30)
    dims = L.AttnDimsC(n_head=16, n_kv=n_kv, head_dim=hd, n_rot=64, cap=64, k_mode=0, v_mode=0, rms_eps=1e-6, rope_base=1e7)
    kvb, scb = ctx.attn_sizes(dims)
    qg, nw, k = rng.standard_normal((16, 2 * hd)).astype(np.float32), np.ones(hd, dtype=np.float32), rng.standard_normal((tokens, n_kv * hd)).astype(np.float32)
    kv, scr, bk, bv, bq, bn = ctx.alloc(kvb), ctx.alloc(scb), *(ctx.from_numpy(x) for x in (k, v, qg, nw))
    ctx.attn_insert(dims, kv, bk, bv, tokens, 5, bq, bn, bn, scr)
    ctx.sync()
    raw = kv.download(np.uint8, kvb)
    n = 64 * n_kv * hd                            # codes of K, scales of K, codes of V, scales of V
    codes = raw[n + n // 16:][:n].view(np.int8).reshape(64, -1)[5:5 + tokens].reshape(-1, 32)
    scales = raw[2 * n + n // 16:][:n // 16].view(np.uint16).reshape(64, -1)[5:5 + tokens].reshape(-1)
    for i, block in enumerate(b):
        want, d = _q8_0(block)
        assert scales[i] == d and np.array_equal(codes[i], want), f"block {i}"
    for x in (kv, scr, bk, bv, bq, bn):
        x.free()
