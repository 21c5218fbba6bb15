"""The multi-sequence pass against the same sequences run one at a time, logits bit for bit, where its own kernels differ from the
single-sequence ones: 20 to 32 columns (the wide projection with its swiglu, residual and prefetch), 1, 8 and 64 splits of the
keys, softmax sums by one and by eight CTAs per head, one and four dims per thread in the values, 1, 2, 4 and 8 query heads per
kv head, both cache kinds, a different position in every column. The caches are filled with ones up to the last position and
hold real rows at the positions that the passes visit."""
import numpy as np
import pytest

from bonsai_vk_b200 import Model, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncol,cap,heads,modes", [
    (20, 64, (4, 1), (0, 0)), (32, 512, (4, 1), (0, 0)), (27, 512, (4, 2), (1, 0)), (24, 4096, (4, 1), (1, 1)),
    (32, 4096, (4, 4), (0, 0)), (21, 4096, (8, 1), (0, 1)), (17, 510, (4, 2), (0, 1)), (2, 4096, (4, 1), (0, 0)), (9, 16384, (4, 2), (1, 0))])
def test_columns_equal_single_sequences(ctx, ncol, cap, heads, modes):
    n_head, n_kv = heads
    kw = dict(n_layer=2, attn_interval=2, hidden=256 * n_head, gdn_heads=2 * n_head, gdn_qk_heads=n_head, n_head=n_head, n_kv=n_kv,
              k_mode=modes[0], v_mode=modes[1], cap=cap, vocab=1040, n_streams=ncol)
    tensors, signs = synth.make_model(synth.tiny(**kw), seed=ncol + cap)
    many, one = Model(ctx, synth.tiny(batch_cols=ncol, **kw), tensors, signs), Model(ctx, synth.tiny(**kw), tensors, signs)
    rng = np.random.default_rng(cap)
    last = [cap - 1 - (c * 37) % max(1, cap // 2) for c in range(ncol)]
    out, single = ctx.alloc(ncol * 4), ctx.alloc(4)
    many.stage_prepare(0, ncol)
    for c in range(ncol):
        one.stage_prepare(c)
        for m in (many, one):
            m.fill_kv(c, last[c])
    for back in (min(last) * 3 // 4, min(last) // 3, 1, 0):
        pos = [p - back for p in last]
        toks = [int(t) for t in rng.integers(0, 1040, size=ncol)]
        many.stage_batch(0, toks, pos, None, out)
        ctx.sync()
        picks = list(out.download(np.int32, ncol))
        for c in range(ncol):
            one.stage(c, toks[c], pos[c], None, single)
            ctx.sync()
            assert np.array_equal(many.logits(c).view(np.uint32), one.logits().view(np.uint32)), f"column {c} at position {pos[c]}"
            assert picks[c] == single.download(np.int32, 1)[0]
    many.close(); one.close()
    out.free(); single.free()
