"""9 to 16 columns on tiles where a CTA's units of two row tiles go to 12 warps: the build has two forms, by when it releases the kernel
behind it. The early one (single projections, and everything but a recurrent block's input) against the single-column
projection, at heights around a whole last tile and two and several tiles a CTA; the late one in the pass of several sequences, whose
recurrent mixer reads ahead of its wait, against the same sequences one at a time. The bits."""
import numpy as np
import pytest

from bonsai_vk_b200 import Model, ptq, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,ncol", [(4096, 4096, 16), (4081, 4096, 9), (7474, 3072, 11), (9000, 2048, 16), (3000, 5120, 13), (30000, 1024, 10)])
def test_early_release(ctx, M, K, ncol):
    rng = np.random.default_rng(M + ncol)
    W = ptq.synth_matrix(rng, M, K)
    x = rng.standard_normal((ncol, K)).astype(np.float32)
    wb, xb = ctx.from_numpy(W), ctx.from_numpy(x)
    image, out = ctx.alloc(ctx.gemm_image_bytes(K, ncol)), ctx.alloc(ncol * M * 4)
    tiles = ctx.gemm_repack(wb, M, K)
    for _ in range(3):                            # (each launch behind another of its kind)
        ctx.gemm_act_quant(xb, K, ncol, image)
        ctx.gemm_q81(tiles, M, K, image, ncol, out, tiled=True)
    ctx.sync()
    got = out.download(np.uint32, ncol * M).reshape(ncol, M)
    pack, one = ctx.alloc(ctx.act_pack_bytes(K)), ctx.alloc(M * 4)
    for c in range(ncol):
        ctx.act_quant_q81(xb, K, pack, x_off=c * K * 4)
        ctx.gemv_q81(wb, M, K, pack, one)
        ctx.sync()
        assert np.array_equal(got[c], one.download(np.uint32, M)), f"column {c}"
    for b in (wb, xb, image, out, tiles, pack, one):
        b.free()


@pytest.mark.parametrize("ncol", [9, 16])
def test_late_release(ctx, ncol):
    kw = dict(n_layer=4, attn_interval=4, hidden=2048, ffn=2048, gdn_heads=16, gdn_qk_heads=8, n_head=8, n_kv=2, cap=64, vocab=1040, n_streams=ncol)
    tensors, signs = synth.make_model(synth.tiny(**kw), seed=ncol)
    many, one = Model(ctx, synth.tiny(batch_cols=ncol, **kw), tensors, signs), Model(ctx, synth.tiny(**kw), tensors, signs)
    rng = np.random.default_rng(ncol)
    out, single = ctx.alloc(ncol * 4), ctx.alloc(4)
    many.stage_prepare(0, ncol)
    for c in range(ncol):
        one.stage_prepare(c)
    for step in range(4):
        toks = [int(t) for t in rng.integers(0, 1040, size=ncol)]
        many.stage_batch(0, toks, [step] * ncol, None, out)
        ctx.sync()
        for c in range(ncol):
            one.stage(c, toks[c], step, None, single)
            ctx.sync()
            assert np.array_equal(many.logits(c).view(np.uint32), one.logits().view(np.uint32)), f"column {c}, step {step}"
    many.close(); one.close()
    out.free(); single.free()
