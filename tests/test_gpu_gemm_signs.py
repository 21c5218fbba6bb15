"""bn_gemm_act_quant rotates H(s . x) for the integers s that it is given: factors other than +-1 scale their values (0 drops them),
as multiplying x by them first does, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hat", [16, 256, 1024])
def test_integer_factors(ctx, hat):
    K, ncol, rng = 3072, 5, np.random.default_rng(hat)
    x = rng.standard_normal((ncol, K)).astype(np.float32)
    s = rng.choice(np.array([1, -1, 0, 2, -3], dtype=np.int32), size=K)
    images = []
    for values, factors in ((x, s), (x * s.astype(np.float32), np.ones(K, dtype=np.int32))):
        xb, sb, im = ctx.from_numpy(values), ctx.from_numpy(factors), ctx.alloc(ctx.gemm_image_bytes(K, ncol))
        ctx.gemm_act_quant(xb, K, ncol, im, signs=sb, hat_block=hat)
        ctx.sync()
        images.append(im.download(np.uint8, ctx.gemm_image_bytes(K, ncol)))
        for b in (xb, sb, im):
            b.free()
    assert np.array_equal(*images)
