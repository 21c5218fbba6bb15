"""Decode attention where the rule for the values kernel's dims per thread (pv_any in attn.cu) changes its mind: eight query heads per
kv head up to three CTAs an SM (two dims, q8_0 and fp16 values) and beyond (four), four heads at 256, 768 (uneven) and 1024 CTAs; keys
that leave a tile of one key in a split, and one more than whole tiles. The oracle's floats."""
import pytest

from tests.test_gpu_attn import test_decode_attention_layer as compare_with_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctx_len,heads,modes", [(16385, (8, 1), (0, 0)), (16450, (8, 1), (1, 1)), (16400, (16, 2), (0, 0)), (16384, (16, 2), (0, 1)),
                                                 (16400, (12, 3), (0, 0)), (16401, (4, 1), (1, 0)), (16640, (16, 4), (0, 1))])
def test_one_token_beyond_the_clusters(ctx, ctx_len, heads, modes):
    compare_with_oracle(ctx, ctx_len, *modes, heads)


@pytest.mark.parametrize("ctx_len,heads,modes", [(4097, (32, 4), (0, 0)), (6200, (32, 4), (0, 1)), (4200, (64, 8), (0, 0)), (4161, (24, 6), (0, 0))])
def test_sixty_four_splits(ctx, monkeypatch, ctx_len, heads, modes):
    monkeypatch.setenv("BONSAI_ATTN_CHAIN", "1")
    compare_with_oracle(ctx, ctx_len, *modes, heads)
