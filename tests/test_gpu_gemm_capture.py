"""The multi-column projection of native rows inside a stream capture: accepted as the first call of a context (there is no scratch
yet and none may be allocated), the replays give the floats of the uncaptured call and of the single-column projection bit for bit, and
they still do after the context's scratch has been replaced by a larger one. One tile and one group of K, a height that is no whole
tile, waves of K that do not fit at once, several passes over the row tiles; uncaptured calls that unpack in place (0 chunks of tiles),
and through one or two chunks of scratch."""
import numpy as np
import pytest

from bonsai_vk_b200 import Context, ptq

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,ncol,chunks", [(16, 1024, 1, 0), (3000, 5120, 11, 0), (130, 13312, 32, 1), (4754, 2048, 17, 0), (40000, 1024, 8, 0), (30001, 1024, 16, 0),
                                             (30000, 2048, 25, 1), (4754, 3072, 17, 1), (3000, 5120, 20, 1), (12289, 7168, 11, 1), (190001, 1024, 18, 2)])
def test_native_rows_under_capture(M, K, ncol, chunks):
    rng = np.random.default_rng(M + K + ncol)
    rows = min(M, 4096)
    W = ptq.synth_matrix(rng, rows, K)
    W.reshape(rows, -1, 28)[0, -1, 26:] = (0x00, 0xFC)      # -inf scale in the last block of row 0
    W = np.ascontiguousarray(np.concatenate([W] * (-(-M // rows)), axis=0)[:M])
    X = rng.standard_normal((ncol, K)).astype(np.float32)
    ctx, st = Context(0), torch.cuda.Stream()
    ctx.use_stream(st.cuda_stream)
    xb, wb, image, out = ctx.from_numpy(X), ctx.from_numpy(W), ctx.alloc(ctx.gemm_image_bytes(K, ncol)), ctx.alloc(ncol * M * 4)
    ctx.gemm_act_quant(xb, K, ncol, image)
    ctx.sync()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        ctx.gemm_q81(wb, M, K, image, ncol, out)
    got = []
    for replay in (True, False, True):
        out.memset(0xFF)
        ctx.sync()
        if replay:
            with torch.cuda.stream(st):
                g.replay()
        else:                                               # outside the capture the scratch comes and, with a larger matrix, goes
            before = ctx.launches
            ctx.gemm_q81(wb, M, K, image, ncol, out)
            assert ctx.launches - before == (2 * chunks or 1)
        ctx.sync()
        got.append(out.download(np.uint32, ncol * M))
        if not replay:
            big, image2, o2 = ctx.alloc(200000 * 8 * 28), ctx.alloc(ctx.gemm_image_bytes(1024, 17)), ctx.alloc(17 * 200000 * 4)
            big.memset(0); image2.memset(0)
            before = ctx.launches
            ctx.gemm_q81(big, 200000, 1024, image2, 17, o2)
            ctx.sync()
            assert ctx.launches - before == 4               # (two chunks of tiles, the first of 48 MB: more than a case of one needs)
            big.free(); image2.free(); o2.free()
    nan = np.isnan(got[1].view(np.float32))
    for i in (0, 2):
        assert np.array_equal(np.isnan(got[i].view(np.float32)), nan) and np.array_equal(got[i][~nan], got[1][~nan]), f"run {i}"
    pack, one = ctx.alloc(ctx.act_pack_bytes(K)), ctx.alloc(M * 4)
    for c in sorted({0, ncol // 2, ncol - 1}):
        ctx.act_quant_q81(xb, K, pack, x_off=c * K * 4)
        ctx.gemv_q81(wb, M, K, pack, one)
        ctx.sync()
        want, n = one.download(np.uint32, M), nan.reshape(ncol, M)[c]
        assert np.array_equal(np.isnan(want.view(np.float32)), n) and np.array_equal(got[1].reshape(ncol, M)[c][~n], want[~n]), f"column {c}"
    pack.free(); one.free()
    del g
    for b in (xb, wb, image, out):
        b.free()
    ctx.close()
