"""The multi-column projection of native rows inside a stream capture: accepted as the first call of a context (there is no scratch
yet and none may be allocated), the replays give the floats of the uncaptured call bit for bit, and they still do after the
context's scratch has been replaced by a larger one. One tile and one group of K, a height that is no whole tile, waves of K that
do not fit at once, several passes over the row tiles."""
import numpy as np
import pytest

from bonsai_vk_b200 import Context, ptq

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,ncol", [(16, 1024, 1), (3000, 5120, 11), (130, 13312, 32), (4754, 2048, 17), (40000, 1024, 8), (30001, 1024, 16), (30000, 2048, 25)])
def test_native_rows_under_capture(M, K, ncol):
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
            ctx.gemm_q81(wb, M, K, image, ncol, out)
        ctx.sync()
        got.append(out.download(np.uint32, ncol * M))
        if not replay:
            big = ctx.alloc(200000 * 8 * 28)
            big.memset(0)
            o2 = ctx.alloc(200000 * 4)
            ctx.gemm_q81(big, 200000, 1024, image, 1, o2)   # (the image holds at least this much)
            ctx.sync()
            big.free(); o2.free()
    nan = np.isnan(got[1].view(np.float32))
    for i in (0, 2):
        assert np.array_equal(np.isnan(got[i].view(np.float32)), nan) and np.array_equal(got[i][~nan], got[1][~nan]), f"run {i}"
    del g
    for b in (xb, wb, image, out):
        b.free()
    ctx.close()
