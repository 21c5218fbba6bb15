"""The timing aids divide by the launches that they made, whatever the environment holds."""
import numpy as np

from bonsai_vk_b200 import kernel_lab


class _Buffer:
    def __init__(self, n=0):
        self.n = n

    def upload(self, a, off=0):
        return self

    def download(self, dtype, count):
        return np.zeros(count, dtype=dtype)

    def free(self):
        pass


class _Context:
    """Counts projections; the clock advances by one millisecond for each."""
    class lib:
        bn_gemm_tiled_bytes = staticmethod(lambda M, K: 64)

    def __init__(self):
        self.count = 0

    def alloc(self, n):
        return _Buffer(n)

    def from_numpy(self, a):
        return _Buffer(a.nbytes)

    def gemm_repack(self, w, M, K, w_off=0):
        return _Buffer(64)

    def gemm_q81(self, *a, **k):
        self.count += 1

    def event(self):
        return [0]

    def record(self, e):
        e[0] = self.count

    def elapsed_ms(self, e0, e1):
        return float(e1[0] - e0[0])

    def gemm_image_bytes(self, K, ncol):
        return 64

    act_pack_bytes = staticmethod(lambda K: 64)

    def gemm_act_quant(self, *a, **k):
        pass

    act_quant_q81 = gemv_q81 = gemm_act_quant

    def sync(self):
        pass


def test_gemm_time_is_per_launch(monkeypatch):
    monkeypatch.setenv("BONSAI_GEMM_REPS", "7")
    ms, nbytes = kernel_lab.gemm_lab(["100000", "1024", "8", "3"], ctx=_Context(), quiet=True)
    assert ms == 1.0 and nbytes == 100000 * 8 * 28
