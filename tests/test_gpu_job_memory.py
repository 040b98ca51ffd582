"""The server's admission estimate is an upper one: under a budget of 1.9 times what a job was measured
to hold (the device memory pool's high-water mark), two such jobs never run at once. In 2D and
3D, at the usual leaf size and at small ones, where trees are large; few entries in P, so that
the estimate's part for P hides nothing."""
import ctypes

import numpy as np
import pytest

from helpers import Engine
from test_gpu_lists import _ring_P

pytestmark = pytest.mark.gpu

ITERS = 4


class _Pool:
    """The default memory pool of device 0, through the driver."""

    USED_HIGH = 8   # CU_MEMPOOL_ATTR_USED_MEM_HIGH

    def __init__(self):
        import torch
        torch.zeros(1, device="cuda")
        self.cu, dev, self.pool = ctypes.CDLL("libcuda.so.1"), ctypes.c_int(), ctypes.c_void_p()
        assert self.cu.cuDeviceGet(ctypes.byref(dev), 0) == 0
        assert self.cu.cuDeviceGetDefaultMemPool(ctypes.byref(self.pool), dev) == 0

    def high(self, reset=False):
        v = ctypes.c_uint64(0)
        if reset:   # to the bytes in use now
            assert self.cu.cuMemPoolSetAttribute(self.pool, self.USED_HIGH, ctypes.byref(v)) == 0
        assert self.cu.cuMemPoolGetAttribute(self.pool, self.USED_HIGH, ctypes.byref(v)) == 0
        return v.value


def _clusters(d, n):
    """Dense cores with a long tail (the exaggeration phase's embeddings, whose trees are deepest)."""
    rng = np.random.default_rng(5)
    w = np.arange(1, 51) ** -1.1
    lab = rng.choice(50, n, p=w / w.sum())
    off = rng.standard_normal((n, d))
    off *= rng.random((n, 1)) ** (1 / d) / np.linalg.norm(off, axis=1, keepdims=True) / np.maximum(rng.random((n, 1)), 3e-4)
    y = 4.0 * rng.uniform(-1, 1, (50, d))[lab] + 0.2 * (w[lab, None] / w.sum()) ** (1 / d) * off
    return np.ascontiguousarray(y.T.astype(np.float32).astype(np.float64))


@pytest.mark.parametrize("d,n,leaf", [(2, 400_000, 100), (2, 60_000, 32), (2, 60_000, 8), (2, 60_000, 2),
                                      (3, 400_000, 100), (3, 100_000, 48), (3, 60_000, 8), (3, 30_000, 2)])
def test_two_jobs_over_the_budget_do_not_overlap(d, n, leaf):
    from tsne_h2pack.serving import EmbeddingServer
    P, Y0 = _ring_P(n), _clusters(d, n)
    tol = 1e-2 if d == 2 else 3e-2
    pool = _Pool()
    before = pool.high(reset=True)
    eng = Engine(P, Y0, n_iter=ITERS, h2_leaf_size=leaf, h2_tol=tol)
    eng.run_all()
    held = pool.high() - before
    eng.close()
    with EmbeddingServer(max_concurrent=2, hbm_budget_gb=1.9 * held / 1e9) as srv:
        ids = [srv.submit(P, n_components=d, init_Y=Y0, n_iter=ITERS, verbose=0, learning_rate=n / 12.0, h2_tol=tol,
                          h2_rebuild_freq=3, h2_rebuild_freq_early=10, h2_leaf_size=leaf) for _ in range(2)]
        a, b = sorted((srv.wait(j)[1] for j in ids), key=lambda r: r.start_s)
    print(f"{d}D {n} points, leaf {leaf}: {held / n:.0f} bytes per point")
    assert a.ok and b.ok
    assert b.start_s >= a.end_s
