"""The 3D near blocks beside the internal bases, whose CTAs hold whole SMs: few and large leaves are
spread over the chip, not sent to the SMs that come free first. 200,000 points on a line, about
360 leaves of up to 700: beside the bases the blocks take at most twice the time that the same sums
(and the finer far entries) take alone on the device. On the first SMs alone it was 4.5 times."""
import threading

import numpy as np
import pytest

from helpers import Engine
from helpers_kernels import kernels_of
from test_gpu_lists import _ring_P

pytestmark = pytest.mark.gpu

RUN = """
y = np.random.default_rng(1).uniform(-30, 30, (3, 200_000))
y[1:] *= 1e-3
Y = np.ascontiguousarray(y.astype(np.float32).astype(np.float64))
eng = Engine(_ring_P(Y.shape[1]), Y, h2_leaf_size=700, h2_tol=3e-2)
for _ in range(4):
    assert eng.rebuild() == 0
    eng.repulsive(Y)   # the build's blocks
    eng.repulsive(Y)   # a second product: the near field by itself
"""


def test_few_large_leaves_are_spread():
    times = kernels_of(RUN)
    blocks, = [t for k, t in times.items() if "k_near<3, 4, 1>" in k]
    alone, = [t for k, t in times.items() if "k_near<3, 4, 0>" in k]
    print(f"near blocks {blocks:.0f} us beside the bases, {alone:.0f} us alone")
    assert blocks <= 2.0 * alone


def test_threads_with_different_shares():
    """Workspaces of different trees build in threads at the same time, each asking for another share
    of an SM, and give the bits that they give alone."""
    rng = np.random.default_rng(2)
    Y = np.ascontiguousarray(rng.uniform(-9, 9, (3, 20_000)).astype(np.float32).astype(np.float64))
    engines = [Engine(_ring_P(Y.shape[1]), Y, h2_leaf_size=leaf, h2_tol=3e-2) for leaf in (30, 100, 250, 500)]
    try:
        leaves = [int((e.h2()["nodes"]["is_leaf"] != 0).sum()) for e in engines]
        assert len({-(-n // 148) for n in leaves}) >= 3 and min(leaves) < 16 * 148
        alone = [e.repulsive(Y) for e in engines]
        bad = []

        def work(e, want):
            for _ in range(100):
                ok = e.rebuild() == 0
                F, Z = e.repulsive(Y)
                if not (ok and Z == want[1] and np.array_equal(F, want[0])):
                    bad.append((e.params.h2_leaf_size, Z, want[1]))
                    return

        threads = [threading.Thread(target=work, args=a) for a in zip(engines, alone)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not bad, bad
    finally:
        for e in engines:
            e.close()
