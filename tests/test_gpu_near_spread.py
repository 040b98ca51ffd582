"""The 3D near blocks beside the internal bases, whose CTAs hold whole SMs: few and large leaves are
spread over the chip, not sent to the SMs that come free first. 200,000 points on a line, about
360 leaves of up to 700: beside the bases the blocks take at most twice the time that the same sums
(and the finer far entries) take alone on the device. On the first SMs alone it was 4.5 times."""
import pytest

from helpers_kernels import kernels_of

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
