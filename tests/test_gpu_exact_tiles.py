"""The exact O(N^2) sums (32 targets a CTA, a 256-source tile a warp, 8 tiles a round) against the oracle: one
iteration's displacement (Z scales its repulsive part) at sizes around a warp of targets, a tile, a round and a ragged last one.

Tolerance: FP32 within a tile of 256 sources (at most 256 x 6e-8 = 1.5e-5 of the sum of magnitudes, the reciprocal
4e-7) and the cancellation of y s - v, at most 3 here: 5e-5 of the displacement's norm."""
import numpy as np
import pytest

import oracle as O
from helpers import Engine, rel2
from test_gpu_lists import _ring_P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [2, 3])
@pytest.mark.parametrize("n", [31, 33, 255, 256, 257, 511, 2_047, 2_048, 2_049, 4_100])
def test_exact_iteration_equals_oracle(d, n):
    Y = np.random.default_rng(n).standard_normal((d, n)).astype(np.float32).astype(np.float64)
    P = _ring_P(n)
    eng = Engine(P, Y, n_iter=1, exact=True)
    try:
        eng.run(0, 1)
        got = eng.embedding()
    finally:
        eng.close()
    want, _ = O.run(P, Y, n_iter=1, use_h2=False)
    assert rel2(got - Y, want - Y) <= 5e-5
