"""Host arrays keep the caller's point order across a renumbering: the embedding set is the one read back, and what
is read after a run is what the oracle's order says (no arithmetic: equal to the FP32 rounding of the input)."""
import numpy as np
import pytest

from helpers import Engine
from test_gpu_lists import _ring_P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n", [(2, 2_001), (2, 70_001), (3, 5_003)])
def test_set_and_get_after_renumbering(d, n):
    rng = np.random.default_rng(n)
    eng = Engine(_ring_P(n), rng.standard_normal((d, n)), n_iter=40)
    try:
        for run in (0, 40):      # before any renumbering, and after the one at iteration 30
            if run:
                eng.run(0, run)
            Y = np.ascontiguousarray(rng.standard_normal((d, n)))
            eng.set_embedding(Y)
            want = Y.astype(np.float32).astype(np.float64)
            assert np.array_equal(eng.embedding(), want)
            assert np.array_equal(eng.state()[0], want)
    finally:
        eng.close()
