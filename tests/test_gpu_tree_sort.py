"""The tree's key sort (sorted tiles and bisected ranks up to 131,072 points, the radix sort above) and
its marks against the oracle's tree, bit for bit: sizes around a tile and around the limit, equal
keys across tiles (their order is the points'), leaf sizes above the staged keys' 256, and point
sets whose nodes end at a block of 1,024 points."""
import numpy as np
import pytest

import oracle as O
from helpers import Engine
from test_gpu_lists import _ring_P

pytestmark = pytest.mark.gpu


def _points(d, n, kind, seed):
    rng = np.random.default_rng(seed)
    y = rng.standard_normal((d, n)) * rng.choice([0.05, 1.0, 6.0], size=(1, n))
    if kind == "equal":        # a third of the points on 5 places, spread over the tiles
        on = rng.random(n) < 0.33
        y[:, on] = y[:, rng.integers(0, 5, on.sum())]
    elif kind == "grid":       # few distinct coordinates: long runs of shared digits
        y = np.round(y * 4) / 4
    return y


CASES = [(2, 2_047, "plain", 100), (2, 2_048, "equal", 100), (2, 2_049, "plain", 40), (3, 4_096, "grid", 64),
         (3, 4_097, "equal", 100), (2, 10_240, "grid", 100), (2, 20_479, "equal", 300), (3, 20_481, "plain", 700),
         (2, 131_072, "equal", 100), (2, 131_073, "equal", 100), (2, 9_000, "plain", 256), (2, 9_001, "plain", 257)]


@pytest.mark.parametrize("d,n,kind,leaf", CASES)
def test_tree_equals_oracle(d, n, kind, leaf):
    Y = np.ascontiguousarray(_points(d, n, kind, n + d).astype(np.float32).astype(np.float64))
    eng = Engine(_ring_P(n), Y, h2_leaf_size=leaf, h2_tol=3e-2)
    try:
        eng.rebuild()
        ref = O.H2(Y, leaf_size=leaf, tol=3e-2)
        g = eng.h2()
        if g is None:
            assert ref.max_level <= 2
            return
        assert np.array_equal(g["perm"], ref.perm())
        for k, v in ref.nodes().items():
            assert np.array_equal(g["nodes"][k], v), k
    finally:
        eng.close()
