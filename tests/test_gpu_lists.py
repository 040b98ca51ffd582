"""The interaction lists of the one-launch count pass (a warp per target) against the oracle's
traversal: bit for bit, at the sizes where the pass changes course: targets with more entries
than their slots (the traversing write pass takes over), inadmissible sets above the set's first
capacity, leaves far coarser than their neighbours (deep expansion), one level of internal nodes,
and segments that are longer than a warp."""
import numpy as np
import pytest

import oracle as O
from helpers import Engine

pytestmark = pytest.mark.gpu


def _ring_P(n):
    from scipy.sparse import csr_matrix
    i = np.arange(n)
    return csr_matrix((np.full(2 * n, 0.5 / n), (np.r_[i, i], np.r_[(i + 1) % n, (i - 1) % n])), shape=(n, n))


def _wall(d, n, sparse, seed):
    """A dense flat wall of points beside a region with a few points: the sparse region's leaves
    are far coarser than the wall's, and touch many of them."""
    rng = np.random.default_rng(seed)
    y = rng.uniform(-8.0, 8.0, (d, n))
    y[0, sparse:] = 1e-3 * rng.uniform(0.0, 1.0, n - sparse)
    y[0, :sparse] = rng.uniform(-8.0, 0.0, sparse)
    y[:, 0], y[:, 1] = -8.0, 8.0      # the wall lies on the root box's middle
    return y


CASES = {
    # about 200 wall leaves beside one sparse leaf: more near entries than slots
    "wall_2d": (2, 24_000, lambda: _wall(2, 24_000, 30, 1), 60),
    "wall_3d": (3, 24_000, lambda: _wall(3, 24_000, 20, 2), 30),
    # the same walls with leaves large enough for the slots
    "wall_2d_fits": (2, 9_000, lambda: _wall(2, 9_000, 40, 3), 160),
    # uniform: every internal set full
    "cube_3d": (3, 30_000, lambda: np.random.default_rng(4).uniform(-9, 9, (3, 30_000)), 40),
    "square_2d": (2, 2_000, lambda: np.random.default_rng(5).uniform(-9, 9, (2, 2_000)), 25),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_lists_equal_oracle(name):
    d, n, make, leaf = CASES[name]
    Y = np.ascontiguousarray(make().astype(np.float32).astype(np.float64))
    eng = Engine(_ring_P(n), Y, h2_leaf_size=leaf, h2_tol=3e-2)
    try:
        g = eng.h2()
        ref = O.H2(Y, leaf_size=leaf, tol=3e-2)
        assert g["n_node"] == ref.n_node
        for k, want in zip(("far_ptr", "far_idx", "near_ptr", "near_idx"), ref.lists()):
            assert np.array_equal(g[k], want), k
        if name in ("wall_2d", "wall_3d"):
            assert np.diff(g["near_ptr"]).max() > 128
    finally:
        eng.close()
