"""The basis kernels at the edges of their row and lane splits: every leaf of a grid of cells holds
exactly `count` points (edges of the CTA sizes, of the lanes per row and of the held rows), and
tolerances small enough that internal nodes pass 64, 128 and (3D) the held rows. Against the
exact FP64 force, within h2_tol (2e-4 at least, for single precision), and the same bits from
a second build."""
import numpy as np
import pytest

import oracle as O
from helpers import Engine, rel2
from test_gpu_lists import _ring_P

pytestmark = pytest.mark.gpu


def _cells(d, side, count, seed, depth=2):
    """side x side cells (3D: x depth), `count` points in the middle of each; two points near the
    outer corners pin the root box, whose cells at that level these are."""
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(*[np.arange(side)] * 2 + [np.arange(depth)] * (d - 2), indexing="ij"), -1).reshape(-1, d)
    half = 5e-5 * 2 ** 17                      # root half-width 6.5536
    w = 2 * half / side
    pts = (g[:, None, :] + rng.uniform(0.2, 0.8, (len(g), count, d))) * w - half
    pts[0, 0, :2], pts[-1, -1, :2] = -half * 0.999, half * 0.999
    return np.ascontiguousarray(pts.reshape(-1, d).T)


CASES = [(3, 16, c, 3e-2) for c in (4, 8, 9, 16, 17)] + \
        [(3, 8, c, 3e-2) for c in (31, 32, 33, 63, 64, 65, 127, 128, 129)] + \
        [(2, 16, c, 1e-2) for c in (8, 31, 32, 33)] + [(2, 8, c, 1e-2) for c in (63, 64, 65, 127, 128, 129)] + \
        [(2, 16, 40, 1e-4), (2, 16, 60, 1e-5), (3, 8, 30, 1e-3), (3, 8, 60, 3e-4), (3, 8, 12, 1.1e-3)]


@pytest.mark.parametrize("d,side,count,tol", CASES)
def test_force_at_the_edges(d, side, count, tol):
    # the last case: a full cube of cells, internal nodes of more candidates than are held
    Y = _cells(d, side, count, 100 * d + count, 8 if tol == 1.1e-3 else 2).astype(np.float32).astype(np.float64)
    n = Y.shape[1]
    assert n >= 2000
    eng = Engine(_ring_P(n), Y, h2_leaf_size=count, h2_tol=tol)
    try:
        g = eng.h2()
        nd = g["nodes"]
        leaf = nd["is_leaf"] != 0
        assert (nd["end"] - nd["start"])[leaf].max() == count
        assert g["ranks"].max() <= 64
        F, Z = eng.repulsive(Y)
        s, v = O.exact_sv(Y)
        Ze, Fe = O.z_force(Y, s, v)
        # the stop rule is relative to a node's own rows; single precision bounds it from below
        bound = max(tol, 2e-4)
        assert rel2(F, Fe) < bound
        assert abs(Z - Ze) < bound * Ze
        # two passes from the same embedding give the same bits
        assert eng.rebuild() == 0
        F2, Z2 = eng.repulsive(Y)
        assert np.array_equal(F, F2) and Z == Z2
    finally:
        eng.close()
