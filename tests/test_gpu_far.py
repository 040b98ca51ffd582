"""The far field with staged sources (k_far_c) and the leaves' finer far entries (k_fine) against
the exact FP64 force, where their loops change course: targets whose sources fill no round of
32, one or several, groups of more than 32 entries, coarse leaves as sources (points, more than
32), finer sources of a coarse leaf, ranks on both sides of 32 (3D: two warps per target), leaves
of more than 32 and more than 128 points. Tolerance: h2_tol, as everywhere for the H2 force."""
import numpy as np
import pytest

import oracle as O
from helpers import Engine, rel2
from test_gpu_lists import _ring_P, _wall

pytestmark = pytest.mark.gpu


def _blobs(d, n, seed):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-30, 30, (d, 12))
    sd = rng.uniform(0.2, 4.0, 12)
    lab = rng.integers(0, 12, n)
    return c[:, lab] + sd[lab] * rng.standard_normal((d, n))


CASES = {
    "blobs_2d": (2, 7_001, lambda: _blobs(2, 7_001, 1), 100, 1e-2),
    "blobs_2d_tight": (2, 2_003, lambda: _blobs(2, 2_003, 2), 30, 1e-3),
    "blobs_2d_leaf_200": (2, 9_000, lambda: _blobs(2, 9_000, 3), 200, 1e-2),
    "wall_2d": (2, 12_000, lambda: _wall(2, 12_000, 150, 4), 160, 1e-2),
    "blobs_3d": (3, 9_001, lambda: _blobs(3, 9_001, 5), 100, 3e-2),
    "blobs_3d_rank_above_32": (3, 12_000, lambda: _blobs(3, 12_000, 6), 64, 3e-3),
    "wall_3d": (3, 12_000, lambda: _wall(3, 12_000, 150, 7), 160, 3e-2),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_force_within_tolerance(name):
    d, n, make, leaf, tol = CASES[name]
    Y = np.ascontiguousarray(make().astype(np.float32).astype(np.float64))
    eng = Engine(_ring_P(n), Y, h2_leaf_size=leaf, h2_tol=tol)
    try:
        F, Z = eng.repulsive(Y)
        g = eng.h2()
        lv = g["nodes"]["level"]
        t = np.repeat(np.arange(g["n_node"]), np.diff(g["far_ptr"]))
        if name.startswith("wall"):
            assert (lv[g["far_idx"]] > lv[t]).any() and (lv[g["far_idx"]] < lv[t]).any()
        if name == "blobs_3d_rank_above_32":
            assert g["ranks"].max() > 32
        s, v = O.exact_sv(Y)
        Ze, Fe = O.z_force(Y, s, v)
        assert rel2(F, Fe) < tol
        assert abs(Z - Ze) < tol * Ze
    finally:
        eng.close()
