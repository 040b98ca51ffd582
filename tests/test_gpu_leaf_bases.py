"""The leaves' bases in 2D at the limits of their three CTA sizes (32, 64 and 128 rows held): a grid
of cells whose counts are those limits and one less and more. With more leaves than one launch
runs at once, each size has a launch of its own; with fewer, one launch of the largest CTAs takes
all. The same cells through both give the same ranks, skeletons and U, bit for bit, and every
leaf's interpolation of its points' kernel rows from its skeleton's holds to the stop rule."""
import ctypes

import numpy as np
import pytest

import oracle as O
from helpers import Engine
from helpers_kernels import kernels_of
from test_gpu_lists import _ring_P

pytestmark = pytest.mark.gpu

HALF = 5e-5 * 2 ** 17     # root half-width
SIDE = 32                 # cells a side, leaves of level 5
LEAF = 128
EDGES = (1, 2, 8, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128)
TOL = 1e-2
ONE_LAUNCH = 148 * 4


def grid(blocks):
    """(2, n) points of the first `blocks` of the 256 blocks of 2 x 2 cells (the two corner blocks,
    which pin the root box, come first), and every cell's count. A block holds one cell of 128
    points, so that it is split, and three of the edge sizes."""
    w = 2 * HALF / SIDE
    order = [0, 255] + list(np.random.default_rng(1).permutation(np.arange(1, 255)))
    pts, counts = [], {}
    for b in order[:blocks]:
        rng = np.random.default_rng(1000 + b)
        sizes = rng.permutation([128, EDGES[b % 14], EDGES[(b + 5) % 14], EDGES[(b // 14 + 9) % 14]])
        for q, count in enumerate(sizes):
            cell = np.array([2 * (b % 16) + q % 2, 2 * (b // 16) + q // 2])
            x = (cell + rng.uniform(0.1, 0.9, (count, 2))) * w - HALF
            if b in (0, 255) and q == (0 if b == 0 else 3):
                x[0] = -0.999 * HALF if b == 0 else 0.999 * HALF
            pts.append(x)
            counts[tuple(cell)] = int(count)
    return np.ascontiguousarray(np.concatenate(pts).T.astype(np.float32).astype(np.float64)), counts


def engine(blocks):
    Y, _ = grid(blocks)
    return Engine(_ring_P(Y.shape[1]), Y, h2_leaf_size=LEAF, h2_tol=TOL)


def _leaves(blocks):
    """cell -> (points, rank, U, skeleton) of every leaf, and the engine's count of leaves"""
    Y, counts = grid(blocks)
    eng = engine(blocks)
    try:
        g = eng.h2()
        h, nd = g["handle"], g["nodes"]
        fn = eng.lib.tsne_h2_get_bases
        fn.argtypes = [ctypes.c_void_p] + [ctypes.c_void_p] * 5
        rows, width = ctypes.c_int(), ctypes.c_int()
        assert fn(h, ctypes.byref(rows), ctypes.byref(width), None, None, None) == 0
        off = np.zeros(g["n_node"] + 1, np.int64)
        U = np.zeros((rows.value, width.value), np.float32)
        skel = np.zeros((g["n_node"], width.value, 2), np.float32)
        assert fn(h, ctypes.byref(rows), ctypes.byref(width), off.ctypes.data, U.ctypes.data, skel.ctypes.data) == 0
        x = Y.T[g["perm"]]
        out = {}
        for t in np.flatnonzero(nd["is_leaf"]):
            a, b = nd["start"][t], nd["end"][t]
            cell = tuple(((x[a] + HALF) * SIDE / (2 * HALF)).astype(int))
            assert nd["level"][t] == 5 and counts[cell] == b - a
            r = g["ranks"][t]
            out[cell] = (x[a:b], r, U[off[t]:off[t] + b - a, :r], skel[t, :r])
        assert len(out) == len(counts) == 4 * blocks
        return out
    finally:
        eng.close()


def _kernel(x, p):
    return (1.0 + ((x[:, None] - p[None]) ** 2).sum(2)) ** -2


def test_sizes_split_and_in_one_launch():
    many, few = _leaves(256), _leaves(100)
    assert len(few) <= ONE_LAUNCH < len(many)
    assert {len(v[0]) for v in many.values()} >= set(EDGES)
    for cell, (x, r, U, skel) in few.items():
        X, R, V, S = many[cell]
        assert np.array_equal(x, X) and r == R, cell
        assert np.array_equal(U, V) and np.array_equal(skel, S), cell
    # K(points, proxies) from the skeleton's rows: the largest residual row is below the stop rule's
    # 0.1 tol of the largest row n0, and single precision adds at most 2^-24 for each of the 64 terms of
    # the dot products of r steps, times what a row of U spreads (4e-6: the entries themselves)
    h = HALF / SIDE
    p = O.proxies(2, h).T
    for cell, (x, r, U, skel) in many.items():
        c = (np.array(cell) + 0.5) * 2 * h - HALF
        A = _kernel(x - c, p)
        n0 = np.linalg.norm(A, axis=1).max()
        assert 1 <= r <= min(len(x), 64)
        U = U.astype(np.float64)
        res = np.linalg.norm(A - U @ _kernel(skel.astype(np.float64) - c, p), axis=1)
        bound = n0 * (0.1 * TOL + (r * 64 * 2.0 ** -24 + 4e-6) * (1.0 + np.abs(U).sum(1)))
        assert (res <= bound).all(), (cell, len(x), r, (res / bound).max())
        # the skeleton is r of the points, with the rows of the identity
        own = [np.flatnonzero((x.astype(np.float32) == s).all(1))[0] for s in skel]
        assert np.array_equal(U[own], np.eye(r))


def test_which_kernels_run():
    sizes = {256: {"64, 1", "128, 1", "128, 2"}, 100: {"128, 2"}}
    for blocks, want in sizes.items():
        names = [k for k in kernels_of(f"import test_gpu_leaf_bases as T\neng = T.engine({blocks})") if "k_id2d<" in k]
        leaves = [k[k.index("<") + 1:k.index(">")] for k in names if "k_id2d<true" in k or "k_id2d<(bool)1" in k]
        assert {k.split(", ", 1)[1] for k in leaves} == want, names
