"""The attractive step with a shared-memory window of Y (k_attr_window, the default 2D form) against
k_attr_update (TSNE_ATTR_PIPE=0): every row's sums run over the same lanes in the same order, so a
run equals the other's through iteration 32 (past the renumbering at 30) to rel 1e-6 (only the
centring mean's FP64 summation order differs), and a repeated run gives the same bits. Sizes
around the window's (12,288 points in 2D, 6,144 in 3D), odd ones, fewer rows than the grid has
half-warps, and a ragged P (empty rows, rows of one entry, a hub row of thousands)."""
import numpy as np
import pytest
from scipy.sparse import csr_matrix

import oracle as O
from helpers import Engine, rel

pytestmark = pytest.mark.gpu


def _P(n, ragged, seed):
    """Symmetric P of about 24 entries per row, near and far columns; ragged: 9 empty rows, rows
    of a single pair, and a hub tied to a third of the points."""
    rng = np.random.default_rng(seed)
    r = np.repeat(np.arange(n), 12)
    c = np.where(rng.random(r.size) < 0.7, (r + rng.integers(1, 40, r.size)) % n, rng.integers(0, n, r.size))
    if ragged:
        keep = ~np.isin(r, np.arange(20, 60)) & ~np.isin(c, np.arange(20, 60))
        r, c = r[keep], c[keep]
        r = np.r_[r, np.arange(30, 60, 2), np.zeros(n // 3, int)]
        c = np.r_[c, np.arange(31, 60, 2), rng.choice(np.arange(100, n), n // 3, replace=False)]
    keep = r != c
    A = csr_matrix((rng.random(keep.sum()) + 0.1, (r[keep], c[keep])), shape=(n, n))
    A = (A + A.T).tocsr()
    A.data /= A.data.sum()
    A.sort_indices()
    return A


CASES = [(2, 300, False), (2, 2_003, True), (2, 12_287, False), (2, 12_288, True), (2, 12_289, False),
         (2, 12_290, True), (2, 30_001, True), (3, 6_144, False), (3, 6_145, True), (3, 13_001, True)]


def _run(P, Y0, pipe, monkeypatch):
    if pipe is None:
        monkeypatch.delenv("TSNE_ATTR_PIPE", raising=False)
    else:
        monkeypatch.setenv("TSNE_ATTR_PIPE", pipe)
    eng = Engine(P, Y0, n_iter=200)
    try:
        eng.run(0, 32)
        return eng.embedding()
    finally:
        eng.close()


@pytest.mark.parametrize("d,n,ragged", CASES)
def test_window_equals_row_form(d, n, ragged, monkeypatch):
    P = _P(n, ragged, n)
    Y0 = O.init_embedding(n, d, 3)
    a = _run(P, Y0, "0", monkeypatch)
    b = _run(P, Y0, None, monkeypatch)
    np.testing.assert_array_equal(b, _run(P, Y0, None, monkeypatch))
    assert rel(b, a) <= 1e-6
