"""Jobs that arrive while another runs, without a premise on how fast a job is: the first job is
orders of magnitude longer than the others' submission (30,000 iterations), and the others,
in 2D and 3D and of the exact method, start and end while it runs, each with the bits that it
gets alone, on streams of their own beside the long job's kernels; so does the long job."""
import pytest

import numpy as np

import oracle as O
from helpers import Engine, problem

pytestmark = pytest.mark.gpu

LONG = 30_000


@pytest.fixture(scope="module")
def jobs():
    out = []
    for n, d, seed in ((2100, 2, 1), (2500, 2, 2), (3000, 3, 3), (1500, 2, 4)):
        P = problem(n, seed=seed, k=30, perplexity=10.0, dim=20, n_clusters=5)[2]
        out.append((P, O.init_embedding(n, d, seed + 10)))
    return out


def _alone(P, Y0, n_iter):
    eng = Engine(P, Y0, n_iter=n_iter)
    eng.run_all()
    Y = eng.embedding()
    eng.close()
    return Y


def test_jobs_submitted_beside_a_long_one(jobs):
    from tsne_h2pack.serving import EmbeddingServer
    ref = [_alone(P, Y0, it) for (P, Y0), it in zip(jobs, (LONG, 60, 60, 60))]

    def submit(srv, P, Y0, n_iter):   # the parameters Engine uses
        d, n = Y0.shape
        return srv.submit(P, n_components=d, init_Y=Y0, n_iter=n_iter, verbose=0, learning_rate=max(n / 12.0, 200.0),
                          h2_tol=1e-2, h2_rebuild_freq=3, h2_rebuild_freq_early=10, h2_leaf_size=100)

    with EmbeddingServer(max_concurrent=4, hbm_budget_gb=100.0) as srv:
        a = submit(srv, *jobs[0], LONG)
        rest = [submit(srv, P, Y0, 60) for P, Y0 in jobs[1:]]
        short = [srv.wait(j) for j in rest]
        Ya, ra = srv.wait(a)
    assert ra.ok and all(r.ok for _, r in short)
    for _, r in short:
        assert r.start_s < ra.end_s and r.end_s < ra.end_s
    for (Y, _), want in zip([(Ya, ra)] + short, ref):
        np.testing.assert_array_equal(Y.T, want)
