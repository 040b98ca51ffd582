"""The attractive step's switches: an empty TSNE_ATTR_PIPE is an unset one (the window form, and no
tile form either, which needs 0), a number asks for the row form of that number."""
import pytest

from helpers_kernels import kernels_of

pytestmark = pytest.mark.gpu

RUN = """
eng = Engine(_ring_P(3000), O.init_embedding(3000, 2, 1), n_iter=6)
eng.run_all()
"""


@pytest.mark.parametrize("pipe,tiles,want", [(None, None, "k_attr_window<2"), ("", None, "k_attr_window<2"),
                                             ("", "1", "k_attr_window<2"), ("0", None, "k_attr_update<2"),
                                             ("0", "1", "k_attr_tile"), ("3", None, "k_attr_update_pf<2")])
def test_form_that_runs(pipe, tiles, want):
    names = [k for k in kernels_of(RUN, TSNE_ATTR_PIPE=pipe, TSNE_ATTR_TILES=tiles, TSNE_ATTR_WINDOW=None,
                                      TSNE_REORDER_ITERS="2", TSNE_ATTR_TILES_FROM="0")
             if "k_attr" in k and "k_attr_ranges" not in k]
    # before the renumbering the tile form is k_attr_update
    assert any(want in k for k in names), names
    assert all(want in k or (want == "k_attr_tile" and "k_attr_update<2" in k) for k in names), names
