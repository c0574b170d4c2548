"""The chosen kNN build at the widths its tensor-core tiles end on: below one
16-dim step (4, 8, 12), which the learned screen keeps, between steps (24, 104), a row of 4 mod 8 halves built on the
zero-padded copy (100, 132, 1020), and the widths around the one-row-per-lane
scoring of the initial rows (256, 264). Every stored distance is the oracle's
exact one, and the graph agrees with the plain join's recall."""
import numpy as np
import pytest

from tagore_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [4, 8, 12, 20, 24, 100, 104, 124, 132, 256, 264, 1020])
def test_chosen_build_at_edge_widths(capi, orc, dim):
    n, K = 2500, 24
    base, _ = synth.mixture("gist" if dim > 200 else "deep", n, dim, 6, 31)
    recall = {}
    for mode in (capi.KNN_CHOSEN, capi.KNN_PLAIN):
        st = capi.gnn_descent_host(base, K, 8, mode=mode)
        assert capi.last_screen().used == (mode == capi.KNN_CHOSEN and dim < 16)
        g, d = st.download(0).reshape(n, K), st.download(3).reshape(n, K)
        half = st.download(2).reshape(n, dim)
        st.free()
        assert (g < n).all() and (np.diff(d, axis=1) >= 0).all()
        assert not (g == np.arange(n)[:, None]).any()
        exp = orc.dist_pairs(half, np.repeat(np.arange(n), K), g.reshape(-1)).reshape(n, K)
        assert np.array_equal(d.view(np.uint32), exp.view(np.uint32))
        truth, tdis = orc.exact_knn(half, K)
        # share of the ten nearest found; equal distances count as found
        recall[mode] = float((d[:, :10] <= tdis[:, 9:10]).mean())
    # 25,000 slots at recall above 0.9: two builds differ by less than 0.02
    assert recall[capi.KNN_CHOSEN] > recall[capi.KNN_PLAIN] - 0.02 and recall[0] > 0.9


@pytest.mark.parametrize("dim", [12, 20, 24, 28, 36])
def test_narrow_builds_are_as_exact_as_the_screen(capi, orc, dim):
    # the relative error of all distances, against the exact lists; two builds of one
    # mode differ by less than 2 %
    n, K = 12000, 32
    base, _ = synth.mixture("sift", n, dim, 6, 37)
    err, exact = {}, None
    for mode in (capi.KNN_CHOSEN, capi.KNN_LEARNED):
        st = capi.gnn_descent_host(base, K, 12, mode=mode)
        d, half = st.download(3).reshape(n, K), st.download(2).reshape(n, dim)
        st.free()
        if exact is None:
            exact = orc.exact_knn(half, K)[1].astype(np.float64)
        err[mode] = np.linalg.norm(d - exact) / np.linalg.norm(exact)
    assert err[capi.KNN_CHOSEN] <= 1.04 * err[capi.KNN_LEARNED], err
