"""The tensor-core joins' screen and tiles: every number of kept partners, lists
that share a tile two by two (small samples) or fill it, and rows that overflow
FP16, whose NaN screens must not cost their neighbours a candidate. Every stored
distance is the oracle's exact one, and the recall is the plain join's."""
import numpy as np
import pytest

from tagore_b200 import synth

pytestmark = pytest.mark.gpu


def recall_and_check(capi, orc, base, K, finite, mode, iters=10, rescale=1, **kw):
    n, dim = base.shape
    st = capi.gnn_descent_host(base, K, iters, mode=mode, rescale=rescale, **kw)
    g, d = st.download(0).reshape(n, K)[finite], st.download(3).reshape(n, K)[finite]
    half = st.download(2).reshape(n, dim)
    st.free()
    rows = np.flatnonzero(finite)
    assert (g < n).all() and not (g == rows[:, None]).any()
    exp = orc.dist_pairs(half, np.repeat(rows, K), g.reshape(-1)).reshape(-1, K)
    assert np.array_equal(d.view(np.uint32), exp.view(np.uint32))
    truth, tdis = orc.exact_knn(half[finite], K)
    return float((d[:, :10] <= tdis[:, 9:10]).mean())


# sample s gives lists of at most 4 s rows: 8 and 16 always share a tile, 17 crosses
# the half's 64 rows, 32 fills the tile
@pytest.mark.parametrize("dim", [64, 128, 200])
@pytest.mark.parametrize("per_row,sample", [(1, 32), (2, 8), (2, 16), (3, 17), (4, 32)])
def test_partners_and_shared_tiles(capi, orc, dim, per_row, sample):
    base, _ = synth.mixture("gist" if dim > 128 else "deep", 2003, dim, 5, 41)
    every = np.ones(len(base), bool)
    r = [recall_and_check(capi, orc, base, 24, every, m, iters=14, sample=sample, per_row=per_row)
         for m in (capi.KNN_CHOSEN, capi.KNN_PLAIN)]
    # 20,000 slots: two builds of one mode differ by less than 0.02
    assert r[0] > r[1] - 0.02, r


@pytest.mark.parametrize("dim", [32, 256])
def test_rows_that_overflow_fp16(capi, orc, dim):
    rng = np.random.default_rng(43)
    base = rng.standard_normal((1500, dim)).astype(np.float32)
    finite = np.ones(1500, bool)
    finite[::100] = False
    base[~finite, ::2] = 1e6
    r = [recall_and_check(capi, orc, base, 24, finite, m, rescale=0)
         for m in (capi.KNN_CHOSEN, capi.KNN_PLAIN)]
    assert r[0] > r[1] - 0.02, r
