"""The prune's collect against the oracle, bit for bit, where its paths part:
distances that tie (the reference's network decides), kNN rows out of order or
with a NaN, lists shorter than the ring, widths of each row reader, and beams
from one entry to the largest."""
import numpy as np
import pytest

from test_prune_gpu import run_pair
from test_screen_gpu import gaussian, graph

pytestmark = pytest.mark.gpu

BOTH = [("path", "dist", 1.0), ("2-hop", "angle", 0.5)]


@pytest.mark.parametrize("mode,metric,thre", BOTH)
@pytest.mark.parametrize("dim", [12, 32])
@pytest.mark.parametrize("top", [2, 60])
def test_ties(capi, orc, mode, metric, thre, dim, top):
    # small whole numbers: most distances tie (top 2; at 12 dims most rows have an
    # equal one), or a few do (top 60)
    x = np.random.default_rng(top).integers(0, top, (600, dim)).astype(np.float16)
    run_pair(capi, orc, graph(orc, x, 32, 3), 20, ("cfs", mode, metric), topm=40, thre=thre)


@pytest.mark.parametrize("mode,metric,thre", BOTH)
def test_rows_out_of_order(capi, orc, mode, metric, thre):
    half, ids, dis, center = graph(orc, gaussian(500, 32, 5), 32, 6)
    ids, dis = ids.copy(), dis.copy()
    ids[::2], dis[::2] = ids[::2, ::-1], dis[::2, ::-1]
    run_pair(capi, orc, (half, ids, dis, center), 20, ("cfs", mode, metric), topm=40, thre=thre)


@pytest.mark.parametrize("dim", [8, 92, 96, 104, 128, 136, 960])
@pytest.mark.parametrize("K,topm", [(24, 1), (33, 32), (65, 100), (128, 256)])
def test_widths_and_beams(capi, orc, dim, K, topm):
    run_pair(capi, orc, graph(orc, gaussian(400, dim, dim), K, 7), min(K, 40),
             ("cfs", "path", "dist"), topm=topm, thre=1.1)


@pytest.mark.parametrize("K,topm", [(24, 16), (24, 40), (96, 64)])
def test_nan_rows(capi, orc, K, topm):
    # every ninth row is NaN: its distances stand anywhere in a beam that the network
    # has sorted. Such a prune is a function of its input, of valid ids
    x = gaussian(700, 32, 21)
    x[::9, 5] = np.nan
    ids, dis = orc.knn_input(gaussian(700, 32, 21), K, noise=0.3, seed=22)
    dis = orc.dist_pairs(x, np.repeat(np.arange(700), K), ids.reshape(-1)).reshape(700, K)
    center = gaussian(1, 32, 23)[0]
    rows = []
    for _ in range(2):
        st = capi.State.from_host(ids, dis, x, center)
        ep = capi.pruning_cfs(st, 20, "path", "dist", topm=topm, thre=1.1)
        g = st.download(0).reshape(700, K)
        st.free()
        assert ep < 700 and (g[:, 0] < K).all()
        assert all((r[1:1 + r[0]] < 700).all() for r in g)
        rows.append(g)
    assert np.array_equal(rows[0], rows[1])
