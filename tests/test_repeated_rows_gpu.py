"""Prunes of bases with repeated vectors, bit for bit against the oracle.

The filter skips the node's own id only while it looks for the first kept
candidate; behind a row equal to the node's it is a candidate like any other. So
the kept sets of nodes with repeated vectors depend on where the id stands. Own ids in
the rows, and distances around those of the empty places, take the same paths."""
import numpy as np
import pytest

from test_prune_gpu import run_pair
from test_screen_gpu import gaussian, graph

pytestmark = pytest.mark.gpu

CALLS = [("index", "NSG", "", 1.0), ("index", "Vamana", "", 1.2), ("index", "NSSG", "", 0.5),
         ("index", "DPG", "", 1.0), ("index", "CAGRA", "", 1.0), ("cfs", "path", "angle", 0.5),
         ("cfs", "path", "dist", 0.9), ("cfs", "2-hop", "dist", 1.0)]
CFS = [("path", "dist", 1.0), ("path", "dist", 1.2), ("path", "angle", 0.5),
       ("2-hop", "angle", 0.5)]


def repeated(n, dim, seed):
    """A twentieth of the rows a second time, and one row ten times."""
    rng = np.random.default_rng(seed)
    x = gaussian(n, dim, seed)
    at = rng.permutation(n)
    k = n // 20
    x[at[:k]] = x[at[k:2 * k]]
    x[at[2 * k:2 * k + 10]] = x[at[-1]]
    return x


def own_ids(ids, dis):
    """Every third node in its own row, at the distance of the entry it replaces."""
    ids = ids.copy()
    ids[::3, 4] = np.arange(len(ids))[::3]
    return ids, dis


@pytest.mark.parametrize("dim", [12, 96, 100, 128, 960])
@pytest.mark.parametrize("call", CALLS)
def test_repeated_rows(capi, orc, dim, call):
    kind, a, b, thre = call
    what = (kind, a, b) if b else (kind, a)
    run_pair(capi, orc, graph(orc, repeated(600, dim, dim), 32, 1), 20, what, topm=40, thre=thre)


@pytest.mark.parametrize("call", CALLS)
def test_two_values_per_dim(capi, orc, call):
    # 12 dims of 0 and 1: most rows have an equal one
    kind, a, b, thre = call
    what = (kind, a, b) if b else (kind, a)
    x = np.random.default_rng(7).integers(0, 2, (600, 12)).astype(np.float16)
    run_pair(capi, orc, graph(orc, x, 32, 2), 20, what, topm=40, thre=thre)


@pytest.mark.parametrize("dim", [100, 128])
@pytest.mark.parametrize("mode,metric,thre", CFS)
def test_own_id_inside_the_row(capi, orc, dim, mode, metric, thre):
    half, ids, dis, center = graph(orc, gaussian(500, dim, 3), 32, 4)
    ids, dis = own_ids(ids, dis)
    run_pair(capi, orc, (half, ids, dis, center), 20, ("cfs", mode, metric), topm=40, thre=thre)


@pytest.mark.parametrize("scale,topm", [(120.0, 30), (300.0, 24), (700.0, 16), (700.0, 30),
                                        (3000.0, 64)])
@pytest.mark.parametrize("mode,metric,thre", CFS)
def test_distances_around_the_empty_places(capi, orc, mode, metric, thre, scale, topm):
    # an unused place of the beam or of the list has the distance 1e7: these distances
    # lie below it, around it and beyond it, those of the own ids too
    half, ids, dis, center = graph(orc, gaussian(300, 64, 8, scale=scale), 24, 9)
    ids, dis = own_ids(ids, dis)
    ids[1::3, 0] = np.arange(len(ids))[1::3]
    run_pair(capi, orc, (half, ids, dis, center), 20, ("cfs", mode, metric), topm=topm, thre=thre)


@pytest.mark.parametrize("dim", [12, 128])
@pytest.mark.parametrize("mode,metric,thre", CFS)
def test_without_allocation(capi, orc, dim, mode, metric, thre):
    half, ids, dis, center = graph(orc, repeated(600, dim, dim), 32, 5)
    ids, dis = own_ids(ids, dis)
    st = capi.State.from_host(ids, dis, half, center)
    buf = orc.Buffers(ids, dis, half, center)
    ep = capi.pruning_cfs_noalloc(st, 20, mode, metric, topm=40, thre=thre)
    assert ep == orc.prune_cfs(buf, 20, mode, metric, topm=40, thre=thre)
    got = st.buffers()
    st.free()
    for name in ("graph", "nei_distance", "reverse_graph", "reverse_distance", "reverse_num"):
        assert np.array_equal(got[name].view(np.uint32), getattr(buf, name).view(np.uint32)), name
