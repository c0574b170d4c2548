"""The screened filter, DPG and CAGRA selects against the oracle, bit for bit,
where their tiles and their error bounds are tried: rows that are not a multiple
of 16 bytes, widths around a 64-dim group, more kept neighbours than one screen
holds, lists of every small length, and bases whose norms are far larger than
their distances or whose distances tie, so that most tests are ambiguous and
fall to the exact distance."""
import numpy as np
import pytest

from test_prune_gpu import run_pair

pytestmark = pytest.mark.gpu


def graph(orc, half, K, seed, noise=0.1):
    ids, dis = orc.knn_input(half, K, noise=noise, seed=seed)
    return half, ids, dis, half.astype(np.float32).mean(0).astype(np.float16)


def gaussian(n, dim, seed, scale=1.0, offset=0.0):
    x = np.random.default_rng(seed).standard_normal((n, dim)) * scale + offset
    return x.astype(np.float16)


EVERY = [("NSG", 1.0), ("Vamana", 1.2), ("NSSG", 0.5), ("DPG", 1.0)]


@pytest.mark.parametrize("dim", [4, 8, 20, 60, 64, 68, 100, 132, 1028])
@pytest.mark.parametrize("itype,thre", EVERY)
def test_widths(capi, orc, dim, itype, thre):
    c = graph(orc, gaussian(500, dim, dim), 32, dim + 1)
    run_pair(capi, orc, c, 20, ("index", itype), topm=32, thre=thre)


@pytest.mark.parametrize("dim", [32, 100])
@pytest.mark.parametrize("itype,thre", EVERY)
def test_far_from_the_origin(capi, orc, dim, itype, thre):
    # coordinates near 100 with steps of 1/16: norms 1e4 per dim, distances of
    # order 1, below the screen's bound for almost every test
    c = graph(orc, gaussian(400, dim, 5, scale=0.3, offset=100.0), 32, 6)
    run_pair(capi, orc, c, 20, ("index", itype), topm=32, thre=thre)


@pytest.mark.parametrize("mode,metric,thre", [("path", "dist", 4.0), ("path", "dist", 0.0),
                                              ("path", "dist", -1.0), ("path", "angle", 0.9),
                                              ("2-hop", "angle", -0.5), ("2-hop", "dist", 1.0)])
def test_thresholds_and_long_kept_lists(capi, orc, mode, metric, thre):
    # alpha 4 drops almost nothing until the degree is full: more than 64 kept
    # neighbours, five screens per tile; FINAL_DEGREE up to K = 128
    c = graph(orc, gaussian(700, 48, 7), 128, 8)
    run_pair(capi, orc, c, 100, ("cfs", mode, metric), topm=100, thre=thre)
    run_pair(capi, orc, c, 128, ("cfs", mode, metric), topm=16, thre=thre)


@pytest.mark.parametrize("fd", [1, 2, 3])
@pytest.mark.parametrize("itype,thre", EVERY[:3])
def test_smallest_degrees(capi, orc, fd, itype, thre):
    c = graph(orc, gaussian(60, 16, 9), 24, 10)
    run_pair(capi, orc, c, fd, ("index", itype), topm=8, thre=thre)


@pytest.mark.parametrize("K,fd", [(3, 1), (31, 16), (32, 16), (33, 16), (47, 24), (64, 32),
                                  (97, 48), (128, 64)])
@pytest.mark.parametrize("itype", ["CAGRA", "DPG"])
def test_rank_prunes_at_tile_edges(capi, orc, itype, K, fd):
    c = graph(orc, gaussian(300, 20, 11), K, 12)
    run_pair(capi, orc, c, fd, ("index", itype))


@pytest.mark.parametrize("itype", ["CAGRA", "DPG", "NSG", "NSSG"])
def test_repeated_ids_in_rows(capi, orc, itype):
    # a row may hold an id several times (an empty slot repeats the first id)
    half, ids, dis, center = graph(orc, gaussian(300, 20, 13), 40, 14)
    ids = ids.copy()
    ids[::3, 20:] = ids[::3, :1]
    ids[1::3, 30:36] = ids[1::3, 3:9]
    run_pair(capi, orc, (half, ids, dis, center), 20, ("index", itype), topm=32, thre=0.5)


def test_noalloc_rows_equal_the_allocating_prune(capi, orc):
    # the static-scratch prune runs collect and filter in one kernel
    for dim in (64, 100):
        half, ids, dis, center = graph(orc, gaussian(900, dim, 15), 40, 16)
        for mode, metric, thre in (("path", "dist", 1.2), ("2-hop", "angle", 0.5)):
            rows = []
            for call in (capi.pruning_cfs, capi.pruning_cfs_noalloc):
                st = capi.State.from_host(ids, dis, half, center)
                call(st, 24, mode, metric, topm=48, thre=thre)
                rows.append(st.buffers())
                st.free()
            for name in rows[0]:
                assert np.array_equal(rows[0][name].view(np.uint8), rows[1][name].view(np.uint8)), name
