"""The search where its visited tables and its tile part from the ordinary case,
id for id against the oracle: lists far longer than the average the shared table is
sized by, so that most ids spill to the global one; a pool that leaves no shared
memory for the tile, or none for the table; widths around one load of a row and one
chunk of the tile."""
import numpy as np
import pytest

from test_search_gpu import both, ragged_graph

pytestmark = pytest.mark.gpu


def base_of(n, dim, seed):
    return np.random.default_rng(seed).integers(0, 200, (n, dim)).astype(np.float32)


@pytest.mark.parametrize("hub", [900, 1100, 5000])
@pytest.mark.parametrize("seed", [0, 11])
def test_spilled_ids(capi, orc, hub, seed):
    # a few hubs on otherwise short lists: 1,024 places for up to 5,000 ids
    rng = np.random.default_rng(hub)
    n = 20000
    lists = [rng.integers(0, n, 1) for _ in range(n)]
    for h in (0, 17, 4242):
        lists[h] = rng.choice(n, hub, replace=False)
    offs = np.zeros(n + 1, np.uint64)
    offs[1:] = np.cumsum([len(x) for x in lists])
    adj = np.concatenate(lists).astype(np.uint32)
    got, want = both(capi, orc, base_of(n, 20, 1), offs, adj, 17, base_of(40, 20, 2), 16, 10, seed)
    assert np.array_equal(got, want)


# of the 232,448 bytes a block may have, 14,000 entries leave 8,256: the tile (4,608)
# and no table; 14,250 entries leave 4,256: neither
@pytest.mark.parametrize("L", [14000, 14250])
def test_pools_that_fill_shared_memory(capi, orc, L):
    n = 3000
    offs, adj = ragged_graph(n, 12, np.random.default_rng(3))
    got, want = both(capi, orc, base_of(n, 16, 3), offs, adj, 5, base_of(3, 16, 4), L, 20, 7)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("dim", [1, 3, 4, 31, 32, 33, 36, 64, 65, 132])
def test_widths(capi, orc, dim):
    n = 2000
    offs, adj = ragged_graph(n, 40, np.random.default_rng(dim))
    got, want = both(capi, orc, base_of(n, dim, 5), offs, adj, 5, base_of(33, dim, 6), 50, 20, 9)
    assert np.array_equal(got, want)


# ids of 25 bits take a shared table of 2,048 buckets so that a remainder fits 14 bits;
# ids of 26 bits leave the shared table out, and every visited id is in global memory
@pytest.mark.parametrize("n", [(1 << 24) + 1, (1 << 25) + 1])
@pytest.mark.parametrize("seed", [0, 5])
def test_bases_at_the_shared_tables_limit(capi, orc, n, seed):
    rng = np.random.default_rng(n)
    base = rng.integers(0, 50, (n, 4), dtype=np.uint8).astype(np.float32)
    offs = np.arange(0, 3 * n + 1, 3, dtype=np.uint64)
    adj = rng.integers(0, n, 3 * n, dtype=np.uint32)
    adj[::5] = n - 1 - adj[::5] % 1000  # the highest ids, met again and again
    q = rng.integers(0, 50, (24, 4)).astype(np.float32)
    for L in (50, 1500):
        got, want = both(capi, orc, base, offs, adj, n - 1, q, L, 20, seed)
        assert np.array_equal(got, want)
