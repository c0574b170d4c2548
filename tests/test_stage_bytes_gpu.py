"""The stage timers' byte and item counts: each stage counts what its own kernels
read and write."""
import ctypes as C

import numpy as np
import pytest

from tagore_b200 import synth

pytestmark = pytest.mark.gpu


def stages(capi, fn):
    L = capi.lib()
    capi.check(L.tagore_reset_counters())
    capi.check(L.tagore_set_profiling(1))
    try:
        out = fn()
    finally:
        capi.check(L.tagore_set_profiling(0))
    arr, cnt = (capi.StageStat * 32)(), C.c_int(0)
    capi.check(L.tagore_stage_stats(arr, 32, C.byref(cnt)))
    return out, {arr[i].name.decode(): arr[i] for i in range(cnt.value)}


@pytest.mark.parametrize("dim", [128, 200])
def test_joins_and_two_hop(capi, dim):
    n, K, fd, iters = 3000, 32, 20, 8
    base, _ = synth.mixture("gist" if dim > 128 else "sift", n, dim, 5, 71)
    st, s = stages(capi, lambda: capi.gnn_descent_host(base, K, iters))
    # a tile holds one node's list or two; the first iterations' lists fill theirs
    assert n < s["knn_join_tiles"].items < n * iters
    assert s["knn_join_tiles"].launches == 0  # a count, not a stage of its own
    _, s = stages(capi, lambda: capi.pruning_cfs(st, fd, "2-hop", "angle", thre=0.5))
    st.free()
    collect, filt = s["prune_select_2hop"], s["prune_filter"]
    rows = n * (480 * 2 * dim + 8 * K)  # 480 rows scored per node, the kNN row
    assert rows < collect.bytes <= rows + n * (480 + K) * 8
    # between one tile of candidates per node and all of them
    out = n * (8 * fd + 4)
    assert 32 * n * (2 * dim + 8) <= filt.bytes - out <= n * (480 + K) * (2 * dim + 8)
    assert collect.items == filt.items == n
