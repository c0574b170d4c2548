"""Calls on a device with little free memory: what a call can do without, it does
without, with the same result."""
import contextlib

import numpy as np
import pytest

from tagore_b200 import synth

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def free_memory(capi, leave):
    """Holds the device's free memory but `leave` bytes."""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    capi.lib().tagore_trim_cache()
    held = [torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")]
    try:
        yield
    finally:
        held.clear()
        torch.cuda.empty_cache()


@pytest.mark.parametrize("mode,metric", [("path", "dist"), ("2-hop", "angle")])
def test_prune_with_short_lists(capi, mode, metric):
    # the candidate lists of 150,000 nodes take 692 MB at K = 96, the rest of the
    # prune's scratch less than 200 MB
    n, K, fd = 150_000, 96, 32
    base, _ = synth.mixture("deep", n, 32, 75, 51)
    st = capi.gnn_descent_host(base, K, 4)
    ids, dis = st.download(0), st.download(3)
    rows = []
    for short in (False, True):
        st.upload(0, ids)
        st.upload(3, dis)
        st.upload(5, np.zeros(n, np.uint32))
        with free_memory(capi, 400 << 20) if short else contextlib.nullcontext():
            capi.pruning_cfs(st, fd, mode, metric, topm=64, thre=0.5)
        rows.append([st.download(i) for i in (0, 1, 3, 4, 5)])
    st.free()
    assert all(np.array_equal(a.view(np.uint32), b.view(np.uint32)) for a, b in zip(*rows))


def test_build_without_the_padded_copy(capi, orc):
    # 1,020 dims are built on a copy of 1,024; what the learned screen needs for the
    # same base leaves no room for the copy's 205 MB
    import torch
    n, dim, K = 100_000, 1020, 32
    base, _ = synth.mixture("gist", n, dim, 50, 53)
    need = 0
    for short in (False, True):
        with free_memory(capi, need + (100 << 20)) if short else contextlib.nullcontext():
            capi.lib().tagore_trim_cache()
            before = torch.cuda.mem_get_info()[0]
            mode = capi.KNN_CHOSEN if short else capi.KNN_LEARNED
            st = capi.gnn_descent_host(base, K, 3, mode=mode)
            need = before - torch.cuda.mem_get_info()[0]  # the pool keeps its peak
            used = capi.last_screen().used
        assert used == 1
        g, d, half = st.download(0), st.download(3), st.download(2).reshape(n, dim)
        st.free()
        some = np.random.default_rng(1).choice(n, 200, replace=False)
        g, d = g.reshape(n, K)[some], d.reshape(n, K)[some]
        exp = orc.dist_pairs(half, np.repeat(some, K), g.reshape(-1)).reshape(-1, K)
        assert np.array_equal(d.view(np.uint32), exp.view(np.uint32))
