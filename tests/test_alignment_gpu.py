"""Prunes of a caller's buffers that start on 8 bytes and not on 16, bit for bit
against the oracle: the rows are then read 8 bytes at a time at every width."""
import numpy as np
import pytest

from test_screen_gpu import gaussian, graph

pytestmark = pytest.mark.gpu

CALLS = [("index", "NSG", "", 1.0), ("index", "Vamana", "", 1.2), ("index", "NSSG", "", 0.5),
         ("index", "DPG", "", 1.0), ("cfs", "2-hop", "dist", 1.0), ("noalloc", "path", "dist", 1.1),
         ("noalloc", "2-hop", "angle", 0.5)]


class Caller:
    """A graph in the caller's buffers, the base and the centre 8 bytes past an
    aligned address."""

    def __init__(self, capi, half, ids, dis, center):
        import torch
        n, k = ids.shape
        self.keep = []

        def put(a, shift=0):
            a = torch.from_numpy(np.ascontiguousarray(a).reshape(-1).view(np.uint8))
            t = torch.zeros(a.numel() + 16, dtype=torch.uint8, device="cuda")
            t[shift:shift + a.numel()] = a.cuda()
            self.keep.append(t)
            return t.data_ptr() + shift

        st = capi.KnnState(n=n, dim=half.shape[1], k=k, device=0, norm_factor=1.0)
        st.data, st.center = put(half, 8), put(center, 8)
        assert st.data % 16 == 8 and st.center % 16 == 8
        st.graph, st.nei_distance = put(ids.astype(np.uint32)), put(dis)
        for name, words in (("reverse_graph", n * 128), ("reverse_distance", n * 128),
                            ("reverse_num", n), ("hybrid_list", n * 128), ("norms", n)):
            setattr(st, name, put(np.zeros(words, np.uint32)))
        self.state = capi.State(st)


@pytest.mark.parametrize("dim", [8, 96, 104, 128, 960])
@pytest.mark.parametrize("call", CALLS)
def test_buffers_on_8_bytes(capi, orc, dim, call):
    import torch
    kind, a, b, thre = call
    half, ids, dis, center = graph(orc, gaussian(400, dim, dim + 1), 32, 1)
    me = Caller(capi, half, ids, dis, center)
    buf = orc.Buffers(ids, dis, half, center)
    torch.cuda.synchronize()
    if kind == "index":
        ep = capi.pruning(me.state, 16, a, topm=40, thre=thre)
        want = orc.prune(buf, 16, a, topm=40, thre=thre)
    else:
        prune = capi.pruning_cfs if kind == "cfs" else capi.pruning_cfs_noalloc
        ep = prune(me.state, 16, a, b, topm=40, thre=thre)
        want = orc.prune_cfs(buf, 16, a, b, topm=40, thre=thre)
    assert ep == want
    got = me.state.buffers()
    for name in ("graph", "nei_distance", "reverse_graph", "reverse_distance", "reverse_num"):
        assert np.array_equal(got[name].view(np.uint32), getattr(buf, name).view(np.uint32)), name


@pytest.mark.parametrize("dim", [96, 128, 136])
def test_connect_on_8_bytes(capi, orc, dim):
    import torch
    half, ids, dis, center = graph(orc, gaussian(400, dim, 9), 32, 2)
    me = Caller(capi, half, ids, dis, center)
    torch.cuda.synchronize()
    ep = capi.pruning(me.state, 6, "NSG", topm=16)
    assert capi.connect(me.state, ep) > 0
    assert capi.connect(me.state, ep) == 0  # every node is reachable now
