"""Rows of a whole-network pass's inputs (cfd_mpnn_net): strided rows are described to the library with
their stride, rows that overlap and feature counts that are not the model's are refused before any launch."""
import ctypes

import numpy as np
import pytest

import cfd_solver_withcuda_b200 as cb
from cfd_solver_withcuda_b200 import warmstart as ws

torch = pytest.importorskip("torch")


class Recorder:
    """The library with its two whole passes replaced by copies of the structures they are given, and the
    single blocks by the engines they are given."""

    def __init__(self, real):
        self.real, self.seen, self.blocks = real, [], []

    def __getattr__(self, name):
        if name in ("cfd_mpnn_mlp_forward", "cfd_mpnn_segment_sum_acc"):
            return lambda *a: self.blocks.append(a[0]._obj.engine if "mlp" in name else None) or 0
        if name not in ("cfd_mpnn_net_forward", "cfd_mpnn_net_backward"):
            return getattr(self.real, name)

        def call(ref, stream):
            a = cb.MpnnNet()
            ctypes.pointer(a)[0] = ref._obj
            self.seen.append(a)
            return 0
        return call


@pytest.fixture
def recorded(monkeypatch):
    r = Recorder(cb.lib())
    monkeypatch.setattr(cb, "lib", lambda: r)
    monkeypatch.setattr(ws, "_stream", lambda t: ctypes.c_void_p(0))
    g = ws.GraphBatch(ws.MeshGraph(ws.make_mesh(5, 3, 0.08)), 1, "cpu")
    return r.seen, ws.Net(layers=1, device="cpu"), g


def test_row_strides_reach_the_library(recorded):
    seen, net, g = recorded
    xn, xe, dp = (torch.zeros(n, w + pad)[:, :w] for n, w, pad in ((g.N, 9, 2), (g.E, 5, 3), (g.N, 4, 1)))
    net.forward(xn, xe, g)
    net.backward(dp)
    for a in seen:
        assert (a.node_in, a.edge_in, a.ld_xn, a.ld_xe) == (9, 5, 11, 8)
    assert seen[1].ld_dpred == 5
    net.forward(torch.zeros(g.N, 9), torch.zeros(g.E, 5), g)
    assert seen[2].ld_xn in (0, 9) and seen[2].ld_xe in (0, 5)


def test_feature_counts_are_the_models(recorded):
    seen, net, g = recorded
    for wn, we in ((10, 5), (9, 4), (8, 5)):
        with pytest.raises(ValueError):
            net.forward(torch.zeros(g.N, wn), torch.zeros(g.E, we), g)
    assert not seen


def test_overlapping_rows_are_refused(recorded):
    seen, net, g = recorded
    net.forward(torch.zeros(1, 9).expand(g.N, 9), torch.zeros(g.E, 5), g)
    net.forward(torch.zeros(g.N, 9), torch.zeros(1, 5).expand(g.E, 5), g)
    net.backward(torch.zeros(1, 4).expand(g.N, 4))
    lib = cb.lib().real
    status = [lib.cfd_mpnn_net_forward(ctypes.byref(seen[0]), None), lib.cfd_mpnn_net_forward(ctypes.byref(seen[1]), None),
              lib.cfd_mpnn_net_backward(ctypes.byref(seen[2]), None)]
    assert status == [cb.CFD_ERR_BAD_ARG] * 3


def test_engines_changed_afterwards_are_used(recorded):
    """A network set to the tcgen05 blocks after it was made runs block by block, and whole passes again when
    it is set back."""
    seen, net, g = recorded
    xn, xe = torch.zeros(g.N, 9), torch.zeros(g.E, 5)
    net.forward(xn, xe, g)
    assert len(seen) == 1 and not cb.lib().blocks
    net.engine = net.bwd_engine = 1
    net.forward(xn, xe, g)
    assert len(seen) == 1 and cb.lib().blocks.count(1) == 5
    net.engine = net.bwd_engine = 0
    net.forward(xn, xe, g)
    net.backward(torch.zeros(g.N, 4))
    assert len(seen) == 3


@pytest.mark.gpu
@pytest.mark.parametrize("pads", [(1, 3, 1), (7, 11, 4)])
def test_strided_rows_equal_packed_rows(pads):
    """Rows of wider buffers (odd strides, and 16-byte aligned ones) give the bits of packed rows."""
    g = ws.MeshGraph(ws.make_mesh(17, 9, 0.08))
    gb = ws.GraphBatch(g, 2, "cuda")
    rng = np.random.default_rng(pads[0])
    wide = [torch.from_numpy(rng.normal(size=(n, w + p)).astype(np.float32)).cuda()
            for n, w, p in ((2 * g.N, 9, pads[0]), (2 * g.E, 5, pads[1]), (2 * g.N, 4, pads[2]))]
    got = []
    for packed in (True, False):
        xn, xe, dp = (t[:, :w].contiguous() if packed else t[:, :w] for t, w in zip(wide, (9, 5, 4)))
        net = ws.Net(layers=2, seed=5)
        pred = net.forward(xn, xe, gb)
        net.backward(dp)
        got.append([t.cpu().numpy().view(np.int32) for t in (pred, net.grad)])
    for a, b in zip(*got):
        assert np.array_equal(a, b)
