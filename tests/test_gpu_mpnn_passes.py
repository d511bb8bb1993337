"""The warm-start network's mma.sync kernels at the shapes where they can go wrong: row counts around
the 16-row warp tiles and the 64-row weight-gradient tiles, input widths with and without the vector
forms, strided rows, one output column; and the whole-network passes against the single calls."""
import numpy as np
import pytest

import cfd_solver_withcuda_b200 as cb
from cfd_solver_withcuda_b200 import warmstart as ws

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm(np.ravel(a) - np.ravel(b)) / max(np.linalg.norm(np.ravel(b)), 1e-30))


@pytest.mark.parametrize("rows", [1, 15, 16, 17, 64, 65, 129, 2500])
@pytest.mark.parametrize("widths,pad,out", [((64, 64, 64), 0, 64), ((16,), 0, 64), ((48, 32), 2, 64), ((9,), 0, 64),
                                            ((64,), 1, 4), ((33, 64), 0, 1)])
def test_dense_block_shapes(rows, widths, pad, out):
    """Forward, data and weight gradients of one block with gathered segments (rows `pad` floats
    apart, odd pads take the element-wise forms) against the CPU restatement with BF16 operands.
    Bounds: FP32 accumulation over at most 192 products (and over the rows for the weights)."""
    import torch
    from oracle import mpnn_ref as R
    rng = np.random.default_rng(rows + 7 * len(widths) + out)
    K = sum(widths)
    p = (rng.normal(size=(64, K)) / 8, rng.normal(size=64), rng.normal(size=(out, 64)) / 8, rng.normal(size=out))
    p = tuple(v.astype(np.float32).astype(np.float64) for v in p)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    segs, cols = [], []
    for i, w in enumerate(widths):
        n = rows if i == len(widths) - 1 else rows + 3
        src = rng.normal(size=(n, w + pad)).astype(np.float32)
        idx = None if i == len(widths) - 1 else rng.integers(0, n, rows).astype(np.int32)
        segs.append((dev(src), None if idx is None else torch.from_numpy(idx).cuda(), 0, w, 0))
        cols.append(src[:, :w][idx if idx is not None else np.arange(rows)])
    x = np.concatenate(cols, axis=1).astype(np.float64)
    net = ws.Net(layers=0, node_in=K, out=out)
    net.dims["blk"] = (K, out)
    net.p["blk"] = tuple(dev(v) for v in p)
    net.g["blk"] = tuple(torch.zeros_like(t) for t in net.p["blk"])
    y = torch.empty((rows, out), device="cuda")
    z1 = torch.empty((rows, 64), device="cuda")
    net._mlp("blk", segs, rows, y, z1)
    yq, zq = R.mlp_forward(x, p, R.bf16)
    assert _rel(z1.cpu().numpy(), zq) < 1e-5
    # The kernels' hidden layer is rounded from their own z1; a rounding that flips moves y by 2^-9.
    assert _rel(y.cpu().numpy(), R.bf16(R.silu(z1.cpu().numpy().astype(np.float64))) @ R.bf16(p[2]).T + p[3]) < 1e-4
    dy = rng.normal(size=(rows, out)).astype(np.float32)
    net._bufs = {"dz": torch.empty((rows, 64), device="cuda")}
    dx = torch.empty((rows, K + pad), device="cuda")
    net._block_grads("blk", dev(dy), z1, rows, segs, dx=dx)
    dxq, gq = R.mlp_backward(x, z1.cpu().numpy().astype(np.float64), dy.astype(np.float64), p, R.bf16)
    assert _rel(dx[:, :K].cpu().numpy(), dxq) < 1e-3
    for a, b in zip(net.g["blk"], gq):
        assert _rel(a.cpu().numpy(), b) < 1e-3


@pytest.mark.parametrize("nx,ny,B,layers,out", [(5, 3, 1, 1, 4), (12, 6, 2, 2, 4), (17, 9, 3, 6, 1), (24, 10, 1, 0, 16)])
def test_whole_passes_equal_the_single_calls(nx, ny, B, layers, out):
    """Prediction, loss and every gradient of the whole-network passes: the same bits as block by
    block."""
    import torch
    g = ws.MeshGraph(ws.make_mesh(nx, ny, 0.08))
    gb = ws.GraphBatch(g, B, "cuda")
    rng = np.random.default_rng(nx)
    dev = lambda *s: torch.from_numpy(rng.normal(size=s).astype(np.float32)).cuda()
    xn, xe, target = dev(B * g.N, 9), dev(B * g.E, 5), dev(B * g.N, out)
    got = []
    for whole in (True, False):
        net = ws.Net(layers=layers, out=out, seed=3)
        assert net.whole
        net.whole = whole
        pred = net.forward(xn, xe, gb)
        loss, dpred = net.loss_grad(target)
        net.backward(dpred)
        got.append([t.cpu().numpy().view(np.int32) for t in (pred, loss, net.grad)])
    for a, b in zip(*got):
        assert np.array_equal(a, b)
