"""cfd_mpnn_mse with the gradient written over the prediction or the target: the loss and the gradient of
separate buffers, bit for bit."""
import numpy as np
import pytest

import cfd_solver_withcuda_b200 as cb
from cfd_solver_withcuda_b200 import warmstart as ws

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1023, 1025, 200000])
@pytest.mark.parametrize("over", ["pred", "target"])
def test_gradient_over_an_input(n, over):
    import torch
    rng = np.random.default_rng(n)
    dev = lambda: torch.from_numpy(rng.normal(size=n).astype(np.float32)).cuda()
    pred, target = dev(), dev()
    loss = torch.zeros(2, device="cuda")
    grad = torch.empty(n, device="cuda")

    def call(p, t, g, i):
        cb._check(cb.lib().cfd_mpnn_mse(ws._ptr(p), ws._ptr(t), n, ws._ptr(g), ws._ptr(loss[i:]), ws._stream(p)))
    call(pred, target, grad, 0)
    for _ in range(20):
        p, t = pred.clone(), target.clone()
        g = p if over == "pred" else t
        call(p, t, g, 1)
        assert loss[0].item() == loss[1].item()
        assert torch.equal(g, grad)
