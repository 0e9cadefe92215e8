"""The network's kernels at the edges of their tiles: outputs narrower and
wider than a 16-, 64- or 128-column tile, inner widths below and just above a
K block, batches of one row, of a tile less and more one row, and of more
tiles than the chip holds CTAs.

Forward and gradients are compared with the FP64 oracle on the same
bf16-rounded operands in relative L2 norm.  Each activation and each dL/dz
carries one bf16 rounding (2^-9) per layer, so three layers give at most
about 3 x 2^-9 = 6e-3 on outputs and, with the rounded dL/dz on top, 1.2e-2
on gradients; the bounds are 1e-2 and 3e-2.  The bases of inputs and outputs
need only a float's alignment and the result does not depend on it.
"""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import mlp_oracle as mo  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,n", [((8, 1), 1), ((16, 17), 129), ((72, 136, 200, 64), 127), ((64, 72, 65), 300),
                                    ((136, 264, 16), 257), ((8, 8, 8, 140), 1), ((64, 512, 24), 10000)])
def test_edges_of_tiles(fz, dims, n):
    import torch
    from firtez_dz_b200 import warmstart as ws
    net = ws.MLP(dims, seed=7)
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, dims[0])).astype(np.float32)
    t = rng.standard_normal((n, dims[-1])).astype(np.float32)
    dx, dt = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    y = torch.empty((n, dims[-1]), dtype=torch.float32, device="cuda")
    net.forward_device(n, dx.data_ptr(), y.data_ptr())
    p = net.get_params()
    yo, _ = mo.forward(p, dims, x)
    assert np.linalg.norm(y.cpu().numpy() - yo) <= 1e-2 * np.linalg.norm(yo)
    # bases one float off a 16-byte boundary
    xb = torch.empty(n * dims[0] + 1, dtype=torch.float32, device="cuda")
    xb[1:] = dx.reshape(-1)
    yb = torch.empty(n * dims[-1] + 1, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    net.forward_device(n, xb.data_ptr() + 4, yb.data_ptr() + 4)
    assert torch.equal(yb[1:], y.reshape(-1))
    net.grad_device(n, dx.data_ptr(), dt.data_ptr())
    g = net.get_params(grads=True)
    _, go = mo.loss_and_grad(p, dims, x, t)
    o = 0
    for i in range(len(dims) - 1):
        for m in (dims[i] * dims[i + 1], dims[i + 1]):
            assert np.linalg.norm(g[o:o + m] - go[o:o + m]) <= 3e-2 * np.linalg.norm(go[o:o + m]), (i, m)
            o += m
