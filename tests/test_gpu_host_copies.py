"""Host arrays reach the device before the kernels that read them start: the
entry points that copy pageable memory and launch on the context's own stream
give the same result call after call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_large_perturbation_repeats(fz):
    """GET_PERTURBATION of 300 nodes (normal equations on the tensor cores,
    CG and SVD): 12 calls each, the same bits (one call in six read data still
    on its way)."""
    lines = fz.lines_parse(fz.atmos.line_database_text())
    reg = fz.regions_from_lines_section(fz.atmos.lines_section(2), lines)
    rng = np.random.default_rng(3)
    npix, npar, nf = 3, 300, 896
    jac = rng.standard_normal((npix, npar, nf)) * np.logspace(0, -1.5, npar)[None, :, None]
    diff = rng.standard_normal((npix, nf))
    lam = np.array([0.01, 0.3, 10.0])
    for dtype in (1, 2):
        first = None
        for _ in range(12):
            ctx = fz.Synthesis(lines, reg, nz=32)
            d = ctx.lm_perturbation(jac, diff, lam, dtype=dtype)
            ctx.close()
            first = d if first is None else first
            np.testing.assert_array_equal(d, first)


def test_network_parameters_repeat(fz):
    """set_params rounds the weights it has just copied to BF16: the same
    forward pass from every copy."""
    import torch
    from firtez_dz_b200 import warmstart as ws
    dims = (896, 1024, 1024, 512, 13)
    rng = np.random.default_rng(4)
    x = torch.from_numpy(rng.standard_normal((64, dims[0])).astype(np.float32)).cuda()
    net = ws.MLP(dims, seed=1)
    p = (rng.standard_normal(net.nparams) * 0.03).astype(np.float32)
    first = None
    for _ in range(12):
        net.set_params(np.zeros_like(p))
        net.set_params(p.copy())
        y = torch.empty((64, dims[-1]), dtype=torch.float32, device="cuda")
        net.forward_device(64, x.data_ptr(), y.data_ptr())
        torch.cuda.synchronize()
        first = y if first is None else first
        assert torch.equal(y, first)
