"""Host arrays on their way to the device: the network's parameters, and
fz_lm_perturbation's batches on both sides of the size from which several
threads copy them in pieces, with a last piece that is not whole.  A pixel's
perturbation does not depend on its batch, and a round trip of parameters
changes no bit, so all comparisons are exact."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(8, 1), (512, 1016, 5), (1024, 512, 13), (896, 1024, 1024, 512, 13)])
def test_parameters_round_trip(fz, dims):
    from firtez_dz_b200 import warmstart as ws
    net = ws.MLP(dims, seed=1)
    for seed in (1, 2):
        p = np.random.default_rng(seed).standard_normal(net.nparams).astype(np.float32)
        net.set_params(p)
        assert np.array_equal(net.get_params(), p)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_perturbation_of_a_batch_is_its_pixels(fz, dtype):
    lines = fz.lines_parse(fz.atmos.line_database_text())
    reg = fz.regions_from_lines_section(fz.atmos.lines_section(2), lines)
    npar, nf = 13, 448
    rng = np.random.default_rng(3)
    n = 301
    jac = (rng.standard_normal((n, npar, nf)) * 0.02).astype(dtype)
    diff = rng.standard_normal((n, nf)) * 0.01
    lam = 10.0 ** rng.uniform(-3, 1, n)
    pen, hss = rng.uniform(0, 0.1, (n, npar)), rng.uniform(0, 0.1, (n, npar, npar))
    hss = hss + hss.transpose(0, 2, 1)
    # batches that grow, shrink and grow again over the kept workspace
    ctx = fz.Synthesis(lines, reg, nz=16)
    small = np.concatenate([ctx.lm_perturbation(jac[i:i + 7], diff[i:i + 7], lam[i:i + 7], reg_pen=pen[i:i + 7],
                                                reg_hss=hss[i:i + 7]) for i in range(0, n, 7)])
    plain = np.concatenate([ctx.lm_perturbation(jac[i:i + 7], diff[i:i + 7], lam[i:i + 7]) for i in range(0, n, 7)])
    assert np.array_equal(ctx.lm_perturbation(jac, diff, lam, reg_pen=pen, reg_hss=hss), small)
    for _ in range(4):   # from the third or fourth through the ring
        assert np.array_equal(ctx.lm_perturbation(jac, diff, lam), plain)
    assert np.array_equal(ctx.lm_perturbation(jac[:5], diff[:5], lam[:5]), plain[:5])
    # two threads on one context
    out = [None, None]

    def call(k):
        out[k] = ctx.lm_perturbation(jac[k:], diff[k:], lam[k:])

    th = [threading.Thread(target=call, args=(k,)) for k in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert np.array_equal(out[0], plain) and np.array_equal(out[1], plain[1:])
