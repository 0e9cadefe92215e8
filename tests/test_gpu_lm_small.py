"""The normal equations and the SVD of up to 16 parameters for every kind of
layout: one parameter, odd and even counts (an odd one leaves a column out of
each round of rotations), the full tile, frequencies that end inside a k-step.

Against (H + lambda diag H)^-1 g in FP64.  The bf16 split of the Jacobian
drops products of 2^-18 of their size, so H is off by less than 2^-17; with
lambda = 1 and at least eight frequencies per parameter the condition number
of the matrix is below 5, and the perturbation within 5 x 2^-17 = 4e-5 of its
norm.  Bound: 1e-4."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npar,nf", [(1, 4), (2, 20), (3, 36), (8, 100), (13, 448), (15, 896), (16, 132)])
def test_perturbation(fz, npar, nf):
    lines = fz.lines_parse(fz.atmos.line_database_text())
    reg = fz.regions_from_lines_section(fz.atmos.lines_section(2), lines)
    ctx = fz.Synthesis(lines, reg, nz=16)
    rng = np.random.default_rng(100 * npar + nf)
    n = 9
    jac = rng.standard_normal((n, npar, nf)).astype(np.float32)
    diff = rng.standard_normal((n, nf))
    got = ctx.lm_perturbation(jac, diff, np.ones(n))
    j = jac.astype(np.float64)
    h = j @ j.transpose(0, 2, 1)
    h[:, np.arange(npar), np.arange(npar)] *= 2.0
    want = np.linalg.solve(h, (j @ diff[:, :, None]))[:, :, 0]
    assert np.all(np.linalg.norm(got - want, axis=1) <= 1e-4 * np.linalg.norm(want, axis=1))
