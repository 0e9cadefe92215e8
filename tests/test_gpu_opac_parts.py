"""Slab rows made in parts (few cells) and by one thread each (many): the
first columns of a large batch and the same columns by themselves give the
same continuum, line and derivative values, hence the same profiles and
Jacobian up to the order of FP32 operations of the synthesis forms that
batches of their sizes take (1e-6 of a profile's and 2e-5 of a Jacobian
column's norm)."""
import numpy as np
import pytest

import lmcase

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nreg,n", [(1, 1), (2, 3), (4, 70)])
def test_small_batch_equals_large(fz, nreg, n):
    nz, big = 16, 5000   # 80,000 cells: more than two CTAs of 256 on each of 148 SMs
    lines = fz.lines_parse(fz.atmos.line_database_text())
    ctx = fz.Synthesis(lines, fz.regions_from_lines_section(fz.atmos.lines_section(nreg, 24), lines), nz=nz)
    m = fz.atmos.make_columns(big, nz, seed=nreg)
    large, mo_l, st_l = ctx.forward(m, hydrostatic=True)
    small, mo_s, st_s = ctx.forward(m[:n], hydrostatic=True)
    assert np.all(st_l == 0) and np.all(st_s == 0)
    assert np.linalg.norm(small - large[:n]) <= 1e-6 * np.linalg.norm(large[:n])
    np.testing.assert_allclose(mo_s, mo_l[:n], rtol=2e-6)
    ctx.rf_nodes(lmcase.NODES)
    _, jl, _, _ = ctx.forward_rf(m, hydrostatic=True)
    _, js, _, _ = ctx.forward_rf(m[:n], hydrostatic=True)
    d = np.linalg.norm((js - jl[:n]).reshape(-1, js.shape[-1]), axis=1)
    assert np.all(d <= 2e-5 * np.linalg.norm(jl[:n].reshape(-1, js.shape[-1]), axis=1) + 1e-12)
