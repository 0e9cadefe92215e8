"""Masked pixels: columns of zeros, or with T = 0 (or next to it) at one height,
have no source function there -- the Planck function of T = 0 is 0, not NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [1, 20, 80])      # 6, 120 and 480 columns: one form of the synthesis each
@pytest.mark.parametrize("he", [False, True])
def test_columns_without_temperature(fz, orc, he, copies):
    lines = fz.lines_parse(fz.atmos.line_database_text())
    reg = fz.regions_from_lines_section("1 33 -344.0 21.5\n2 32 -344.0 21.5\n", lines)
    g, _ = orc.gain(lines, reg)
    nz = 24
    m = fz.atmos.make_columns(6, nz, seed=5)
    m[0] = 0.0
    m[1, 0] = 0.0
    m[2, 0, 10] = 0.0
    m[3, 0, 10] = 1e-6
    m[4, 0] = 1e-6
    ref, _, sref = orc.forward(lines, reg, g, m, hydrostatic=he)
    ctx = fz.Synthesis(lines, reg, nz=nz, gain=g)
    ctx.rf_nodes({1: 2, 5: 1})
    big = np.concatenate([m] * copies)
    for syn, st in (ctx.forward(big, hydrostatic=he)[::2], ctx.forward_rf(big, hydrostatic=he)[::3]):
        assert np.all(np.isfinite(syn))
        syn, st = syn.reshape(copies, 6, 4, -1), st.reshape(copies, 6)
        assert np.all(syn[:, [0, 1, 4]] == 0.0)
        assert np.all((st == 0) == (sref == 0))
        # a gap's opacity is not a number: here the height counts as a boundary
        # without source, which the oracle has no rule for
        assert np.all(np.abs(syn[:, [2, 3], 0]).max(axis=2) > 0)
        assert np.max(np.abs(syn[:, 5, 0] / ref[5, 0] - 1)) < 1e-5
        assert np.max(np.abs(syn[:, 5, 1:] - ref[5, 1:])) < 1e-6
