"""Responses of the deep heights that the spectrum hardly sees: the products of
the operators above them keep their relative accuracy, far below the largest
response (same bound as the node Jacobian's, at every height for itself)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RF_TOL = 2e-4


@pytest.mark.parametrize("he", [True, False])
@pytest.mark.parametrize("seed", [5, 6])
def test_deep_heights_to_their_own_scale(fz, orc, he, seed):
    nz = 24
    lines = fz.lines_parse(fz.atmos.line_database_text())
    reg = fz.regions_from_lines_section("1 33 -344.0 21.5\n2 32 -344.0 21.5\n", lines)
    g, _ = orc.gain(lines, reg)
    m = fz.atmos.make_columns(1, nz, seed=seed)
    if not he:
        _, m, _ = orc.forward(lines, reg, g, m, hydrostatic=True)
    ctx = fz.Synthesis(lines, reg, nz=nz, gain=g)
    _, rf, _, st = ctx.forward_rf_full(m, hydrostatic=he)
    _, ref, _, _ = orc.forward_rf(lines, reg, g, m, {1: nz, 2: nz}, hydrostatic=he)   # a node at every height
    assert np.all(st == 0)
    ref = ref[0].reshape(2, nz, -1)
    scale = np.abs(ref).max(axis=2)
    # up to the largest response: the uppermost heights' local responses have
    # roundings of their own (small differences of large derivatives)
    seen = (scale > 1e-25) & (np.arange(nz)[None, :] <= scale.argmax(axis=1)[:, None])
    assert scale[seen].min() < 1e-12
    err = np.abs(rf[0, :2] - ref).max(axis=2)
    assert np.max(err[seen] / scale[seen]) <= RF_TOL
