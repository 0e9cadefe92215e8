"""The global temperature term of hydrostatic equilibrium skips layers of
O(1,1) <= 1e-5: H goes through them unchanged, whatever their response."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("section", ["1 33 -344.0 21.5\n2 32 -344.0 21.5\n", "1,2 41 -700.0 60.0\n"])
def test_a_skipped_layer_keeps_its_response_to_itself(fz, section):
    """T = 700 K at one height: its chemistry derivatives leave the range of
    FP32 and its layer is opaque.  The heights above keep finite responses."""
    nz, k = 24, 10
    lines = fz.lines_parse(fz.atmos.line_database_text())
    ctx = fz.Synthesis(lines, fz.regions_from_lines_section(section, lines), nz=nz)
    m = fz.atmos.make_columns(1, nz, seed=5)
    m[0, 0, k] = 700.0
    syn, rf, _, _ = ctx.forward_rf_full(m, hydrostatic=True)
    assert np.all(np.isfinite(syn))
    assert not np.all(np.isfinite(rf[0, 0, k]))          # the case is met
    assert np.all(np.isfinite(rf[0, :, k + 1:]))
    assert np.all(np.abs(rf[0, :, k + 1:]).max(axis=2) > 0)
