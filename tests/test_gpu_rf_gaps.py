"""A layer whose absorption matrix is not finite counts as the identity and has
no response: the column's other responses are those of the same column with
a layer of no thickness in its place."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NZ, K = 24, 10
NODES = {1: 3, 2: 2, 4: 1, 5: 1, 6: 1, 7: 2}
GAPS = [(5, np.nan), (7, np.inf), (10, np.inf), (10, np.nan)]   # Bx, Bz, v_z


def _columns(fz):
    """(columns with a gap at height K, the same columns with z(K+1) = z(K) there);
    heights in whole km, so that every other dz keeps its value."""
    a = np.repeat(fz.atmos.make_columns(1, NZ, seed=5), len(GAPS), 0)
    a[:, 12] = 20.0 * np.arange(NZ) - 100.0
    b = a.copy()
    b[:, 12, :K + 1] += 20.0
    for i, (row, v) in enumerate(GAPS):
        a[i, row, K] = v
    return a, b


def _context(fz, section):
    lines = fz.lines_parse(fz.atmos.line_database_text())
    return fz.Synthesis(lines, fz.regions_from_lines_section(section, lines), nz=NZ)


@pytest.mark.parametrize("section", ["1 33 -344.0 21.5\n2 32 -344.0 21.5\n", "1 32 -344.0 21.5\n"])
def test_a_gap_is_a_layer_of_no_thickness(fz, section):
    a, b = _columns(fz)
    ctx = _context(fz, section)
    ctx.rf_nodes(NODES)
    syn_a, jac_a, _, st = ctx.forward_rf(a, hydrostatic=False)
    syn_b, jac_b, _, st_b = ctx.forward_rf(b, hydrostatic=False)
    assert np.all(st != 0) and np.all(st_b == 0)
    np.testing.assert_array_equal(syn_a, syn_b)
    np.testing.assert_array_equal(jac_a, jac_b)
    assert np.all(np.abs(jac_a).max(axis=2) > 0)
    syn_a, rf_a, _, _ = ctx.forward_rf_full(a, hydrostatic=False)
    syn_b, rf_b, _, _ = ctx.forward_rf_full(b, hydrostatic=False)
    np.testing.assert_array_equal(syn_a, syn_b)
    np.testing.assert_array_equal(rf_a, rf_b)
    assert np.all(rf_a[:, :, K] == 0.0)


@pytest.mark.parametrize("section", ["1 33 -344.0 21.5\n2 32 -344.0 21.5\n", "1,2 41 -700.0 60.0\n"])
def test_a_gap_leaves_the_jacobian_finite(fz, section):
    a, _ = _columns(fz)
    a[:, 1] *= 1e-3
    ctx = _context(fz, section)
    ctx.rf_nodes({1: 3, 4: 1, 5: 1, 6: 1, 7: 2})
    for he in (False, True):
        syn, jac, _, st = ctx.forward_rf(a, hydrostatic=he)
        assert np.all(st != 0)
        assert np.all(np.isfinite(syn)) and np.all(np.isfinite(jac)) and np.all(np.abs(jac).max(axis=2) > 0)
