"""One layer's evolution operator across its branches: the series of thin
layers, the roots above, the limits between, and degenerate matrices."""
import numpy as np
import pytest
from scipy.linalg import expm

pytestmark = pytest.mark.gpu


def _matrix(t):
    i, q, u, v, a, b, c = t   # eta_I, Q, U, V, rho_Q, U, V
    return np.array([[i, q, u, v], [q, i, -c, b], [u, c, i, -a], [v, -b, a, i]])


def _solve(fz, t, src):
    """fz_rte_solve and its FP64 value for optical depths t (nw, 7) in each of
    two layers above a boundary, sources src (3,)."""
    nw = t.shape[0]
    zz = np.array([0.0, 1.0, 2.0])            # dz = 1e5 cm everywhere
    eta = np.tile((t / 1e5).astype(np.float32).T[None, None], (1, 3, 1, 1))
    s = np.tile(src.astype(np.float32)[None, :, None], (1, 1, nw))
    got = fz.rte_solve(eta, s, zz)[0]
    t32 = (eta[0, 0].astype(np.float64) * 1e5).astype(np.float32).astype(np.float64).T
    want = np.zeros((nw, 4))
    e0 = np.array([1.0, 0.0, 0.0, 0.0])
    for w in range(nw):
        m = expm(-_matrix(t32[w]))
        st = src[0] * e0
        for k in (1, 2):
            st = src[k] * e0 + m @ (st - src[k] * e0)
        want[w] = st
    return got, want


@pytest.mark.parametrize("scale", [1e-6, 1e-3, 0.05, 0.45, 0.5, 0.55, 1.0, 3.0, 10.0])
def test_operator_across_the_series_limit(fz, scale):
    """Random matrices with |eta|, |rho| around the given optical depth: the
    series end at |d|, |e| = 1/4.  FP32: a few ulp of the intensity, and the
    roots' own rounding times their size in the angle."""
    rng = np.random.default_rng(int(1e6 * scale))
    n = 128
    t = rng.standard_normal((n, 7)) * scale
    t[:, 0] = 1.1 * np.linalg.norm(t[:, 1:4], axis=1) + 0.1 * scale
    got, want = _solve(fz, t, np.array([1.0, 2.0, 0.5]))
    assert np.max(np.abs(got - want)) <= 2e-6 * (1.0 + scale)


def test_degenerate_layers(fz):
    """No polarisation, absorption only, dispersion only, |eta| = |rho| at right
    angles, a strong Faraday rotation (the argument reduction's own branch
    above 6e4 rad is not compared: FP32 does not hold its phase)."""
    t = np.array([[0.3, 0, 0, 0, 0, 0, 0], [0.3, 0.2, 0, 0.1, 0, 0, 0], [0.3, 0, 0, 0, 0.2, 0, 0.1],
                  [1.0, 0.5, 0, 0, 0, 0.5, 0], [0.5, 0.1, 0, 0, 0, 0, 40.0], [60.0, 20.0, 0, 0, 0, 0, 0.0],
                  [0.0, 0, 0, 0, 0, 0, 0]])
    got, want = _solve(fz, t, np.array([1.0, 2.0, 0.5]))
    assert np.max(np.abs(got - want)) <= 1e-5
    assert np.all(got[0, 1:] == 0.0) and np.all(got[6] == [1.0, 0.0, 0.0, 0.0])
    big = np.array([[1.0, 0.1, 0, 0, 0, 0, 1.0e5]])
    g, _ = _solve(fz, big, np.array([1.0, 2.0, 0.5]))
    assert np.all(np.isfinite(g)) and np.max(np.abs(g)) < 3.0


def test_equal_lande_factors_share_a_component(fz, orc):
    """A line between levels of equal Lande factors (15648.5, g = 3) has one
    shift per type: its components are summed before the Voigt function."""
    lines = fz.lines_parse(fz.atmos.line_database_text())
    reg = fz.regions_from_lines_section("3 31 -322.5 21.5\n", lines)
    g, _ = orc.gain(lines, reg)
    m = fz.atmos.make_columns(5, 33, seed=2)
    syn, _, st = fz.Synthesis(lines, reg, nz=33, gain=g).forward(m, hydrostatic=True)
    ref, _, _ = orc.forward(lines, reg, g, m, hydrostatic=True)
    assert np.all(st == 0)
    assert np.max(np.abs(syn[:, 0] / ref[:, 0] - 1)) < 1e-5
    assert np.max(np.abs(syn[:, 1:] - ref[:, 1:])) < 1e-6


@pytest.mark.parametrize("n1,n2", [(1, 1), (2, 3), (63, 2), (64, 65), (130, 1), (511, 513)])
def test_wavelength_pairs_of_any_region_sizes(fz, orc, n1, n2):
    """Two wavelengths a thread: odd regions end in a single one, regions start
    inside or at the start of a warp, up to the largest NUMW."""
    lines = fz.lines_parse(fz.atmos.line_database_text())
    reg = fz.regions_from_lines_section("1 %d -300.0 2.5\n2 %d -200.0 3.5\n" % (n1, n2), lines)
    g, _ = orc.gain(lines, reg)
    m = fz.atmos.make_columns(2, 12, seed=3)
    syn, _, st = fz.Synthesis(lines, reg, nz=12, gain=g).forward(m, hydrostatic=True)
    ref, _, _ = orc.forward(lines, reg, g, m, hydrostatic=True)
    assert np.all(st == 0)
    assert np.max(np.abs(syn[:, 0] / ref[:, 0] - 1)) < 1e-5
    assert np.max(np.abs(syn[:, 1:] - ref[:, 1:])) < 1e-6


@pytest.mark.parametrize("section", ["1 112 -1193.25 21.5\n2 112 -1193.25 21.5\n", "1,2 75 -700.0 33.0\n",
                                     "1 96 -1021.25 21.5\n2 96 -1021.25 21.5\n3 96 -1021.25 21.5\n4 96 -1021.25 21.5\n",
                                     "2 5 -43.0 21.5\n"])
@pytest.mark.parametrize("nz", [2, 5, 8, 9, 33])
def test_every_batch_size_takes_the_same_steps(fz, section, nz):
    """Layers of several heights at once (two launches up to 64 columns, groups of
    a CTA up to two columns per SM) against one height after the other: the same
    bits, at the sizes where a form begins or ends."""
    lines = fz.lines_parse(fz.atmos.line_database_text())
    ctx = fz.Synthesis(lines, fz.regions_from_lines_section(section, lines), nz=nz)
    m = fz.atmos.make_columns(640, nz, seed=nz)
    syn, mo, st = ctx.forward(m, hydrostatic=False)
    assert np.all(st == 0)
    for n in (1, 3, 64, 65, 148, 149, 296, 297):
        s, o, t = ctx.forward(m[:n], hydrostatic=False)
        np.testing.assert_array_equal(s, syn[:n])
        np.testing.assert_array_equal(o, mo[:n])
        np.testing.assert_array_equal(t, st[:n])
