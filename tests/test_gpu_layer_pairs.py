"""One layer's operator where the two wavelengths of a thread take different
branches: thin beside thick, degenerate, transparent or not finite, each in
either place of the pair."""
import numpy as np
import pytest

import test_gpu_layer as layer

pytestmark = pytest.mark.gpu

NAN = np.nan
# eta_I, eta_Q, U, V, rho_Q, U, V
THIN = {
    "transparent": [0, 0, 0, 0, 0, 0, 0],
    "unpolarised": [0.3, 0, 0, 0, 0, 0, 0],
    "weak": [0.01, 1e-3, 2e-3, -1e-3, 5e-4, 1e-3, 2e-3],
    "at right angles": [1.0, 0.4, 0, 0, 0, 0.4, 0],             # d = e = 0, far from vanishing
    "nearly at right angles": [1.0, 0.4, 1e-4, 0, 0, 0.4, 3e-5],
    "small": [0.2, 0.08, 0.05, 0.02, 0.03, 0.06, 0.08],
    "below the limit": [0.8, 0.3, 0.2, 0.1, 0.1, 0.2, 0.3],
}
THICK = {
    "above the limit": [1.5, 0.5, 0.3, 0.4, 0.2, -0.1, 0.3],
    "polarised": [3.0, 2.0, 0.5, -1.0, 0.3, 0.1, -0.2],
    "rotating": [0.5, 0.1, 0, 0, 0, 0, 20.0],
}


@pytest.mark.parametrize("thick", list(THICK))
@pytest.mark.parametrize("thin", list(THIN))
def test_halves_on_either_side_of_the_series_limit(fz, thin, thick):
    a, b = THIN[thin], THICK[thick]
    t = np.array([a, b, b, a, a, a, b, b, a], dtype=np.float64)   # the last one alone
    got, want = layer._solve(fz, t, np.array([1.0, 2.0, 0.5]))
    scale = np.abs(t).max(axis=1)
    # FP32: a few ulp of the intensity, and the roots' own rounding times their
    # size in the angle
    assert np.all(np.abs(got - want).max(axis=1) <= 2e-6 * (1.0 + scale))


@pytest.mark.parametrize("bad", [[NAN] * 7, [1.0, 0, 0, 0, NAN, 0, 0], [np.inf, 0, 0, 0, 0, 0, 0],
                                 [1.0, np.inf, 0, 0, 0, 0, 0]])
def test_a_half_that_is_not_finite_is_the_identity(fz, bad):
    for a in list(THIN.values()) + list(THICK.values()):
        t = np.array([a, bad, bad, a, bad], dtype=np.float64)
        _, want = layer._solve(fz, np.where(np.isfinite(t), t, 0.0), np.array([1.0, 2.0, 0.5]))
        gap, _ = _raw(fz, t)
        assert np.max(np.abs(gap[[0, 3]] - want[[0, 3]])) <= 2e-6 * (1.0 + np.abs(a).max())
        np.testing.assert_array_equal(gap[[1, 2, 4]], np.tile([1.0, 0.0, 0.0, 0.0], (3, 1)))


def _raw(fz, t):
    eta = np.tile((t / 1e5).astype(np.float32).T[None, None], (1, 3, 1, 1))
    src = np.tile(np.array([1.0, 2.0, 0.5], dtype=np.float32)[None, :, None], (1, 1, len(t)))
    return fz.rte_solve(eta, src, np.array([0.0, 1.0, 2.0]))[0], eta


def test_voigt_pairs_of_different_damping(fz):
    """Each argument with its own damping, an odd number of them."""
    from scipy.special import wofz
    rng = np.random.default_rng(2)
    a = np.exp(rng.uniform(np.log(1e-4), np.log(3.0), 1001)).astype(np.float32)
    v = rng.uniform(-25.0, 25.0, 1001).astype(np.float32)
    h, f = fz.voigt(a, v)
    w = wofz(v.astype(np.float64) + 1j * a.astype(np.float64))
    assert np.max(np.abs(h - w.real)) < 6e-6 and np.max(np.abs(f - w.imag)) < 6e-6
