"""Layers of any optical thickness: e^-tI is 0 long before its FP32 argument
reduction would lose the remainder, and the layer then gives its own source."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SRC = np.array([1.0, 2.0, 0.5])


def _solve(fz, t):
    """Two layers of optical depths t (n, 7) above a boundary."""
    eta = np.tile((t / 1e5).astype(np.float32).T[None, None], (1, 3, 1, 1))
    src = np.tile(SRC.astype(np.float32)[None, :, None], (1, 1, len(t)))
    return fz.rte_solve(eta, src, np.array([0.0, 1.0, 2.0]))[0]


@pytest.mark.parametrize("lo,hi", [(1e2, 1e10), (1e10, 1e20), (1e20, 1e30)])
def test_thick_unpolarised_layers_give_their_source(fz, lo, hi):
    """Against e^-100 the layer below has no weight: the top layer's source to
    the rounding of its three operations."""
    t = np.zeros((101, 7))
    t[:, 0] = np.geomspace(lo, hi, 101)
    got = _solve(fz, t)
    assert np.max(np.abs(got[:, 0] - SRC[2])) <= 3e-7
    assert np.all(got[:, 1:] == 0.0)


def test_thick_polarised_layers_give_their_source(fz):
    """|eta| < eta_I: every eigenvalue of the matrix is as thick; up to the size
    where the square of |eta|^2 leaves FP32."""
    rng = np.random.default_rng(1)
    t = rng.standard_normal((300, 7))
    t[:, 1:] *= 0.5 / np.linalg.norm(t[:, 1:4], axis=1)[:, None]
    t[:, 0] = 1.0
    t *= np.geomspace(1e3, 1e8, 300)[:, None]
    got = _solve(fz, t)
    assert np.max(np.abs(got[:, 0] - SRC[2])) <= 3e-7
    assert np.max(np.abs(got[:, 1:])) <= 3e-7


def test_the_exponential_goes_over_into_its_limit(fz):
    """Around the smallest normal value of e^-tI and around the limit of the
    argument, and a matrix of NaN (the identity)."""
    t = np.zeros((6, 7))
    t[:, 0] = [87.0, 87.6, 88.5, 103.9, 104.1, np.nan]
    got = _solve(fz, t)
    assert np.max(np.abs(got[:5, 0] - SRC[2])) <= 3e-7
    assert got[5, 0] == SRC[0]
