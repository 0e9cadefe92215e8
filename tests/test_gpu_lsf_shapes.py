"""The LSF kernel where its tiles end: a lane's four outputs and a warp's 128
cut at every remainder, one to five warps, and steps left over after the last
four.  An asymmetric kernel (a shifted Gaussian plus noise) against the
oracle's convolution of the same unconvolved profiles, with the bounds of
test_gpu_lsf.py."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import lsf_oracle as lo  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw", [5, 31, 126, 127, 128, 129, 257, 514])
def test_every_remainder(fz, nw):
    lines = fz.lines_parse(fz.atmos.line_database_text())
    reg = fz.regions_from_lines_section("1,2 %d -700.0 %.4f\n" % (nw, 2500.0 / nw), lines)
    ctx = fz.Synthesis(lines, reg, nz=16)
    m = fz.atmos.make_columns(3, 16, seed=nw)
    syn0, _, _ = ctx.forward(m, hydrostatic=True)
    rng = np.random.default_rng(nw)
    x = (np.arange(nw) + nw // 2) % nw - nw // 2
    k = np.exp(-0.5 * ((x - 0.7) / max(1.0, 0.02 * nw)) ** 2) * rng.uniform(0.8, 1.2, nw)
    k /= k.sum()
    assert ctx.lsf_kernel(0, k)
    valid, ki = lo.install(k)
    assert valid
    syn1, _, _ = ctx.forward(m, hydrostatic=True)
    np.testing.assert_allclose(syn1, lo.convolve(syn0, [nw], [ki], [True]), rtol=2.4e-7, atol=1e-15)
