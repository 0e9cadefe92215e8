"""Contexts side by side: what one context sets up for its own sizes must not
take from another that was made before it."""
import numpy as np
import pytest

import lmcase

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("section,nz,other,counts", [
    # layers of four and of two heights at once
    ("1 112 -1193.25 21.5\n2 112 -1193.25 21.5\n", 128, 96, (65, 148, 296)),
    # one height after the other, slabs above 48 KB
    ("1 40 -430.0 21.5\n2 40 -430.0 21.5\n", 1000, 700, (300,)),
])
def test_a_second_context_leaves_the_first_as_it_was(fz, section, nz, other, counts):
    lines = fz.lines_parse(fz.atmos.line_database_text())
    reg = fz.regions_from_lines_section(section, lines)
    m = fz.atmos.make_columns(max(counts), nz, seed=5)
    a = fz.Synthesis(lines, reg, nz=nz)
    before = [a.forward(m[:n], hydrostatic=False) for n in counts]
    b = fz.Synthesis(lines, reg, nz=other)
    for n, want in zip(counts, before):
        for x, y in zip(a.forward(m[:n], hydrostatic=False), want):
            np.testing.assert_array_equal(x, y)
    b.close()


def test_a_second_context_beside_jacobian_and_inversion(fz):
    nz, npix = 64, 90
    lines = fz.lines_parse(fz.atmos.line_database_text())
    reg = fz.regions_from_lines_section("1 112 -1193.25 21.5\n2 112 -1193.25 21.5\n", lines)
    m = fz.atmos.make_columns(npix, nz, seed=6)
    opts = fz.LMOpts(maxit=3, isigma=1e-3)

    def work(c):
        c.rf_nodes(lmcase.NODES)
        obs, true, _ = c.forward(m, hydrostatic=True)
        _, jac, _, _ = c.forward_rf(m[:70], hydrostatic=True)
        return (jac,) + tuple(c.invert(obs, lmcase.initial_guess(true, seed=1), hydrostatic=True, opts=opts))

    a = fz.Synthesis(lines, reg, nz=nz)
    before = work(a)
    b = fz.Synthesis(lines, reg, nz=40)
    b.rf_nodes({1: 2})
    for x, y in zip(work(a), before):
        np.testing.assert_array_equal(x, y)
    b.close()
