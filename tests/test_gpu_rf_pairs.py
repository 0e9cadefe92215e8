"""The response functions of regions of one line each (two wavelengths per
thread) against the general kernel, which regions with blended lines run: a
second line too weak to matter (log gf -90) sends the same region there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NODES = {1: 5, 2: 1, 4: 2, 5: 2, 6: 2, 7: 2}
TOL = 2e-4    # of a column's largest entry, the oracle tests' node-Jacobian tolerance


def _pair(fz, n1, n2, nz):
    lines = fz.lines_parse(fz.atmos.line_database_text())
    weak = lines.copy()
    weak["loggf"][2] = -90.0
    rows = "%s %d -%.2f 21.5\n%s %d -%.2f 21.5\n"
    one = fz.regions_from_lines_section(rows % ("1", n1, 10.75 * (n1 - 1), "2", n2, 10.75 * (n2 - 1)), lines)
    two = fz.regions_from_lines_section(rows % ("1,3", n1, 10.75 * (n1 - 1), "2,3", n2, 10.75 * (n2 - 1)), weak)
    a = fz.Synthesis(lines, one, nz=nz)
    return a, fz.Synthesis(weak, two, nz=nz, gain=a.gain)


def _close(got, want):
    scale = np.abs(want).max(axis=-1, keepdims=True)
    top = np.abs(want).max(axis=(-2, -1), keepdims=True)
    assert np.max(np.abs(got - want) / np.maximum(scale, 1e-4 * top)) < TOL


@pytest.mark.parametrize("he", [True, False])
@pytest.mark.parametrize("n1,n2", [(1, 1), (2, 3), (31, 33), (64, 64), (112, 112), (65, 190), (255, 257)])
def test_node_jacobian(fz, he, n1, n2):
    a, b = _pair(fz, n1, n2, 24)
    m = fz.atmos.make_columns(3, 24, seed=n1)
    for nodes in (NODES, {7: 1}):
        a.rf_nodes(nodes)
        b.rf_nodes(nodes)
        s1, j1, _, st1 = a.forward_rf(m, hydrostatic=he)
        s2, j2, _, st2 = b.forward_rf(m, hydrostatic=he)
        assert np.all(st1 == 0) and np.all(st2 == 0)
        assert np.max(np.abs(s1 - s2)) < 1e-5
        _close(j1, j2)


@pytest.mark.parametrize("he", [True, False])
@pytest.mark.parametrize("n1,n2", [(1, 2), (33, 32), (112, 112)])
def test_every_height(fz, he, n1, n2):
    a, b = _pair(fz, n1, n2, 16)
    m = fz.atmos.make_columns(2, 16, seed=n2)
    _, r1, _, _ = a.forward_rf_full(m, hydrostatic=he)
    _, r2, _, _ = b.forward_rf_full(m, hydrostatic=he)
    assert np.max(np.abs(r1 - r2) / np.abs(r2).max(axis=(2, 3), keepdims=True)) < 2e-3   # the oracle test's


def test_output_at_any_word(fz):
    """Pairs are stored as 8-byte words only where the output allows it."""
    import torch
    a, _ = _pair(fz, 112, 112, 16)
    np_ = a.rf_nodes(NODES)
    m = torch.from_numpy(fz.atmos.make_columns(2, 16, seed=1)).cuda()
    syn = torch.empty((2, 4, a.numw), dtype=torch.float64, device="cuda")
    mo = torch.empty_like(m)
    n = 2 * np_ * 4 * a.numw
    buf = torch.zeros(n + 1, dtype=torch.float32, device="cuda")
    out = []
    for off in (0, 1):
        buf.zero_()
        a.forward_rf_device(m.data_ptr(), 2, syn.data_ptr(), buf.data_ptr() + 4 * off, mo.data_ptr(), hydrostatic=True)
        torch.cuda.synchronize()
        out.append(buf[off:off + n].clone())
    assert torch.equal(*out)


@pytest.mark.parametrize("scale", [0.55, 0.8, 1.0, 1.3, 1.9])
def test_chemistry_derivatives_across_the_partition_functions(fz, orc, scale):
    """The T response with temperatures from 2,400 to 18,000 K: every interval
    of the partition functions' value and derivative pieces, one column at a
    threshold of theirs (6,000 K) at every height."""
    lines = fz.lines_parse(fz.atmos.line_database_text())
    reg = fz.regions_from_lines_section("1 21 -215.0 21.5\n", lines)
    g, _ = orc.gain(lines, reg)
    nz = 33
    m = fz.atmos.make_columns(4, nz, seed=6)
    m[:, 0] *= np.float32(scale)
    m[3, 0] = 6000.0
    ctx = fz.Synthesis(lines, reg, nz=nz, gain=g)
    nodes = {1: 3, 2: 2}
    ctx.rf_nodes(nodes)
    _, jac, _, st = ctx.forward_rf(m, hydrostatic=False)
    _, ojac, _, _ = orc.forward_rf(lines, reg, g, m, nodes, hydrostatic=False)
    assert np.all(st == 0)
    scale_ = np.abs(ojac).max(axis=2, keepdims=True)
    assert np.max(np.abs(jac - ojac) / np.maximum(scale_, 1e-3 * scale_.max(axis=1, keepdims=True))) < TOL
