"""No device allocation while a stream is being captured: the tail of an
inversion whose loop the host drives (line spread function, more than 16
nodes) captures an iteration for every pool size, and a caller may capture a
small batch after a large one."""
import numpy as np
import pytest

import lmcase

pytestmark = pytest.mark.gpu


def _case(fz, nz, npix, lsf):
    lines = fz.lines_parse(fz.atmos.line_database_text())
    ctx = fz.Synthesis(lines, fz.regions_from_lines_section("1 48 -505.25 21.5\n2 48 -505.25 21.5\n", lines), nz=nz)
    if lsf:
        for r in range(2):
            ctx.lsf_gaussian(r, 35.0, 0.0)
    obs, true, st = ctx.forward(fz.atmos.make_columns(npix, nz, seed=23), hydrostatic=True)
    assert np.all(st == 0)
    obs = obs + np.random.default_rng(3).normal(0.0, 1e-3, obs.shape)
    init = lmcase.initial_guess(true, seed=1)
    init[::2] = true[::2]      # half of the pixels end early: the pool is compacted on the way
    return ctx, obs, init


@pytest.mark.parametrize("lsf,nodes", [(True, lmcase.NODES), (False, {1: 5, 4: 4, 5: 4, 6: 3, 7: 1})])
def test_the_pool_of_a_host_driven_inversion_shrinks(fz, lsf, nodes):
    """100 pixels iterated until all are done, the pool of 100 slots ending
    below 65; the same pixels in a pool of 48 take the same steps."""
    nz, npix = 32, 100
    got = []
    for slots in (100, 48):
        ctx, obs, init = _case(fz, nz, npix, lsf)
        ctx.rf_nodes(nodes)
        opts = fz.LMOpts(maxsteps=3, maxit=12, isigma=1e-3, slots=slots)
        got.append(ctx.invert(obs, init, hydrostatic=True, opts=opts))
        ctx.close()
    assert np.all(got[0][3] == 0)
    assert got[0][2].min() < got[0][2].max()
    for x, y in zip(*got):
        np.testing.assert_array_equal(x, y)


def test_a_captured_small_batch_after_a_large_one(fz):
    import torch
    nz = 32
    lines = fz.lines_parse(fz.atmos.line_database_text())
    ctx = fz.Synthesis(lines, fz.regions_from_lines_section("1 48 -505.25 21.5\n2 48 -505.25 21.5\n", lines), nz=nz)
    m = torch.from_numpy(fz.atmos.make_columns(100, nz, seed=2)).cuda()
    syn = torch.empty((100, 4, ctx.numw), dtype=torch.float64, device="cuda")
    out, st = torch.empty_like(m), torch.zeros(100, dtype=torch.int32, device="cuda")

    def run(n):
        s = torch.cuda.current_stream().cuda_stream
        ctx.forward_device(m.data_ptr(), n, syn.data_ptr(), out.data_ptr(), st.data_ptr(), stream=s, hydrostatic=True)

    run(100)
    torch.cuda.synchronize()
    want = syn[:7].clone(), out[:7].clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        run(7)
    syn.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(syn[:7], want[0]) and torch.equal(out[:7], want[1])
    run(7)      # outside a capture the layers are there again
    torch.cuda.synchronize()
    assert torch.equal(syn[:7], want[0]) and torch.equal(out[:7], want[1])


def test_a_captured_batch_keeps_its_layers(fz):
    """A graph captured while the context holds layers for 7 columns, replayed after
    batches that needed more of them."""
    import torch
    nz, n = 32, 60
    lines = fz.lines_parse(fz.atmos.line_database_text())
    ctx = fz.Synthesis(lines, fz.regions_from_lines_section("1 48 -505.25 21.5\n2 48 -505.25 21.5\n", lines), nz=nz)
    m = torch.from_numpy(fz.atmos.make_columns(100, nz, seed=2)).cuda()
    syn = torch.empty((100, 4, ctx.numw), dtype=torch.float64, device="cuda")
    out = torch.empty_like(m)

    def run(k):
        s = torch.cuda.current_stream().cuda_stream
        ctx.forward_device(m.data_ptr(), k, syn.data_ptr(), out.data_ptr(), stream=s, hydrostatic=True)

    run(100)
    run(7)
    torch.cuda.synchronize()
    want = syn[:7].clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        run(7)
    for k in (9, 30, n):
        run(k)
    torch.cuda.synchronize()
    big = syn[:n].clone()
    syn.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(syn[:7], want) and torch.equal(big[:7], want)
