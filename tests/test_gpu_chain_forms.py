"""The chemistry chain's forms: the precomputed Saha factors against the ones
computed in the chain, at the sizes where a form starts or ends."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ctx(fz, nz):
    lines = fz.lines_parse(fz.atmos.line_database_text())
    return fz.Synthesis(lines, fz.regions_from_lines_section("1 9 -86.0 21.5\n", lines), nz=nz)


@pytest.mark.parametrize("he", [False, True])
@pytest.mark.parametrize("nz,ncol", [(2, 1), (3, 5), (33, 99), (33, 149), (128, 3), (3, 2367), (3, 2368), (3, 5921)])
def test_precomputed_factors_equal_the_chains_own(fz, nz, ncol, he):
    """fz_forward_device_static computes the Saha factors inside the chain,
    fz_forward_device takes k_saha's rows: the same bits.  Temperatures reach
    from 1,500 K to 45,000 K, through every piece of the partition functions,
    and a column at a piece's own threshold (6,000 K) everywhere.  2,368
    columns is where the chain changes from 32 to 16 lanes, 5,921 the first size of two
    chunks of rows."""
    import torch
    ctx = _ctx(fz, nz)
    m = fz.atmos.make_columns(ncol, nz, seed=5)
    m[:, 0] *= np.geomspace(0.35, 4.75, ncol, dtype=np.float32)[:, None] if ncol > 1 else np.float32(1.0)
    m[-1, 0] = 6000.0
    d = torch.from_numpy(m).cuda()
    out = []
    for call in (ctx.forward_device, ctx.forward_device_static):
        syn = torch.zeros((ncol, 4, ctx.numw), dtype=torch.float64, device="cuda")
        mo, st = torch.empty_like(d), torch.zeros(ncol, dtype=torch.int32, device="cuda")
        call(d.data_ptr(), ncol, syn.data_ptr(), mo.data_ptr(), st.data_ptr(), hydrostatic=he)
        torch.cuda.synchronize()
        out.append((syn.cpu().numpy(), mo.cpu().numpy(), st.cpu().numpy()))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
