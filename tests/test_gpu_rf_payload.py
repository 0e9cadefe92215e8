"""The response functions' file payload, (pixel, height, wavelength, Stokes,
parameter) from (pixel, parameter, height, Stokes, wavelength): a permutation,
so every comparison is exact.  Payload bases on and 8 bytes off a 16-byte
boundary, wavelengths that do not fill a warp."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off", [0, 2])
@pytest.mark.parametrize("npix,nz,nw", [(1, 1, 1), (3, 5, 31), (2, 7, 224), (5, 3, 500)])
def test_permutation(fz, npix, nz, nw, off):
    import torch
    rf = torch.randn(npix, 6, nz, 4, nw, device="cuda")
    out = torch.full((off + rf.numel() + 4,), -7.0, device="cuda")
    torch.cuda.synchronize()
    p = ctypes.c_void_p
    assert fz.lib().fz_rf_to_v3_device(npix, nz, nw, p(rf.data_ptr()), p(out.data_ptr() + 4 * off), None) == 0
    torch.cuda.synchronize()
    body = out[off:off + rf.numel()].reshape(npix, nz, nw, 4, 6)
    assert torch.equal(body, rf.permute(0, 2, 4, 3, 1))
    assert torch.all(out[:off] == -7.0) and torch.all(out[off + rf.numel():] == -7.0)
