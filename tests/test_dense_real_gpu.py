"""Real transforms whose real side is dense rows (VDX_FFT_FLAG_DENSE_REAL): the
torch front end's even-length rows run out of place without packing copies;
odd lengths and misaligned views keep the packed path."""

import numpy as np
import pytest

from helpers import rel_l2, tol_fp32

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import vkdispatch_gb300 as vd  # noqa: E402
from vkdispatch_gb300 import _lib as L  # noqa: E402
from vkdispatch_gb300.fft import plan as P  # noqa: E402


@pytest.mark.parametrize("n", [2, 6, 30, 64, 512, 1000, 1920, 2048, 8190, 15, 81])
@pytest.mark.parametrize("rows", [1, 5, 67])
def test_rfft_irfft_rows(n, rows):
    x = np.random.default_rng(n + rows).uniform(-1, 1, (rows, n)).astype(np.float32)
    base = torch.from_numpy(np.concatenate([np.zeros(1, np.float32), x.ravel()])).cuda()
    for t in (torch.from_numpy(x).cuda(), base[1:].view(rows, n)):  # aligned, and 4 bytes off
        y = vd.torch_fft.rfft(t)
        assert rel_l2(y.cpu().numpy(), np.fft.rfft(x.astype(np.float64))) <= tol_fp32(max(2, n))
        keep = y.clone()
        z = vd.torch_fft.irfft(y, n)
        assert z.shape == t.shape and z.is_contiguous()
        assert rel_l2(z.cpu().numpy(), x) <= 2 * tol_fp32(max(2, n))
        assert torch.equal(y, keep)  # the spectrum is an input


def test_double_and_signals_of_three_dimensions():
    x = torch.randn((3, 6, 100), dtype=torch.float64, device="cuda")
    y = vd.torch_fft.rfft2(x)
    want = torch.fft.rfft2(x)
    assert float((y - want).abs().max() / want.abs().max()) < 1e-13
    z = vd.torch_fft.irfft2(y, s=(6, 100))
    assert float((z - x).abs().max()) < 1e-13


def test_refusals():
    s = 0
    x = torch.zeros(4 * 66 + 1, device="cuda")
    with pytest.raises(ValueError):
        P.get_plan((4, 65), 1, L.VDX_KIND_R2C, False, False, L.VDX_C64, L.VDX_C64, flags=L.VDX_FFT_FLAG_DENSE_REAL)
    with pytest.raises(ValueError):
        P.get_plan((4, 64), 1, L.VDX_KIND_C2C, False, False, L.VDX_C64, L.VDX_C64, flags=L.VDX_FFT_FLAG_DENSE_REAL)
    p = P.get_plan((4, 64), 1, L.VDX_KIND_R2C, False, False, L.VDX_C64, L.VDX_C64, flags=L.VDX_FFT_FLAG_DENSE_REAL)
    out = torch.zeros((4, 33), dtype=torch.complex64, device="cuda")
    with pytest.raises(ValueError):
        p.exec(x.data_ptr(), x.data_ptr(), None, s)
    with pytest.raises(ValueError):
        p.exec(x.data_ptr() + 4, out.data_ptr(), None, s)
