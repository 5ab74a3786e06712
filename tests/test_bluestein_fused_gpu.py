"""One-launch Bluestein transforms: every storage type and both layouts, rows and
column tiles with a remainder, convolution lengths from the shortest two-pass
plan to the longest that one CTA holds, in place and out of place."""

import numpy as np
import pytest

import vkdispatch_gb300 as vd

from helpers import crandn, rel_l2, tol_fp32

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# n with a prime factor above 13; the convolution runs at the power of two from 2n - 1 up
CASES = [17, 31, 34, 257, 509, 1009, 2039, 4099, 8191]


@pytest.mark.parametrize("n", CASES)
def test_c64_rows_and_columns(n):
    rng = np.random.default_rng(n)
    for shape, axis in (((7, n), 1), ((2, n, 11), 1)):
        x = crandn(rng, shape)
        # forward and inverse convolutions of the chirp at up to 4n points
        tol = 3 * tol_fp32(4 * n)
        want = np.fft.fft(x.astype(np.complex128), axis=axis)
        b = vd.asbuffer(x)
        vd.fft.fft(b, axis=axis)
        assert rel_l2(b.read(0), want) <= tol
        vd.fft.ifft(b, axis=axis)
        assert rel_l2(b.read(0), x) <= 2 * tol
        y = vd.torch_fft.fft(torch.from_numpy(x).cuda(), dim=axis)
        assert rel_l2(y.cpu().numpy(), want) <= tol


@pytest.mark.parametrize("storage,tol", [(vd.complex32, 2.5e-3), (vd.complexbf16, 1.6e-2), (vd.complex128, 1e-12)])
@pytest.mark.parametrize("n", [17, 262, 1009])
def test_other_storage(n, storage, tol):
    rng = np.random.default_rng(n)
    for shape, axis in (((5, n), 1), ((2, n, 9), 1)):
        b = vd.Buffer(shape, storage)
        b.write(crandn(rng, shape, np.complex128) * 0.25)
        q = np.asarray(b.read(0)).astype(np.complex128)
        vd.fft.fft(b, axis=axis)
        assert rel_l2(b.read(0), np.fft.fft(q, axis=axis)) <= tol
