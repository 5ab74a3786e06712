"""Bluestein transforms under the environment's plan choices: the convolution
length M is 512 or 1024, where plans of 8, 16 and 32 points per thread exist,
but not for every storage type and layout."""

import numpy as np
import pytest

import vkdispatch_gb300 as vd
from vkdispatch_gb300.fft import plan as P

from helpers import crandn, rel_l2, tol_fp32

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["8", "16", "32", "runtime"])
def choice(request, monkeypatch):
    if request.param == "runtime":
        monkeypatch.setenv("VDX_NO_FIXED", "1")
    else:
        monkeypatch.setenv("VDX_POINTS_PER_THREAD", request.param)
    P.cache_clear()
    yield request.param
    P.cache_clear()


def _check(n, storage, tol):
    rng = np.random.default_rng(n)
    for shape, axis in (((5, n), 1), ((2, n, 9), 1)):
        b = vd.Buffer(shape, storage)
        b.write(crandn(rng, shape, np.complex128) * 0.25)
        q = np.asarray(b.read(0)).astype(np.complex128)
        vd.fft.fft(b, axis=axis)
        assert rel_l2(b.read(0), np.fft.fft(q, axis=axis)) <= tol


@pytest.mark.parametrize("storage,tol", [(vd.complex32, 2.5e-3), (vd.complexbf16, 1.6e-2)])
@pytest.mark.parametrize("n", [131, 262, 509])
def test_half_storage(choice, n, storage, tol):
    _check(n, storage, tol)


@pytest.mark.parametrize("n", [131, 211, 262, 509])
def test_c64(choice, n):
    # forward and inverse convolutions of the chirp at up to 4n points
    _check(n, vd.complex64, 3 * tol_fp32(4 * n))


@pytest.mark.parametrize("storage,tol", [(vd.complex32, 2.5e-3), (vd.complexbf16, 1.6e-2), (vd.complex128, 1e-12)])
@pytest.mark.parametrize("n", [211, 2053, 4093])
def test_default_plans(n, storage, tol):
    """M = 512, whose rows default to the two-pass plan on complex64, and 8192,
    the longest convolution of fp64."""
    P.cache_clear()
    _check(n, storage, tol)
