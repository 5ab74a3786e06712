"""Choices of the planner for runtime lengths, and the kernels on them: in lists
of even radices the pass whose scatter conflicts least runs first; rows of 33 to
48 threads share a CTA where they are short; long columns of many transforms keep
to 512 threads; tiles of 3, 5, 6 or 7 columns give way to 2 or 4."""

import numpy as np
import pytest

import vkdispatch_gb300 as vd
from vkdispatch_gb300 import _lib as L
from vkdispatch_gb300.fft import plan as P

from helpers import crandn, rel_l2, tol_fp32

pytestmark = pytest.mark.gpu


def _plan(shape, axis=1):
    return P.get_plan(shape, axis, L.VDX_KIND_C2C, False, False, L.VDX_C64, L.VDX_C64).describe()


@pytest.mark.parametrize("n,first", [(2304, 12), (2688, 14), (2240, 14), (144, 12), (80, 10)])
def test_first_radix(n, first):
    radices = [int(r) for r in _plan((64, n))["radices"].split("x")]
    assert int(np.prod(radices)) == n
    if all(r % 2 == 0 for r in radices):
        assert radices[0] == first


@pytest.mark.parametrize("n", [144, 192, 1000, 2240, 2304, 2688])
def test_transforms(n):
    rng = np.random.default_rng(n)
    for shape, axis in (((5, n), 1), ((2, n, 11), 1)):
        x, k = crandn(rng, shape), crandn(rng, shape)
        b = vd.asbuffer(x)
        vd.fft.fft(b, axis=axis)
        want = np.fft.fft(x.astype(np.complex128), axis=axis)
        assert rel_l2(b.read(0), want) <= tol_fp32(n)
        vd.fft.ifft(b, axis=axis)
        assert rel_l2(b.read(0), x) <= 2 * tol_fp32(n)
        c = vd.asbuffer(x)
        vd.fft.convolve(c, vd.asbuffer(k), axis=axis)
        assert rel_l2(c.read(0), np.fft.ifft(want * np.conj(k), axis=axis)) <= 2 * tol_fp32(n)
    r = rng.standard_normal((5, 2 * n)).astype(np.float32)
    rb = vd.asrfftbuffer(r)
    vd.fft.rfft(rb)
    assert rel_l2(rb.read_fourier(0), np.fft.rfft(r.astype(np.float64), axis=-1)) <= tol_fp32(2 * n)
    vd.fft.irfft(rb)
    assert rel_l2(rb.read_real(0), r) <= 2 * tol_fp32(2 * n)


@pytest.mark.parametrize("n,rows_per_cta", [(297, 3), (363, 3), (405, 2), (504, 1), (546, 1)])
def test_rows_per_cta(n, rows_per_cta):
    d = _plan((200, n))
    if 32 < d["threads_per_transform"] <= 48:
        assert d["transforms_per_cta"] == rows_per_cta
    rng = np.random.default_rng(n)
    for rows in (1, 2, 7):
        x = crandn(rng, (rows, n))
        b = vd.asbuffer(x)
        vd.fft.fft(b)
        assert rel_l2(b.read(0), np.fft.fft(x.astype(np.complex128))) <= tol_fp32(n)
        vd.fft.ifft(b)
        assert rel_l2(b.read(0), x) <= 2 * tol_fp32(n)
    r = rng.standard_normal((7, 2 * n)).astype(np.float32)
    rb = vd.asrfftbuffer(r)
    vd.fft.rfft(rb)
    assert rel_l2(rb.read_fourier(0), np.fft.rfft(r.astype(np.float64), axis=-1)) <= tol_fp32(2 * n)


@pytest.mark.parametrize("n,wide", [(5200, 520), (5600, 560), (6400, 640), (6000, 600)])
def test_columns_per_tile(n, wide):
    rng = np.random.default_rng(n)
    for inner, threads in ((5, wide), (400, 512)):
        d = _plan((1, n, inner))
        assert d["threads_per_transform"] <= threads
        x = crandn(rng, (1, n, inner))
        b = vd.asbuffer(x)
        vd.fft.fft(b, axis=1)
        assert rel_l2(b.read(0), np.fft.fft(x.astype(np.complex128), axis=1)) <= tol_fp32(n)
        vd.fft.ifft(b, axis=1)
        assert rel_l2(b.read(0), x) <= 2 * tol_fp32(n)


@pytest.mark.parametrize("n", [1500, 2000, 2100, 2205, 4095])
@pytest.mark.parametrize("inner", [1, 3, 33, 700])
def test_column_tiles(n, inner):
    rng = np.random.default_rng(n + inner)
    x = crandn(rng, (1, n, inner))
    if inner == 33:  # fewer tiles than SMs, whatever their width
        assert _plan((1, n, inner))["transforms_per_cta"] in (2, 4, 8)
    b = vd.asbuffer(x)
    vd.fft.fft(b, axis=1)
    assert rel_l2(b.read(0), np.fft.fft(x.astype(np.complex128), axis=1)) <= tol_fp32(n)
    k = crandn(rng, (1, n, inner))
    c = vd.asbuffer(x)
    vd.fft.convolve(c, vd.asbuffer(k), axis=1)
    want = np.fft.ifft(np.fft.fft(x.astype(np.complex128), axis=1) * np.conj(k), axis=1)
    assert rel_l2(c.read(0), want) <= 2 * tol_fp32(n)
