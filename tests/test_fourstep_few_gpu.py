"""Four-step passes of runtime plans on both sides of the rule for launches of
few CTAs: sub-lengths of one, two, three and four radix passes, rows and column
tiles with a remainder, every storage type."""

import numpy as np
import pytest

import vkdispatch_gb300 as vd
from vkdispatch_gb300.fft import plan as P

from helpers import crandn, rel_l2, tol_fp32

pytestmark = pytest.mark.gpu

# short lengths 9 x 9, 13 x 13, 49 x 175, 49 x 343, 125 x 125, 165 x 182, 343 x 343
LENGTHS = [81, 169, 8575, 16807, 15625, 30030, 117649]


@pytest.fixture(autouse=True)
def fourstep_always(monkeypatch):
    monkeypatch.setenv("VDX_FOURSTEP_MIN", "64")
    P.cache_clear()
    yield
    P.cache_clear()


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("many", [False, True])
def test_c64(n, many):
    rng = np.random.default_rng(n)
    # a pass fills the chip at 152 CTAs of up to 512 threads: 2^21 points do, one transform does not
    rows = max(3, (1 << 21) // n) if many else 1
    for shape, axis in (((rows, n), 1), ((1, n, 5 * rows // 3 if many else 3), 1)):
        x = crandn(rng, shape)
        b = vd.asbuffer(x)
        vd.fft.fft(b, axis=axis)
        want = np.fft.fft(x.astype(np.complex128), axis=axis)
        assert rel_l2(b.read(0), want) <= tol_fp32(n)
        vd.fft.ifft(b, axis=axis)
        assert rel_l2(b.read(0), x) <= 2 * tol_fp32(n)


@pytest.mark.parametrize("storage,tol", [(vd.complex32, 2.5e-3), (vd.complexbf16, 1.6e-2)])
@pytest.mark.parametrize("n", [81, 8575, 16807])
def test_half_storage(n, storage, tol):
    rng = np.random.default_rng(n)
    for shape, axis in (((2, n), 1), ((1, n, 5), 1)):
        b = vd.Buffer(shape, storage)
        b.write(crandn(rng, shape, np.complex128) * 0.25)
        q = np.asarray(b.read(0)).astype(np.complex128)
        vd.fft.fft(b, axis=axis)
        assert rel_l2(b.read(0), np.fft.fft(q, axis=axis)) <= tol
