"""Runtime-radix passes of the composite radices (6, 10, 12, 14, 15) and the
pass roles around them: one-pass plans, first, middle and last passes, the
forward / inverse turn of a convolution, packed real rows, strided tiles with a
partial last tile, and batches of uneven lengths; against FP64 numpy."""

import numpy as np
import pytest

import vkdispatch_gb300 as vd

from helpers import crandn, rel_l2, tol_fp32

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# one pass each; two passes; three and more, with a composite radix in every role; even radices only
LENGTHS = [6, 10, 12, 14, 15, 45, 84, 96, 150, 182, 210, 1440, 1500, 2100, 2730, 4095, 5040, 7800]


@pytest.mark.parametrize("n", LENGTHS)
def test_c2c_and_convolution(n):
    rng = np.random.default_rng(n)
    for shape, axis in (((5, n), 1), ((2, n, 11), 1)):
        x = crandn(rng, shape)
        b = vd.asbuffer(x)
        vd.fft.fft(b, axis=axis)
        assert rel_l2(b.read(0), np.fft.fft(x.astype(np.complex128), axis=axis)) <= tol_fp32(n)
        vd.fft.ifft(b, axis=axis)
        assert rel_l2(b.read(0), x) <= 2 * tol_fp32(n)
        k = crandn(rng, shape)
        b, kb = vd.asbuffer(x), vd.asbuffer(k)
        vd.fft.convolve(b, kb, axis=axis)
        want = np.fft.ifft(np.fft.fft(x.astype(np.complex128), axis=axis) * np.conj(k.astype(np.complex128)), axis=axis)
        assert rel_l2(b.read(0), want) <= 2 * tol_fp32(n)


@pytest.mark.parametrize("n", LENGTHS)
def test_real_rows(n):
    """Even rows of 2n reals run n complex points; odd n runs the full-length rule."""
    rng = np.random.default_rng(n)
    for m in (2 * n,) + ((n,) if n % 2 else ()):
        x = rng.uniform(-1, 1, (3, m)).astype(np.float32)
        b = vd.asrfftbuffer(x)
        vd.fft.rfft(b)
        assert rel_l2(b.read_fourier(0), np.fft.rfft(x.astype(np.float64), axis=-1)) <= tol_fp32(m)
        vd.fft.irfft(b)
        assert rel_l2(b.read_real(0), x) <= 2 * tol_fp32(m)


@pytest.mark.parametrize("storage,tol", [(vd.complex32, 2.5e-3), (vd.complexbf16, 1.6e-2)])
@pytest.mark.parametrize("n", [16, 32, 48, 64, 128, 150, 256, 512, 1024, 1500, 2048, 4096])
def test_half_storage(n, storage, tol):
    """16-bit storage: compile-time plans of powers of two up to 4096 points, runtime passes besides."""
    rng = np.random.default_rng(n)
    for shape, axis in (((5, n), 1), ((2, n, 9), 1)):
        x = crandn(rng, shape) * 0.25
        b = vd.Buffer(shape, storage)
        b.write(x)
        q = b.read(0).astype(np.complex128)
        vd.fft.fft(b, axis=axis)
        assert rel_l2(b.read(0), np.fft.fft(q, axis=axis)) <= tol
        q = b.read(0).astype(np.complex128)
        vd.fft.ifft(b, axis=axis)
        assert rel_l2(b.read(0), np.fft.ifft(q, axis=axis)) <= tol


def test_uneven_batch_of_composite_radices():
    from vkdispatch_gb300.batch import BatchPlan

    lengths = LENGTHS + [16, 64, 1024, 20736, 21000, 65536]
    items, off = [], 0
    for n in lengths:
        items.append((off, n, 3))
        off += 3 * n
    x = crandn(np.random.default_rng(1), (off,))
    d = torch.from_numpy(x).cuda()
    plan = BatchPlan(items)
    plan(d, plan.make_workspace())
    torch.cuda.synchronize()
    assert plan.status() == 0
    got = d.cpu().numpy()
    for o, n, c in items:
        ref = np.fft.fft(x[o:o + n * c].reshape(c, n).astype(np.complex128), axis=-1)
        assert rel_l2(got[o:o + n * c].reshape(c, n), ref) <= 2 * tol_fp32(n), n
