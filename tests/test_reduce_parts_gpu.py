"""Reductions at the edges of their parts: steps of four elements, one to eight
warps per part, short last parts, one or many partials per row; and the same
bits from an aligned and from a misaligned array, since a result depends on n
alone."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import vkdispatch_gb300 as vd  # noqa: E402
import vkdispatch_gb300.codegen as vc  # noqa: E402


@vd.reduce.reduce(0, axes=[1])
def add_f32(a: vc.f32, b: vc.f32) -> vc.f32:
    return a + b


@vd.reduce.reduce("-inf", axes=[1])
def max_f32(a: vc.f32, b: vc.f32) -> vc.f32:
    return vc.max(a, b)


@vd.reduce.reduce(0, axes=[1])
def xor_i32(a: vc.i32, b: vc.i32) -> vc.i32:
    return a ^ b


@vd.reduce.map_reduce(vd.reduce.SubgroupAdd, axes=[1])
def abs_c64(buffer: vc.Buff[vd.complex64]) -> vd.float32:
    v = buffer[vd.reduce.mapped_io_index()]
    return vc.sqrt(v.real * v.real + v.imag * v.imag)


def _views(a):
    """The array on a 16-byte boundary, and one element past it."""
    t = torch.from_numpy(a).cuda()
    big = torch.empty(a.size + 1, dtype=t.dtype, device="cuda")
    off = big[1:].view(t.shape)
    off.copy_(t)
    return t, off


def _rows(fn, t, vt):
    return fn(vd.from_cuda_array(t, var_type=vt)).tensor.reshape(-1)[: t.shape[0]].cpu().numpy()


@pytest.mark.parametrize("n", [1, 3, 4, 5, 127, 128, 511, 4095, 4096, 4097, 8193, 16384, 65536, 65537, 131075, 262147])
@pytest.mark.parametrize("rows", [2, 37])
def test_edges(n, rows):
    rng = np.random.default_rng(n + rows)
    x = rng.standard_normal((rows, n)).astype(np.float32)
    t, off = _views(x)
    got = _rows(add_f32, t, vd.float32)
    eps = np.finfo(np.float32).eps
    bound = 2 * eps * max(1.0, np.log2(n)) * np.abs(x).astype(np.float64).sum(axis=1) + 1e-30
    # the serial part of the fold: at most 16 steps of a thread's accumulator and its tail
    assert np.all(np.abs(got - x.astype(np.float64).sum(axis=1)) <= 2 * bound)
    assert np.array_equal(got, _rows(add_f32, off, vd.float32))
    assert np.array_equal(_rows(max_f32, t, vd.float32), x.max(axis=1))
    assert np.array_equal(_rows(max_f32, off, vd.float32), x.max(axis=1))
    i = rng.integers(-(1 << 31), 1 << 31, (rows, n), dtype=np.int64).astype(np.int32)
    ti, offi = _views(i)
    want = np.bitwise_xor.reduce(i, axis=1)
    assert np.array_equal(_rows(xor_i32, ti, vd.int32), want) and np.array_equal(_rows(xor_i32, offi, vd.int32), want)
    c = (x + 1j * x[:, ::-1]).astype(np.complex64)
    tc, offc = _views(c)
    gc = _rows(abs_c64, tc, vd.complex64)
    ref = np.abs(c.astype(np.complex128)).sum(axis=1)
    assert np.all(np.abs(gc - ref) <= 1e-6 * ref + 1e-30)
    assert np.array_equal(gc, _rows(abs_c64, offc, vd.complex64))


def test_single_large_row_and_infinities():
    x = torch.randn(1, (1 << 24) + 5, device="cuda")
    x[0, 12345] = float("inf")
    assert _rows(max_f32, x, vd.float32)[0] == np.inf
    assert _rows(add_f32, x, vd.float32)[0] == np.inf
    x[0, 777] = float("nan")
    assert np.isnan(_rows(add_f32, x, vd.float32)[0])
