"""Results of a row do not depend on the rows beside it, whose number sets how
many warps fold a part (one, two, four or eight) and which parts share a CTA:
the same rows reduced alone and at the front and the end of many give the same
bits."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import vkdispatch_gb300 as vd  # noqa: E402
import vkdispatch_gb300.codegen as vc  # noqa: E402


@vd.reduce.reduce(0, axes=[1])
def add_f32(a: vc.f32, b: vc.f32) -> vc.f32:
    return a + b


@vd.reduce.map_reduce(vd.reduce.SubgroupAdd, axes=[1])
def abs_c64(buffer: vc.Buff[vd.complex64]) -> vd.float32:
    v = buffer[vd.reduce.mapped_io_index()]
    return vc.sqrt(v.real * v.real + v.imag * v.imag)


def _rows(fn, t, vt):
    return fn(vd.from_cuda_array(t, var_type=vt)).tensor.reshape(-1)[: t.shape[0]]


# (rows, n): 64 elements, a whole block, one part of two warps, of one warp by
# its number, two parts, and 16 parts of two warps; n odd where rows misalign.
# The last: rows that leave places of a CTA empty (5 and 18 parts in fours) and
# that do not
SHAPES = [(16384, 64), (20001, 65), (9000, 512), (4097, 2048), (5000, 1023), (6001, 4096), (2501, 4099), (333, 8191),
          (1024, 65536), (1500, 18001), (400, 70000), (148, 21716), (33, 100001)]


@pytest.mark.parametrize("rows,n", SHAPES)
@pytest.mark.parametrize("kind", ["add", "abs"])
def test_rows_alone_and_among_others(rows, n, kind):
    g = torch.Generator(device="cuda").manual_seed(rows + n)
    if kind == "add":
        x, fn, vt = torch.randn((rows, n), generator=g, device="cuda"), add_f32, vd.float32
        want, mag = x.double().sum(1), x.double().abs().sum(1)
    else:
        x = torch.view_as_complex(torch.randn((rows, n, 2), generator=g, device="cuda"))
        fn, vt = abs_c64, vd.complex64
        want = mag = x.to(torch.complex128).abs().sum(1)
    got = _rows(fn, x, vt)
    # a fold of at most 12 levels in a part, 10 over parts, and the magnitude's own rounding
    assert float(((got.double() - want).abs() / mag).max()) <= 25 * 2.0 ** -24
    for lo, m in ((0, 1), (0, 2), (rows - 3, 3), (rows // 2, 7)):
        alone = _rows(fn, x[lo:lo + m].contiguous(), vt)
        assert torch.equal(alone, got[lo:lo + m])
