"""Multi-kernel convolutions against one convolution per kernel in numpy: runtime
lengths of one, two, three and four radix passes, and the lengths whose plain
convolutions default to two-pass plans; rows and column tiles with a remainder,
both products, fp32 and fp64."""

import numpy as np
import pytest

from helpers import crandn, rel_l2, tol_fp32

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from vkdispatch_gb300 import _lib as L  # noqa: E402
from vkdispatch_gb300.fft import plan as P  # noqa: E402


@pytest.mark.parametrize("n", [7, 11, 24, 45, 360, 363, 512, 625, 1000, 1024, 2187, 4095])
@pytest.mark.parametrize("inner", [1, 11])
@pytest.mark.parametrize("double", [False, True])
def test_against_numpy(n, inner, double):
    rng = np.random.default_rng(n + inner)
    rows, K = 3, 3
    shape = (rows, n) + ((inner,) if inner > 1 else ())
    dt, code = (np.complex128, L.VDX_C128) if double else (np.complex64, L.VDX_C64)
    x, k = crandn(rng, shape, dt), crandn(rng, (K,) + shape, dt)
    xt, kt = torch.from_numpy(x).cuda(), torch.from_numpy(k).cuda()
    y = torch.empty((K,) + shape, dtype=xt.dtype, device="cuda")
    stride = x.size
    f = np.fft.fft(x.astype(np.complex128), axis=1)
    for kop, kk in ((L.VDX_KOP_MUL_CONJ, np.conj(k)),) + (() if double else ((L.VDX_KOP_MUL, k),)):
        if double and (n % 11 == 0 or n % 13 == 0):  # a fp64 thread holds 8 points
            with pytest.raises(ValueError):
                P.get_plan(shape, 1, L.VDX_KIND_CONV, False, True, code, code, None, kop, code)
            return
        p = P.get_plan(shape, 1, L.VDX_KIND_CONV, False, True, code, code, None, kop, code)
        s = torch.cuda.current_stream().cuda_stream
        if not p.exec_multi(xt.data_ptr(), y.data_ptr(), kt.data_ptr(), K, stride, stride, s):
            assert double and n > 1000
            pytest.skip("the kept spectrum of long fp64 transforms does not fit in shared memory")
        want = np.fft.ifft(f[None] * kk, axis=2)
        assert rel_l2(y.cpu().numpy(), want) <= (1e-13 if double else 2 * tol_fp32(n))
