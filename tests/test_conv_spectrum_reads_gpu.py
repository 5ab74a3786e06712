"""Fused convolutions of 512 and 1024 points by how they read the kernel
spectrum: one per batch or one for all, plain or with the forward spectrum
written (mode 1) or its product with a second one (mode 2), rows and column
tiles with a remainder."""

import numpy as np
import pytest

from helpers import crandn, rel_l2, tol_fp32

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from vkdispatch_gb300 import _lib as L  # noqa: E402
from vkdispatch_gb300.autograd import _ops  # noqa: E402
from vkdispatch_gb300.fft import plan as P  # noqa: E402


@pytest.mark.parametrize("n", [256, 512, 1024])
@pytest.mark.parametrize("inner", [1, 11])
@pytest.mark.parametrize("shared", [False, True])
def test_modes(n, inner, shared):
    rng = np.random.default_rng(n + inner)
    shape = (3, n) + ((inner,) if inner > 1 else ())
    x, aux = crandn(rng, shape), crandn(rng, shape)
    k = crandn(rng, ((1,) if shared else (3,)) + shape[1:])
    xt, kt, at = (torch.from_numpy(v).cuda() for v in (x, k, aux))
    s = torch.cuda.current_stream().cuda_stream
    f = np.fft.fft(x.astype(np.complex128), axis=1)
    for kop, kk in ((L.VDX_KOP_MUL_CONJ, np.conj(k)), (L.VDX_KOP_MUL, k)):
        p = P.get_plan(shape, 1, L.VDX_KIND_CONV, False, True, L.VDX_C64, L.VDX_C64, None, kop, L.VDX_C64, shared)
        want = np.fft.ifft(f * kk, axis=1)
        y = torch.empty_like(xt)
        p.exec(xt.data_ptr(), y.data_ptr(), kt.data_ptr(), s)
        assert rel_l2(y.cpu().numpy(), want) <= 2 * tol_fp32(n)
        spec = torch.empty_like(xt)
        if kop == L.VDX_KOP_MUL_CONJ:
            p.exec_ops(xt.data_ptr(), y.data_ptr(), kt.data_ptr(), _ops(spec_out=spec.data_ptr()), s)
            sw = f
        else:
            p.exec_ops(xt.data_ptr(), y.data_ptr(), kt.data_ptr(),
                       _ops(spec_out=spec.data_ptr(), spec_aux=at.data_ptr(), spec_scale=0.5), s)
            sw = aux * np.conj(f) * 0.5
        assert rel_l2(y.cpu().numpy(), want) <= 2 * tol_fp32(n)
        assert rel_l2(spec.cpu().numpy(), sw) <= tol_fp32(n)
