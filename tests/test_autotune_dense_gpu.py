"""Autotuned real transforms: dense rows out of place and packed rows in place
are searched and cached apart, each as it runs."""

import numpy as np
import pytest

import vkdispatch_gb300 as vd
from vkdispatch_gb300.fft import plan as P

from helpers import rel_l2, tol_fp32

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_dense_and_packed_rows_are_searched_apart(tmp_path):
    rows, n = 37, 2 * 1170
    x = np.random.default_rng(n).standard_normal((rows, n)).astype(np.float32)
    want = np.fft.rfft(x.astype(np.float64), axis=1)
    P.cache_clear()
    with vd.fft.autotune():
        searches = [P.autotune_stats()[1]]
        y = vd.torch_fft.rfft(torch.from_numpy(x).cuda())
        searches.append(P.autotune_stats()[1])
        z = vd.torch_fft.irfft(y, n)
        searches.append(P.autotune_stats()[1])
        b = vd.asrfftbuffer(x)
        vd.fft.rfft(b)
        searches.append(P.autotune_stats()[1])
        vd.fft.irfft(b)
        searches.append(P.autotune_stats()[1])
    assert np.all(np.diff(searches) == 1)
    assert rel_l2(y.cpu().numpy(), want) <= tol_fp32(n)
    assert rel_l2(z.cpu().numpy(), x) <= 2 * tol_fp32(n)
    assert rel_l2(b.read_real(0), x) <= 2 * tol_fp32(n)
    path = tmp_path / "tune.txt"
    P.autotune_save(path)
    P.autotune_load(path)
    P.cache_clear()
    with vd.fft.autotune():  # both kinds of entry come back from the file
        vd.torch_fft.rfft(torch.from_numpy(x).cuda())
        vd.fft.rfft(vd.asrfftbuffer(x))
        assert P.autotune_stats()[1] == searches[-1]
    P.cache_clear()
