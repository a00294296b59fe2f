"""Calls of the spectra besides the usual one: oversampling factors whose
window is far beyond the spectrum (no running median then), through both entry
points.

Bars: the same bits as with any other window of at least half the spectrum.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chi2(n):
    return 1000.0 + np.random.default_rng(n).normal(0, 3, n)


def _noalloc(chi2, osf):
    import torch
    from gtls_b200 import _lib
    x = torch.from_numpy(chi2).cuda()
    out = [torch.empty_like(x) for _ in range(3)]
    sde = [ctypes.c_double(), ctypes.c_double()]
    lib = _lib.load()
    rc = lib.gtls_spectra_noalloc(x.data_ptr(), None, len(chi2), osf, *(o.data_ptr() for o in out),
                                  ctypes.byref(sde[0]), ctypes.byref(sde[1]),
                                  torch.cuda.current_stream().cuda_stream)
    assert rc == 0, lib.gtls_noalloc_last_error()
    return [o.cpu().numpy() for o in out] + [s.value for s in sde]


@pytest.mark.parametrize("osf", [1e9, 4e13, 1e14, 1e17])
def test_windows_far_beyond_the_spectrum(cuda, osf):
    import torch
    from gtls_b200 import _lib
    chi2 = _chi2(500)
    want = _lib.spectra(torch.from_numpy(chi2).cuda(), None, 100)
    got = _lib.spectra(torch.from_numpy(chi2).cuda(), None, osf)
    other = _noalloc(chi2, osf)
    for a, b, c in zip(want[:3], got[:3], other[:3]):
        np.testing.assert_array_equal(b.cpu().numpy(), a.cpu().numpy())
        np.testing.assert_array_equal(c, a.cpu().numpy())
    assert tuple(got[3:]) == tuple(want[3:]) == tuple(other[3:])
