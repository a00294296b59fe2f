"""Calls of the spectra besides the usual one: oversampling factors whose
window is far beyond the spectrum (no running median then), and one array for several
outputs (as of a caller that wants the power alone), through both entry
points.

Bars: the same bits as with any other window of at least half the spectrum;
the last output written to a shared array within 1e-9 (of its largest value) of the
one that has an array to itself.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chi2(n):
    return 1000.0 + np.random.default_rng(n).normal(0, 3, n)


def _noalloc(chi2, osf, arrays=(0, 1, 2), ctx=None):
    """gtls_spectra_noalloc (with a context gtls_spectra) with output i in array arrays[i]."""
    import torch
    from gtls_b200 import _lib
    x = torch.from_numpy(chi2).cuda()
    bufs = [torch.empty_like(x) for _ in range(3)]
    out = [bufs[a] for a in arrays]
    sde = [ctypes.c_double(), ctypes.c_double()]
    lib = _lib.load()
    args = (x.data_ptr(), None, len(chi2), osf, *(o.data_ptr() for o in out), ctypes.byref(sde[0]),
            ctypes.byref(sde[1]), torch.cuda.current_stream().cuda_stream)
    rc = lib.gtls_spectra_noalloc(*args) if ctx is None else lib.gtls_spectra(ctx, *args)
    assert rc == 0, lib.gtls_noalloc_last_error()
    torch.cuda.synchronize()
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


@pytest.mark.parametrize("n", [60, 2592, 30000])
@pytest.mark.parametrize("arrays", [(0, 1, 1), (1, 0, 1), (1, 1, 0), (0, 0, 0)])
@pytest.mark.parametrize("entry", ["gtls_spectra", "gtls_spectra_noalloc"])
def test_outputs_that_share_an_array(cuda, entry, arrays, n):
    from gtls_b200 import _lib
    chi2 = _chi2(n)
    ctx = _lib.context(0) if entry == "gtls_spectra" else None
    want = _noalloc(chi2, 3.0, (0, 1, 2), ctx)
    got = _noalloc(chi2, 3.0, arrays, ctx)
    for i in range(3):   # SR, raw power and power are written in this order
        if arrays[i] not in arrays[i + 1:]:
            np.testing.assert_allclose(got[i], want[i], rtol=1e-9, atol=1e-9 * np.abs(want[i]).max())
    np.testing.assert_allclose(got[3:], want[3:], rtol=1e-9)
