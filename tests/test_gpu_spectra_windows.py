"""The spectra's sorted-tile running median against numpy.ma, at the edges of
its tiles: windows of 3, 127/129, 255/257 and 511/513 periods (the last beyond the
tiles), spectra of one row, of whole tiles and of one more, masked runs longer
than a window, and ties.

Bars: as the spectra's against the reference's module, 1e-9 relative (plus
1e-9 of the largest power for values near 0).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(chi2, mask, k):
    sr = np.ma.array(chi2.min() / chi2 if mask is None else np.ma.array(chi2, mask=mask).min() / chi2, mask=mask)
    sde_raw = (1 - sr.mean()) / sr.std()
    praw = (sr - sr.mean()) * (sde_raw / (sr - sr.mean()).max())
    n = len(chi2)
    if n <= 2 * k:
        return np.ma.getdata(sr), praw, praw, sde_raw, sde_raw
    rows = np.lib.stride_tricks.sliding_window_view(np.arange(n), k)
    med = np.ma.median(praw[rows], axis=1)
    front = (n - len(med)) // 2
    at = np.clip(np.arange(n) - front, 0, len(med) - 1)
    p = praw - np.ma.getdata(med)[at]
    p = p - p.mean()
    sde = (p / p.std()).max()
    return np.ma.getdata(sr), praw, p * (sde / p.max()), sde_raw, sde


@pytest.mark.parametrize("k,n", [
    (3, 7), (3, 700), (31, 63), (127, 255), (127, 256 + 129), (129, 3000), (255, 5 * 258 + 254), (257, 2000),
    (511, 1500), (513, 1200), (91, 166 * 40 + 90), (91, 166 * 40 + 91),
])
@pytest.mark.parametrize("masked", [False, True])
def test_running_median_windows(cuda, k, n, masked):
    import torch
    from gtls_b200 import _lib
    rng = np.random.default_rng(k * 100_000 + n)
    chi2 = 1000.0 + np.round(rng.normal(0, 3, n), 1)   # rounded: ties
    mask = None
    if masked:
        mask = rng.random(n) < 0.1
        mask[n // 2:n // 2 + max(1, k // 2)] = True
        mask[0] = False
    osf = (k - 1) / 30.0 if (k - 1) / 30.0 * 30 == k - 1 else k / 30.0   # k - 1 is even: one is added
    want = _reference(chi2, mask, k)
    got = _lib.spectra(torch.from_numpy(chi2).cuda(),
                       torch.from_numpy(mask.astype(np.uint8)).cuda() if masked else None, osf)
    keep = slice(None) if mask is None else ~mask
    for a, b in zip(got[:3], want[:3]):
        b = np.ma.getdata(b)[keep]
        np.testing.assert_allclose(a.cpu().numpy()[keep], b, rtol=1e-9, atol=1e-9 * np.abs(b).max())
    np.testing.assert_allclose(got[3:], want[3:], rtol=1e-9)
