"""Curves whose baseline E = sum v^2 w is not finite: an uncertainty of 0 (or
one whose square is), an infinite flux, a NaN.  No start that passes the depth test has
a finite value then, so the minimum is n at the first start that fails, or
infinite at the first start of all.  Nothing needs to be summed for that.

Bars: values and locations exactly; at most a hundredth of the passing
starts' multiply-adds (a quarter, the narrowest of five durations, where no weight is
finite and none fails; a start for each of the warps where a period is cut into many
ranges).  An infinite flux leaves the mean of all windows open: no bar but the
whole there.
"""
import numpy as np
import pytest

from test_gpu_bounds import _case

pytestmark = pytest.mark.gpu


def _run(y, dy, c, periods, all_, precision, skip):
    import torch
    from gtls_b200 import _lib
    t, widths, tm, ov, maxd = c[0], c[3], c[4], c[5], c[6]
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to("cuda:0")
    tm_ = _lib.Timing()
    chi2, loc = _lib.search(dict(t=up(t), y=up(y), dy=up(dy), span=float(np.float32(t.max() - t.min()))), up(periods),
                            dict(widths=up(widths), overshoot=up(ov), templates=up(tm), max_width=maxd), 1e-5, skip, 1,
                            _lib.GTLS_PASS_ALL if all_ else _lib.GTLS_PASS_MAIN, precision, timing=tm_,
                            flags=_lib.GTLS_SEARCH_ALL_DURATIONS)
    return chi2.cpu().numpy(), loc.cpu().numpy(), tm_


def _first_failing(t, y, period, widths, all_, skip):
    x = t / period
    v = y[np.argsort(x - np.trunc(x), kind="stable")] - 1.0
    n = len(v)
    v = np.concatenate([v, v])
    for d, w in enumerate(widths):
        s = 1 if all_ or w <= skip else w // skip
        mean = -np.convolve(v[:n + w - 1], np.ones(w), "valid") / w
        bad = np.nonzero(~(mean > 1e-5) | (np.arange(n) % s != 0))[0]
        if len(bad):
            return d * n + bad[0]
    return -1


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("all_", [False, True])
@pytest.mark.parametrize("kind", ["zero_dy", "tiny_dy", "all_zero_dy"])
@pytest.mark.parametrize("fails", [True, False])
@pytest.mark.parametrize("periods", [3, 300])
def test_an_infinite_baseline(cuda, kind, all_, precision, fails, periods):
    n = 9000
    c = _case(n, [40, 60, 100, 200, 400], seed=3)
    y = 1.0 - 0.05 + 1e-3 * np.random.default_rng(1).standard_normal(n)   # every start passes
    if fails:
        y[n // 3:n // 3 + 100] = 1.2
    dy = c[2].copy()
    if kind == "all_zero_dy":
        dy[:] = 0.0
    else:
        dy[n // 2] = 0.0 if kind == "zero_dy" else 1e-170
    P = np.linspace(0.61, 3.4, periods)
    skip = 8 if fails else 1000   # (a skipped start has the value n too)
    chi2, loc, tm_ = _run(y, dy, c, P, all_, precision, skip)
    for i in (0, periods // 2, periods - 1):
        at = _first_failing(c[0], y, P[i], c[3], all_, skip)
        assert chi2[i] == (n if at >= 0 else np.inf)
        if at >= 0 or kind != "all_zero_dy":
            assert loc[i] == max(at, 0)
        else:   # every start's sums are infinite: none has a value
            assert loc[i] == np.iinfo(np.int64).max
    assert tm_.chi2_issued_fma <= (0.25 if kind == "all_zero_dy" else 0.01 if periods > 3 else 0.05) * tm_.chi2_active_fma


@pytest.mark.parametrize("all_", [False, True])
def test_a_flux_that_is_not_finite(cuda, all_):
    n = 9000
    c = _case(n, [40, 60, 100, 200, 400], seed=3)
    for value in (np.nan, np.inf, -np.inf):
        y = c[1].copy()
        y[n // 2] = value
        chi2, loc, tm_ = _run(y, c[2], c, np.linspace(0.61, 3.4, 300), all_, "fp64", 8)
        assert (chi2 == n).all()
        assert tm_.chi2_issued_fma <= tm_.chi2_active_fma
