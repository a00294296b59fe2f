"""Curves whose samples are far from alike, as they come: flares, a glitch,
uncertainties of which a few are far too small.
The bounds must still rule out most of the starts there (the multiply-adds of
the starts that are summed, against those of all that pass the depth
test), and the minimum is the oracle's.

Bars: at most a tenth of the multiply-adds (a list that runs over sums every
start, some of them twice; on clean curves one start in a hundred is summed);
FP64 chi2 within 1e-9 relative of the FP64 oracle, FP32 within 2e-6, locations
identical in FP64.
"""
import numpy as np
import pytest

import tls_oracle as O
from test_gpu_bounds import _case

pytestmark = pytest.mark.gpu

PERIODS = np.linspace(0.61, 3.4, 300)   # (a few periods are cut into short ranges of starts)
CHECKED = [0, 117, 299]


def _odd(kind, n, widths):
    t, y, dy, widths, tm, ov, maxd = _case(n, widths, seed=n + len(kind), depth=1e-3)
    y, dy = y.copy(), dy.copy()
    rng = np.random.default_rng(n)
    if kind == "flares":
        for i in rng.integers(100, n - 200, 6):
            y[i:i + 60] += 0.5 * np.exp(-np.arange(60) / 12.0)
    elif kind == "glitch":
        y[n // 3] = 50.0
    elif kind == "sure":         # one sample surer than the others, a million times their weight
        dy[n // 3] /= 1000.0
    elif kind == "sure_flat":    # and one of v = 0
        dy[[n // 3, n // 2]] /= 3000.0
        y[n // 2] = 1.0
    elif kind in ("glitches", "crowd"):   # up to 400 times the flux; a crowd: more than are left out of the prefix sums
        k = 700 if kind == "glitches" else 6000
        y[rng.integers(0, n, k)] *= np.exp(rng.uniform(0.0, 6.0, k))
    elif kind == "lost":         # one sample whose weight FP32 does not hold beside the others'
        y[n // 3], dy[n // 3] = 1e30, dy[n // 3] * 1e20
    elif kind == "ties":         # every start of a duration has the same value
        y[:] = 1.0 - 1e-3
        dy[:] = 1e-3
    return t, y, dy, widths, tm, ov, maxd


def _run(c, all_, precision, periods=PERIODS):
    import torch
    from gtls_b200 import _lib
    t, y, dy, widths, tm, ov, maxd = c
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to("cuda:0")
    tm_ = _lib.Timing()
    chi2, loc = _lib.search(dict(t=up(t), y=up(y), dy=up(dy), span=float(np.float32(t.max() - t.min()))), up(periods),
                            dict(widths=up(widths), overshoot=up(ov), templates=up(tm), max_width=maxd), 1e-5, 8, 1,
                            _lib.GTLS_PASS_ALL if all_ else _lib.GTLS_PASS_MAIN, precision, timing=tm_,
                            flags=_lib.GTLS_SEARCH_ALL_DURATIONS)
    return chi2.cpu().numpy(), loc.cpu().numpy(), tm_


def _widths(lo, hi, ratio):
    return np.unique(np.round(np.geomspace(lo, hi, int(np.log(hi / lo) / np.log(ratio)) + 1)).astype(int))


@pytest.mark.parametrize("kind", ["flares", "glitch", "sure", "sure_flat"])
@pytest.mark.parametrize("all_,n,widths", [
    (False, 19728, _widths(20, 1400, 1.06)),
    (False, 40000, _widths(40, 4500, 1.08)),
    (True, 9000, _widths(60, 800, 1.3)),
])
def test_most_starts_are_ruled_out(cuda, kind, all_, n, widths):
    c = _odd(kind, n, widths)
    back = O.NumpyBackend()
    t, y, dy, widths, tm, ov, maxd = c
    ref = [back.noskip_pass(t, y, dy, p, widths, tm, ov, maxd, 1e-5) if all_ else
           back.main_pass(t, y, dy, p, widths, tm, ov, maxd, 1e-5, 8) for p in PERIODS[CHECKED]]
    for precision, rtol in (("fp64", 1e-9), ("fp32", 2e-6)):
        chi2, loc, tm_ = _run(c, all_, precision)
        np.testing.assert_allclose(chi2[CHECKED], [r[0] for r in ref], rtol=rtol)
        if precision == "fp64":
            np.testing.assert_array_equal(loc[CHECKED], [r[1] for r in ref])
        assert tm_.chi2_issued_fma <= 0.1 * tm_.chi2_active_fma, (precision, tm_.as_dict())


@pytest.mark.parametrize("kind", ["ties", "glitches", "crowd", "lost"])
@pytest.mark.parametrize("n,widths", [(19728, _widths(20, 1400, 1.06)), (40000, _widths(40, 4500, 1.08))])
def test_what_the_list_cannot_hold_is_summed_once_at_most(cuda, kind, n, widths):
    """Where the list of a CTA runs over: starts that all tie (the widest duration
    rules out the others in the end), many glitches, more than are set apart, and
    a sample whose v is known to no window.  Not more is summed than starts that pass."""
    c = _odd(kind, n, widths)
    t, y, dy, widths, tm, ov, maxd = c
    back = O.NumpyBackend()
    ref = [back.main_pass(t, y, dy, p, widths, tm, ov, maxd, 1e-5, 8) for p in PERIODS[CHECKED]]
    for precision, rtol in (("fp64", 1e-9), ("fp32", 2e-6)):
        chi2, loc, tm_ = _run(c, False, precision)
        np.testing.assert_allclose(chi2[CHECKED], [r[0] for r in ref], rtol=rtol)
        if precision == "fp64" and kind != "ties":
            np.testing.assert_array_equal(loc[CHECKED], [r[1] for r in ref])
        assert tm_.chi2_issued_fma <= (0.1 if kind == "ties" else 1.0) * tm_.chi2_active_fma, (precision, tm_.as_dict())


def test_fp32_sums_as_few_starts_as_fp64(cuda):
    """On a curve 1% below 1, where every start passes, many come close to the
    minimum.  FP32 sums of the main pass round by 37 half ulps at 4,500 samples,
    a ninth of the bounds' own 2e-5, so that hardly more starts stay than in FP64."""
    n, widths = 40000, _widths(40, 4500, 1.08)
    c = list(_odd("offset", n, widths))
    c[1] = c[1] - 0.01
    tm_ = [_run(c, False, p)[2] for p in ("fp64", "fp32")]
    assert tm_[1].chi2_issued_fma <= 1.02 * tm_[0].chi2_issued_fma, [t.as_dict() for t in tm_]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("kind", ["ties", "glitches", "crowd", "flares"])
def test_a_value_does_not_depend_on_who_sums_it(cuda, kind, precision):
    """The same period among 300 (whole ranges, and where the list ran over list by
    list, a warp a window) and alone (short ranges, wide windows by the CTA): the same bits."""
    n, widths = 19728, _widths(20, 1400, 1.06)
    c = _odd(kind, n, widths)
    chi2 = _run(c, False, precision)[0]
    for i in CHECKED:
        assert _run(c, False, precision, PERIODS[i:i + 1])[0][0] == chi2[i]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_second_searches_in_chunks_and_sets_of_curves(cuda, precision):
    """Curves of which some have spikes and some periods' lists run over, searched
    together and in small chunks: the bits of each curve's own search."""
    import torch
    from gtls_b200 import _lib
    kinds = ["flares", "ties", "glitch", "crowd", "sure"]
    widths = _widths(20, 1400, 1.06)
    cs = [_odd(k, n, widths) for k, n in zip(kinds, (19728, 15001, 9000, 19728, 12345))]
    periods = [PERIODS[i::3] for i in range(len(cs))]
    alone = [_run(c, False, precision, p)[:2] for c, p in zip(cs, periods)]
    cat = lambda k: torch.from_numpy(np.concatenate([np.ascontiguousarray(c[k]).reshape(-1) for c in cs])).to("cuda:0")
    off = lambda sizes: np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    curves = dict(t=cat(0), y=cat(1), dy=cat(2), sample_off=off([len(c[0]) for c in cs]),
                  span=np.array([np.float32(c[0].max() - c[0].min()) for c in cs], dtype=np.float32))
    tables = dict(widths=cat(3), overshoot=cat(5), templates=cat(4), dur_off=off([len(c[3]) for c in cs]),
                  tmpl_off=off([c[4].size for c in cs])[:-1], max_width=np.array([c[6] for c in cs], dtype=np.int32))
    p_off = off([len(p) for p in periods])
    p_dev = torch.from_numpy(np.concatenate(periods)).to("cuda:0")
    try:
        for budget in (8 << 30, 12 << 20):
            _lib.set_chunk_budget(budget)
            chi2, loc = _lib.search_batch(curves, p_dev, p_off, tables, 1e-5, 8, np.ones(len(cs), dtype=np.int32),
                                          _lib.GTLS_PASS_MAIN, precision, flags=_lib.GTLS_SEARCH_ALL_DURATIONS)
            chi2, loc = chi2.cpu().numpy(), loc.cpu().numpy()
            for i, (c, l) in enumerate(alone):
                np.testing.assert_array_equal(chi2[p_off[i]:p_off[i + 1]], c, err_msg=kinds[i])
                if kinds[i] != "ties":
                    np.testing.assert_array_equal(loc[p_off[i]:p_off[i + 1]], l, err_msg=kinds[i])
    finally:
        _lib.set_chunk_budget(8 << 30)
