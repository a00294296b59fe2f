"""The all-starts pass where its bounds cannot settle a start.

* A start whose window mean lies within the screening's rounding of the depth
  threshold is decided by its block of samples; where it fails there it still
  carries the value n (GPUFun.py:407,437).
* Uncertainties far from one: the weights alone are beyond FP32.

Bars: the value n exactly, and the location of the only start that has it;
chi2 times a power of two exactly, and the same locations.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DEPTH_MIN = 0.01


def _search(t, y, dy, widths, P, pass_, precision="fp64", skip=8):
    import torch
    from gtls_b200 import _lib
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to("cuda:0")
    widths = np.array(widths, dtype=np.int32)
    maxd = int(widths.max()) + int(widths.max()) % 2
    tm = np.ones((len(widths), maxd))
    for d, w in enumerate(widths):
        x = np.linspace(-1, 1, w) if w > 1 else np.zeros(1)
        tm[d, :w] = 0.5 * np.sqrt(np.clip(1 - 0.99 * x * x, 0, None)) ** 0.5
    curve = dict(t=up(t), y=up(y), dy=up(dy), span=float(np.float32(t.max() - t.min())))
    tables = dict(widths=up(widths), overshoot=up(np.full(len(widths), 1.07)), templates=up(tm), max_width=maxd)
    c, l = _lib.search(curve, up(np.atleast_1d(P)), tables, DEPTH_MIN, skip, 1, pass_, precision,
                       flags=_lib.GTLS_SEARCH_ALL_DURATIONS)
    return c.cpu().numpy(), l.cpu().numpy()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("at", [64 * 70 + 17, 7999, 8999])
def test_a_start_just_below_the_threshold_has_the_value_n(cuda, at, precision):
    """Every sample lies 0.0101 below 1 and passes on its own but one, 5e-7
    below the threshold: the sum of all samples before it, some 80, rounds
    the screening's mean by 1e-5, the sample itself by 1e-9.  E is 100 n, so n
    is the minimum.  (P is longer than the curve: the folded order is that of
    the times.)"""
    from gtls_b200 import _lib
    n = 9000
    t = 1.0 + np.arange(n) * 1e-3
    y = np.full(n, 1.0 - 0.0101)
    y[at] = 1.0 - (DEPTH_MIN - 5e-7)
    c, l = _search(t, y, np.full(n, 0.0101 / 10.0), [1, 2, 3], 1000.0, _lib.GTLS_PASS_ALL, precision)
    assert c[0] == n
    assert l[0] == at


@pytest.mark.parametrize("bits", [73, -70])
@pytest.mark.parametrize("pass_", ["GTLS_PASS_MAIN", "GTLS_PASS_ALL"])
def test_scaled_uncertainties_scale_chi2(cuda, pass_, bits):
    """dy divided by 2^bits multiplies every weight, and so E and every delta,
    by 4^bits without a rounding (weights of 1e50 and 1e-36).  Every start passes
    the depth test and none is skipped, so that n is no candidate.  (The first
    sweep of the all-starts pass looks at every second start and more.)"""
    from gtls_b200 import _lib
    n = 9000
    rng = np.random.default_rng(5)
    t = 1.0 + np.arange(n) * 1e-3
    sigma = rng.uniform(0.5e-3, 1.5e-3, n)
    y = 1.0 - 0.05 + sigma * rng.standard_normal(n)
    args = ([35, 60, 101], np.array([0.7, 1000.0]), getattr(_lib, pass_), "fp64", 200)
    c0, l0 = _search(t, y, sigma, *args)
    c1, l1 = _search(t, y, sigma * 2.0 ** -bits, *args)
    np.testing.assert_array_equal(c1, c0 * 4.0 ** bits)
    np.testing.assert_array_equal(l1, l0)
