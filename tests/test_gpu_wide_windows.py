"""Windows that the CTA sums together: widths around the split (1,024), around
the samples in shared memory at a time (4,096) and beyond two of those, on a
curve with dips (their windows overlap) and on one where every start ties
(windows far apart, many more than are summed together).

Bars: FP64 chi2 within 1e-9 relative of the FP64 oracle, identical locations
where the minimum is unique, and the same bits with and without neighbours.
"""
import numpy as np
import pytest

import tls_oracle as O
from test_gpu_bounds import _case, _search

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("n,widths", [
    (9001, [1024, 1025, 1031, 1409]),
    (20000, [1025, 2049, 4095, 4096, 4097, 4480]),
    (26001, [3000, 8191, 8192, 8193, 9000]),
    (28500, [4095, 4096, 4097, 4200]),      # all of them valid at P = 0.61: at most 0.15 n
    (56001, [8191, 8192, 8193]),
])
def test_wide_windows_match_the_oracle(cuda, n, widths, flat):
    t, y, dy, widths, tm, ov, maxd = _case(n, widths, seed=n, dy=not flat, flat=flat)
    P = np.array([0.61, 1.7, 3.4])
    c, l = _search(t, y, dy, widths, tm, ov, P, False, "fp64", 1)
    c_ref, l_ref = O.search_periods(O.NumpyBackend(), P, t, y, dy, widths, tm, ov, maxd, 1e-5, 8, 1)
    assert np.isfinite(c[0])
    np.testing.assert_allclose(c, c_ref, rtol=1e-9)
    if not flat:
        np.testing.assert_array_equal(l, l_ref)
    for i, p in enumerate(P):
        one, lone = _search(t, y, dy, widths, tm, ov, np.array([p]), False, "fp64", 1)
        assert one[0] == c[i] or np.isnan([one[0], c[i]]).all()   # no valid duration: NaN
        assert flat or lone[0] == l[i]


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("n,durations", [(8300, 190), (8300, 200), (3000, 64)])
def test_blocks_of_all_starts_match_the_oracle(cuda, n, durations, flat):
    """All starts of 64 to 200 durations: blocks of one and of two durations
    (the table holds 192 of 128 blocks), and with every start tying more blocks
    than are taken up at a time."""
    t, y, dy, widths, tm, ov, maxd = _case(n, list(range(9, 9 + durations)), seed=n, dy=not flat, flat=flat)
    P = np.array([1.7])
    c_ref, l_ref = O.search_periods(O.NumpyBackend(), P, t, y, dy, widths, tm, ov, maxd, 1e-5, 8, 1, noskip=True)
    for precision, rtol in (("fp64", 1e-9), ("fp32", 2e-6)):
        c, l = _search(t, y, dy, widths, tm, ov, P, True, precision, 1)
        np.testing.assert_allclose(c, c_ref, rtol=rtol)
        if precision == "fp64" and not flat:
            np.testing.assert_array_equal(l, l_ref)


@pytest.mark.parametrize("n,widths", [(14500, [2047, 2048, 2049]), (28500, [2000, 4095, 4097, 4200])])
def test_wide_chains_of_all_starts_match_the_oracle(cuda, n, widths):
    """FP32, every start: the blocks' chains over samples in shared memory
    (2,048 at a time), and the same bits with and without neighbours."""
    t, y, dy, widths, tm, ov, maxd = _case(n, widths, seed=n)
    P = np.array([0.61, 0.7])
    c, _ = _search(t, y, dy, widths, tm, ov, P, True, "fp32", 1)
    c_ref, _ = O.search_periods(O.NumpyBackend(), P, t, y, dy, widths, tm, ov, maxd, 1e-5, 8, 1, noskip=True)
    assert np.isfinite(c).all()
    np.testing.assert_allclose(c, c_ref, rtol=2e-6)
    for i, p in enumerate(P):
        assert _search(t, y, dy, widths, tm, ov, np.array([p]), True, "fp32", 1)[0][0] == c[i]
