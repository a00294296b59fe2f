"""The scratch budget of a search is one: a single period of a long curve
takes no more than it (a small search is cut into many ranges of starts, each with
lists of its own, where there is room for them), and what it finds does not
depend on it.

Bars: the context's scratch at most the budget, an eighth and 2 MB (how it
grows) and the curve's own arrays; chi2 and locations bit for bit.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def curve(cuda):
    from test_gpu_bounds import _case
    widths = [40, 100, 300, 1000, 1407, 1409, 3000, 8400]
    return _case(70000, widths, seed=9)


def _scratch(curve, budget, pass_, precision):
    """(chi2, loc, bytes of scratch) of one period in a context of its own."""
    import torch
    from gtls_b200 import _lib
    t, y, dy, widths, tm, ov, maxd = curve
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to("cuda:0")
    args = (dict(t=up(t), y=up(y), dy=up(dy), span=float(np.float32(t.max() - t.min()))), up(np.array([1.7])),
            dict(widths=up(widths), overshoot=up(ov), templates=up(tm), max_width=maxd), 1e-5, 8, 1,
            getattr(_lib, pass_), precision)
    _lib.search(*args, flags=_lib.GTLS_SEARCH_ALL_DURATIONS)   # torch's own memory and the kernels are in place
    h = ctypes.c_void_p()
    assert _lib.load().gtls_ctx_create(0, ctypes.byref(h)) == 0
    saved = _lib._ctxs[0]
    _lib._ctxs[0] = h
    try:
        if budget:
            _lib.set_chunk_budget(budget)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        c, l = _lib.search(*args, flags=_lib.GTLS_SEARCH_ALL_DURATIONS)
        torch.cuda.synchronize()
        used = before - torch.cuda.mem_get_info()[0]
        return c.cpu().numpy(), l.cpu().numpy(), used
    finally:
        _lib._ctxs[0] = saved
        assert _lib.load().gtls_ctx_destroy(h) == 0


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("pass_", ["GTLS_PASS_MAIN", "GTLS_PASS_ALL"])
def test_one_period_of_a_long_curve_stays_within_the_budget(curve, pass_, precision):
    from gtls_b200 import _lib
    n, widths, maxd = len(curve[0]), curve[3], curve[6]
    pair = 24 if precision == "fp64" else 16
    least = 8 * n + (n + maxd + 1) * pair
    own = 16 * n + 16 * int(widths.sum()) + 64 * 200 * len(widths) + (1 << 16)   # (v, w), template rows, cells, the rest
    c0, l0, _ = _scratch(curve, 0, pass_, precision)
    for budget in (least, 2 * least):
        c, l, used = _scratch(curve, budget, pass_, precision)
        np.testing.assert_array_equal(c, c0)
        np.testing.assert_array_equal(l, l0)
        assert used <= (budget + own) * 9 / 8 + (2 << 20), (used, budget, own)
    with pytest.raises(_lib.GtlsError):
        _scratch(curve, least - 1, pass_, precision)
