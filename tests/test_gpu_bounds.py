"""The chi2 minimum with ruled-out starts against the oracle, at the sizes
where the kernel changes its way: batches of 2,688 samples, widths of the
sample ring (1,407) and the coarse prefix, windows summed by one warp or by the
CTA (1,024), the skips of 32, blocks of 64 starts in the all-starts pass, and
a curve on which every start ties (the list of starts overflows).

Bars: FP64 chi2 within 1e-9 relative of the FP64 oracle and identical argmin
(duration, start) locations; FP32 chi2 within 2e-6 relative.
"""
import numpy as np
import pytest

import tls_oracle as O

pytestmark = pytest.mark.gpu


def _case(n, widths, seed=0, depth=2e-3, dy=True, flat=False):
    rng = np.random.default_rng(seed)
    t = 10.0 + np.arange(n) * (20.0 / n)
    sigma = rng.uniform(0.5e-3, 1.5e-3, n) if dy else np.full(n, 1e-3)
    y = 1.0 + (0.0 if flat else 1.0) * sigma * rng.standard_normal(n)
    if flat:
        y -= 1e-3
    else:
        y[((t - 10.3) % 1.7) < 0.12] -= depth
    widths = np.array([w for w in widths if w <= n], dtype=np.int32)
    maxd = int(widths.max()) + int(widths.max()) % 2
    tm = np.ones((len(widths), maxd))
    for d, w in enumerate(widths):
        x = np.linspace(-1, 1, w) if w > 1 else np.zeros(1)
        tm[d, :w] = 0.5 * np.sqrt(np.clip(1 - 0.99 * x * x, 0, None)) ** 0.5
    ov = np.full(len(widths), 1.07)
    return t, y, sigma / sigma.mean(), widths, tm, ov, maxd


def _search(t, y, dy, widths, tm, ov, P, all_, precision, batch):
    import torch
    from gtls_b200 import _lib
    dev = torch.device("cuda:0")
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    curve = dict(t=up(t), y=up(y), dy=up(dy), span=float(np.float32(t.max() - t.min())))
    tables = dict(widths=up(widths), overshoot=up(ov), templates=up(tm), max_width=tm.shape[1])
    c, l = _lib.search(curve, up(P), tables, 1e-5, 8, batch, _lib.GTLS_PASS_ALL if all_ else _lib.GTLS_PASS_MAIN,
                       precision)
    return c.cpu().numpy(), l.cpu().numpy()


@pytest.mark.parametrize("all_", [False, True])
@pytest.mark.parametrize("n,widths", [
    (40, [1, 2, 3, 5]),
    (2687, [17, 31, 32, 33, 127, 128, 129, 300]),
    (2689, [16, 64, 255, 256, 257, 400]),
    (5376, [40, 63, 65, 511, 513, 640]),
    (12288, [150, 1023, 1024, 1025, 1406, 1407, 1500]),
    (13003, [200, 1407, 1408, 1409, 1700]),
])
def test_minimum_and_location_match_the_oracle(cuda, n, widths, all_):
    t, y, dy, widths, tm, ov, maxd = _case(n, widths, seed=n, dy=n % 2 == 1)
    P = np.array([0.61, 0.85, 1.7, 3.4])[: 2 if all_ and n > 6000 else 4]
    c, l = _search(t, y, dy, widths, tm, ov, P, all_, "fp64", 4)
    c_ref, l_ref = O.search_periods(O.NumpyBackend(), P, t, y, dy, widths, tm, ov, maxd, 1e-5, 8, 4, noskip=all_)
    np.testing.assert_allclose(c, c_ref, rtol=1e-9)
    np.testing.assert_array_equal(l, l_ref)
    c32, _ = _search(t, y, dy, widths, tm, ov, P, all_, "fp32", 4)
    np.testing.assert_allclose(c32, c_ref, rtol=2e-6)


@pytest.mark.parametrize("all_,n", [(False, 12288), (True, 2689)])
def test_every_start_ties(cuda, all_, n):
    t, y, dy, widths, tm, ov, maxd = _case(n, [16, 17, 18, 19, 20, 22, 24, 200, 300], dy=False, flat=True)
    P = np.array([0.61, 1.7])
    c, _ = _search(t, y, dy, widths, tm, ov, P, all_, "fp64", 1)
    c_ref, _ = O.search_periods(O.NumpyBackend(), P, t, y, dy, widths, tm, ov, maxd, 1e-5, 8, 1, noskip=all_)
    np.testing.assert_allclose(c, c_ref, rtol=1e-9)
