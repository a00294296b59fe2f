"""The model chi2 and its gradient at the sizes where their kernel changes its
way: samples of a step (128), of a warp's segment, of a round (12,288), curves
of one sample and of none, few curves (split over 64 CTAs) and many (one CTA
each), a transit that covers every sample, and a depth of 0.

Bars: chi2 within 1e-12 relative of the torch model, the gradient within 1e-6
relative of its autograd (as tests/test_adjoint.py), each gradient component's
floor 1e-12 of the sum of its terms' magnitudes.
"""
import numpy as np
import pytest

import adjoint_reference as AR

pytestmark = pytest.mark.gpu


def _curve(n, rng, P=2.3, D=0.11, depth=1.1e-3):
    t = 100.0 + np.sort(rng.uniform(0.0, max(1.0, n / 700.0), n))
    y = 1.0 + 1e-3 * rng.standard_normal(n)
    w = 1.0 / (1e-3 * rng.uniform(0.5, 1.5, n)) ** 2
    return t, y, w, [P, 100.0 + 0.3 * P, D, depth, 0.41, 0.23]


@pytest.mark.parametrize("lengths", [
    [1], [127, 128, 129], [1535, 0, 1537], [12287], [12289, 12288], [30001], [600] * 1200 + [5000],
])
def test_sizes(cuda, lengths):
    import torch
    from gtls_b200 import _lib
    rng = np.random.default_rng(sum(lengths) + len(lengths))
    shapes = [dict(), dict(P=0.9, D=0.44), dict(depth=0.0), dict(depth=0.2, D=0.3)]   # short, long, none, deep
    curves = [_curve(n, rng, **shapes[i % 4]) for i, n in enumerate(lengths)]
    up = lambda k: torch.from_numpy(np.concatenate([np.asarray(c[k], dtype=np.float64) for c in curves])).cuda()
    off = torch.from_numpy(np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)).cuda()
    params = torch.tensor([c[3] for c in curves], dtype=torch.float64)
    t, y, w = up(0), up(1), up(2)
    chi2 = _lib.model_chi2(t, y, w, off, params.cuda()).cpu().numpy()
    scale = torch.from_numpy(rng.uniform(0.5, 2.0, len(lengths)))
    grad = _lib.model_chi2_grad(t, y, w, off, params.cuda(), scale.cuda()).cpu().numpy() / scale.numpy()[:, None]
    for i in ([*range(8), len(lengths) - 1] if len(lengths) > 8 else range(len(lengths))):
        tt, yy, ww = (torch.from_numpy(np.asarray(a)) for a in curves[i][:3])
        if lengths[i] == 0:
            assert chi2[i] == 0.0 and not grad[i].any()
            continue
        if curves[i][3][3] == 0.0 or bool((AR.model(tt, params[i]) == 1).all()):   # no planet, or none in transit
            np.testing.assert_allclose(chi2[i], float((ww * (yy - 1) ** 2).sum()), rtol=1e-12)
            assert not grad[i].any()
            continue
        c, g = AR.autograd_grad(tt, yy, ww, params[i])
        np.testing.assert_allclose(chi2[i], float(c), rtol=1e-12)
        floor = 1e-12 * float((2 * ww * (yy - 1).abs()).sum()) * np.array([1e3, 1e3, 1e2, 1e2, 1.0, 1.0])
        assert np.all(np.abs(grad[i] - g.numpy()) <= 1e-6 * np.abs(g.numpy()) + floor), (i, grad[i], g)
