"""How the model chi2 and its gradient may be called: they do not wait for
their kernels, so they may be captured in a graph that outlives whatever the
context does afterwards, and may overlap on several streams.  And samples that
are not finite: chi2 and the whole gradient of their curve are NaN, in transit or out.

Bars: the same bits as the calls made alone; NaN where the model's own formula
gives it, the other curves' bits unchanged.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _set(C, n, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    f = dict(dtype=torch.float64, device="cuda")
    t = (100.0 + torch.arange(n, **f) * (2.0 / 1440.0)).repeat(C)
    y = 1.0 + 1e-3 * torch.randn(C * n, generator=g, **f)
    w = torch.full((C * n,), 1e6, **f)
    off = torch.arange(C + 1, device="cuda") * n
    p = torch.tensor([[2.3, 100.7, 0.11, 1.1e-3, 0.41, 0.23]], **f).repeat(C, 1)
    p[:, 1] += torch.linspace(0.0, 1.0, C, **f)
    return dict(t=t, y=y, w=w, off=off, p=p, C=C, chi2=torch.empty(C, **f), grad=torch.empty(C, 6, **f),
                one=torch.ones(C, **f))


def _call(ctx, s, stream):
    from gtls_b200 import _lib
    lib = _lib.load()
    ptr = [s[k].data_ptr() for k in ("t", "y", "w", "off")]
    rc = lib.gtls_model_chi2(ctx, *ptr, s["C"], s["p"].data_ptr(), s["chi2"].data_ptr(), stream)
    assert rc == 0, lib.gtls_last_error(ctx)
    rc = lib.gtls_model_chi2_grad(ctx, *ptr, s["C"], s["p"].data_ptr(), s["one"].data_ptr(), s["grad"].data_ptr(), stream)
    assert rc == 0, lib.gtls_last_error(ctx)


@pytest.fixture
def fresh(cuda):
    import torch
    from gtls_b200 import _lib
    h = ctypes.c_void_p()
    assert _lib.load().gtls_ctx_create(0, ctypes.byref(h)) == 0
    yield h
    torch.cuda.synchronize()
    assert _lib.load().gtls_ctx_destroy(h) == 0


def _alone(s):
    import torch
    from gtls_b200 import _lib
    _call(_lib.context(0), s, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return s["chi2"].clone(), s["grad"].clone()


@pytest.mark.parametrize("C,n", [(1, 3000), (40, 20000), (1500, 300)])
def test_captured_as_the_first_call_and_replayed_after_searches(fresh, C, n):
    import torch
    from gtls_b200 import _lib
    s = _set(C, n, 1)
    want = _alone(s)
    s["chi2"].zero_(), s["grad"].zero_()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        _call(fresh, s, torch.cuda.current_stream().cuda_stream)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(s["chi2"], want[0]) and torch.equal(s["grad"], want[1])
    # the context allocates and frees scratch; the parameters change in place
    out, cnt = torch.empty(4_000_000, dtype=torch.float64, device="cuda"), ctypes.c_int64()
    for points in (1000, 4_000_000):
        assert _lib.load().gtls_period_grid(fresh, 1e-9, 1e-3, points, 0.0, 1e9, out.data_ptr(), ctypes.byref(cnt),
                                            torch.cuda.current_stream().cuda_stream) == 0
    s["p"][:, 1] += 0.01
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    got = s["chi2"].clone(), s["grad"].clone()
    want = _alone(s)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    del g


def test_calls_overlap_on_two_streams_of_one_context(fresh):
    import torch
    sets = [_set(3, 20000, 2), _set(200, 5000, 3)]
    want = [_alone(s) for s in sets]
    streams = [torch.cuda.Stream() for _ in sets]
    for s in sets:
        s["chi2"].zero_(), s["grad"].zero_()
    torch.cuda.synchronize()
    for _ in range(20):
        for s, st in zip(sets, streams):
            _call(fresh, s, st.cuda_stream)
    torch.cuda.synchronize()
    for s, (c, gr) in zip(sets, want):
        assert torch.equal(s["chi2"], c) and torch.equal(s["grad"], gr)


@pytest.mark.parametrize("key,value", [("y", float("nan")), ("y", float("inf")), ("w", float("nan")), ("w", float("inf"))])
@pytest.mark.parametrize("sample", [0, 4999, 9999])   # of the second curve; all out of transit
def test_a_sample_that_is_not_finite_shows_in_the_gradient(cuda, key, value, sample):
    s = _set(3, 10000, 4)
    s["p"][:, 1] = 100.0 + 1.9
    q = ((s["t"][10000 + sample] - s["p"][1, 1]) / s["p"][1, 0]).item()
    assert abs(q - round(q)) * 2.3 > 0.11   # the sample lies outside every transit
    c0, g0 = _alone(s)
    s[key][10000 + sample] = value
    c1, g1 = _alone(s)
    assert g1[1].isnan().all() and not c1[1].isfinite()
    for i in (0, 2):
        assert c1[i] == c0[i] and (g1[i] == g0[i]).all()
