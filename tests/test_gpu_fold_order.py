"""The fold order where its rounds and its bucket sorts can go wrong: index
words of 17 to 20 bits, curves at the edges of those, and periods that are
multiples of the cadence, whose buckets hold from 31 to thousands of samples.
Bit for bit np.argsort(phase, kind="stable") of foldFast's phases
(GPUFun.py:30-41)."""
import numpy as np
import pytest

import tls_oracle as O

pytestmark = pytest.mark.gpu


def _times(kind, n, rng):
    cad = 2.0 / 1440.0
    if kind == "from_zero":        # the first turn's phases are finer than the later ones'
        return np.arange(n) * cad, cad
    if kind == "binary":           # exact phases: clusters of equal ones
        return 3.0 + np.arange(n) * 2.0 ** -9, 2.0 ** -9
    if kind == "repeated":         # equal times, out of order
        return rng.permutation(np.repeat(50.0 + np.arange((n + 3) // 4) * cad, 4)[:n]), cad
    return 1300.0 + np.sort(rng.uniform(0.0, n * cad, n)), cad


@pytest.mark.parametrize("kind", ["from_zero", "binary", "repeated", "irregular"])
@pytest.mark.parametrize("n", [33, 3001, 32769, 131072, 131073, 160001, 524289, 1048575, 1048576])
def test_order_of_clustered_and_long_curves(cuda, n, kind):
    import torch
    from gtls_b200 import _lib
    rng = np.random.default_rng(n)
    t, cad = _times(kind, n, rng)
    span = n * cad
    P = [span / 7.3, span / 41.9 + cad / 3]
    if n < 1048576:   # whole turns of 31 to 65 samples a phase, and of hundreds
        P += [cad * max(2, n // k) for k in (31, 32, 33, 64, 65, 400)]
        P += [cad * (n // 33 + 1) * (1.0 + 1e-10), cad * (n // 200 + 1) * (1.0 - 3e-9)]
    P = np.array(P)
    got = _lib.fold_order(torch.from_numpy(t).cuda(), torch.from_numpy(P).cuda()).cpu().numpy()
    for i, p in enumerate(P):
        np.testing.assert_array_equal(got[i], np.argsort(O.fold_phases(t, p), kind="stable"), err_msg="period %r" % p)
