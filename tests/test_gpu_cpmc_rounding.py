"""The CPMC one-body step divides a pivot row by its pivot with one rounding (not by a product with a rounded
reciprocal): the overlaps are those of the same elimination in exact rational arithmetic, rounded where the kernel
rounds."""

from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def determinant(c, w):
    n, o = c.shape
    s = [[0.0] * o for _ in range(o)]
    for i in range(o):
        for k in range(o):
            for p in range(n):
                s[i][k] = fma(float(c[p, i]), float(w[p, k]), s[i][k])
    det = 1.0
    for j in range(o):
        pr = max(range(j, o), key=lambda r: (abs(s[r][j]), -r))
        if pr != j:
            s[j], s[pr] = s[pr], s[j]
            det = -det
        pv = s[j][j]
        det *= pv
        s[j] = [x / pv for x in s[j]]
        for r in range(o):
            if r != j:
                f = s[r][j]
                s[r] = [fma(-f, x, y) for x, y in zip(s[j], s[r])]
    return det


def test_overlaps():
    import torch
    from cs_afqmc_gb300 import _lib
    from cs_afqmc_gb300._engine import stream_ptr

    n, no, nw = 9, (4, 3), 60
    rng = np.random.default_rng(5)
    mo = [np.linalg.qr(rng.standard_normal((n, n)))[0][:, :k] for k in no]
    w = [m[None] + 0.2 * rng.standard_normal((nw,) + m.shape) for m in mo]
    dev = [torch.as_tensor(np.ascontiguousarray(x), device="cuda") for x in mo + w]
    ovl = torch.empty(nw, dtype=torch.float64, device="cuda")
    greens = torch.empty((nw, 2, n, n), dtype=torch.float64, device="cuda")
    _lib.call("afq_cpmc_init", n, no[0], no[1], nw, *(x.data_ptr() for x in dev), ovl.data_ptr(), greens.data_ptr(), stream_ptr())
    want = [determinant(mo[0], w[0][i]) * determinant(mo[1], w[1][i]) for i in range(nw)]
    assert np.array_equal(ovl.cpu().numpy(), np.array(want))
