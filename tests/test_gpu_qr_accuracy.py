"""Distance of the FP64 QR's Q from the exact one (extended precision on the host), root mean square over
the elements. The bounds are those of Householder sums by 32 lanes a column with every reflector's scale
to one or two roundings; seeds and sizes are fixed, so that the figures repeat."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

X = np.clongdouble


def exact_q(a):
    a = a.astype(X)
    nw, m, k = a.shape
    vs, taus = [], []
    for j in range(k):
        x = a[:, j:, j]
        norm = np.sqrt(np.sum(x.real ** 2 + x.imag ** 2, 1))
        alpha = x[:, 0].copy()
        beta = np.where(alpha.real >= 0, -norm, norm).astype(X)
        v = x / (alpha - beta)[:, None]
        v[:, 0] = 1
        tau = (beta - alpha) / beta
        a[:, j:, j:] -= (np.conj(tau)[:, None] * v)[:, :, None] * np.einsum("wr,wrc->wc", np.conj(v), a[:, j:, j:])[:, None]
        vs.append(v)
        taus.append(tau)
    q = np.broadcast_to(np.eye(m, k, dtype=X), a.shape).copy()
    for j in reversed(range(k)):
        v = vs[j]
        q[:, j:, j:] -= (taus[j][:, None] * v)[:, :, None] * np.einsum("wr,wrc->wc", np.conj(v), q[:, j:, j:])[:, None]
    return q


@pytest.mark.parametrize("norb,n_el,nw,bound", [(60, 10, 100, 2.72e-16), (60, 28, 40, 3.78e-16)])
def test_q_is_as_near_as_with_plain_sums(norb, n_el, nw, bound):
    from tests.helpers import Case, to_np

    case = Case(kind="rhf", norb=norb, nelec=(n_el, n_el), nchol=12, nw=nw, restricted=True, precision="fp64",
                orthonormal=True, perturb=0.03, seed=norb)
    rng = np.random.default_rng(n_el)
    w = case.walkers0 + 0.1 * (rng.standard_normal(case.walkers0.shape) + 1j * rng.standard_normal(case.walkers0.shape)) / 2 ** 0.5
    pg = case.gpu_prop_data()
    pg["walkers"] = case.gpu_walkers(w)
    before = to_np(pg["walkers"])
    q = to_np(case.prop.orthonormalize_walkers(pg)["walkers"]).astype(X)
    ref = exact_q(before)
    err = np.sqrt(np.sum(np.abs(q - ref) ** 2) / np.sum(np.abs(ref) ** 2))
    assert float(err) < bound, float(err)
