"""QR of the walker slabs over the sizes where the kernel's split changes: electrons around the multiples of
4 (columns per lane), rows around one warp's share and several warps, and FP64 slabs of the same sizes and larger,
against numpy's Householder QR."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# FP32: 64 rows a warp, 4 columns a lane. FP64: a warp per slab.
FP64 = [(2, 1, 1), (3, 3, 2), (5, 4, 4), (64, 3, 1), (65, 4, 3), (40, 7, 6), (64, 12, 9), (65, 11, 5), (56, 13, 13), (57, 16, 14),
        (48, 17, 20), (49, 20, 18), (40, 21, 24), (41, 24, 24), (32, 25, 28), (33, 29, 32), (48, 33, 36), (73, 40, 37),
        (192, 36, 36), (193, 36, 33), (60, 41, 44), (400, 8, 7)]
MIXED = [(2, 1, 1), (7, 5, 4), (64, 8, 8), (65, 9, 7), (64, 16, 13), (128, 20, 20), (64, 28, 28), (66, 32, 31), (129, 33, 33),
         (150, 36, 35), (170, 40, 37), (256, 10, 12)]


@pytest.mark.parametrize("precision,norb,n_up,n_dn", [("fp64", *s) for s in FP64] + [("mixed", *s) for s in MIXED])
def test_qr(precision, norb, n_up, n_dn):
    from tests.helpers import Case, to_np

    case = Case(kind="uhf", norb=norb, nelec=(n_up, n_dn), nchol=3 + norb // 6, nw=5, restricted=False, precision=precision,
                orthonormal=False, perturb=0.3, seed=norb + n_up)
    eps = np.finfo(np.float64 if precision == "fp64" else np.float32).eps
    pg = case.gpu_prop_data()
    before = [to_np(x).astype(np.complex128) for x in pg["walkers"]]
    pg = case.prop.orthonormalize_walkers(pg)
    for w, q in zip(before, pg["walkers"]):
        q, k = to_np(q).astype(np.complex128), w.shape[2]
        # rounding of k reflectors; Q itself is as sensitive as W's condition number
        tol = 4 * (k + 2) * eps
        gram = np.einsum("wpi,wpj->wij", q.conj(), q)
        assert np.max(np.abs(gram - np.eye(k))) < tol
        for a, b in zip(w, q):
            assert np.max(np.abs(np.linalg.qr(a)[0] - b)) < tol * np.linalg.cond(a)
