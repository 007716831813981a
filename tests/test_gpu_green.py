"""Green's function and overlap kernels over the electron counts where their code changes: every padded
size (multiples of 4), one warp for two slabs up to 16 electrons, one or two matrix rows per
lane, several block passes of S, against numpy in FP64."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def setup(norb, n_up, n_dn, nw, restricted, precision):
    from tests.helpers import Case

    kind = "rhf" if n_up == n_dn else "uhf"
    return Case(kind=kind, norb=norb, nelec=(n_up, n_dn), nchol=norb + 3, nw=nw, restricted=restricted,
                precision=precision, orthonormal=True, perturb=0.3, seed=norb + n_up)


def expected(case):
    mo = case.sys.mo_coeff
    mos = mo if isinstance(mo, list) else [mo, mo]
    ws = case.walkers0 if isinstance(case.walkers0, list) else [case.walkers0]
    ovl, green = 1.0, []
    for w, c in zip(ws, mos):
        s = np.einsum("pi,wpk->wik", c[:, : w.shape[2]], w)
        ovl = ovl * np.linalg.det(s)
        green.append(np.einsum("wpk,wki->wip", w, np.linalg.inv(s)))
    if len(ws) == 1:
        ovl = ovl * ovl
    rc = case.o_ham["rot_chol"]
    rcs = rc if isinstance(rc, list) else [rc] * len(green)
    fb = sum(np.einsum("gip,wip->wg", r, g) for r, g in zip(rcs, green))
    return ovl, fb * (2 if len(ws) == 1 else 1)


SIZES = [(5, 1, 1), (9, 4, 4), (13, 5, 3), (17, 8, 8), (23, 12, 9), (33, 16, 16), (34, 17, 2), (41, 20, 20), (47, 23, 22),
         (50, 24, 24), (58, 28, 27), (66, 32, 32)]


@pytest.mark.parametrize("restricted", [True, False], ids=["one-slab", "two-slab"])
@pytest.mark.parametrize("norb,n_up,n_dn", SIZES + [(70, 33, 33), (84, 40, 40)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_green_and_overlap(norb, n_up, n_dn, restricted, precision):
    from tests.helpers import rel_err, to_np

    if restricted and n_up != n_dn:
        pytest.skip("restricted walkers have equal spins")
    if precision == "mixed" and n_up > 32:
        norb = 130  # the mixed path takes more than 32 electrons per spin above 128 orbitals
    case = setup(norb, n_up, n_dn, 5, restricted, precision)
    w = case.gpu_walkers()
    ovl = to_np(case.trial.calc_overlap(w, case.wave_data))
    fb = to_np(case.trial.calc_force_bias(w, case.ham_data, case.wave_data))
    o, f = expected(case)
    # S^-1 amplifies rounding by its condition number (some 1e2 to 1e3 for these perturbed walkers)
    tol = 1e-10 if precision == "fp64" else 2e-4
    assert np.max(np.abs(ovl - o) / np.abs(o)) < tol
    assert rel_err(fb, f) < tol


def test_singular_and_non_finite_walkers_stay_their_own():
    """A walker orthogonal to the trial, one of zeros, one with a NaN: no other walker changes."""
    from tests.helpers import to_np

    case = setup(20, 5, 5, 6, True, "fp64")
    good = to_np(case.trial.calc_overlap(case.gpu_walkers(), case.wave_data))
    w = case.walkers0.copy()
    w[1] = 0.0
    w[3, 2, 1] = np.nan
    w[4] = np.linalg.svd(case.sys.mo_coeff)[0][:, 5:10]
    got = to_np(case.trial.calc_overlap(case.gpu_walkers(w), case.wave_data))
    keep = [0, 2, 5]
    assert np.array_equal(got[keep], good[keep])
    assert not np.abs(got[1]) > 0 and np.isnan(got[3]) and not np.abs(got[4]) > 1e-20
