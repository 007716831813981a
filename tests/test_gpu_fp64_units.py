"""The two forms of the FP64 contractions, digit products on the tensor cores (default) and sums on the FP64
units (ham_data["fp64_units"]): the error each promises on graded operands, and that whole calls agree where
the digit plans change (walkers in chunks, sums in several segments, batches, non-finite walkers)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def units(case):
    """A copy of the case's Hamiltonian that asks for the FP64 units."""
    return {**{k: v for k, v in case.ham_data.items() if not k.startswith("_")}, "fp64_units": True}


@pytest.mark.parametrize("grade", [0, 20, 40])
def test_force_bias_of_graded_operands(grade):
    """One electron and the first orbital as trial make G[p] = W[p] / W[0]; its elements fall by 2^-grade while the
    Cholesky rows rise by as much, so that every term of a sum counts."""
    import torch
    from cs_afqmc_gb300 import wavefunctions
    from tests.helpers import to_np

    n, nchol, nw = 64, 40, 9
    rng = np.random.default_rng(grade)
    fall = np.ldexp(1.0, -np.round(grade * np.arange(n) / (n - 1)).astype(int))
    w = (rng.standard_normal((nw, n, 1)) + 1j * rng.standard_normal((nw, n, 1))) * fall[:, None]
    w[:, 0] = 1.0
    rc = rng.standard_normal((nchol, 1, n)) * fall[::-1]
    mo = np.eye(n)[:, :1]
    trial = wavefunctions.rhf(n, (1, 1))
    dev = lambda x: torch.as_tensor(np.ascontiguousarray(x), device="cuda")  # noqa: E731
    ham = {"h0": 0.0, "h1": dev(np.zeros((2, n, n))), "chol": dev(np.zeros((nchol, n * n))), "rot_chol": dev(rc),
           "rot_h1": dev(np.zeros((1, n)))}
    x, y = w[:, :, 0], rc[:, 0]
    terms = 2 * x.astype(np.clongdouble)[:, None, :] * y[None]
    want, size = terms.sum(-1), np.abs(terms).sum(-1)
    fb = to_np(trial.calc_force_bias(dev(w), {**ham, "fp64_units": True}, {"mo_coeff": dev(mo)}))
    # n roundings of a sum, and those of G
    assert np.all(np.abs(fb - want) <= (n + 8) * 2.0 ** -53 * size)
    fb = to_np(trial.calc_force_bias(dev(w), ham, {"mo_coeff": dev(mo)}))
    # remainders of 2^-57 of a row's largest element and products left out below 7 2^-58, a part each of a complex
    # number; the rounding of the result, and those of G
    top = np.abs(x).max(1)[:, None] * np.abs(y).max(1)[None]
    assert np.all(np.abs(fb - want) <= 8 * 2.0 ** -53 * size + 2 * 2 * n * (2 * 2.0 ** -57 + 7 * 2.0 ** -58) * 4 * top)


# name: case, what it reaches
PLANS = {
    "chunks above 128 orbitals": dict(kind="rhf", restricted=True, norb=130, nelec=(4, 4), nchol=36, nw=160),
    "chunks up to 64 orbitals": dict(kind="uhf", restricted=False, norb=60, nelec=(2, 1), nchol=16, nw=1300),
    "V cotangents in two segments, stacked": dict(kind="uhf", restricted=False, norb=40, nelec=(28, 27), nchol=30, nw=12),
    "V cotangents in two segments": dict(kind="uhf", restricted=False, norb=70, nelec=(30, 26), nchol=30, nw=6),
    "batches": dict(kind="uhf", restricted=False, norb=66, nelec=(9, 8), nchol=60, nw=48, n_batch=2),
    "steps on the units, reverse mode on digits": dict(kind="uhf", restricted=False, norb=20, nelec=(5, 4), nchol=24, nw=400),
    "derivatives on digits": dict(kind="rhf", restricted=False, norb=28, nelec=(7, 7), nchol=24, nw=30),
    "all on digits from 200 slabs on": dict(kind="uhf", restricted=False, norb=33, nelec=(7, 6), nchol=30, nw=100),
    "all on digits, few walkers": dict(kind="rhf", restricted=True, norb=47, nelec=(12, 12), nchol=30, nw=3),
    "one walker": dict(kind="rhf", restricted=False, norb=33, nelec=(6, 6), nchol=50, nw=1),
}


def close(a, b, tol):
    a, b = np.asarray(a), np.asarray(b)
    assert np.array_equal(np.isfinite(a), np.isfinite(b))
    ok = np.isfinite(b)
    top = np.max(np.abs(b[ok]), initial=0.0)
    assert np.max(np.abs(a[ok] - b[ok]), initial=0.0) <= tol * top


def draws(case, steps):
    import torch

    rng = np.random.default_rng(case.nw)
    f = torch.as_tensor(rng.standard_normal((1, 1, steps, case.nw, case.nchol)), device="cuda")
    return f, torch.as_tensor(rng.random(1), device="cuda")


def run(case, ham, call, steps, walkers=None):
    from cs_afqmc_gb300 import sampling
    from tests.helpers import to_np

    pg = case.gpu_prop_data()
    if walkers is not None:
        pg["walkers"] = case.gpu_walkers(walkers)
    samp = sampling.sampler(n_prop_steps=steps, n_ene_blocks=1, n_sr_blocks=1, n_blocks=1)
    f, z = draws(case, steps)
    args = (case.ham, ham)
    rest = (case.prop, pg, case.trial, case.wave_data)
    out = []
    if call == "block":
        e, pg = samp.propagate_phaseless(*args, *rest, fields=f, zetas=z)
        out = [e]
    elif call == "jvp":
        op = np.diag(np.linspace(-1.0, 1.0, case.norb))
        e, de, pg = samp.propagate_phaseless_ad_norot_jvp(*args, op, *rest, fields=f, zetas=z)
        out = [e, de]
    else:
        e, rdm1, pg = samp.propagate_phaseless_ad_norot_vjp(*args, *rest, fields=f, zetas=z)
        out = [e, rdm1]
    w = pg["walkers"]
    return [np.asarray(to_np(x)) for x in out + [pg["weights"], pg["overlaps"]] + (w if isinstance(w, list) else [w])]


@pytest.mark.parametrize("call", ["block", "jvp", "vjp"])
@pytest.mark.parametrize("plan", list(PLANS))
def test_both_forms_agree(plan, call):
    from tests.helpers import Case

    case = Case(orthonormal=True, perturb=0.05, **PLANS[plan])
    for a, b in zip(run(case, case.ham_data, call, 2), run(case, units(case), call, 2)):
        close(a, b, 1e-10)


def test_free_projection_and_measurements_agree():
    from cs_afqmc_gb300 import sampling
    from tests.helpers import Case, to_np

    case = Case(kind="uhf", restricted=False, norb=60, nelec=(9, 8), nchol=50, nw=30, orthonormal=True, perturb=0.05)
    samp = sampling.sampler(n_prop_steps=2, n_ene_blocks=1, n_sr_blocks=1, n_blocks=2)
    f = np.random.default_rng(1).standard_normal((2, 2, case.nw, case.nchol))
    got = []
    for ham in (case.ham_data, units(case)):
        pg, be, bw, _ = samp.propagate_free(case.ham, ham, case.prop, case.gpu_prop_data(), case.trial, case.wave_data, fields=f)
        w = pg["walkers"]
        got.append([to_np(x) for x in (be, bw, pg["norms"], pg["normed_overlaps"], w[0], w[1],
                                       case.trial.calc_energy(w, ham, case.wave_data),
                                       case.trial.calc_force_bias(w, ham, case.wave_data))])
    for a, b in zip(*got):
        close(a, b, 1e-10)


@pytest.mark.parametrize("call", ["block", "jvp", "vjp"])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_a_walker_that_is_not_finite(bad, call):
    """Its weight falls to 0 in both forms, and nothing else differs between them."""
    from tests.helpers import Case

    case = Case(kind="uhf", restricted=False, norb=66, nelec=(9, 8), nchol=60, nw=40, orthonormal=True, perturb=0.05)
    w = [x.copy() for x in case.walkers0]
    w[0][7, 3, 2] = bad
    for a, b in zip(run(case, case.ham_data, call, 2, w), run(case, units(case), call, 2, w)):
        close(a, b, 1e-10)
