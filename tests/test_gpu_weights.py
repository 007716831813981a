"""Weights and population control over the population sizes where their kernels change: one launch on a cluster of
eight blocks (uneven shares, one to four warps a block) up to 1024 walkers, two launches above, against the
oracle's step."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw", [1, 7, 8, 9, 255, 256, 257, 520, 1023, 1024, 1025])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_weights_and_shift(nw, precision):
    from tests.helpers import Case, rel_err, to_np

    case = Case(kind="rhf", norb=6, nelec=(2, 2), nchol=5, nw=nw, restricted=True, precision=precision, seed=3)
    fields = np.random.default_rng(nw).standard_normal((nw, 5))
    po = case.o_prop.propagate(case.o_trial, case.o_ham, case.oracle_prop_data(), fields, case.sys.mo_coeff)
    pg = case.prop.propagate(case.trial, case.ham_data, case.gpu_prop_data(), fields, case.wave_data)
    tol = 1e-9 if precision == "fp64" else 2e-4
    weights = to_np(pg["weights"])
    assert rel_err(weights, po["weights"]) < tol
    # the shift from the weights as they are: sums of up to 1025 terms, one logarithm
    shift = to_np(pg["e_estimate"]) - 0.1 * np.log(np.sum(weights) / nw) / case.dt
    assert abs(pg["pop_control_ene_shift"].item() - shift) < 1e-10 * max(1.0, abs(shift))
