"""A Hamiltonian or trial changed in place between two calls: contexts hold copies of it, and the second call has to
see the new values."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def copied(x):
    return [copied(y) for y in x] if isinstance(x, (list, tuple)) else x.clone() if hasattr(x, "clone") else x


def fresh(case):
    return {k: copied(v) for k, v in case.ham_data.items() if not k.startswith("_")}


def step(case, ham):
    from tests.helpers import to_np

    pg = case.gpu_prop_data()
    f = np.random.default_rng(2).standard_normal((case.nw, case.nchol))
    pg = case.prop.propagate(case.trial, ham, pg, f, case.wave_data)
    w = pg["walkers"]
    return [to_np(x) for x in ([w] if not isinstance(w, list) else w) +
            [pg["weights"], case.trial.calc_force_bias(w, ham, case.wave_data), case.trial.calc_energy(w, ham, case.wave_data)]]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("what", ["chol", "rot_chol", "exp_h1"])
@pytest.mark.parametrize("kind", ["rhf", "uhf"])
def test_changed_in_place(kind, what, precision):
    import torch
    from tests.helpers import Case

    nelec = (4, 4) if kind == "rhf" else (4, 2)
    case = Case(kind=kind, norb=11, nelec=nelec, nchol=23, nw=6, restricted=kind == "rhf", precision=precision,
                orthonormal=True, perturb=0.1)
    ham = case.ham_data
    ham["chol"] = torch.as_tensor(np.asarray(ham["chol"].cpu() if hasattr(ham["chol"], "cpu") else ham["chol"]), device="cuda").clone()
    before = step(case, ham)
    x = ham[what]
    for t in x if isinstance(x, (list, tuple)) else [x]:
        t.mul_(1.01)
    after = step(case, ham)
    want = step(case, fresh(case))
    assert any(not np.array_equal(a, b) for a, b in zip(before, after))
    for a, b in zip(after, want):
        assert np.array_equal(a, b)
    again = step(case, ham)
    assert all(np.array_equal(a, b) for a, b in zip(after, again))
    assert len(ham["_afq_engines"]) <= 2  # the stale ones are gone
