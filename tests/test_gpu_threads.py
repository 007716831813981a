"""Contexts of different sizes driven from two host threads: the dynamic shared memory that a kernel may take is a
property of the function, shared by the threads, and none may lower it between another's setting and launch."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_small_context_does_not_lower_the_limit():
    from cs_afqmc_gb300 import _lib
    from tests.helpers import Case

    large, small = (Case(kind="rhf", restricted=True, norb=n, nelec=(o, o), nchol=g, nw=nw)
                    for n, o, g, nw in ((40, 13, 32, 70), (9, 2, 7, 3)))
    lib = _lib.load()
    large.trial.calc_force_bias(large.gpu_walkers(), large.ham_data, large.wave_data)
    before = lib.afq_test_digits_smem_limit()
    small.trial.calc_force_bias(small.gpu_walkers(), small.ham_data, small.wave_data)
    assert lib.afq_test_digits_smem_limit() >= before > 0


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_two_threads_of_different_sizes(precision):
    import torch
    from tests.helpers import Case, to_np

    sizes = [dict(norb=9, nelec=(2, 2), nchol=7, nw=3), dict(norb=40, nelec=(13, 13), nchol=80, nw=70)]
    cases = [Case(kind="rhf", restricted=True, precision=precision, **s) for s in sizes]
    walkers = [c.gpu_walkers() for c in cases]

    def call(c, w):
        return c.trial.calc_energy(w, c.ham_data, c.wave_data)

    want = [to_np(call(c, w)) for c, w in zip(cases, walkers)]
    torch.cuda.synchronize()
    got, errors = [[], []], []
    start = threading.Barrier(2)

    def run(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait()
                for _ in range(1000):
                    e = call(cases[k], walkers[k])
                got[k] = to_np(e)
        except Exception as e:  # noqa: BLE001 (reported below)
            errors.append(repr(e))

    threads = [threading.Thread(target=run, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
