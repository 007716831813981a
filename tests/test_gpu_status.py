"""A wait of an FP64 tensor-core contraction that runs out is reported by every call that contracts on them:
in scalars[AFQ_S_STATUS] where there is a state, as NaN where there is none. The guard word is set by hand."""

import numpy as np
import pytest

from cs_afqmc_gb300 import _lib

pytestmark = pytest.mark.gpu

BIT = 8


def preset(eng):
    from cs_afqmc_gb300._engine import stream_ptr

    _lib.call("afq_test_preset_status", eng.ctx, BIT, stream_ptr())


def system():
    from tests.helpers import Case

    case = Case(kind="uhf", norb=11, nelec=(4, 2), nchol=23, nw=6, restricted=False)
    pg = case.gpu_prop_data()
    return case, pg, case.prop._engine(case.trial, case.ham_data, case.wave_data, pg["walkers"])


def status(pg):
    return int(pg["_scalars"].cpu()[_lib.AFQ_S_STATUS])


def field_block(case, pg, samp, f):
    from cs_afqmc_gb300 import corr_sample
    import torch

    two = case.gpu_prop_data()
    sums = torch.empty(4, dtype=torch.float64, device="cuda")
    corr_sample.cs_block_scan(pg, case.ham_data, case.prop, case.trial, case.wave_data, two, case.ham_data, case.prop,
                              case.trial, case.wave_data, samp, fields=f, sums=sums)


CALLS = {
    "step": lambda c, pg, s, f, z: c.prop.propagate(c.trial, c.ham_data, pg, f[0, 0, 0], c.wave_data),
    "block": lambda c, pg, s, f, z: s.propagate_phaseless(c.ham, c.ham_data, c.prop, pg, c.trial, c.wave_data, fields=f, zetas=z),
    "pair": lambda c, pg, s, f, z: field_block(c, pg, s, f),
    "jvp": lambda c, pg, s, f, z: s.propagate_phaseless_ad_norot_jvp(c.ham, c.ham_data, np.eye(c.norb), c.prop, pg, c.trial,
                                                                     c.wave_data, fields=f, zetas=z),
    "vjp": lambda c, pg, s, f, z: s.propagate_phaseless_ad_norot_vjp(c.ham, c.ham_data, c.prop, pg, c.trial, c.wave_data,
                                                                     fields=f, zetas=z),
    "free step": lambda c, pg, s, f, z: c.prop.propagate_free(c.trial, c.ham_data, pg, f[0, 0, 0], c.wave_data),
    "free": lambda c, pg, s, f, z: s.propagate_free(c.ham, c.ham_data, c.prop, pg, c.trial, c.wave_data, fields=f[0]),
}


@pytest.mark.parametrize("bits", [0, BIT])
@pytest.mark.parametrize("call", list(CALLS))
def test_state_reports_it(call, bits):
    import torch
    from cs_afqmc_gb300 import sampling

    case, pg, eng = system()
    rng = np.random.default_rng(3)
    f = torch.as_tensor(rng.standard_normal((1, 1, 2, case.nw, case.nchol)), device="cuda")
    z = torch.as_tensor(rng.random(1), device="cuda")
    if bits:
        preset(eng)
    CALLS[call](case, pg, sampling.sampler(n_prop_steps=2, n_ene_blocks=1, n_sr_blocks=1, n_blocks=1), f, z)
    assert status(pg) == bits


def test_measurements_are_nan():
    from cs_afqmc_gb300 import _engine
    from tests.helpers import to_np

    case, pg, _ = system()
    w = pg["walkers"]
    eng = _engine.engine_for(case.trial, case.ham_data, case.wave_data, w)
    calls = [case.trial.calc_force_bias, case.trial.calc_energy]
    assert all(np.all(np.isfinite(to_np(c(w, case.ham_data, case.wave_data)))) for c in calls)
    preset(eng)
    assert all(np.all(np.isnan(to_np(c(w, case.ham_data, case.wave_data)))) for c in calls)
