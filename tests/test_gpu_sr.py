"""Comb resampling over population sizes around the scan's limits (serial sums below 256 walkers, 32 elements ahead of the
chunks, chunks of 1024, sums in shared or, above 5888, global memory) and weights that try its roundings: the new
weight and the indices are those of numpy.cumsum, bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def weights(kind, nw):
    rng = np.random.default_rng(nw)
    w = rng.uniform(0.6, 1.4, nw)
    if kind == "equal":  # every element at the same distance from a half
        w[:] = 1.0 + 2.0 ** -50 + 2.0 ** -52
    elif kind == "halves":  # few bits: halves wherever the sums have grown past the last one
        w = rng.integers(1, 8, nw) * 2.0 ** -44 + 1.0 + rng.integers(0, 2, nw) * 2.0 ** -52
    elif kind == "killed":  # zeros, also in front
        w[rng.random(nw) < 0.4] = 0.0
        w[:40] = 0.0
    elif kind == "wide":
        w = np.exp(rng.uniform(-60.0, 60.0, nw))
    elif kind == "steep":  # each element larger than the sum of the earlier ones, up to the last octave
        w = 2.0 ** -np.minimum(np.arange(nw)[::-1], 90.0) * rng.uniform(1.0, 2.0, nw)
    elif kind == "negative":
        w *= rng.choice([-1.0, 1.0], nw)
    elif kind == "infinite":
        w[nw // 2] = np.inf
    return w


@pytest.mark.parametrize("nw", [1, 33, 127, 128, 129, 255, 256, 257, 1055, 1056, 1057, 2048, 5888, 5889, 6144, 6145, 9000])
@pytest.mark.parametrize("kind", ["random", "equal", "halves", "killed", "wide", "steep", "negative", "infinite"])
def test_indices_and_weight_of_numpy_cumsum(kind, nw):
    import torch

    from tests.helpers import Case, to_np

    case = Case(kind="rhf", norb=2, nelec=(1, 1), nchol=2, nw=nw, restricted=True, precision="fp64", seed=1)
    w = weights(kind, nw)
    pg = case.gpu_prop_data()
    pg["weights"].copy_(torch.as_tensor(w))
    zeta = 0.37
    pg = case.prop.stochastic_reconfiguration_local(pg, case.trial, case.ham_data, case.wave_data, zeta=np.array([zeta]))
    cum = np.cumsum(np.abs(w))
    new = to_np(pg["weights"])
    with np.errstate(invalid="ignore"):
        assert np.array_equal(new, np.full(nw, cum[-1] / nw))
        z = cum[-1] * (np.arange(nw) + zeta) / nw
        expected = np.minimum(np.searchsorted(cum, z), nw - 1)
    if kind != "infinite":
        assert np.array_equal(to_np(pg["sr_indices"]), expected)
