"""Workspace of FP64 contexts (no GPU): what the options leave out, and what a population costs."""

import ctypes
import os

import pytest

from cs_afqmc_gb300 import _lib

pytestmark = pytest.mark.skipif(not os.path.exists(_lib.LIB_PATH), reason="library not built")


def size(norb, nocc, nchol, nw, option=0, uhf=0):
    d = _lib.Dims(norb=norb, n_up=nocc, n_dn=nocc, nchol=nchol, n_walkers=nw, walker_type=uhf, trial_type=uhf,
                  precision=_lib.AFQ_PREC_FP64, n_exp_terms=6, n_batch=1, mixed_config=option, dt=0.005)
    n = _lib.load().afq_workspace_size(ctypes.byref(d))
    assert n > 0
    return n


def digits(rows, k):
    return 16 * rows * k


@pytest.mark.parametrize("norb,nocc,nchol", [(20, 5, 100), (60, 10, 300), (120, 20, 600), (198, 33, 990)])
@pytest.mark.parametrize("nw", [1, 4, 50, 256])
def test_options(norb, nocc, nchol, nw):
    full, measure, units = (size(norb, nocc, nchol, nw, o) for o in (0, _lib.FP64_MEASURE, _lib.FP64_UNITS))
    assert units < measure < full
    # the walkers' arrays alone: vhs, G, the fields and biases, the walkers, the energies' partial sums
    arrays = 16 * nw * (norb * norb + nocc * norb + 2 * nchol + norb * nocc + 5 * ((nchol + 15) // 16) + 16)
    assert units < arrays + 20 * 256
    assert full - measure > digits(norb * norb, nchol)


def test_one_walker_needs_no_exchange_matrix():
    chol, rot, u = digits(198 * 198, 990), digits(990, 198 * 33), digits(198 * 33, 198 * 33)
    assert size(198, 33, 990, 1) < 1.1 * (chol + rot)
    assert size(198, 33, 990, 1, _lib.FP64_MEASURE) < 1.2 * rot
    assert size(198, 33, 990, 4) > chol + rot + u


def test_forming_the_exchange_matrix_takes_no_room_of_its_own():
    """Its scratch lies where the walkers' is: nothing above the operands and the walkers' arrays."""
    nw, norb, nocc, nchol = 256, 198, 33, 990
    kept = digits(norb * norb, nchol) + digits(nchol, norb * nocc) + digits(norb * nocc, norb * nocc)
    # per walker: vhs, its digits for 152 walkers, columns, arrays
    walkers = nw * (16 * norb * norb + 64 * norb * nocc + 32 * 2 * nchol + 32 * 2 * nocc * norb) + 152 * 32 * 256 * 1.7 * norb
    assert size(norb, nocc, nchol, nw) < 1.05 * kept + walkers
