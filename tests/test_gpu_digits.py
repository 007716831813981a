"""The digit-sliced FP64 GEMM (afq_test_gemm_digits) against extended-precision products.

Bound, from the slicing alone: with 2^e >= max|row|, each operand's remainder is at most
2^-57 2^e per element (two of them: 2^-56), and the digit products left out (i + j >= 8) sum to
at most 7 * 64 * 64 * 2^-70 (1 + 2^-6) < 2^-55 per term, so |error| <= K 2^(ea + eb) 2^-54 plus
half an ulp of the result.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(a, b, tr):
    import torch

    from cs_afqmc_gb300 import _lib
    from cs_afqmc_gb300._engine import stream_ptr

    m, k = a.shape
    n = b.shape[0]
    ta, tb = (torch.as_tensor(np.ascontiguousarray(x), device="cuda") for x in (a, b))
    d = torch.full((m, n), 7.0, dtype=torch.float64, device="cuda")
    ws = torch.empty(_lib.load().afq_test_gemm_digits_bytes(m, n, k, tr), dtype=torch.uint8, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.call("afq_test_gemm_digits", ta.data_ptr(), tb.data_ptr(), d.data_ptr(), m, n, k, tr, ws.data_ptr(),
              status.data_ptr(), stream_ptr())
    torch.cuda.synchronize()
    assert status.item() == 0
    return d.cpu().numpy()


def longdouble_product(a, b):
    out = np.zeros((a.shape[0], b.shape[0]), dtype=np.longdouble)
    al, bl = a.astype(np.longdouble), b.astype(np.longdouble)
    for k in range(a.shape[1]):
        out += al[:, k][:, None] * bl[:, k][None, :]
    return out


def bound(a, b, ref):
    def scale(x):
        return np.exp2(np.frexp(np.abs(x).max(1))[1].astype(np.float64))

    return a.shape[1] * np.outer(scale(a), scale(b)) * 2.0 ** -54 + np.abs(ref).astype(np.float64) * 2.0 ** -52


@pytest.mark.parametrize("tr", [16, 32, 48, 64])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (128, 128, 16), (129, 130, 17), (300, 257, 513), (64, 200, 1100)])
def test_against_extended_precision(m, n, k, tr):
    rng = np.random.default_rng(m + n + k)
    a, b = rng.standard_normal((m, k)), rng.standard_normal((n, k))
    a *= np.exp2(rng.integers(-40, 40, m))[:, None]          # rows of any size
    b *= np.exp(-12.0 * np.arange(k) / k)[None, :]           # falling along K, as Cholesky vectors
    ref = longdouble_product(a, b)
    assert np.all(np.abs(run(a, b, tr) - ref) <= bound(a, b, ref))


@pytest.mark.parametrize("tr", [16, 32, 64])
def test_extreme_digits_are_exact(tr):
    """Every digit at its largest with one sign: the accumulators reach their bound."""
    k = 512
    digits = np.float64(sum((128 if j == 0 else 63) * 2.0 ** (-7 - 7 * j) for j in range(7)) - 2.0 ** -40)
    a, b = np.full((3, k), digits * 0.999), np.full((5, k), digits * 0.999)
    ref = longdouble_product(a, b)
    assert np.all(np.abs(run(a, b, tr) - ref) <= bound(a, b, ref))
    ones = run(np.ones((3, k)), np.ones((5, k)), tr)
    assert np.array_equal(ones, np.full((3, 5), float(k)))


@pytest.mark.parametrize("tr", [48, 64])
def test_zeros_tiny_huge_and_non_finite_rows(tr):
    rng = np.random.default_rng(3)
    a, b = rng.standard_normal((6, 40)), rng.standard_normal((7, 40))
    a[1] = 0.0
    a[2] *= 2.0 ** -1000
    a[3] *= 1e300
    a[4, 7] = np.nan
    a[5, 3] = np.inf
    b[2] *= 2.0 ** -1060  # denormals
    b[3] = 0.0
    d = run(a, b, tr)
    ok = [0, 1, 2, 3]
    ref = longdouble_product(a[ok], b)
    lim = bound(a[ok], b, ref) + 5e-324
    with np.errstate(over="ignore"):
        assert np.all(np.abs(d[ok] - ref.astype(np.float64)) <= lim)
    assert np.all(np.isnan(d[4:])) and not np.any(np.isnan(d[:4]))
    assert np.all(d[1] == 0.0) and np.all(d[:4, 3] == 0.0)


def test_error_against_a_plain_fp64_sum():
    """Not further from the exact product than FP64 arithmetic, over the library's K range."""
    for k in (40, 256, 600, 2400):
        rng = np.random.default_rng(k)
        a, b = rng.standard_normal((64, k)), rng.standard_normal((48, k))
        ref = longdouble_product(a, b)
        plain = np.zeros((64, 48))
        for i in range(k):  # one FP64 accumulator per element, as a scalar loop
            plain += a[:, i][:, None] * b[:, i][None, :]
        err = lambda x: float(np.sqrt(np.mean((x - ref).astype(np.float64) ** 2)))  # noqa: E731
        assert err(run(a, b, 64)) <= err(plain), k


# Sizes just above the line where the Taylor products go to the digit GEMM (nw * columns * norb^2 >=
# 1e6); with the walkers in four chunks (n_batch) the same call stays on the FP64 units.
ROUTES = [
    dict(kind="rhf", restricted=True, norb=33, nelec=(6, 6), nchol=40, nw=160),     # one slab, ragged
    dict(kind="uhf", restricted=False, norb=33, nelec=(6, 5), nchol=40, nw=88),     # two slabs, unequal
    dict(kind="rhf", restricted=False, norb=64, nelec=(3, 3), nchol=50, nw=44),     # tile edge, few columns
    dict(kind="uhf", restricted=False, norb=65, nelec=(9, 2), nchol=60, nw=24),     # past the stacked form
    dict(kind="rhf", restricted=True, norb=48, nelec=(24, 24), nchol=60, nw=20),    # a 48-column tile
    dict(kind="uhf", restricted=False, norb=50, nelec=(24, 20), nchol=60, nw=16),   # two column tiles
    dict(kind="rhf", restricted=True, norb=130, nelec=(33, 33), nchol=140, nw=4),   # two row and column tiles
    dict(kind="uhf", restricted=False, norb=128, nelec=(20, 19), nchol=130, nw=4),
]


def route_case(cfg, n_batch):
    from tests.helpers import Case

    case = Case(precision="fp64", n_batch=n_batch, orthonormal=True, perturb=0.05, **cfg)
    return case, case.gpu_prop_data()


def draws(case, n_prop):
    rng = np.random.default_rng(9)
    return rng.standard_normal((1, 1, n_prop, case.nw, case.nchol)), rng.uniform(size=1)


def close(x, y, tol=1e-11):
    from tests.helpers import rel_err, to_np

    if isinstance(x, (list, tuple)):
        return all(close(a, b, tol) for a, b in zip(x, y))
    return rel_err(to_np(x), to_np(y)) < tol


def ids(c):
    return f"{c['kind']}{'r' if c['restricted'] else 'u'}-n{c['norb']}"


# Both routes round each product to FP64: relative differences are some 1e-15 per step, far
# below 1e-11 after two of them.
@pytest.mark.parametrize("cfg", ROUTES, ids=ids)
def test_block_routes_agree(cfg):
    from cs_afqmc_gb300 import sampling

    out = []
    for n_batch in (1, 4):
        case, pd = route_case(cfg, n_batch)
        f, z = draws(case, 2)
        e, pd = sampling.sampler(2, 1, 1).propagate_phaseless(case.ham, case.ham_data, case.prop, pd, case.trial,
                                                              case.wave_data, fields=f, zetas=z)
        out.append((e, pd["walkers"], pd["weights"], pd["overlaps"]))
    assert close(out[0], out[1])


@pytest.mark.parametrize("mode", ["jvp", "vjp"])
@pytest.mark.parametrize("cfg", ROUTES[:6], ids=ids)
def test_derivative_routes_agree(cfg, mode):
    from cs_afqmc_gb300 import sampling

    out = []
    for n_batch in (1, 4):
        case, pd = route_case(cfg, n_batch)
        f, z = draws(case, 2)
        s = sampling.sampler(2, 1, 1)
        args = (case.prop, pd, case.trial, case.wave_data)
        if mode == "jvp":
            op = np.random.default_rng(4).standard_normal((case.norb, case.norb))
            e, d, pd = s.propagate_phaseless_ad_norot_jvp(case.ham, case.ham_data, op + op.T, *args, fields=f, zetas=z)
        else:
            e, d, pd = s.propagate_phaseless_ad_norot_vjp(case.ham, case.ham_data, *args, fields=f, zetas=z)
        out.append((e, d, pd["walkers"], pd["weights"]))
    assert close(out[0], out[1])


@pytest.mark.parametrize("cfg", [
    dict(kind="rhf", restricted=True, norb=17, nelec=(3, 3), nchol=3, nw=5),     # U form, ragged
    dict(kind="rhf", restricted=False, norb=22, nelec=(5, 5), nchol=4, nw=70),
    dict(kind="uhf", restricted=False, norb=21, nelec=(4, 1), nchol=3, nw=6),
    dict(kind="uhf", restricted=False, norb=29, nelec=(4, 3), nchol=4, nw=6),    # too few vectors: sums over f_g
], ids=["u-restricted", "u-two-slab", "u-uhf", "sums"])
def test_energy_forms_against_the_oracle(cfg):
    """Both forms of the local energy at the line between them (norb = 7 nchol)."""
    from tests.helpers import rel_err, to_np

    case, pd = route_case(cfg, 1)
    e = to_np(case.trial.calc_energy(pd["walkers"], case.ham_data, case.wave_data))
    w = [x.copy() for x in case.walkers0] if isinstance(case.walkers0, list) else case.walkers0
    assert rel_err(e, case.o_trial.energy(w, case.o_ham, case.sys.mo_coeff)) < 1e-11
