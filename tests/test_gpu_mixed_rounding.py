"""The order and the rounding of the mixed path's FP32 sums (Green's function elimination, QR).

Resampling compares sums of weights with the comb's teeth, so an FP32 rounding in a walker's overlap can
exchange a whole walker. The overlaps and Q are therefore compared with the same sums in the same order
on the CPU, bit for bit, not within a tolerance: an element of S and a column sum over the rows in
their order, the pivot row divided before the others take multiples of it."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32
W = np.longdouble  # a product of two FP32 numbers and its sum with a third


def fma(a, b, c):
    return (np.asarray(a, F).astype(W) * np.asarray(b, F).astype(W) + np.asarray(c, F).astype(W)).astype(F)


def mul(a, b):
    return fma(a[0], b[0], -(a[1] * b[1])), fma(a[0], b[1], a[1] * b[0])


def sub(a, b):
    return a[0] - b[0], a[1] - b[1]


def parts(w):
    return np.ascontiguousarray(w.real.astype(F)), np.ascontiguousarray(w.imag.astype(F))


def determinant(c, w, widest):
    """det(C^T W) of every walker as the elimination rounds it; the product of the pivots in FP64."""
    n, o = c.shape
    c, (wx, wy), nw = c.astype(F), parts(w), w.shape[0]
    s = [np.zeros((nw, o, o), F), np.zeros((nw, o, o), F)]
    for p in range(n):
        s = [fma(c[p][None, :, None], x[:, p, None, :], t) for x, t in zip((wx, wy), s)]
    mask = np.uint32(31 if widest <= 32 else 63)  # row index in the low bits of the pivot key
    used, rows, piv, at = np.zeros((nw, o), bool), [], [], np.arange(nw)
    for j in range(o):
        mag = np.abs(s[0][:, :, j]) + np.abs(s[1][:, :, j])
        key = (mag.view(np.uint32) & ~mask) | (mask - np.arange(o, dtype=np.uint32))
        key[used] = 0
        pr = key.argmax(1)
        used[at, pr] = True
        rows.append(pr)
        px, py = s[0][at, pr, j], s[1][at, pr, j]
        piv.append(px.astype(np.float64) + 1j * py)
        _, ex = np.frexp(np.maximum(np.abs(px), np.abs(py)))
        x, y = np.ldexp(px, -ex), np.ldexp(py, -ex)
        d = np.ldexp((W(1) / fma(x, x, y * y).astype(W)).astype(F), -ex)
        inv = (x * d, -y * d)
        row = mul((s[0][at, pr], s[1][at, pr]), (inv[0][:, None], inv[1][:, None]))
        row[0][:, j], row[1][:, j] = inv
        f = s[0][:, :, j, None].copy(), s[1][:, :, j, None].copy()
        s[0][:, :, j] = 0
        s[1][:, :, j] = 0
        s = list(sub(s, mul(f, (row[0][:, None], row[1][:, None]))))
        s[0][at, pr], s[1][at, pr] = row
    rows = np.array(rows).T
    sign = np.array([(-1) ** sum(x > y for i, x in enumerate(r) for y in r[i + 1:]) for r in rows])
    return sign * np.prod(np.array(piv), 0)


@pytest.mark.parametrize("norb,n_up,n_dn", [(6, 2, 1), (9, 5, 4), (20, 8, 7), (33, 12, 9), (50, 16, 13), (64, 20, 17),
                                            (65, 24, 21), (64, 28, 25), (70, 32, 31), (130, 33, 29), (140, 40, 37)])
def test_overlaps_round_as_sums_in_order(norb, n_up, n_dn):
    from tests.helpers import Case, to_np

    case = Case(kind="uhf", norb=norb, nelec=(n_up, n_dn), nchol=5, nw=6, restricted=False, precision="mixed",
                orthonormal=True, perturb=0.1, seed=norb)
    ovl = to_np(case.trial.calc_overlap(case.gpu_walkers(), case.wave_data))
    want = 1.0
    for c, w in zip(case.sys.mo_coeff, case.walkers0):
        want = want * determinant(np.asarray(c)[:, : w.shape[2]], w.astype(np.complex64), max(n_up, n_dn))
    # the pivots are the same numbers; 70 FP64 products of them
    assert np.max(np.abs(ovl - want) / np.abs(want)) < 70 * 2.3e-16


def lanes_sum(x, y, lanes, ascending):
    """Sums of rows r, r + lanes, .. and then the shuffle tree over the lanes."""
    nw, m, nc = x.shape
    out = []
    for v in (x, y):
        s = np.zeros((nw, lanes, nc), F)
        for r in range(m):
            s[:, r % lanes] += v[:, r]
        offs = [1 << i for i in range(lanes.bit_length() - 1)]
        for o in offs if ascending else offs[::-1]:
            s = s + s[:, np.arange(lanes) ^ o]
        out.append(s[:, 0])
    return out


def column_sums(x, y, j, by_warp):
    k = x.shape[2]
    lanes = 1 if by_warp else 32
    while by_warp and 2 * lanes * (k - j - 1) <= 32:
        lanes *= 2
    ax, ay, bx, by = x[:, j:, j + 1:], y[:, j:, j + 1:], x[:, j:, j:j + 1], y[:, j:, j:j + 1]
    return lanes_sum(fma(ax, bx, ay * by), fma(ay, bx, -(ax * by)), lanes, by_warp)


def norm2(a, by_warp):
    """The squares below the diagonal: a float pair over 32 lanes, or FP64 over a block's threads."""
    nw, m = a.shape
    if not by_warp:
        v = np.zeros((nw, 8, 32))
        v.reshape(nw, 256)[:, :m] = a
        for o in (16, 8, 4, 2, 1):
            v = v + v[:, :, np.arange(32) ^ o]
        t = np.zeros((nw, 32))
        t[:, :8] = v[:, :, 0]
        for o in (16, 8, 4, 2, 1):
            t = t + t[:, np.arange(32) ^ o]
        return t[:, 0].astype(F)
    h, l = np.zeros((nw, 32), F), np.zeros((nw, 32), F)
    for i in range(m):
        c = i % 32
        s = h[:, c] + a[:, i]
        b = s - h[:, c]
        l[:, c] += (h[:, c] - (s - b)) + (a[:, i] - b)
        h[:, c] = s
    for o in (16, 8, 4, 2, 1):
        at = np.arange(32) ^ o
        s = h + h[:, at]
        b = s - h
        l, h = l + (l[:, at] + ((h - (s - b)) + (h[:, at] - b))), s
    return (h + l)[:, 0]


def update(x, y, j, f, sums):
    v, (sx, sy) = (x[:, j:, j:j + 1], y[:, j:, j:j + 1]), sums
    sx, sy = sx[:, None], sy[:, None]
    p = mul((f[0][:, None, None], f[1][:, None, None]), (fma(v[0], sx, -(v[1] * sy)), fma(v[1], sx, v[0] * sy)))
    x[:, j:, j + 1:] -= p[0]
    y[:, j:, j + 1:] -= p[1]


def householder_q(w, by_warp):
    x, y = parts(w)
    nw, m, k = x.shape
    taus = []
    for j in range(k):
        xn = norm2(fma(x[:, j + 1:, j], x[:, j + 1:, j], y[:, j + 1:, j] * y[:, j + 1:, j]), by_warp)
        ax, ay = x[:, j, j].copy(), y[:, j, j].copy()
        n2 = np.sqrt(fma(ax, ax, ay * ay) + xn)
        b = np.where(ax >= 0, -n2, n2)
        t = ((b - ax) / b, -ay / b)
        dx = ax - b  # 1 / (alpha - b), |Re| >= |Im|; the block's divisor is rounded twice
        r = ay / dx
        den = fma(ay, r, dx) if by_warp else dx + ay * r
        scale = F(1) / den, -r / den
        x[:, j + 1:, j], y[:, j + 1:, j] = mul((x[:, j + 1:, j], y[:, j + 1:, j]), (scale[0][:, None], scale[1][:, None]))
        x[:, j, j], y[:, j, j] = 1, 0
        taus.append(t)
        if j < k - 1:
            update(x, y, j, (t[0], -t[1]), column_sums(x, y, j, by_warp))
    for j in reversed(range(k)):
        t = taus[j]
        x[:, j, j], y[:, j, j] = 1, 0
        if j < k - 1:
            update(x, y, j, t, column_sums(x, y, j, by_warp))
        vx, vy, tx, ty = x[:, j + 1:, j].copy(), y[:, j + 1:, j].copy(), t[0][:, None], t[1][:, None]
        x[:, j + 1:, j], y[:, j + 1:, j] = fma(ty, vy, -(tx * vx)), fma(-ty, vx, -(tx * vy))
        x[:, j, j], y[:, j, j] = F(1) - t[0], -t[1]
        x[:, :j, j] = 0
        y[:, :j, j] = 0
    return x + 1j * y


# above 32 columns, or where four slabs do not fit a block's shared memory, a block takes a slab, and the second one too
@pytest.mark.parametrize("norb,n_up,n_dn", [(2, 1, 1), (9, 5, 1), (20, 3, 2), (40, 12, 9), (64, 28, 17), (90, 32, 16),
                                            (130, 33, 4), (170, 40, 37), (256, 17, 27), (140, 30, 35)])
def test_qr_rounds_as_sums_in_order(norb, n_up, n_dn):
    from tests.helpers import Case, to_np

    case = Case(kind="uhf", norb=norb, nelec=(n_up, n_dn), nchol=5, nw=6, restricted=False, precision="mixed",
                orthonormal=False, perturb=0.3, seed=norb)
    pg = case.gpu_prop_data()
    before = [to_np(w) for w in pg["walkers"]]
    pg = case.prop.orthonormalize_walkers(pg)
    for w, q in zip(before, pg["walkers"]):
        k = w.shape[2]
        by_warp = all(j <= 32 and 32 * (norb * (j | 1) + 64) <= 227 * 1024 for j in (n_up, k))
        assert np.array_equal(householder_q(w, by_warp), to_np(q)), k
