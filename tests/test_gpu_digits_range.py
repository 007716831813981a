"""The accumulators of the digit-sliced FP64 GEMM at the top of their range, against exact integers.

An operand is built from its digits, x = sum_j d_j 2^(-7-7j) with d_0 <= 128 and the others in [-64, 63], so that
the kernel's slicing gives these digits back. The kernel sums the products with i + j = c <= 7, in units of
2^(-14-7c): below 2^24 for c <= 5 over 512 terms, where FP32 sums are exact; c = 6 and 7 may pass that and
round. Sums above 2^22 take the epilogue's slow reading. More than 512 terms come in segments added in FP64."""

import numpy as np
import pytest

from tests.test_gpu_digits import run

pytestmark = pytest.mark.gpu

# the last digit a multiple of 8: 53 bits
LARGE = [127] + [63] * 6 + [56]
TOP = [128] + [0] * 6 + [-8]
LOW = [-127] + [-64] * 7
MIXED = [127, -64, 63, -64, 63, -64, 63, -64]


def value(d):
    q = sum(x << (49 - 7 * j) for j, x in enumerate(d))
    assert abs(q) <= 1 << 56 and float(q) == q
    return np.ldexp(float(q), -56)


def groups(a, b, k):
    """Sums of the products with i + j = c over k terms, as exact integers."""
    return [k * sum(a[i] * b[c - i] for i in range(max(0, c - 7), min(c, 7) + 1)) for c in range(15)]


def scaled(g, last):
    """sum_{c <= last} g_c 2^(-14-7c), in units of 2^-112."""
    return sum(x << (98 - 7 * c) for c, x in enumerate(g) if c <= last)


@pytest.mark.parametrize("tr", [16, 32, 64])
@pytest.mark.parametrize("k", [16, 480, 511, 512, 513, 1024, 1531])
@pytest.mark.parametrize("a,b", [(LARGE, LARGE), (LARGE, LOW), (LOW, LOW), (TOP, TOP), (TOP, LARGE), (MIXED, MIXED), (MIXED, LOW)],
                         ids=["large", "opposite", "low", "top", "top-large", "mixed", "mixed-low"])
def test_sums_at_the_top_of_the_range(a, b, k, tr):
    d = run(np.full((3, k), value(a)), np.full((5, k), value(b)), tr)
    assert np.all(d == d[0, 0])
    seg = min(k, 512)
    g = groups(a, b, seg)
    assert all(abs(x) <= 1 << 24 for x in g[:6])
    if seg >= 480 and (a, b) in ((LARGE, LARGE), (LOW, LOW), (TOP, TOP)):
        assert abs(g[0]) > 1 << 22  # the slow reading
    want = scaled(groups(a, b, k), 7)
    err = abs(int(np.ldexp(d[0, 0], 60)) * (1 << 52) - want)
    assert np.ldexp(d[0, 0], 60) == int(np.ldexp(d[0, 0], 60))
    # a rounding per segment and per sum of two, and one unit of 2^-56 (2^-63) for each of the tensor core's sums of
    # c = 6 (7): 7 (8) a block of 16 terms; none where these stay below 2^24
    nseg = -(-k // 512)
    limit = (2 * nseg - 1) * (abs(want) >> 53) + (1 << 40)
    if abs(g[6]) > 1 << 24 or abs(g[7]) > 1 << 24:
        limit += nseg * 32 * 8 * (1 << 56)
    assert err <= limit, (err, limit)
