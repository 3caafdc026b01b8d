"""The one-launch LU panel and the interchanges that follow it against the
oracle, bit for bit: every shape of the recursion, rows at the edges of a
CTA's and a cluster's share, ties, zeros, NaN and infinities in the pivot
search, tiny pivots."""
import numpy as np
import pytest

from tests.oracle_lib import rand, same_bits, first_diff

pytestmark = pytest.mark.gpu


def check(hb, orc, p, m, n, a, lda, recursive=False):
    a1, a2 = a.copy(order="F"), a.copy(order="F")
    p1, p2 = np.zeros(min(m, n), np.int32), np.zeros(min(m, n), np.int32)
    name = f"{p}getrf{'2' if recursive else ''}"
    i1 = getattr(hb, name)(m, n, a1, lda, p1)
    i2 = getattr(orc, name)(m, n, a2, lda, p2)
    assert i1 == i2
    assert np.array_equal(p1, p2), np.flatnonzero(p1 != p2)[:4]
    assert same_bits(a1, a2), first_diff(a1, a2)


@pytest.mark.parametrize("p", ["d", "s"])
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 32, 33, 47, 52, 63, 64])
@pytest.mark.parametrize("m", [64, 65, 256, 257, 700])
def test_panel_widths(hb, orc, p, m, n):
    rng = np.random.default_rng(m * 100 + n)
    check(hb, orc, p, m, n, rand(rng, m + 1, n, np.float64 if p == "d" else np.float32), m + 1,
          recursive=True)


@pytest.mark.parametrize("p,m", [("d", 2048), ("d", 2816), ("d", 2817), ("d", 5632), ("d", 5633),
                                 ("s", 4096), ("s", 4097), ("s", 8192), ("s", 8193)])
def test_panel_heights(hb, orc, p, m):
    """Full clusters of 8 and 16 CTAs, and one row more."""
    rng = np.random.default_rng(m)
    check(hb, orc, p, m, 64, rand(rng, m, 64, np.float64 if p == "d" else np.float32), m)


@pytest.mark.parametrize("p", ["d", "s"])
@pytest.mark.parametrize("m,n", [(300, 300), (1000, 1000), (700, 130), (130, 700), (500, 500)])
def test_ties_and_zeros(hb, orc, p, m, n):
    """Entries -1, 0, 1: most pivot searches end in a tie, many columns become
    zero (INFO, no interchange)."""
    rng = np.random.default_rng(m + n)
    a = rng.integers(-1, 2, (m, n)).astype(np.float64 if p == "d" else np.float32)
    a[:, 5] = a[:, 3]
    check(hb, orc, p, m, n, np.asfortranarray(a), m)


@pytest.mark.parametrize("p", ["d", "s"])
@pytest.mark.parametrize("m", [40, 600])
@pytest.mark.parametrize("place", ["first", "middle", "all"])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_special_values(hb, orc, p, m, place, value):
    rng = np.random.default_rng(m)
    a = rand(rng, m, 36, np.float64 if p == "d" else np.float32)
    rows = {"first": [0], "middle": [m // 2], "all": list(range(m))}[place]
    a[rows, 20] = value
    check(hb, orc, p, m, 36, a, m)


@pytest.mark.parametrize("p", ["d", "s"])
def test_tiny_pivots(hb, orc, p):
    rng = np.random.default_rng(3)
    t = np.float64 if p == "d" else np.float32
    a = rand(rng, 400, 64, t)
    a *= t(np.finfo(t).tiny)
    check(hb, orc, p, 400, 64, a, 400)


@pytest.mark.parametrize("p", ["d", "s"])
@pytest.mark.parametrize("m,n", [(65, 64), (128, 97), (1000, 1003), (2900, 700), (300, 2000)])
def test_blocked(hb, orc, p, m, n):
    rng = np.random.default_rng(m + 3 * n)
    check(hb, orc, p, m, n, rand(rng, m + 5, n, np.float64 if p == "d" else np.float32), m + 5)
