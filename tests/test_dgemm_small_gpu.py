"""Small FP64 products (staged tiles, KC chunks over a cluster) against the
oracle, bit for bit: edges of the 32 x 32 tiles, of the 64-deep slabs and of the
256-deep chunks, either order of each operand, any alignment, signed zeros."""
import numpy as np
import pytest

from tests.oracle_lib import rand, same_bits, first_diff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta", ["N", "T"])
@pytest.mark.parametrize("tb", ["N", "T"])
@pytest.mark.parametrize("m,n,k,pad", [
    (1, 1, 1, 0), (31, 33, 63, 1), (32, 32, 64, 0), (33, 47, 65, 2), (64, 8, 255, 0),
    (40, 70, 256, 3), (65, 31, 257, 0), (3, 200, 511, 1), (64, 64, 513, 0), (33, 35, 2049, 1),
    (20, 20, 5000, 0), (300, 1, 3000, 0), (256, 256, 256, 0), (64, 96, 2560, 0),
    # Either side of the lines for a long k: two to eight chunks a CTA.
    (128, 100, 4096, 1), (128, 100, 4097, 1), (40, 33, 6144, 1), (40, 33, 6145, 1),
    (31, 1, 8192, 0), (31, 1, 8193, 0), (1, 32, 10240, 1), (2, 40, 10241, 0), (8, 8, 16384, 0),
    (8, 8, 16385, 0), (16, 32, 17000, 2), (31, 16, 17000, 0), (64, 1, 33000, 0),
])
def test_dgemm_small_bitexact(hb, orc, ta, tb, m, n, k, pad):
    rng = np.random.default_rng(m + 7 * n + 11 * k)
    ra, ca = (m, k) if ta == "N" else (k, m)
    rb, cb = (k, n) if tb == "N" else (n, k)
    a, b, c = rand(rng, ra + pad, ca), rand(rng, rb + pad, cb), rand(rng, m + pad, n)
    for alpha, beta in ((1.5, 0.3), (-1.0, 1.0), (1.0, 0.0)):
        c1, c2 = c.copy(order="F"), c.copy(order="F")
        if beta == 0.0:
            c1[:m], c2[:m] = np.nan, np.nan  # C is not read
        hb.dgemm(ta, tb, m, n, k, alpha, a, ra + pad, b, rb + pad, beta, c1, m + pad)
        orc.dgemm(ta, tb, m, n, k, alpha, a, ra + pad, b, rb + pad, beta, c2, m + pad)
        assert same_bits(c1, c2), (alpha, beta, first_diff(c1, c2))


@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("n,k", [(33, 20), (64, 700), (100, 64), (64, 2100)])
def test_dsyrk_small_bitexact(hb, orc, uplo, n, k):
    rng = np.random.default_rng(n + k)
    a, c = rand(rng, n, k), rand(rng, n, n)
    for beta in (1.0, 0.3):
        c1, c2 = c.copy(order="F"), c.copy(order="F")
        hb.dsyrk(uplo, "N", n, k, -1.0, a, n, beta, c1, n)
        orc.dsyrk(uplo, "N", n, k, -1.0, a, n, beta, c2, n)
        assert same_bits(c1, c2), first_diff(c1, c2)


def test_dgemm_small_negative_zero(hb, orc):
    """Products that underflow to -0: the padding of k must not turn them into +0."""
    m, n, k = 5, 6, 3
    a = np.full((m, k), -1e-200, order="F")
    b = np.full((k, n), 1e-200, order="F")
    c1, c2 = np.zeros((m, n), order="F"), np.zeros((m, n), order="F")
    hb.dgemm("N", "N", m, n, k, 1.0, a, m, b, k, 0.0, c1, m)
    orc.dgemm("N", "N", m, n, k, 1.0, a, m, b, k, 0.0, c2, m)
    assert np.array_equal(np.signbit(c1), np.signbit(c2))
