"""Cholesky blocks, triangular base solves and the complex LU panel against the
oracle, bit for bit, at the edges of their tiles."""
import numpy as np
import pytest

from tests.oracle_lib import rand, same_bits, first_diff

pytestmark = pytest.mark.gpu
REAL = {"d": np.float64, "s": np.float32}


@pytest.mark.parametrize("p", ["d", "s"])
@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("n", [1, 2, 7, 31, 32, 33, 40, 63, 64, 65, 150])
@pytest.mark.parametrize("bad", [None, 0, "half", "last"])
def test_potrf_blocks(hb, orc, p, uplo, n, bad):
    rng = np.random.default_rng(n)
    g = rand(rng, n, n)
    a = (g @ g.T / n + np.eye(n)).astype(REAL[p])
    if bad is not None:
        i = {"half": n // 2, "last": n - 1}.get(bad, bad)
        a[i, i] = np.nan if n % 2 else -1.0
    a1, a2 = np.asfortranarray(a), np.asfortranarray(a.copy())
    i1 = getattr(hb, f"{p}potrf")(uplo, n, a1, n)
    i2 = getattr(orc, f"{p}potrf")(uplo, n, a2, n)
    assert i1 == i2
    assert same_bits(a1, a2), first_diff(a1, a2)


@pytest.mark.parametrize("p", ["d", "s"])
@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("n", [700, 1500, 3000])
@pytest.mark.parametrize("block", ["second", "middle", "last"])
def test_potrf_fails_beside_an_update(hb, orc, p, uplo, n, block):
    """The block that fails is factored beside the rest of the step before it, which
    the reference has done by then: A and INFO are its bits, whatever the two
    streams' timing (hence the repetitions), and POSV leaves B alone."""
    rng = np.random.default_rng(n)
    g = rand(rng, n, n)
    a = (g @ g.T / n + np.eye(n)).astype(REAL[p])
    i = 64 * {"second": 1, "middle": n // 128, "last": (n - 1) // 64}[block] + 17
    a[i, i] = -1.0
    a = np.asfortranarray(a)
    want = a.copy(order="F")
    assert getattr(orc, f"{p}potrf")(uplo, n, want, n) == i + 1
    b = rand(rng, n, 2, REAL[p])
    for trial in range(10):
        got, x = a.copy(order="F"), b.copy(order="F")
        if trial % 2:
            info = getattr(hb, f"{p}posv")(uplo, n, 2, got, n, x, n)
        else:
            info = getattr(hb, f"{p}potrf")(uplo, n, got, n)
        assert info == i + 1
        assert same_bits(got, want), (trial, first_diff(got, want))
        assert same_bits(x, b)


@pytest.mark.parametrize("p", ["d", "s"])
@pytest.mark.parametrize("side", ["L", "R"])
@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("diag", ["N", "U"])
@pytest.mark.parametrize("r", [31, 32, 33, 47, 63, 64, 65, 97])
def test_trsm_bases(hb, orc, p, side, uplo, trans, diag, r):
    rng = np.random.default_rng(r)
    for other in (1, 16, 35):
        m, n = (r, other) if side == "L" else (other, r)
        a = rand(rng, r + 1, r, REAL[p]) / REAL[p](np.sqrt(r))
        a[:r] += np.diag(np.full(r, 1.5)).astype(REAL[p])
        a = np.asfortranarray(a)
        b = rand(rng, m + 2, n, REAL[p])
        x1, x2 = b.copy(order="F"), b.copy(order="F")
        getattr(hb, f"{p}trsm")(side, uplo, trans, diag, m, n, 1.0, a, r + 1, x1, m + 2)
        getattr(orc, f"{p}trsm")(side, uplo, trans, diag, m, n, REAL[p](1.0), a, r + 1, x2, m + 2)
        assert same_bits(x1, x2), (other, first_diff(x1, x2))


@pytest.mark.parametrize("p", ["d", "s"])
@pytest.mark.parametrize("side", ["L", "R"])
@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("diag", ["N", "U"])
@pytest.mark.parametrize("r", [1, 2, 15, 31, 32, 33, 47, 64])
def test_trsm_bases_many_rows(hb, orc, p, side, uplo, diag, r):
    """Either side of the lines between a lane an element and a thread a row, and
    between one launch and three."""
    lines = {("d", "L"): (12000, 24000), ("d", "R"): (8000, 16000), ("s", "L"): (24000, 64000),
             ("s", "R"): (12000, 32000)}[p, side]
    rng = np.random.default_rng(r)
    a = rand(rng, r, r, REAL[p]) / REAL[p](np.sqrt(r))
    a = np.asfortranarray(a + np.diag(np.full(r, 1.5)).astype(REAL[p]))
    for other in (lines[r > 32] - 1, lines[r > 32] + 1):
        m, n = (r, other) if side == "L" else (other, r)
        b = rand(rng, m + 1, n, REAL[p])
        x1, x2 = b.copy(order="F"), b.copy(order="F")
        getattr(hb, f"{p}trsm")(side, uplo, "N", diag, m, n, 1.0, a, r, x1, m + 1)
        getattr(orc, f"{p}trsm")(side, uplo, "N", diag, m, n, REAL[p](1.0), a, r, x2, m + 1)
        assert same_bits(x1, x2), (other, first_diff(x1, x2))


def check_zgetrf(hb, orc, p, a, recursive, columns=None):
    m, n = a.shape
    a1, a2 = a.copy(order="F"), a.copy(order="F")
    p1, p2 = np.zeros(min(m, n), np.int32), np.zeros(min(m, n), np.int32)
    i1 = hb.zgetrf(p, m, n, a1, m, p1, recursive=recursive)
    i2 = orc.zgetrf(m, n, a2, m, p2, recursive=recursive)
    assert i1 == i2
    assert np.array_equal(p1, p2), np.flatnonzero(p1 != p2)[:4]
    r = REAL["d" if p == "z" else "s"]
    b1, b2 = a1.T.view(r)[:columns], a2.T.view(r)[:columns]  # row by row: column by column of a
    assert same_bits(b1, b2), first_diff(b1, b2)


def crand(rng, p, m, n):
    t = np.complex128 if p == "z" else np.complex64
    return np.asfortranarray((rng.uniform(-1, 1, (m, n)) + 1j * rng.uniform(-1, 1, (m, n))).astype(t))


@pytest.mark.parametrize("p", ["z", "c"])
@pytest.mark.parametrize("m", [64, 130, 300, 1000])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 33, 50, 63, 64])
def test_complex_panel_widths(hb, orc, p, m, n):
    check_zgetrf(hb, orc, p, crand(np.random.default_rng(m + n), p, m, n), True)


@pytest.mark.parametrize("p,m", [("z", 1152), ("z", 1153), ("z", 2304), ("z", 2320), ("c", 2700),
                                 ("c", 5300)])
def test_complex_panel_heights(hb, orc, p, m):
    check_zgetrf(hb, orc, p, crand(np.random.default_rng(m), p, m, 64), False)


@pytest.mark.parametrize("p", ["z", "c"])
@pytest.mark.parametrize("m,n", [(200, 200), (65, 64), (300, 130), (130, 300), (600, 600)])
@pytest.mark.parametrize("ties", [False, True])
def test_complex_blocked(hb, orc, p, m, n, ties):
    rng = np.random.default_rng(m + 2 * n)
    a = crand(rng, p, m, n)
    if ties:  # magnitudes from a few values, columns that become zero
        a = np.asfortranarray((rng.integers(-1, 2, (m, n)) + 1j * rng.integers(-1, 2, (m, n)))
                              .astype(a.dtype))
        a[:, 5] = a[:, 3]
    check_zgetrf(hb, orc, p, a, False)


@pytest.mark.parametrize("p", ["z", "c"])
@pytest.mark.parametrize("m", [40, 600])
@pytest.mark.parametrize("place", ["first", "middle", "all"])
@pytest.mark.parametrize("re,im", [(np.nan, 0), (0, np.nan), (np.inf, 1), (0, -np.inf),
                                   (np.inf, np.nan)])
def test_complex_panel_special_values(hb, orc, p, m, place, re, im):
    """NaN anywhere; infinities in the last column, whose search they go through (what
    the C runtime recovers from quotients of infinities is not reproduced)."""
    rng = np.random.default_rng(m)
    infinite = np.isinf([re, im]).any()
    a = crand(rng, p, m, 21 if infinite else 36)
    rows = {"first": [0], "middle": [m // 2], "all": list(range(m))}[place]
    a[rows, 20] = complex(re, im)
    check_zgetrf(hb, orc, p, a, True, columns=20 if infinite else None)


@pytest.mark.parametrize("p", ["d", "s"])
@pytest.mark.parametrize("side", ["L", "R"])
@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("r,other", [(65, 1), (96, 9), (288, 64), (450, 3), (500, 70), (511, 8),
                                     (512, 130), (700, 17), (200, 960), (200, 961)])
def test_trsm_subtrees(hb, orc, p, side, uplo, trans, r, other):
    """Subtrees in one launch: partial blocks, more right-hand sides than a
    cluster takes, updates deeper than a KC chunk (upper, r = 500 and 511), as many
    right-hand sides as fit a wave of clusters and one more."""
    rng = np.random.default_rng(r + other)
    m, n = (r, other) if side == "L" else (other, r)
    a = rand(rng, r, r, REAL[p]) / REAL[p](np.sqrt(r))
    a = np.asfortranarray(a + np.diag(np.full(r, 1.5)).astype(REAL[p]))
    b = rand(rng, m + 1, n, REAL[p])
    for diag in "NU":
        x1, x2 = b.copy(order="F"), b.copy(order="F")
        getattr(hb, f"{p}trsm")(side, uplo, trans, diag, m, n, 1.0, a, r, x1, m + 1)
        getattr(orc, f"{p}trsm")(side, uplo, trans, diag, m, n, REAL[p](1.0), a, r, x2, m + 1)
        assert same_bits(x1, x2), (diag, first_diff(x1, x2))
