"""Bounded device waits that run out (GPU): the LU panels' pivot exchanges (the
one-launch panel's messages between the CTAs of a cluster, the cooperative
leaf's global tags) are given a low poll limit through the test hook, so that
their waits give up. The call must return, report the timeout
(cudaErrorLaunchTimeout through hwyblas_last_cuda_error), leave the context
usable, and, with the default limit restored, the next factorization must be
bit-identical to the oracle again. The failure is made on purpose only through
the limit: no fault, trap or endless wait. The cooperative leaf's loads are plain
loads (no asynchronous copies are in flight when a wait gives up); the one-launch
panel waits for the messages in flight before its CTAs exit."""
import numpy as np
import pytest

from tests.oracle_lib import rand, same_bits

pytestmark = pytest.mark.gpu

CUDA_ERROR_LAUNCH_TIMEOUT = 702  # cudaErrorLaunchTimeout
DEFAULT_POLLS = 1 << 26


@pytest.mark.parametrize("n", [16, 40])
def test_leaf_wait_times_out_reports_and_recovers(hb, orc, n):
    lib = hb.lib()
    rng = np.random.default_rng(12)
    # 59 CTAs of 1024 rows: beyond the 16-CTA cluster, so the cooperative
    # variant with polled global slots runs. One leaf, and leaves with
    # interchanges by their pivots between them.
    m = 60000
    a0 = rand(rng, m, n)
    lib.hwyblas_last_cuda_error()  # clear
    prev = lib.hwyblas_set_leaf_wait_limit(1)
    try:
        assert prev == DEFAULT_POLLS
        a = a0.copy(order="F")
        ipiv = np.zeros(n, np.int32)
        hb.dgetrf2(m, n, a, m, ipiv)
        assert lib.hwyblas_last_cuda_error() == CUDA_ERROR_LAUNCH_TIMEOUT
        assert ipiv.min() >= 1 and ipiv.max() <= m
    finally:
        assert lib.hwyblas_set_leaf_wait_limit(0) == 1
    a1, a2 = a0.copy(order="F"), a0.copy(order="F")
    p1, p2 = np.zeros(n, np.int32), np.zeros(n, np.int32)
    info1 = hb.dgetrf2(m, n, a1, m, p1)
    assert lib.hwyblas_last_cuda_error() == 0
    info2 = orc.dgetrf2(m, n, a2, m, p2)
    assert info1 == info2 == 0
    assert np.array_equal(p1, p2)
    assert same_bits(a1, a2)


def test_leaf_wait_limit_default_is_restored(hb):
    lib = hb.lib()
    assert lib.hwyblas_set_leaf_wait_limit(0) == DEFAULT_POLLS


@pytest.mark.parametrize("p", ["d", "s", "z", "c"])
@pytest.mark.parametrize("m,n", [(300, 64), (2000, 64), (2300, 40), (700, 700)])
@pytest.mark.parametrize("polls", [1, 10, 30, 100, 300, 1000])
def test_panel_wait_times_out_reports_and_recovers(hb, orc, p, m, n, polls):
    """The one-launch panel's waits for the other CTAs' candidates: a cluster of 2, of 8
    and of 9 to 16 CTAs, and panels with their interchanges after them. One poll gives
    up at the first column; with more, some CTAs may give up in mid-panel while others
    go on. A CTA that gave up stays for the candidates that are on their way to it."""
    lib = hb.lib()
    rng = np.random.default_rng(m + n)
    if p in "zc":
        a0 = np.asfortranarray((rng.uniform(-1, 1, (m, n)) + 1j * rng.uniform(-1, 1, (m, n)))
                               .astype(np.complex128 if p == "z" else np.complex64))
    else:
        a0 = rand(rng, m, n, np.float64 if p == "d" else np.float32)

    def factor(a, ipiv):
        if p in "zc":
            return hb.zgetrf(p, m, n, a, m, ipiv)
        return getattr(hb, f"{p}getrf")(m, n, a, m, ipiv)

    want, pivots = a0.copy(order="F"), np.zeros(n, np.int32)
    if p in "zc":
        info = orc.zgetrf(m, n, want, m, pivots)
    else:
        info = getattr(orc, f"{p}getrf")(m, n, want, m, pivots)
    real = np.float64 if p in "dz" else np.float32

    def check(a, ipiv, got):
        assert got == info
        assert np.array_equal(ipiv, pivots)
        assert same_bits(a.T.view(real), want.T.view(real))

    lib.hwyblas_last_cuda_error()  # clear
    lib.hwyblas_set_leaf_wait_limit(polls)
    try:
        for _ in range(3):
            a, ipiv = a0.copy(order="F"), np.zeros(n, np.int32)
            got = factor(a, ipiv)
            error = lib.hwyblas_last_cuda_error()
            assert error == CUDA_ERROR_LAUNCH_TIMEOUT or (error == 0 and polls > 1)
            if error == 0:
                check(a, ipiv, got)
            else:  # pivots stay in range
                assert ipiv.min() >= 1 and ipiv.max() <= m
    finally:
        lib.hwyblas_set_leaf_wait_limit(0)
    a, ipiv = a0.copy(order="F"), np.zeros(n, np.int32)
    got = factor(a, ipiv)
    assert lib.hwyblas_last_cuda_error() == 0
    check(a, ipiv, got)
