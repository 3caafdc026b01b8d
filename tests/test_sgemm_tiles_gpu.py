"""FP32 GEMM tiles against the oracle, bit for bit: edges of the 64- and
128-wide tiles, of the 16-deep slabs and of the 384-deep chunks, aligned and
unaligned operands, both orders of each operand."""
import numpy as np
import pytest

from tests.oracle_lib import rand, same_bits, first_diff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta", ["N", "T"])
@pytest.mark.parametrize("tb", ["N", "T"])
@pytest.mark.parametrize("m,n,k,pad", [
    (1, 1, 1, 0), (63, 31, 15, 1), (64, 32, 16, 0), (65, 33, 17, 3), (130, 129, 383, 2),
    (128, 64, 384, 4), (129, 100, 385, 0), (200, 70, 800, 5),
    # 128 x 64 tiles, either side of the 24 from which they are taken.
    (512, 384, 64, 0), (512, 385, 33, 1), (640, 320, 385, 4), (513, 449, 385, 3),
    (640, 640, 400, 0), (129, 770, 50, 2),
    (1601, 1540, 20, 3), (1664, 1536, 400, 0),  # at least 148 tiles of 128 x 128
])
def test_sgemm_tiles_bitexact(hb, orc, ta, tb, m, n, k, pad):
    rng = np.random.default_rng(m + 7 * n + 11 * k)
    ra, ca = (m, k) if ta == "N" else (k, m)
    rb, cb = (k, n) if tb == "N" else (n, k)
    a, b = rand(rng, ra + pad, ca, np.float32), rand(rng, rb + pad, cb, np.float32)
    c = rand(rng, m + pad, n, np.float32)
    for alpha, beta in ((1.5, 0.3), (-1.0, 1.0), (1.0, 0.0)):
        c1, c2 = c.copy(order="F"), c.copy(order="F")
        if beta == 0.0:
            c1[:m], c2[:m] = np.nan, np.nan  # C is not read
        hb.sgemm(ta, tb, m, n, k, alpha, a, ra + pad, b, rb + pad, beta, c1, m + pad)
        orc.sgemm(ta, tb, m, n, k, np.float32(alpha), a, ra + pad, b, rb + pad,
                  np.float32(beta), c2, m + pad)
        assert same_bits(c1, c2), (alpha, beta, first_diff(c1, c2))


@pytest.mark.parametrize("offset", [0, 1, 2])
def test_sgemm_tiles_device_alignment(hb, orc, cuda, offset):
    """Device operands whose base is not 16-byte aligned take the narrow loads."""
    rng = np.random.default_rng(offset)
    m, n, k = 132, 68, 52
    a, b = rand(rng, m, k, np.float32), rand(rng, k, n, np.float32)
    want = np.zeros((m, n), np.float32, order="F")
    orc.sgemm("N", "N", m, n, k, np.float32(1), a, m, b, k, np.float32(0), want, m)

    def dev(x):
        buf = cuda.zeros(x.size + 4, dtype=cuda.float32, device="cuda")
        buf[offset:offset + x.size] = cuda.from_numpy(x.ravel(order="F")).cuda()
        return buf[offset:offset + x.size]

    c = dev(want * 0)
    hb.sgemm("N", "N", m, n, k, 1.0, dev(a), m, dev(b), k, 0.0, c, m)
    assert same_bits(c.cpu().numpy().reshape((m, n), order="F"), want)


@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("n,k", [(65, 17), (300, 400), (600, 385), (2000, 30)])
def test_ssyrk_tiles_bitexact(hb, orc, uplo, n, k):
    rng = np.random.default_rng(n + k)
    a, c = rand(rng, n, k, np.float32), rand(rng, n, n, np.float32)
    c1, c2 = c.copy(order="F"), c.copy(order="F")
    hb.ssyrk(uplo, "N", n, k, 1.5, a, n, 0.3, c1, n)
    orc.ssyrk(uplo, "N", n, k, np.float32(1.5), a, n, np.float32(0.3), c2, n)
    assert same_bits(c1, c2), first_diff(c1, c2)
