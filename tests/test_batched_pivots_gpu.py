"""Batched LU of matrices that need interchanges: every problem equal to the
single-problem routine, in repeated runs (the pivot of a column reaches all of a
CTA's warps before the rows are interchanged)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", ["d", "s"])
def test_batched_lu_interchanges(hb, cuda, p):
    torch = cuda
    t = torch.float64 if p == "d" else torch.float32
    gen = torch.Generator(device="cuda").manual_seed(3)
    sizes = [60 + (37 * i) % 240 for i in range(300)]
    a = [torch.rand(n * n, dtype=t, device="cuda", generator=gen) * 2 - 1 for n in sizes]
    want, wpiv = [x.clone() for x in a], [torch.zeros(n, dtype=torch.int32, device="cuda")
                                          for n in sizes]
    f = hb.dgetrf if p == "d" else hb.sgetrf
    for n, x, q in zip(sizes, want, wpiv):
        assert f(n, n, x, n, q) == 0
    for _ in range(3):
        got = [x.clone() for x in a]
        piv = [torch.zeros_like(q) for q in wpiv]
        assert hb.getrf_batched(sizes, got, sizes, piv, precision=p) == [0] * len(sizes)
        torch.cuda.synchronize()
        for n, x, y, q, r in zip(sizes, got, want, piv, wpiv):
            assert torch.equal(q, r), n
            assert torch.equal(x, y), n


@pytest.mark.parametrize("p", ["d", "s"])
@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("config", [64, 256])
def test_batched_solve_interchanges(hb, cuda, p, trans, config):
    """Whole columns a batch (small n, many right-hand sides), one column or less a
    thread, more rows than the order in shared memory holds; no interchange at all."""
    torch = cuda
    t = torch.float64 if p == "d" else torch.float32
    gen = torch.Generator(device="cuda").manual_seed(4)
    sizes = [1, 2, 7, 16, 63, 64, 65, 255, 256, 257, 512, 513, 1000, 1024, 1025, 100]
    rhs = [40, 33, 40, 17, 3, 40, 5, 2, 9, 3, 2, 3, 1, 2, 2, 6]
    a = [torch.rand(n * n, dtype=t, device="cuda", generator=gen) * 2 - 1 for n in sizes]
    a[-1].view(100, 100).diagonal().add_(200)  # pivots on the diagonal
    piv = [torch.zeros(n, dtype=torch.int32, device="cuda") for n in sizes]
    b = [torch.rand(n * r, dtype=t, device="cuda", generator=gen) for n, r in zip(sizes, rhs)]
    getrf, getrs = (hb.dgetrf, hb.dgetrs) if p == "d" else (hb.sgetrf, hb.sgetrs)
    want = [x.clone() for x in b]
    for n, r, x, q, y in zip(sizes, rhs, a, piv, want):
        assert getrf(n, n, x, n, q) == 0
        assert getrs(trans, n, r, x, n, q, y, n) == 0
    old = hb.lib().hwyblas_batched_set_config(config)
    try:
        assert hb.getrs_batched(trans, sizes, rhs, a, sizes, piv, b, sizes, precision=p) == 0
    finally:
        hb.lib().hwyblas_batched_set_config(old)
    torch.cuda.synchronize()
    for n, x, y in zip(sizes, b, want):
        assert torch.equal(x, y), n


@pytest.mark.parametrize("p", ["d", "s"])
@pytest.mark.parametrize("config", [256, 1002])
@pytest.mark.parametrize("count", [290, 300, 450])
def test_batched_ctas_an_sm(hb, cuda, p, config, count):
    """Batches that two CTAs of 256 threads an SM hold, that three do, and larger ones:
    LU, solve and TRSM equal to the 64-thread configuration's."""
    torch = cuda
    if p == "s" and config == 1002:
        pytest.skip("FP64 only")
    t = torch.float64 if p == "d" else torch.float32
    gen = torch.Generator(device="cuda").manual_seed(5)
    n = 72
    a0 = torch.rand(count, n, n, dtype=t, device="cuda", generator=gen) * 2 - 1
    b0 = torch.rand(count, 5, n, dtype=t, device="cuda", generator=gen)
    sizes, rhs = [n] * count, [5] * count

    def run(cfg):
        a, b, x = a0.clone(), b0.clone(), b0.clone()
        piv = torch.zeros(count, n, dtype=torch.int32, device="cuda")
        old = hb.lib().hwyblas_batched_set_config(cfg)
        try:
            info = hb.getrf_batched(sizes, list(a), sizes, list(piv), precision=p)
            hb.getrs_batched("N", sizes, rhs, list(a), sizes, list(piv), list(b), sizes, precision=p)
            hb.trsm_batched("L", "L", "N", "U", sizes, rhs, 1.0, list(a), sizes, list(x), sizes,
                            precision=p)
        finally:
            hb.lib().hwyblas_batched_set_config(old)
        torch.cuda.synchronize()
        assert info == [0] * count
        return a, piv, b, x

    for got, want in zip(run(config), run(64)):
        assert torch.equal(got, want)
