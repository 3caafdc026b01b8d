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
