"""The work whose time matters to a user of this library, as measurable cases.

Every case goes through the package's public wrappers (the C ABI with the
reference's routine names). Matrices are column-major: a tensor of shape
(columns, ld) holds one, so ``t[:, :rows].T`` is the matrix itself. Device
tensors are used in place; a ``host`` case passes NumPy arrays, which the
library stages through the device, as a program relinked from the reference
does. Routines that work in place get a fresh copy of their input in every
pass, as a program that keeps its matrix makes one.
"""
import math

import numpy as np
import torch

import hwyblas_b200 as hb

TYPES = {"d": torch.float64, "s": torch.float32, "z": torch.complex128, "c": torch.complex64}


def listed():
    return [
        # One product of a few dozen rows: a call's fixed cost.
        {"name": "dgemm_small", "do": "gemm", "p": "d", "ta": "N", "tb": "N", "m": 33, "n": 47,
         "k": 65, "pad": 0, "alpha": 1.5, "beta": 0.5},
        # The mid-sized square product of the plain FP64 configuration.
        {"name": "dgemm_1024", "do": "gemm", "p": "d", "ta": "N", "tb": "N", "m": 1024,
         "n": 1024, "k": 1024, "pad": 0, "alpha": 1.5, "beta": 0.5},
        # A large ragged product with a transposed operand and padded leading dimensions.
        {"name": "dgemm_large_tn", "do": "gemm", "p": "d", "ta": "T", "tb": "N", "m": 4099,
         "n": 3001, "k": 5003, "pad": 5, "alpha": 1.0, "beta": 0.0},
        # Single precision, ragged, the other operand transposed.
        {"name": "sgemm_nt", "do": "gemm", "p": "s", "ta": "N", "tb": "T", "m": 3001, "n": 2047,
         "k": 2500, "pad": 3, "alpha": 1.0, "beta": 1.0},
        # The triangular solve of the configurations: many right-hand sides.
        {"name": "dtrsm_4096x512", "do": "trsm", "p": "d", "side": "L", "uplo": "L", "trans": "N",
         "diag": "U", "m": 4096, "n": 512},
        # LU with partial pivoting, the configurations' size.
        {"name": "dgetrf_4096", "do": "getrf", "p": "d", "m": 4096, "n": 4096, "pad": 0},
        # A whole small solve on host arrays: the drop-in call of a relinked program.
        {"name": "dgesv_host_500", "do": "gesv", "p": "d", "n": 500, "nrhs": 1, "host": True},
        # Cholesky solve of a ragged SPD system with a few right-hand sides.
        {"name": "dposv_3001", "do": "posv", "p": "d", "uplo": "L", "n": 3001, "nrhs": 16},
        # Complex LU solve.
        {"name": "zgesv_1500", "do": "gesv", "p": "z", "n": 1500, "nrhs": 8, "host": False},
        # The FP64-accurate product on the INT8 tensor cores, slice count chosen by the call.
        {"name": "dgemm_emulated_8192", "do": "emulated", "m": 8192, "n": 8192, "k": 8192,
         "spread": 8},
        # The mixed-precision solver at its headline size.
        {"name": "dgesv_mixed_16384", "do": "mixed", "kind": "gesv", "n": 16384, "nrhs": 1,
         "cond": 1e6},
        # Thousands of small uneven problems, each LU + solve + product, three calls in all.
        {"name": "batched_10000", "do": "batched", "p": "d", "count": 10000, "low": 8,
         "high": 512},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """One more case: a family, then sizes spread over the logarithm of its range."""
    do = rng.choice(["gemm", "gemm", "trsm", "getrf", "gesv", "posv", "emulated", "mixed",
                     "batched"])
    if do == "gemm":
        p = rng.choice("dds" "dzc")
        top = 5000 if p in "ds" else 2500
        return {"do": do, "p": p, "ta": rng.choice("NT" if p in "ds" else "NTC"),
                "tb": rng.choice("NT"), "m": _log(rng, 16, top), "n": _log(rng, 16, top),
                "k": _log(rng, 16, top), "pad": rng.choice([0, 0, 1, 6]),
                "alpha": rng.choice([1.0, -1.0, 1.5]), "beta": rng.choice([0.0, 1.0, 0.5])}
    if do == "trsm":
        m, n = _log(rng, 32, 4096), _log(rng, 1, 1024)
        side = rng.choice("LR")
        if side == "R":
            m, n = n, m
        return {"do": do, "p": rng.choice("dds"), "side": side, "uplo": rng.choice("LU"),
                "trans": rng.choice("NT"), "diag": rng.choice("NU"), "m": m, "n": n}
    if do == "getrf":
        p = rng.choice("ddsz")
        return {"do": do, "p": p, "m": _log(rng, 64, 4096), "n": _log(rng, 64, 4096),
                "pad": rng.choice([0, 0, 3])}
    if do == "gesv":
        return {"do": do, "p": rng.choice("ddsz"), "n": _log(rng, 32, 3000),
                "nrhs": _log(rng, 1, 64), "host": rng.random() < 0.25}
    if do == "posv":
        return {"do": do, "p": rng.choice("ddsz"), "uplo": rng.choice("LU"),
                "n": _log(rng, 32, 4000), "nrhs": _log(rng, 1, 64)}
    if do == "emulated":
        return {"do": do, "m": _log(rng, 256, 8192), "n": _log(rng, 256, 8192),
                "k": _log(rng, 256, 8192), "spread": rng.randint(0, 16)}
    if do == "mixed":
        return {"do": do, "kind": rng.choice(["gesv", "posv"]), "n": _log(rng, 1024, 10000),
                "nrhs": _log(rng, 1, 64), "cond": rng.choice([1e2, 1e4, 1e6])}
    high = _log(rng, 32, 512)
    return {"do": "batched", "p": rng.choice("ds"), "count": _log(rng, 200, 8000),
            "low": rng.randint(4, 16), "high": high}


# ---------------------------------------------------------------------------
# Inputs.


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _uniform(gen, shape, dtype):
    """Entries uniform in [-1, 1] (both parts of a complex one)."""
    if dtype.is_complex:
        real = torch.float64 if dtype == torch.complex128 else torch.float32
        return torch.view_as_complex(_uniform(gen, tuple(shape) + (2,), real))
    return torch.rand(shape, dtype=dtype, device="cuda", generator=gen).mul_(2).sub_(1)


def _matrix(gen, rows, cols, dtype, pad=0):
    return _uniform(gen, (cols, rows + pad), dtype)


def _spread(gen, rows, cols, spread):
    """Entries u * 2^e, u uniform in [-1, 1], e a whole number in [-spread, spread]."""
    u = _matrix(gen, rows, cols, torch.float64)
    e = torch.randint(-spread, spread + 1, u.shape, device="cuda", generator=gen)
    return u.mul_(torch.exp2(e.to(torch.float64)))


def _spd(gen, n, dtype):
    """G G^H / n + 1e-3 I, G Gaussian."""
    g = torch.randn((n, n), dtype=dtype, device="cuda", generator=gen)
    a = g @ g.mH
    a /= n
    a.diagonal().add_(1e-3)
    return a


def _conditioned(gen, n, cond):
    """H1 diag(s) H2: H1, H2 products of 4 Householder reflectors from Gaussian
    vectors, s geometric from 1 to 1/cond."""
    a = torch.diag(torch.logspace(0.0, -math.log10(cond), n, dtype=torch.float64, device="cuda"))
    for side in range(2):
        for _ in range(4):
            v = torch.randn(n, dtype=torch.float64, device="cuda", generator=gen)
            v /= torch.linalg.norm(v)
            if side == 0:
                a.addr_(v, v @ a, alpha=-2.0)
            else:
                a.addr_(a @ v, v, alpha=-2.0)
    return a


def _batch_sizes(case, seed):
    """The batch's sizes: a program's own, the same from step to step."""
    rng = np.random.default_rng(case["count"])
    low, high = case["low"], case["high"]
    n = np.exp(rng.uniform(np.log(low), np.log(high), case["count"])).astype(int)
    return n.clip(low, high), rng.integers(1, 17, case["count"])


class _State:
    pass


def prepare(case, seed):
    s, g = _State(), _gen(seed)
    s.case = case
    do = case["do"]
    if do in ("gemm", "trsm", "getrf", "gesv", "posv"):
        t = TYPES[case["p"]]
    if do == "gemm":
        m, n, k, pad = case["m"], case["n"], case["k"], case["pad"]
        s.a = _matrix(g, *((m, k) if case["ta"] == "N" else (k, m)), t, pad)
        s.b = _matrix(g, *((k, n) if case["tb"] == "N" else (n, k)), t, pad)
        s.c0 = _matrix(g, m, n, t, pad)
        s.c = s.c0.clone()
    elif do == "trsm":
        # Entries scaled so that the solution neither grows nor vanishes with
        # the order; the diagonal of a non-unit triangle is in [1, 2].
        r = case["m"] if case["side"] == "L" else case["n"]
        s.a = _matrix(g, r, r, t).mul_(2.0 / math.sqrt(r))
        s.a.diagonal().copy_(torch.rand(r, dtype=t, device="cuda", generator=g).add_(1))
        s.b = _matrix(g, case["m"], case["n"], t)
        s.x = torch.empty_like(s.b)
    elif do == "getrf":
        s.a = _matrix(g, case["m"], case["n"], t, case["pad"])
        s.lu = torch.empty_like(s.a)
        s.ipiv = torch.zeros(min(case["m"], case["n"]), dtype=torch.int32, device="cuda")
    elif do in ("gesv", "posv"):
        n = case["n"]
        s.a = _matrix(g, n, n, t) if do == "gesv" else _spd(g, n, t)
        s.b = _matrix(g, n, case["nrhs"], t)
        if case.get("host"):
            s.a, s.b = s.a.cpu().numpy(), s.b.cpu().numpy()
            s.f, s.x = np.empty_like(s.a), np.empty_like(s.b)
            s.ipiv = np.zeros(n, np.int32)
        else:
            s.f, s.x = torch.empty_like(s.a), torch.empty_like(s.b)
            s.ipiv = torch.zeros(n, dtype=torch.int32, device="cuda")
    elif do == "emulated":
        s.a = _spread(g, case["m"], case["k"], case["spread"])
        s.b = _spread(g, case["k"], case["n"], case["spread"])
        s.c = _matrix(g, case["m"], case["n"], torch.float64).zero_()
    elif do == "mixed":
        n = case["n"]
        s.a = (_conditioned(g, n, case["cond"]) if case["kind"] == "gesv"
               else _spd(g, n, torch.float64))
        s.b = _matrix(g, n, case["nrhs"], torch.float64)
        s.x = torch.zeros_like(s.b)
        s.ipiv = torch.zeros(n, dtype=torch.int32, device="cuda")
    else:
        t = torch.float64 if case["p"] == "d" else torch.float32
        s.n, s.r = _batch_sizes(case, seed)
        s.at = np.concatenate([[0], np.cumsum(s.n * s.n)])
        s.bt = np.concatenate([[0], np.cumsum(s.n * s.r)])
        s.pt = np.concatenate([[0], np.cumsum(s.n)])
        s.a, s.g1, s.g2 = (_uniform(g, (int(s.at[-1]),), t) for _ in range(3))
        # Diagonally dominant systems, as blocks of discretised equations are: a
        # batch of matrices near singularity would weigh a few of its problems only.
        n = np.repeat(s.n, s.n)
        step = np.arange(len(n)) - np.repeat(s.pt[:-1], s.n)
        diagonal = torch.as_tensor(np.repeat(s.at[:-1], s.n) + step * (n + 1), device="cuda")
        s.a[diagonal] += torch.as_tensor(n + 1, device="cuda", dtype=t)
        s.b = _uniform(g, (int(s.bt[-1]),), t)
        s.lu, s.x, s.c = torch.empty_like(s.a), torch.empty_like(s.b), torch.zeros_like(s.a)
        s.ipiv = torch.zeros(int(s.pt[-1]), dtype=torch.int32, device="cuda")

        def at(buf, offsets):
            return hb.ptr_array([buf.data_ptr() + int(o) * buf.element_size()
                                 for o in offsets[:-1]])

        # The C arrays of sizes and device pointers, kept as a C caller keeps its own.
        s.cn, s.cr = hb.int_array(s.n), hb.int_array(s.r)
        s.pa, s.px, s.pp = at(s.lu, s.at), at(s.x, s.bt), at(s.ipiv, s.pt)
        s.p1, s.p2, s.p3 = at(s.g1, s.at), at(s.g2, s.at), at(s.c, s.at)
    return s


# ---------------------------------------------------------------------------
# One pass.


def _gemm(s):
    c = s.case
    args = (c["ta"], c["tb"], c["m"], c["n"], c["k"], c["alpha"], s.a, s.a.shape[1], s.b,
            s.b.shape[1], c["beta"], s.c, s.c.shape[1])
    if c["beta"] != 0.0:
        s.c.copy_(s.c0)
    if c["p"] == "d":
        hb.dgemm(*args)
    elif c["p"] == "s":
        hb.sgemm(*args)
    else:
        hb.zgemm(c["p"], *args)
    return s.c


def _trsm(s):
    c = s.case
    s.x.copy_(s.b)
    f = hb.dtrsm if c["p"] == "d" else hb.strsm
    f(c["side"], c["uplo"], c["trans"], c["diag"], c["m"], c["n"], 1.0, s.a, s.a.shape[1], s.x,
      s.x.shape[1])
    return s.x


def _getrf(s):
    c = s.case
    s.lu.copy_(s.a)
    args = (c["m"], c["n"], s.lu, s.lu.shape[1], s.ipiv)
    if c["p"] == "z":
        info = hb.zgetrf("z", *args)
    else:
        info = (hb.dgetrf if c["p"] == "d" else hb.sgetrf)(*args)
    return {"lu": s.lu, "ipiv": s.ipiv, "info": info}


def _copy(dst, src):
    if isinstance(dst, np.ndarray):
        np.copyto(dst, src)
    else:
        dst.copy_(src)


def _gesv(s):
    c = s.case
    n = c["n"]
    _copy(s.f, s.a)
    _copy(s.x, s.b)
    args = (n, c["nrhs"], s.f, n, s.ipiv, s.x, n)
    if c["p"] == "z":
        info = hb.zgesv("z", *args)
    else:
        info = (hb.dgesv if c["p"] == "d" else hb.sgesv)(*args)
    return {"lu": s.f, "ipiv": s.ipiv, "x": s.x, "info": info}


def _posv(s):
    c = s.case
    n = c["n"]
    _copy(s.f, s.a)
    _copy(s.x, s.b)
    args = (c["uplo"], n, c["nrhs"], s.f, n, s.x, n)
    if c["p"] == "z":
        info = hb.zposv("z", *args)
    else:
        info = (hb.dposv if c["p"] == "d" else hb.sposv)(*args)
    return {"f": s.f, "x": s.x, "info": info}


def _emulated(s):
    c = s.case
    hb.dgemm_emulated("N", "N", c["m"], c["n"], c["k"], 1.0, s.a, c["m"], s.b, c["k"], 0.0, s.c,
                      c["m"])
    return s.c


def _mixed(s):
    # A is left as it was (the factors are not returned), so X is the result.
    c = s.case
    n = c["n"]
    if c["kind"] == "gesv":
        info, _ = hb.dgesv_mixed(n, c["nrhs"], s.a, n, s.ipiv, s.b, n, s.x, n)
    else:
        info, _ = hb.dposv_mixed("L", n, c["nrhs"], s.a, n, s.b, n, s.x, n)
    return {"x": s.x, "info": info}


def _batched(s):
    p = s.case["p"]
    s.lu.copy_(s.a)
    s.x.copy_(s.b)
    info = hb.getrf_batched(s.cn, s.pa, s.cn, s.pp, precision=p)
    hb.getrs_batched("N", s.cn, s.cr, s.pa, s.cn, s.pp, s.px, s.cn, precision=p)
    hb.gemm_batched("N", "N", s.cn, s.cn, s.cn, 1.0, s.p1, s.cn, s.p2, s.cn, 0.0, s.p3, s.cn,
                    precision=p)
    return {"lu": s.lu, "ipiv": s.ipiv, "x": s.x, "c": s.c, "info": np.array(info, np.int32)}


_RUN = {"gemm": _gemm, "trsm": _trsm, "getrf": _getrf, "gesv": _gesv, "posv": _posv,
        "emulated": _emulated, "mixed": _mixed, "batched": _batched}


def run(state):
    return _RUN[state.case["do"]](state)


# ---------------------------------------------------------------------------
# What a pass cannot do without, and how close another implementation comes.


def work(case):
    do, p = case["do"], case.get("p", "d")
    size = {"d": 8, "s": 4, "z": 16, "c": 8}[p]
    mul = 4 if p in "zc" else 1  # real flops of a complex multiply-add over a real one's
    if do in ("gemm", "emulated"):
        m, n, k = case["m"], case["n"], case["k"]
        c = 2 if case.get("beta", 0.0) != 0.0 else 1
        return {"bytes": size * (m * k + k * n + c * m * n), "flops": mul * 2 * m * n * k}
    if do == "trsm":
        m, n = case["m"], case["n"]
        r = m if case["side"] == "L" else n
        return {"bytes": size * (r * r / 2 + 2 * m * n), "flops": m * n * r}
    if do == "getrf":
        hi, lo = max(case["m"], case["n"]), min(case["m"], case["n"])
        return {"bytes": size * 2 * hi * lo, "flops": mul * (hi * lo ** 2 - lo ** 3 / 3)}
    if do in ("gesv", "posv", "mixed"):
        n, r = case["n"], case["nrhs"]
        chol = do == "posv" or case.get("kind") == "posv"
        one = n ** 3 / 3 if chol else 2 * n ** 3 / 3
        passes = 1 if do == "mixed" else 2  # the mixed solvers do not write A
        half = 0.5 if chol else 1
        return {"bytes": size * (passes * half * n * n + 2 * n * r),
                "flops": mul * (one + 2 * n * n * r)}
    n, r = (v.astype(float) for v in _batch_sizes(case, 0))
    return {"bytes": size * float(np.sum(5 * n * n + 2 * n * r)),
            "flops": float(np.sum(2 / 3 * n ** 3 + 2 * n * n * r + 2 * n ** 3))}


def tolerance(case):
    """The plain routines give the reference's own bits, each element's sums
    in the reference's order: nothing else is right. The emulated product and
    the mixed solvers promise FP64 accuracy: the product differs from FP64 sums
    in another order by 3e-15 of the result at k = 8192, and X is the solution
    to about its last bit."""
    if case["do"] == "emulated":
        return {"rel": 1.2e-14}
    if case["do"] == "mixed":
        return {"rel": 4e-15}
    return "exact"


# ---------------------------------------------------------------------------
# The same outputs from 64-bit library routines.


def _wide(t):
    return t.to(torch.complex128 if t.is_complex() else torch.float64)


def _lu(a):
    """Compact LU factors (rows x columns), None if their pivots may differ."""
    return torch.linalg.lu_factor(a)[0]


def _put(buf, rows, value):
    """`buf`'s layout with its matrix replaced."""
    out = _wide(buf).clone()
    out[:, :rows] = value.T
    return out


def exact(case, seed):
    s, do = prepare(case, seed), case["do"]
    if do in ("gemm", "emulated"):
        def op(t, flag, rows):
            a = _wide(t[:, :rows].T)
            return a if flag == "N" else a.T if flag == "T" else a.mH

        m, k, n = case["m"], case["k"], case["n"]
        ta, tb = case.get("ta", "N"), case.get("tb", "N")
        v = op(s.a, ta, m if ta == "N" else k) @ op(s.b, tb, k if tb == "N" else n)
        v = case.get("alpha", 1.0) * v
        if do == "gemm" and case["beta"] != 0.0:
            v += case["beta"] * _wide(s.c0[:, :m].T)
        return _put(s.c if do == "emulated" else s.c0, m, v)
    if do == "trsm":
        a, b = _wide(s.a.T), _wide(s.b.T)
        a = torch.tril(a) if case["uplo"] == "L" else torch.triu(a)
        upper = case["uplo"] == "U"
        if case["trans"] == "T":
            a, upper = a.T, not upper
        x = torch.linalg.solve_triangular(a, b, upper=upper, left=case["side"] == "L",
                                          unitriangular=case["diag"] == "U")
        return _put(s.b, case["m"], x)
    if do == "getrf":
        # In single precision another rounding picks other pivots: no such factors.
        lu = None if case["p"] == "s" else _put(s.a, case["m"], _lu(s.a[:, :case["m"]].T))
        return {"lu": lu, "ipiv": None, "info": 0}
    if do in ("gesv", "posv"):
        at, bt = (torch.as_tensor(v, device="cuda") for v in (s.a, s.b))
        a, b = _wide(at.T), _wide(bt.T)
        if do == "gesv":
            x = _put(bt, case["n"], torch.linalg.solve(a, b))
            lu = None if case["p"] == "s" else _put(at, case["n"], _lu(a))
            return {"lu": lu, "ipiv": None, "x": x, "info": 0}
        # The stored triangle's mirror image is the matrix that is factored.
        tri = torch.tril(a) if case["uplo"] == "L" else torch.triu(a)
        full = tri + tri.mH
        full.diagonal().copy_(a.diagonal().real)
        low = torch.linalg.cholesky(full)
        f = a.clone()
        if case["uplo"] == "L":
            f = torch.tril(low) + torch.triu(f, 1)
        else:
            f = torch.triu(low.mH) + torch.tril(f, -1)
        return {"f": _put(at, case["n"], f),
                "x": _put(bt, case["n"], torch.cholesky_solve(b, low)), "info": 0}
    if do == "mixed":
        return {"x": _put(s.b, case["n"], torch.linalg.solve(s.a.T, s.b.T)), "info": 0}
    lu, x, c = _wide(s.a).clone(), _wide(s.b).clone(), _wide(s.c).clone()
    for n in np.unique(s.n):
        ids = np.nonzero(s.n == n)[0]
        n = int(n)

        def take(buf, off, size):
            at = torch.as_tensor(off[ids], device="cuda")[:, None]
            return at + torch.arange(size, device="cuda")[None, :]

        ia = take(s.a, s.at, n * n)
        mats = [_wide(v[ia]).view(-1, n, n).mT for v in (s.a, s.g1, s.g2)]
        f, piv = torch.linalg.lu_factor(mats[0])
        lu[ia] = f.mT.reshape(len(ids), -1)
        c[ia] = (mats[1] @ mats[2]).mT.reshape(len(ids), -1)
        top = int(s.r[ids].max())
        ib = torch.as_tensor(s.bt[ids], device="cuda")[:, None] + torch.arange(n * top,
                                                                             device="cuda")
        mine = torch.arange(n * top, device="cuda") < torch.as_tensor(n * s.r[ids],
                                                                     device="cuda")[:, None]
        rhs = torch.where(mine, _wide(s.b)[ib.clamp(max=s.b.numel() - 1)], 0.0)
        v = torch.linalg.lu_solve(f, piv, rhs.view(-1, top, n).mT).mT.reshape(len(ids), -1)
        x[ib[mine]] = v[mine]
    return {"lu": lu, "ipiv": None, "x": x, "c": c, "info": None}
