"""The work this library is measured on: its dense-solve entry points over the
sizes, types and options its users call them with.

A case is a dict of plain values; ``kind`` names the entry point:

  lu_one       DeviceMatrix.lu() and LU.solve() of one general system
  lu_batch     DeviceBatch.lu() and LUBatch.solve_mut() of many equal systems
  refined      solve_refined() of one large system (FP32 factor, FP64 refinement)
  chol         a captured CholeskyBatch factor + solve + log-determinant (FP64)
  chol_refined CholeskyBatch.solve_refined_into() (FP32 factor, FP64 refinement)
  adjoint      PosvLogdet.forward() and .backward()
  gemm         gemm() in FP64, or its BF16-split form (slices = 3)
  ls           DeviceBatch.qr() and QRBatch.solve_mut(), ragged least squares

Inputs are synthetic, on the GPU, from the seed alone.  Entry points that
factor in place get their input copied into the buffers the caller keeps, as a
program that streams new systems through them does.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import nalgebra_gb300 as na


def listed():
    return [
        # one small system, the reference's 100 x 100 solve bench: latency of a single call
        {"name": "lu_one_100", "kind": "lu_one", "n": 100, "nrhs": 1},
        # thousands of small dense systems in one launch
        {"name": "lu_batch_4096x64", "kind": "lu_batch", "count": 4096, "n": 64, "nrhs": 1, "shift": 64.0},
        # one large FP64 system
        {"name": "lu_one_8192", "kind": "lu_one", "n": 8192, "nrhs": 1},
        # the same kind of system through the precision form
        {"name": "refined_4096", "kind": "refined", "n": 4096, "cond": 100.0},
        # ragged SPD batch, FP64, replayed from a CUDA graph
        {"name": "chol_20000", "kind": "chol", "count": 20000, "lo": 8, "hi": 256, "nrhs": 4},
        # the same batch through the precision form
        {"name": "chol_refined_20000", "kind": "chol_refined", "count": 20000, "lo": 8, "hi": 256, "nrhs": 4},
        # gradients through an SPD solve and log-determinant, factor stored, FP64
        {"name": "adjoint_f64_2048x128", "kind": "adjoint", "batch": 2048, "n": 128, "f64": True, "recompute": False},
        # the same in FP32 at an odd order, factor recomputed to save memory
        {"name": "adjoint_f32_1000x97", "kind": "adjoint", "batch": 1000, "n": 97, "f64": False, "recompute": True},
        # an ordinary product of odd sizes, accumulated into C
        {"name": "gemm_1000x777x1333", "kind": "gemm", "m": 1000, "n": 777, "k": 1333, "alpha": -1.0, "beta": 1.0,
         "spread": 0, "slices": 0},
        # a large product with rows and columns of very different magnitude, FP64
        {"name": "gemm_8192", "kind": "gemm", "m": 8192, "n": 8192, "k": 8192, "alpha": 1.0, "beta": 0.0,
         "spread": 20, "slices": 0},
        # the same product through the split-precision form
        {"name": "gemm_split_8192", "kind": "gemm", "m": 8192, "n": 8192, "k": 8192, "alpha": 1.0, "beta": 0.0,
         "spread": 20, "slices": 3},
        # thousands of tall least-squares problems of uneven height
        {"name": "ls_8192", "kind": "ls", "count": 8192, "lo": 128, "hi": 512, "n": 64},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mean(lo, hi, p):
    """Mean of n^p over the whole numbers lo..hi."""
    return float((np.arange(lo, hi + 1, dtype=np.float64) ** p).mean())


def draw(rng):
    kind = rng.choice(["lu_one", "lu_batch", "refined", "chol", "chol_refined", "adjoint", "gemm", "ls"])
    if kind == "lu_one":
        n = _log(rng, 32, 6000)
        return {"kind": kind, "n": n, "nrhs": 1 if n > 1500 else rng.choice([1, 1, 3, 10])}
    if kind == "lu_batch":
        n = rng.randint(8, 128)
        return {"kind": kind, "count": _log(rng, 200, 4096 if n > 64 else 16384), "n": n,
                "nrhs": rng.choice([1, 1, 2, 5]), "shift": rng.choice([0.0, float(n)])}
    if kind == "refined":
        return {"kind": kind, "n": _log(rng, 500, 5000), "cond": 10.0 ** rng.uniform(1.0, 3.0)}
    if kind in ("chol", "chol_refined"):
        hi = _log(rng, 24, 384)
        lo = rng.choice([max(4, hi // 32), hi // 2, hi])
        most = 20000 * _mean(8, 256, 3) / _mean(lo, hi, 3)
        return {"kind": kind, "count": _log(rng, 100, min(20000, most)), "lo": lo, "hi": hi,
                "nrhs": rng.choice([1, 2, 4, 4])}
    if kind == "adjoint":
        return {"kind": kind, "batch": _log(rng, 64, 2048), "n": rng.randint(16, 128), "f64": rng.random() < 0.6,
                "recompute": rng.random() < 0.4}
    if kind == "gemm":
        m, n, k = (_log(rng, 48, 5000) for _ in range(3))
        alpha, beta = rng.choice([(1.0, 0.0), (1.0, 0.0), (-1.0, 1.0), (0.5, -0.25)])
        return {"kind": kind, "m": m, "n": n, "k": k, "alpha": alpha, "beta": beta, "spread": rng.choice([0, 0, 20]),
                "slices": rng.choice([0, 0, 3])}
    n = rng.randint(8, 128)
    lo = rng.randint(n, 4 * n)
    hi = rng.randint(lo, max(lo, min(8 * n, 1024)))
    most = 8192 * 320 * 64 ** 2 / ((lo + hi) / 2 * n * n)
    return {"kind": kind, "count": _log(rng, 100, max(120, min(8192, most))), "lo": lo, "hi": hi, "n": n}


# -- inputs --------------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape, dtype=torch.float64):
    return torch.randn(*shape, dtype=dtype, device="cuda", generator=g)


def _sizes(c):
    """The orders (or heights) of a ragged batch: the case's own, whatever the seed of the values."""
    return np.random.default_rng([c["count"], c["lo"], c["hi"]]).integers(c["lo"], c["hi"] + 1, size=c["count"])


def _offsets(sizes):
    return np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.int64)


def _general(c, seed):
    """One n x n system: (A column-major, flat; B column-major, flat)."""
    g = _gen(seed)
    return _randn(g, c["n"] * c["n"]), _randn(g, c["n"] * c["nrhs"])


def _general_batch(c, seed):
    g = _gen(seed)
    n = c["n"]
    a = _randn(g, c["count"], n, n)
    a.diagonal(dim1=1, dim2=2).add_(c["shift"])
    return a, _randn(g, c["count"], c["nrhs"], n)


def _conditioned(c, seed):
    """A = U diag(s) V^T, U and V orthogonal, s log-uniform in [1/cond, 1]."""
    g = _gen(seed)
    n = c["n"]
    u, _ = torch.linalg.qr(_randn(g, n, n))
    v, _ = torch.linalg.qr(_randn(g, n, n))
    e = torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    e[0], e[-1] = 0.0, 1.0
    return (u * c["cond"] ** (-e)) @ v.T, _randn(g, n)


def _groups(ns, off):
    """The matrices of each order: (order, their offsets on the GPU)."""
    for n in np.unique(ns):
        yield int(n), torch.from_numpy(off[ns == n]).cuda()


def _at(off, length):
    return off[:, None] + torch.arange(length, device="cuda")[None, :]


def _ragged_spd(c, seed):
    """Packed SPD matrices A = B B^T + n I and their right-hand sides."""
    g = _gen(seed)
    ns = _sizes(c)
    aoff, boff = _offsets(ns * ns), _offsets(ns * c["nrhs"])
    a = torch.empty(int((ns * ns).sum()), dtype=torch.float64, device="cuda")
    b = _randn(g, int(ns.sum()) * c["nrhs"])
    for n, off in _groups(ns, aoff):
        f = _randn(g, off.numel(), n, n)
        m = torch.bmm(f, f.transpose(1, 2))
        m.diagonal(dim1=1, dim2=2).add_(float(n))
        a[_at(off, n * n)] = m.reshape(off.numel(), n * n)
    return ns, aoff, a, boff, b


def _spd(c, seed):
    g = _gen(seed)
    n, dt = c["n"], torch.float64 if c["f64"] else torch.float32
    f = _randn(g, c["batch"], n, n)
    a = torch.bmm(f, f.transpose(1, 2))
    a.diagonal(dim1=1, dim2=2).add_(float(n))
    b, w = _randn(g, c["batch"], n), _randn(g, c["batch"], n)
    return a.to(dt).reshape(c["batch"], n * n), b.to(dt), w.to(dt)


def _factors(c, seed):
    """A and B (as their column-major images) and C of one product."""
    g = _gen(seed)
    a, b, d = _randn(g, c["k"], c["m"]), _randn(g, c["n"], c["k"]), _randn(g, c["n"], c["m"])
    if c["spread"]:
        s = c["spread"]
        a *= torch.exp2(torch.randint(-s, s + 1, (c["m"],), device="cuda", generator=g).double())[None, :]
        b *= torch.exp2(torch.randint(-s, s + 1, (c["n"],), device="cuda", generator=g).double())[:, None]
    return a, b, d


def _tall(c, seed):
    g = _gen(seed)
    ms = _sizes(c)
    aoff, boff = _offsets(ms * c["n"]), _offsets(ms)
    return ms, aoff, _randn(g, int(ms.sum()) * c["n"]), boff, _randn(g, int(ms.sum()))


# -- state and one pass --------------------------------------------------------------------------------

def _t(buf):
    return torch.as_tensor(buf, device="cuda")


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"case": c}
    if kind == "lu_one":
        s["a"], s["b"] = _general(c, seed)
        s["work"] = na.DeviceBuffer.empty(c["n"] * c["n"])
        s["rhs"] = na.DeviceMatrix(s["b"], c["n"], c["nrhs"])
    elif kind == "lu_batch":
        s["a"], s["b"] = _general_batch(c, seed)
        n, cnt = c["n"], c["count"]
        s["batch"] = na.DeviceBatch(torch.empty_like(s["a"]).reshape(-1), [n] * cnt)
        s["rhs"] = na.DeviceBatch(torch.empty_like(s["b"]).reshape(-1), [n] * cnt, [c["nrhs"]] * cnt)
    elif kind == "refined":
        a, b = _conditioned(c, seed)
        s["a"] = na.DeviceMatrix(a.T.contiguous().reshape(-1), c["n"], c["n"])
        s["rhs"] = na.DeviceMatrix(b, c["n"], 1)
    elif kind in ("chol", "chol_refined"):
        ns, aoff, s["a"], boff, s["b"] = _ragged_spd(c, seed)
        cols = np.full(c["count"], c["nrhs"])
        if kind == "chol":
            s["batch"] = na.DeviceBatch(s["a"].clone(), ns, offsets=aoff)
            s["rhs"] = na.DeviceBatch(s["b"].clone(), ns, cols, boff)
            s["chol"] = s["batch"].cholesky()
            s["graph"] = s["chol"].capture(s["rhs"])
        else:
            s["chol"] = na.DeviceBatch(s["a"], ns, offsets=aoff).cholesky()
            s["rhs"] = na.DeviceBatch(s["b"], ns, cols, boff)
            s["out"] = na.DeviceBatch(torch.empty_like(s["b"]), ns, cols, boff)
    elif kind == "adjoint":
        s["a"], s["b"], s["w"] = _spd(c, seed)
        s["form"] = na.PosvLogdet(c["n"], c["batch"], "float64" if c["f64"] else "float32", c["recompute"])
    elif kind == "gemm":
        a, b, s["c0"] = _factors(c, seed)
        s["a"] = na.DeviceMatrix(a.reshape(-1), c["m"], c["k"])
        s["b"] = na.DeviceMatrix(b.reshape(-1), c["k"], c["n"])
        s["c"] = na.DeviceMatrix(s["c0"].clone().reshape(-1), c["m"], c["n"])
    else:
        ms, aoff, s["a"], boff, s["b"] = _tall(c, seed)
        s["batch"] = na.DeviceBatch(torch.empty_like(s["a"]), ms, np.full(c["count"], c["n"]), aoff)
        s["rhs"] = na.DeviceBatch(torch.empty_like(s["b"]), ms, np.ones(c["count"], np.int64), boff)
    return s


def run(state):
    s, c = state, state["case"]
    kind = c["kind"]
    if kind == "lu_one":
        s["work"].copy_(s["a"])
        lu = na.DeviceMatrix(s["work"], c["n"], c["n"]).lu()
        x = lu.solve(s["rhs"])
        return [_t(x.data), _t(lu.lu.data), _t(lu.ipiv)]
    if kind == "lu_batch":
        s["batch"].data.copy_(s["a"])
        s["rhs"].data.copy_(s["b"])
        lu = s["batch"].lu()
        info = lu.solve_mut(s["rhs"])
        return [_t(s["rhs"].data), _t(s["batch"].data), _t(lu.ipiv), _t(info)]
    if kind == "refined":
        x, _ = na.solve_refined(s["a"], s["rhs"])
        return [_t(x.data)]
    if kind == "chol":
        s["batch"].data.copy_(s["a"])
        s["rhs"].data.copy_(s["b"])
        s["graph"].replay()
        return [_t(s["rhs"].data), _t(s["batch"].data), _t(s["chol"].logdet), _t(s["chol"].info)]
    if kind == "chol_refined":
        s["chol"].solve_refined_into(s["rhs"], s["out"])
        return [_t(s["out"].data), _t(s["chol"].info)]
    if kind == "adjoint":
        x, logdet = s["form"].forward(s["a"], s["b"])
        da, db = s["form"].backward(s["w"])
        return [_t(x), _t(logdet), _t(da), _t(db)]
    if kind == "gemm":
        if c["beta"] != 0.0:
            s["c"].data.copy_(s["c0"])
        na.gemm(s["c"], c["alpha"], s["a"], s["b"], c["beta"], split_slices=c["slices"])
        return [_t(s["c"].data)]
    s["batch"].data.copy_(s["a"])
    s["rhs"].data.copy_(s["b"])
    qr = s["batch"].qr()
    x = qr.solve_mut(s["rhs"])
    return [_t(x), _t(s["batch"].data), _t(qr.diag), _t(s["rhs"].data), _t(qr.info)]


# -- what a pass cannot do without ---------------------------------------------------------------------

def work(case):
    c, kind = case, case["kind"]
    if kind in ("lu_one", "refined", "lu_batch"):
        n, cnt, r = c["n"], c.get("count", 1), c.get("nrhs", 1)
        factors = 0 if kind == "refined" else n * n
        return {"bytes": cnt * 8 * (n * n + factors + 2 * n * r), "flops": cnt * (2 / 3 * n ** 3 + 2 * n * n * r)}
    if kind in ("chol", "chol_refined"):
        n, r = _sizes(c).astype(np.float64), c["nrhs"]
        tri = n * (n + 1) / 2
        return {"bytes": 8 * float((tri * (2 if kind == "chol" else 1) + 2 * r * n).sum()),
                "flops": float((n ** 3 / 3 + 2 * r * n ** 2).sum())}
    if kind == "adjoint":
        n, cnt, size = c["n"], c["batch"], 8 if c["f64"] else 4
        return {"bytes": cnt * size * (n * (n + 1) // 2 * 2 + n * n + 4 * n),
                "flops": cnt * (n ** 3 * (4 / 3 if c["recompute"] else 1.0) + 8 * n * n)}
    if kind == "gemm":
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": 8 * (m * k + k * n + m * n * (2 if c["beta"] else 1)), "flops": 2 * m * n * k}
    m, n = _sizes(c).astype(np.float64), c["n"]
    return {"bytes": 8 * float((2 * m * n + 2 * m + 2 * n).sum()),
            "flops": float((2 * m * n * n - 2 / 3 * n ** 3 + 4 * m * n + n * n).sum())}


# -- the same outputs in plain 64-bit torch ------------------------------------------------------------

def _exact_chol(c, seed):
    ns, aoff, a, boff, b = _ragged_spd(c, seed)
    logdet = torch.empty(c["count"], dtype=torch.float64, device="cuda")
    for n, off in _groups(ns, aoff):
        which = torch.from_numpy(np.nonzero(ns == n)[0]).cuda()
        rows, rhs = _at(off, n * n), _at(torch.from_numpy(boff[ns == n]).cuda(), n * c["nrhs"])
        m = a[rows].reshape(-1, n, n)
        low = torch.linalg.cholesky(m)
        x = torch.cholesky_solve(b[rhs].reshape(-1, c["nrhs"], n).transpose(1, 2), low)
        b[rhs] = x.transpose(1, 2).reshape(-1, c["nrhs"] * n)
        logdet[which] = 2.0 * low.diagonal(dim1=1, dim2=2).log().sum(1)
        # column-major image: the factor's column j is row j of its transpose; the input stays above it
        a[rows] = (low.transpose(1, 2) + torch.tril(m, -1)).reshape(-1, n * n)
    return b, a, logdet


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "lu_one":
        n = c["n"]
        a, b = _general(c, seed)
        lu, piv = torch.linalg.lu_factor(a.reshape(n, n).T)
        x = torch.linalg.lu_solve(lu, piv, b.reshape(c["nrhs"], n).T)
        return [x.T.reshape(-1), lu.T.reshape(-1), None]
    if kind == "lu_batch":
        a, b = _general_batch(c, seed)
        lu, piv = torch.linalg.lu_factor(a.transpose(1, 2))
        x = torch.linalg.lu_solve(lu, piv, b.transpose(1, 2))
        return [x.transpose(1, 2).reshape(-1), lu.transpose(1, 2).reshape(-1), None, None]
    if kind == "refined":
        return [torch.linalg.solve(*_conditioned(c, seed))]
    if kind == "chol":
        return [*_exact_chol(c, seed), None]
    if kind == "chol_refined":
        return [_exact_chol(c, seed)[0], None]
    if kind == "adjoint":
        a, b, w = (t.double() for t in _spd(c, seed))
        n = c["n"]
        low = torch.linalg.cholesky(a.reshape(-1, n, n))
        inv = torch.cholesky_inverse(low)
        x = torch.cholesky_solve(b[:, :, None], low)[:, :, 0]
        v = torch.cholesky_solve(w[:, :, None], low)[:, :, 0]
        # the gradient of the lower entries: an off-diagonal one stands for A_ij and A_ji
        g = inv - v[:, :, None] * x[:, None, :]
        g = torch.tril(g + g.transpose(1, 2), -1) + torch.diag_embed(g.diagonal(dim1=1, dim2=2))
        return [x, 2.0 * low.diagonal(dim1=1, dim2=2).log().sum(1), g.transpose(1, 2).reshape(-1, n * n), v]
    if kind == "gemm":
        a, b, d = _factors(c, seed)
        r = torch.zeros_like(d)
        for k in range(0, c["k"], 256):  # short sums first: fewer roundings than one long one
            r += b[:, k:k + 256] @ a[k:k + 256]
        r *= c["alpha"]
        if c["beta"] != 0.0:
            r += c["beta"] * d
        return [r.reshape(-1)]
    # least squares: two Cholesky-QR passes over the problems padded with zero rows
    ms, aoff, a, boff, b = _tall(c, seed)
    n, hi = c["n"], int(ms.max())
    q = torch.zeros(c["count"], n, hi, dtype=torch.float64, device="cuda")
    y = torch.zeros(c["count"], hi, dtype=torch.float64, device="cuda")
    for m, off in _groups(ms, aoff):
        which = torch.from_numpy(np.nonzero(ms == m)[0]).cuda()
        q[which, :, :m] = a[_at(off, m * n)].reshape(-1, n, m)
        y[which, :m] = b[_at(torch.from_numpy(boff[ms == m]).cuda(), m)]
    r = torch.eye(n, dtype=torch.float64, device="cuda").expand(c["count"], n, n)
    for _ in range(2):
        low = torch.linalg.cholesky(torch.bmm(q, q.transpose(1, 2)))
        q = torch.linalg.solve_triangular(low, q, upper=False)
        r = torch.bmm(low.transpose(1, 2), r)
    x = torch.linalg.solve_triangular(r, torch.bmm(q, y[:, :, None]), upper=True)
    return [x.reshape(-1), None, None, None, None]
