"""GPU checks of the large FP64 LU on matrices whose rows and columns have very
different scales, by powers of two.  Partial pivoting does not see column scaling,
and every elimination step commutes with both kinds, so the factors keep the
componentwise accuracy of the unscaled matrix's.

Tolerance: |P A - L U| <= n u |L||U| for the elimination in FP64 (Higham, Accuracy
and Stability, 9.2; u = 2^-53).  A 32-deep digit product adds at most 2^-50 of the
sum of its magnitudes, a 128-deep residue product 2^-60.3 sqrt(128) 2^7 = 2^-49.8, so
2^-49 |L||U| in all; numpy's own product n u |L||U|.  That is below 2 n u + 2^-49 <=
1.1 n eps64 from n = 129 on.  The solve, with its two triangular systems: three times
the bound on |L||U||x|."""
import numpy as np
import pytest

import oracle as O
from tests.conftest import EPS64
from tests.test_getrf_large_gpu import _getrf

pytestmark = pytest.mark.gpu


def _scales(rng, n, kind, spread):
    r = 2.0 ** rng.integers(-spread, spread + 1, size=(n, 1)) if kind != "columns" else np.ones((n, 1))
    c = 2.0 ** rng.integers(-spread, spread + 1, size=(1, n)) if kind != "rows" else np.ones((1, n))
    return r, c


def _check(cuda, a, b):
    n = a.shape[0]
    lu, ipiv, info, x, info2 = _getrf(cuda, a, b)
    _, ipiv_o, _ = O.lu(a)
    assert info == 0 and info2 == 0 and np.array_equal(ipiv, ipiv_o)
    low, up = np.tril(lu, -1) + np.eye(n), np.triu(lu)
    pa, pb = a.copy(), b.copy()
    for i, p in enumerate(ipiv):
        if p != i:
            pa[[i, p]], pb[[i, p]] = pa[[p, i]], pb[[p, i]]
    mags = np.abs(low) @ np.abs(up)
    assert np.all(np.abs(pa - low @ up) <= 1.1 * n * EPS64 * mags)
    mags = np.abs(low) @ (np.abs(up) @ np.abs(x))
    assert np.all(np.abs(pb - pa @ x) <= 3.3 * n * EPS64 * mags)
    return lu, ipiv


@pytest.mark.parametrize("spread", [20, 200])
@pytest.mark.parametrize("kind", ["rows", "columns", "both"])
@pytest.mark.parametrize("n", [160, 420, 1025])
def test_scaled_matrices(cuda, n, kind, spread):
    rng = np.random.default_rng(n + spread)
    a, b = rng.standard_normal((n, n)), rng.standard_normal(n)
    r, c = _scales(rng, n, kind, spread)
    _, ipiv = _check(cuda, a * r * c, b * r[:, 0])
    if kind == "columns":
        assert np.array_equal(ipiv, O.lu(a)[1])


@pytest.mark.parametrize("kind,spread", [("columns", 600), ("both", 300)])
def test_scales_whose_quotients_overflow(cuda, kind, spread):
    n = 300
    rng = np.random.default_rng(spread)
    a, b = rng.standard_normal((n, n)), rng.standard_normal(n)
    r, c = _scales(rng, n, kind, spread)
    _check(cuda, a * r * c, b * r[:, 0])


@pytest.mark.parametrize("density", [0.05, 0.5])
def test_scaled_columns_with_zeros(cuda, density):
    """A row of U may be zero in its largest columns: no one exponent serves it."""
    n = 420
    rng = np.random.default_rng(9)
    a = rng.standard_normal((n, n)) * (rng.random((n, n)) < density) + np.diag(rng.standard_normal(n))
    for kind in ("columns", "both"):
        r, c = _scales(rng, n, kind, 100)
        _check(cuda, a * r * c, rng.standard_normal(n) * r[:, 0])


def test_past_the_register_panels(cuda):
    """Order 8200 with scaled rows and columns; the solution on the device."""
    import nalgebra_gb300 as ng

    torch, n = cuda, 8200
    g = torch.Generator(device="cuda").manual_seed(3)
    # column-major matrices as their row-major transposes
    at = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g)
    e = torch.randint(-100, 101, (2, n), device="cuda", generator=g).to(torch.float64)
    at *= torch.exp2(e[0])[:, None] * torch.exp2(e[1])[None, :]
    b = torch.randn(n, dtype=torch.float64, device="cuda", generator=g) * torch.exp2(e[1])
    f, xs = at.clone(), b.clone()
    lu = ng.DeviceMatrix(f.reshape(-1), n, n).lu()
    assert lu.solve_mut(ng.DeviceMatrix(xs, n, 1))  # in place: f[j, i] = LU_ij
    perm = np.arange(n)
    for i, p in enumerate(lu.ipiv.to_numpy()[:n]):
        perm[[i, p]] = perm[[p, i]]
    perm = torch.from_numpy(perm).cuda()
    mags = f.abs().tril().T @ xs.abs()  # |U||x|
    mags = f.abs().triu(1).T @ mags + mags
    resid = (b - at.T @ xs)[perm].abs()
    assert bool((resid <= 3.3 * n * EPS64 * mags).all())


def test_forward_error_no_larger_than_the_fp64_loop(cuda):
    """Sixty systems of order 200 against solutions refined in extended precision:
    the geometric mean of the error is no larger than that of nalgebra's own loop
    (the digit products keep eight levels: about 0.5 of it; seven: 1.2)."""
    import scipy.linalg

    n, logs = 200, []
    for seed in range(60):
        rng = np.random.default_rng([n, seed])
        a, b = rng.standard_normal((n, n)), rng.standard_normal(n)
        x = _getrf(cuda, a, b)[3]
        lu, piv, _ = O.lu(a)
        x_o = O.lu_solve(lu, piv, b)
        f = scipy.linalg.lu_factor(a)
        ref, al = x_o.astype(np.longdouble), a.astype(np.longdouble)
        for _ in range(4):
            ref = ref + scipy.linalg.lu_solve(f, (b - al @ ref).astype(float))
        logs.append(np.log(float(np.max(np.abs(x - ref)) / np.max(np.abs(x_o - ref)))))
    assert np.mean(logs) <= 0.0
