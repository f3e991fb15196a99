"""GPU checks of the SPD solves on matrices of very different row scales,
A = D A0 D with D powers of two: every step of the factorization and of the solves
commutes with D, so what comes out is the unscaled system's result scaled, to the
bit.  And on matrices whose factors are graded in other ways (smooth kernels,
bands), the solution's residual row by row.

Tolerance of the latter: (3 n + 1) u |L||L^T||x| for the factorization and the two
triangular solves in FP64 (Higham, Accuracy and Stability, 10.4; u = 2^-53); the digit
products stay within the loops' bounds there (at most 2^-50 of the sum of the
magnitudes per 16 terms), for which the bound is doubled."""
import numpy as np
import pytest

from tests.conftest import EPS64
from tests.test_adjoint_gpu import _gpu
from tests.test_chol_gpu import _posv_ragged

pytestmark = pytest.mark.gpu


def _flat(ms):
    return np.concatenate([np.asfortranarray(m).ravel(order="F") for m in ms])


@pytest.mark.parametrize("spread", [20, 200])
@pytest.mark.parametrize("nrhs", [1, 4, 9, 16])
def test_solution_scales_with_the_matrix(cuda, nrhs, spread):
    ns = [33, 47, 64, 70, 129, 150, 256, 260]
    rng = np.random.default_rng(nrhs + spread)
    mats, rhs, d = [], [], []
    for n in ns:
        f = rng.standard_normal((n, n))
        mats.append(f @ f.T + 0.5 * np.eye(n))
        rhs.append(rng.standard_normal((n, nrhs)))
        d.append(2.0 ** rng.integers(-spread, spread + 1, size=(n, 1)))
    A0, B0, info, logdet, aoff, boff = _posv_ragged(cuda, ns, _flat(mats), _flat(rhs), nrhs)
    A1, B1, info1, *_ = _posv_ragged(cuda, ns, _flat([m * s * s.T for m, s in zip(mats, d)]),
                                     _flat([r * s for r, s in zip(rhs, d)]), nrhs)
    assert np.all(info == 0) and np.all(info1 == 0)
    for i, n in enumerate(ns):
        l0, l1 = (np.tril(x[aoff[i]:aoff[i] + n * n].reshape(n, n).T) for x in (A0, A1))
        x0, x1 = (x[boff[i]:boff[i] + n * nrhs].reshape(nrhs, n).T for x in (B0, B1))
        assert np.array_equal(l1, l0 * d[i]) and np.array_equal(x1 * d[i], x0), n


@pytest.mark.parametrize("recompute", [0, 1])
@pytest.mark.parametrize("spread", [20, 200])
def test_adjoint_scales_with_the_matrix(cuda, spread, recompute):
    for n in (48, 97, 128):
        rng = np.random.default_rng(n + spread)
        f = rng.standard_normal((2, n, n))
        a = f @ np.transpose(f, (0, 2, 1)) + np.array([n, 0.5])[:, None, None] * np.eye(n)
        b, w = rng.standard_normal((2, n)), rng.standard_normal((2, n))
        d = 2.0 ** rng.integers(-spread, spread + 1, size=(2, n))
        X0, ld, dA0, db0, info = _gpu(cuda, a.reshape(2, n * n), b, w, n, np.float64, recompute)
        dd = d[:, :, None] * d[:, None, :]
        X1, _, dA1, db1, info1 = _gpu(cuda, (a * dd).reshape(2, n * n), b * d, w * d, n, np.float64, recompute)
        assert np.all(info == 0) and np.all(info1 == 0)
        assert np.array_equal(X1 * d, X0)
        assert np.array_equal(db1 * d, db0) and np.array_equal(dA1 * dd, dA0)


@pytest.mark.parametrize("spread", [0, 30])
def test_graded_factors(cuda, spread):
    rng = np.random.default_rng(spread)
    n, mats, rhs = 200, [], []
    t = np.linspace(0.0, 1.0, n)
    mats.append(np.exp(-((t[:, None] - t[None, :]) / 0.3) ** 2) + 1e-10 * np.eye(n))  # L_rr falls to 1e-5
    rhs.append(np.stack([np.ones(n), np.sin(6 * t), t ** 3], 1))
    band = rng.standard_normal((n, n)) * (np.abs(np.subtract.outer(np.arange(n), np.arange(n))) <= 5)
    mats.append(band @ band.T + 1e-6 * np.eye(n))
    rhs.append(rng.standard_normal((n, 3)))
    arrow = np.diag(rng.uniform(1.0, 2.0, n))
    arrow[-3:, :-3] = rng.standard_normal((3, n - 3)) * 0.01
    arrow = np.tril(arrow) + np.tril(arrow, -1).T
    mats.append(arrow)
    rhs.append(rng.standard_normal((n, 3)))
    d = [2.0 ** rng.integers(-spread, spread + 1, size=(n, 1)) for _ in mats]
    mats = [m * s * s.T for m, s in zip(mats, d)]
    # right-hand sides scaled as the rows are, and not
    rhs = [np.concatenate([r * s, r], 1) for r, s in zip(rhs, d)]
    A, B, info, _, aoff, boff = _posv_ragged(cuda, [n] * len(mats), _flat(mats), _flat(rhs), 6)
    assert np.all(info == 0)
    for i, (a, b) in enumerate(zip(mats, rhs)):
        low = np.abs(np.tril(A[aoff[i]:aoff[i] + n * n].reshape(n, n).T))
        x = B[boff[i]:boff[i] + 6 * n].reshape(6, n).T
        resid = np.abs(b - a.astype(np.longdouble) @ x)
        assert np.all(resid <= (3 * n + 1) * EPS64 * (low @ (low.T @ np.abs(x)))), i
