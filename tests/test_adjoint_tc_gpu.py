"""GPU checks of the FP64 adjoint's backward pass at orders above 32, whose
inverse is formed on the tensor cores: block edges, factor stored and
recomputed, a failing matrix among good ones.

Tolerance: the computed inverse of an SPD matrix by L^-T L^-1 has a relative
residual of about n u kappa (Higham, Accuracy and Stability, 14.3); the reference
is formed in extended precision from the same data, so the gradients agree to
8 n eps64 kappa relative to the largest entry."""
import numpy as np
import pytest

from tests.conftest import EPS64
from tests.test_adjoint_gpu import _gpu

pytestmark = pytest.mark.gpu


def _reference(a, b, w):
    inv = np.linalg.inv(a.astype(np.float64)).astype(np.longdouble)
    al = a.astype(np.longdouble)
    inv = inv + inv @ (np.eye(a.shape[0], dtype=np.longdouble) - al @ inv)  # one Newton step in extended precision
    x, v = inv @ b, inv @ w
    g = inv - np.outer(v, x)
    return np.tril(g + g.T, -1) + np.diag(np.diag(g)), v


@pytest.mark.parametrize("recompute", [0, 1])
@pytest.mark.parametrize("n", [33, 47, 48, 49, 64, 65, 96, 97, 112, 127, 128])
def test_gradient_at_block_edges(cuda, n, recompute):
    rng = np.random.default_rng(n)
    count = 3
    f = rng.standard_normal((count, n, n))
    a = f @ np.transpose(f, (0, 2, 1)) + np.array([n, 1.0, 0.1])[:, None, None] * np.eye(n)
    b, w = rng.standard_normal((count, n)), rng.standard_normal((count, n))
    X, logdet, dA, db, info = _gpu(cuda, a.reshape(count, n * n), b, w, n, np.float64, recompute)
    assert np.all(info == 0)
    for s in range(count):
        g, v = _reference(a[s], b[s], w[s])
        got = dA[s]
        tol = 8 * n * EPS64 * np.linalg.cond(a[s])
        assert np.max(np.abs(db[s] - v)) <= tol * np.max(np.abs(v))
        assert np.max(np.abs(got - g)) <= tol * np.max(np.abs(g))
        assert np.all(np.triu(got, 1) == 0.0)


@pytest.mark.parametrize("recompute", [0, 1])
@pytest.mark.parametrize("n", [4, 5, 6, 15, 16, 17, 31, 32, 33, 48, 97, 112, 127, 128])
def test_f32_gradient_at_block_edges(cuda, n, recompute):
    """The FP32 form in blocks of 16: the same bound with FP32's rounding."""
    eps32 = 2.0 ** -23
    rng = np.random.default_rng(n)
    count = 2
    f = rng.standard_normal((count, n, n))
    a = (f @ np.transpose(f, (0, 2, 1)) + np.array([n, 4.0])[:, None, None] * np.eye(n)).astype(np.float32)
    b, w = rng.standard_normal((count, n)).astype(np.float32), rng.standard_normal((count, n)).astype(np.float32)
    X, logdet, dA, db, info = _gpu(cuda, a.reshape(count, n * n), b, w, n, np.float32, recompute)
    assert np.all(info == 0)
    for s in range(count):
        ad, bd, wd = a[s].astype(np.float64), b[s].astype(np.float64), w[s].astype(np.float64)
        g, v = _reference(ad, bd, wd)
        x = np.linalg.solve(ad, bd)
        tol = 8 * n * eps32 * np.linalg.cond(ad)
        assert np.max(np.abs(X[s] - x)) <= tol * np.max(np.abs(x))
        assert abs(logdet[s] - np.linalg.slogdet(ad)[1]) <= tol * n
        assert np.max(np.abs(db[s] - v)) <= tol * np.max(np.abs(v))
        assert np.max(np.abs(dA[s] - g)) <= tol * np.max(np.abs(g))
        assert np.all(np.triu(dA[s], 1) == 0.0)


def test_not_spd_in_the_recompute_form(cuda):
    n, count = 80, 4
    rng = np.random.default_rng(0)
    f = rng.standard_normal((count, n, n))
    a = f @ np.transpose(f, (0, 2, 1)) + n * np.eye(n)
    a[2, 40, 40] = -1.0
    b, w = rng.standard_normal((count, n)), rng.standard_normal((count, n))
    for dtype in (np.float64, np.float32):
        *_, info = _gpu(cuda, a.reshape(count, n * n), b, w, n, dtype, 1)
        assert list(info) == [0, 0, 41, 0]
