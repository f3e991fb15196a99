"""GPU checks of the Cholesky form whose trailing updates run on the tensor
cores (FMA form, orders above 32): block and tile edges, right-hand sides up to
and past the ones that ride along, failing pivots, NaN and infinities, extreme
scales, the untouched strict upper triangle.

Tolerance: the componentwise backward error of a Cholesky factorization,
|L L^T - A|_ij <= (n + 1) u sqrt(a_ii a_jj) to first order (Higham, Accuracy and
Stability, 10.1), holds for any summation of the inner products; the digit
products add at most n 2^-53 sqrt(a_ii a_jj) (16-deep blocks whose rows are
bounded by sqrt(a_ii)).  The tests allow (2 n + 8) eps64."""
import numpy as np
import pytest

import oracle as O
from nalgebra_gb300 import FLAG_SUBSTITUTE
from tests.conftest import EPS64
from tests.test_chol_gpu import _posv_ragged

pytestmark = pytest.mark.gpu


def _batch(ns, nrhs, seed, scale=None):
    rng = np.random.default_rng(seed)
    mats, rhs = [], []
    for i, n in enumerate(ns):
        f = rng.standard_normal((n, n))
        a = f @ f.T + (n if i % 2 else 0.5) * np.eye(n)
        if scale is not None:
            d = 2.0 ** rng.integers(-scale, scale + 1, size=n)
            a = a * d[:, None] * d[None, :]
        a[np.triu_indices(n, 1)] = rng.standard_normal(n * (n - 1) // 2)  # never read
        mats.append(a)
        rhs.append(rng.standard_normal((n, nrhs)))
    flat = lambda ms: np.concatenate([np.asfortranarray(m).ravel(order="F") for m in ms] + [np.zeros(0)])
    return mats, rhs, flat(mats), flat(rhs)


def _check_factor(a, l, n):
    sym = np.tril(a) + np.tril(a, -1).T
    low = np.tril(l).astype(np.longdouble)
    d = np.sqrt(np.diag(sym))
    err = np.abs((low @ low.T).astype(np.longdouble) - sym)
    assert np.all(err <= (2 * n + 8) * EPS64 * d[:, None] * d[None, :])
    assert np.array_equal(np.triu(l, 1), np.triu(a, 1))
    return sym


@pytest.mark.parametrize("nrhs", [0, 1, 4, 5, 16, 17])
@pytest.mark.parametrize("ns", [[33, 34, 47, 48, 49, 63, 64], [65, 80, 81, 111, 127, 128], [129, 143, 145, 200, 255, 256],
                                [257, 300, 384, 500, 511, 512], [1, 2, 15, 16, 17, 40]])
def test_factor_and_solve(cuda, ns, nrhs):
    mats, rhs, a_flat, b_flat = _batch(ns, nrhs, sum(ns) + nrhs)
    order = np.arange(len(ns)) if ns[0] == 1 else None  # one launch for all orders: small ones on this form too
    A, B, info, logdet, aoff, boff = _posv_ragged(cuda, np.array(ns, np.int32), a_flat, b_flat, nrhs, 0, order=order)
    assert np.all(info == 0)
    for s, n in enumerate(ns):
        sym = np.tril(mats[s]) + np.tril(mats[s], -1).T
        if nrhs in (0, 4, 17):  # the factor does not depend on how many ride along otherwise
            _check_factor(mats[s], A[aoff[s]:aoff[s] + n * n].reshape(n, n).T, n)
        assert abs(logdet[s] - np.linalg.slogdet(sym)[1]) <= 1e-11 * n
        if nrhs:
            x = B[boff[s]:boff[s] + n * nrhs].reshape(nrhs, n).T
            assert O.backward_error(sym, x, rhs[s]) <= n * EPS64


def test_row_scales(cuda):
    """Rows and columns scaled by powers of two up to 2^+-200: the factor scales
    with them, componentwise."""
    ns = [70, 150, 260]
    mats, rhs, a_flat, b_flat = _batch(ns, 2, 3, scale=200)
    A, B, info, logdet, aoff, boff = _posv_ragged(cuda, np.array(ns, np.int32), a_flat, b_flat, 2, 0)
    assert np.all(info == 0)
    for s, n in enumerate(ns):
        _check_factor(mats[s], A[aoff[s]:aoff[s] + n * n].reshape(n, n).T, n)


@pytest.mark.parametrize("power", [-1000, -400, 400, 1000])
def test_whole_matrix_scales(cuda, power):
    n = 100
    mats, rhs, a_flat, b_flat = _batch([n], 1, 9)
    A0, B0, *_ = _posv_ragged(cuda, np.array([n], np.int32), a_flat, b_flat, 1, 0)
    A1, B1, info, *_ = _posv_ragged(cuda, np.array([n], np.int32), np.ldexp(a_flat, power), b_flat, 1, 0)
    assert info[0] == 0
    low = np.tril(np.ones((n, n), bool)).T.ravel()  # column-major image of the lower triangle
    assert np.array_equal(A1[low], np.ldexp(A0[low], power // 2))


def test_failing_pivots_and_special_values(cuda):
    ns = np.array([100, 100, 100, 100, 150, 150], np.int32)
    mats, rhs, _, b_flat = _batch(ns, 2, 5)
    mats[0][37, 37] = -1.0
    mats[1][99, 99] = 0.0
    mats[2][50, 20] = np.nan
    mats[3][60, 60] = np.nan
    mats[4][120, 3] = np.inf
    a_flat = np.concatenate([np.asfortranarray(m).ravel(order="F") for m in mats])
    A, B, info, logdet, aoff, boff = _posv_ragged(cuda, ns, a_flat, b_flat, 2, 0)
    want = O.posv_ragged(ns, aoff, a_flat, boff, b_flat, 2)[2]
    assert np.array_equal(info, want) and info[5] == 0
    assert np.all(np.isnan(logdet[:5]))
    for s in range(5):  # right-hand sides of a failed system stay as given
        n = ns[s]
        assert np.array_equal(B[boff[s]:boff[s] + 2 * n], b_flat[boff[s]:boff[s] + 2 * n])


def test_substitute(cuda):
    n = 90
    mats, rhs, _, b_flat = _batch([n], 1, 6)
    mats[0][30, 30] = -5.0
    a_flat = np.asfortranarray(mats[0]).ravel(order="F")
    A, B, info, *_ = _posv_ragged(cuda, np.array([n], np.int32), a_flat, b_flat, 1, FLAG_SUBSTITUTE, substitute=1e3)
    Lo, info_o = O.cholesky(mats[0], substitute=1e3)
    assert info[0] == info_o == 0
    low = np.tril(np.ones((n, n), bool)).T.ravel()
    assert np.allclose(A[low], np.asfortranarray(Lo).ravel(order="F")[low], rtol=1e-8, atol=1e-8)


def test_reciprocal_square_root(cuda):
    """1 x 1 systems: L = a * rsqrt(a) over the range, within 2 ulps of sqrt(a)
    (rsqrt to about an ulp, and the product's rounding)."""
    rng = np.random.default_rng(1)
    a = np.ldexp(rng.uniform(1.0, 4.0, 20000), 2 * rng.integers(-510, 511, 20000))
    a[:8] = [1.0, 4.0, 2.0 ** -1022, 2.0 ** -1074, np.finfo(float).max, 2.0 ** 1000, 2.0 ** -1000, 3.0]
    A, B, info, *_ = _posv_ragged(cuda, np.ones(a.size, np.int32), a, np.ones(a.size), 1, 0)
    assert np.all(info == 0)
    assert np.all(np.abs(A - np.sqrt(a)) <= 2 * np.spacing(np.sqrt(a)))
