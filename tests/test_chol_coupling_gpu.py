"""GPU checks of SPD systems of two parts that lie interleaved, coupled by 2^-60 of
their own entries or not at all, with right-hand sides 2^-70 apart.  Elimination
keeps the small coupling and the small part entry by entry: |A - L L^T| and |b - A x|
are bounded by multiples of |L||L^T| and |L||L^T||x| (Higham, Accuracy and Stability,
10.3 and 10.4).

Tolerance: (n + 1) u and (3 n + 1) u for the loops in FP64 (u = 2^-53), doubled for the
digit products (slices.cuh)."""
import numpy as np
import pytest

from tests.test_chol_gpu import _posv_ragged

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
NS = [33, 48, 65, 100, 129, 200]


def _q(x):
    return x.astype(np.longdouble)


@pytest.mark.parametrize("nrhs", [1, 4, 12])
@pytest.mark.parametrize("coupling", [2.0 ** -60, 0.0])
def test_small_parts_are_kept(cuda, coupling, nrhs):
    rng = np.random.default_rng(nrhs)
    mats, rhs = [], []
    for n in NS:
        f = rng.standard_normal((n, n))
        a = f @ f.T + n * np.eye(n)
        part = rng.random(n) < 0.5
        a[part[:, None] != part[None, :]] *= coupling
        b = rng.standard_normal((n, nrhs))
        b[part] *= 2.0 ** -70
        mats.append(a)
        rhs.append(b)
    flat = lambda ms: np.concatenate([m.ravel(order="F") for m in ms])
    A, B, info, _, aoff, boff = _posv_ragged(cuda, NS, flat(mats), flat(rhs), nrhs)
    assert np.all(info == 0)
    for i, n in enumerate(NS):
        low = np.tril(A[aoff[i]:aoff[i] + n * n].reshape(n, n).T)
        x = B[boff[i]:boff[i] + n * nrhs].reshape(nrhs, n).T
        size = np.abs(low) @ np.abs(low.T)
        rows = rng.choice(n, 33, replace=False)
        assert np.all(np.abs(_q(mats[i][rows]) - _q(low[rows]) @ _q(low.T)) <= 2 * (n + 1) * U * size[rows]), n
        res = _q(rhs[i][rows]) - _q(mats[i][rows]) @ _q(x)
        assert np.all(np.abs(res) <= 2 * (3 * n + 1) * U * (size[rows] @ np.abs(x))), n
