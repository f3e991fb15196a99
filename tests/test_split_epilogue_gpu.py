"""The split GEMM's read of C, 32 columns ahead of the tile it updates: edges of the
128 x 256 tiles and of the chunks, more than one tile per CTA, and scales whose
sum leaves the range of one power of two.  Bound as the form's other tests: 1e-5
of |A||B| for three slices, and the roundings of beta C."""
import numpy as np
import pytest

from tests.conftest import EPS64
from tests.test_gemm_gpu import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (127, 31, 64), (128, 32, 70), (129, 33, 128), (33, 255, 20), (257, 257, 65),
                                   (4100, 1300, 40)])
@pytest.mark.parametrize("alpha,beta", [(2.0, -1.0), (-0.5, 0.25)])
def test_beta(cuda, m, n, k, alpha, beta):
    rng = np.random.default_rng(m + n + k)
    a, b, c = rng.standard_normal((m, k)), rng.standard_normal((k, n)), rng.standard_normal((m, n))
    got = _run(cuda, "split", a, b, c, alpha, beta, 3)
    bound = 1e-5 * abs(alpha) * (np.abs(a) @ np.abs(b)) + 4 * EPS64 * abs(beta) * np.abs(c)
    assert np.all(np.abs(got - (alpha * (a @ b) + beta * c)) <= bound)


def test_scales_that_cancel_or_leave_the_range(cuda):
    rng = np.random.default_rng(1)
    m, n, k = 40, 40, 32
    a, b = rng.uniform(1, 2, (m, k)), rng.uniform(1, 2, (k, n))
    a[:20] *= 2.0 ** 700
    a[20:] *= 2.0 ** -700
    b[:, :20] *= 2.0 ** -700
    b[:, 20:] *= 2.0 ** 700
    c = np.ones((m, n))
    got = _run(cuda, "split", a, b, c, 1.0, 1.0, 3)
    with np.errstate(over="ignore", under="ignore"):
        want = a @ b + c
    assert np.all(np.isinf(got[:20, 20:])) and np.all(got[20:, :20] == 1.0)
    for s in (np.s_[:20, :20], np.s_[20:, 20:]):
        assert np.all(np.abs(got[s] - want[s]) <= 2e-5 * np.abs(want[s]))
