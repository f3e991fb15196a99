"""GPU checks of the FP64 GEMM by residues where the FP32 sums of one chunk reach
their 2^24: rows and columns of one value each, whose residue products all have
one sign, with K on both sides of the limits of the single-chunk form.

Tolerance: the products are k a b.  The scaled integers contribute
sqrt(k) 2^-60.3 |a||b| with |a||b| = k |a b| the product of the 2-norms, the
conversion and the update 4 eps64 k |a b|."""
import numpy as np
import pytest

from tests.test_gemm_crt_gpu import EPS64, _run

pytestmark = pytest.mark.gpu

# residues that agree in every term and sums past 2^23 (their quotients by 255 lie next to a tie)
PAIRS = [(191.0, 91.0), (0.03605407017761904, -1.1247242642203534), (0.07225526464417992, 1.6176015886087278),
         (0.35730532898036416, -0.2633927429673586)]


@pytest.mark.parametrize("k", [512, 513, 576, 640, 853, 967, 1021, 1024, 1025])
def test_constant_rows_and_columns(cuda, k):
    m = n = 512
    rng = np.random.default_rng(k)
    u, v = rng.standard_normal(m), rng.standard_normal(n)
    for i, (p, q) in enumerate(PAIRS):
        u[40 * i], v[70 * i] = p, q
    got = _run(cuda, np.repeat(u[:, None], k, 1), np.repeat(v[None, :], k, 0), np.zeros((m, n)), 1.0, 0.0)
    want = np.outer(u.astype(np.longdouble), v) * k
    bound = (np.sqrt(k) * 2.0 ** -60.3 + 4 * EPS64) * np.abs(want)
    worst = np.abs(got - want) / bound
    assert np.all(worst <= 1.0), (int((worst > 1.0).sum()), float(worst.max()))


@pytest.mark.parametrize("k", [853, 1024])
def test_few_valued_operands(cuda, k):
    """Blocks of equal entries and their negatives, the 191 x 91 pair among them."""
    m, n = 300, 270
    rng = np.random.default_rng(k)
    a = rng.choice([191.0, 91.0, -191.0], size=(m, 1)) * np.where(np.arange(k) < 1000, 1.0, -1.0)
    b = rng.choice([91.0, 191.0, 254.0], size=(1, n)) * np.where(np.arange(k) < 1000, 1.0, -1.0)[:, None]
    got = _run(cuda, a, b, np.zeros((m, n)), 1.0, 0.0)
    assert np.array_equal(got, a @ b)  # integers below 2^53
