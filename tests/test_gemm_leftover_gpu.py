"""GPU check of the tiles that the FP64 GEMM's modular form leaves to the FP64 kernel:
whatever tile size they take, the bits of nacu_dgemm.  Rows beyond the modular form's
exponents leave every tile; a permutation's products are exact in both forms."""
import numpy as np
import pytest

from nalgebra_gb300 import _lib
from tests.test_gemm_crt_gpu import _run

pytestmark = pytest.mark.gpu


def _fp64(torch, a, b, c, alpha, beta):
    m, k = a.shape
    n = b.shape[1]
    A, B, C = (torch.from_numpy(np.asfortranarray(x).ravel(order="F")).cuda() for x in (a, b, c))
    _lib.call("nacu_dgemm", m, n, k, alpha, A.data_ptr(), m, B.data_ptr(), k, beta, C.data_ptr(), m,
              torch.cuda.current_stream().cuda_stream)
    return C.cpu().numpy().reshape(n, m).T


@pytest.mark.parametrize("m,n,k", [(1, 1, 64), (17, 33, 70), (65, 127, 300), (129, 128, 129), (700, 1100, 257),
                                   (1700, 1601, 200)])
def test_left_over_tiles_have_the_fp64_kernels_bits(cuda, m, n, k):
    rng = np.random.default_rng(m + n + k)
    a, b, c = rng.standard_normal((m, k)), rng.standard_normal((k, n)), rng.standard_normal((m, n))
    a *= 1e250
    c *= 1e250
    for alpha, beta in ((1.0, 0.0), (-0.5, 2.0)):
        assert np.array_equal(_run(cuda, a, b, c, alpha, beta), _fp64(cuda, a, b, c, alpha, beta))
    p = np.zeros((m, k))
    p[np.arange(m), rng.integers(0, k, m)] = 1.0
    assert np.array_equal(_run(cuda, p, b, c, 1.0, 0.0), p @ b)
