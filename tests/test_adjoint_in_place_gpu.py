"""GPU check of the adjoint's backward pass written over its input (dA the factor's, or
the matrix's, own buffer): the same bits as with a buffer of its own."""
import numpy as np
import pytest

from nalgebra_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("recompute", [0, 1])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n", [3, 16, 32, 33, 64, 97, 128])
def test_gradient_over_its_input(cuda, n, dtype, recompute):
    torch = cuda
    rng = np.random.default_rng(n)
    count = 400
    f = rng.standard_normal((count, n, n))
    a = f @ np.transpose(f, (0, 2, 1)) + n * np.eye(n)
    d = lambda x: torch.from_numpy(np.ascontiguousarray(x, dtype=dtype)).cuda()
    A, B, W = d(a), d(rng.standard_normal((count, n))), d(rng.standard_normal((count, n)))
    X, L, db = torch.zeros_like(B), torch.zeros_like(A), torch.zeros_like(B)
    logdet, info = torch.zeros_like(B[:, 0]), torch.zeros(count, dtype=torch.int32, device="cuda")
    pre, s = "d" if dtype == np.float64 else "s", torch.cuda.current_stream().cuda_stream
    _lib.call(f"nacu_{pre}posv_logdet_forward", n, A.data_ptr(), n * n, B.data_ptr(), X.data_ptr(),
              0 if recompute else L.data_ptr(), logdet.data_ptr(), info.data_ptr(), count, s)
    source = A if recompute else L

    def backward(al, da):
        _lib.call(f"nacu_{pre}posv_logdet_backward", n, al.data_ptr(), n * n, recompute, X.data_ptr(), W.data_ptr(),
                  None, da.data_ptr(), db.data_ptr(), info.data_ptr(), count, s)
        return da.cpu().numpy(), db.cpu().numpy()

    want = backward(source, torch.empty_like(A))
    both = source.clone()
    got = backward(both, both)
    assert np.all(info.cpu().numpy() == 0)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
