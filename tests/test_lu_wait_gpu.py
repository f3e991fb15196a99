"""GPU check of the large LU's bounded waits: panels whose waits give up at once
report it, the mirror passes it on, and the next factorization is right."""
import numpy as np
import pytest

import oracle as O
from nalgebra_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [129, 300, 1100])
def test_wait_that_runs_out_is_reported(cuda, n):
    import nalgebra_gb300 as ng

    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    good = ng.DeviceMatrix.from_numpy(a).lu()
    b = ng.DeviceMatrix.from_numpy(np.ones((n, 2)))
    assert good.solve(b) is not None

    w = ng.DeviceMatrix.from_numpy(a)
    wsb = _lib.load().nacu_getrf_workspace_bytes(n)
    ws, ipiv, info = (ng.DeviceBuffer.zeros(*x) for x in ((wsb, np.uint8), (n, np.int32), (2, np.int32)))
    _lib.call("nacu_test_dgetrf_wait_limit", n, w.data.data_ptr(), n, ipiv.data_ptr(), info.data_ptr(), 0,
              ws.data_ptr(), wsb, ng.current_stream())
    ng.synchronize()
    assert info.to_numpy()[0] == -1000
    piv = ipiv.to_numpy()
    assert np.all((piv >= np.arange(n)) & (piv < n))  # pivots stay rows of the matrix

    failed = ng.DeviceMatrix.from_numpy(a).lu()
    failed.info.copy_(np.array([-1000, 0], np.int32))
    assert not failed.is_invertible() and failed.solve(b) is None

    again = ng.DeviceMatrix.from_numpy(a).lu()
    assert np.array_equal(again.ipiv.to_numpy()[:n], O.lu(a)[1])
    assert np.array_equal(again.lu.to_numpy(), good.lu.to_numpy())


def test_limits(cuda):
    L = _lib.load()
    assert L.nacu_test_dgetrf_wait_limit(-1, None, 0, None, None, 0, None, 0, None) == -1
    assert L.nacu_test_dgetrf_wait_limit(4, None, 4, None, None, -1, None, 0, None) == -6
    assert L.nacu_test_dgetrf_wait_limit(4, None, 4, None, None, (1 << 20) + 1, None, 0, None) == -6
