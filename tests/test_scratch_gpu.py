"""Scratch kept between calls: another allocator of the process gets it back."""
import numpy as np
import pytest

import nalgebra_gb300 as na

pytestmark = pytest.mark.gpu


def test_release_gives_the_scratch_back(cuda):
    torch = cuda
    n = 4096
    m = na.DeviceMatrix.from_numpy(np.eye(n))
    c = na.DeviceMatrix.from_numpy(np.zeros((n, n)))
    na.release_scratch()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    na.gemm(c, 1.0, m, m, 0.0)  # scratch of 1.4 GB
    torch.cuda.synchronize()
    na.release_scratch()
    # but for code that the first launches load
    assert torch.cuda.mem_get_info()[0] > free - (256 << 20)
    na.gemm(c, 1.0, m, m, 0.0)  # and the pool serves again
    assert np.array_equal(c.to_numpy(), np.eye(n))
