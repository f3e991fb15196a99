"""The batched solve's form for one right-hand side against the form for several:
the same operations in the same order, so the same bits, in both modes and types
of arithmetic, singular systems included."""
import numpy as np
import pytest

from nalgebra_gb300 import _lib

pytestmark = pytest.mark.gpu
FLAG_EXACT = 1


@pytest.mark.parametrize("flags", [0, FLAG_EXACT])
@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 63, 64, 65, 96, 97, 127, 128])
def test_same_bits_as_the_form_for_several(cuda, n, flags):
    torch = cuda
    rng = np.random.default_rng(n)
    count = 3
    a = rng.standard_normal((count, n, n))
    a[2, :, n // 2] = 0.0  # exactly singular: information, and the forward solve's result left in B
    b = rng.standard_normal((count, 1, n))
    s = torch.cuda.current_stream().cuda_stream
    A = torch.from_numpy(np.ascontiguousarray(a.transpose(0, 2, 1))).cuda()
    ipiv = torch.zeros(count * n, dtype=torch.int32, device="cuda")
    info = torch.zeros(count, dtype=torch.int32, device="cuda")
    _lib.call("nacu_dgetrf_batched", n, A.data_ptr(), n * n, ipiv.data_ptr(), info.data_ptr(), count, flags, s)
    got, infos = [], []
    for nrhs in (1, 2):
        B = torch.from_numpy(np.repeat(b, nrhs, axis=1).copy()).cuda()
        inf = torch.full((count,), -7, dtype=torch.int32, device="cuda")
        _lib.call("nacu_dgetrs_batched", n, nrhs, A.data_ptr(), n * n, ipiv.data_ptr(), B.data_ptr(), n * nrhs,
                  inf.data_ptr(), count, flags, s)
        torch.cuda.synchronize()
        got.append(B.cpu().numpy()[:, 0])
        infos.append(inf.cpu().numpy())
    assert np.array_equal(infos[0], infos[1]) and infos[0][2] != 0
    assert np.array_equal(got[0].view(np.int64), got[1].view(np.int64))
