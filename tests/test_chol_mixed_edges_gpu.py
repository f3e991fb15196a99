"""The refinement form at the edges of its pieces: 32-row blocks of the FP32 solve
and the tiles fetched ahead of it, 8-column pieces of the residual dealt to four
warps, staged columns in one or two passes (256 rows).  Each solution meets the
form's own target, a normwise backward error of n eps64."""
import numpy as np
import pytest

import oracle as O
from tests.conftest import EPS64
from tests.test_chol_mixed_gpu import _mixed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs", [1, 3, 4])
@pytest.mark.parametrize("ns", [[1, 2, 7, 8, 9, 16, 17, 31], [32, 33, 39, 63, 64, 65, 40], [95, 96, 97, 127, 129, 160, 193],
                                [255, 256, 224, 5], [257, 288, 300, 33], [511, 512, 1, 385]])
def test_edges(cuda, ns, nrhs):
    rng = np.random.default_rng(sum(ns) + nrhs)
    mats = []
    for n in ns:
        f = rng.standard_normal((n, n))
        mats.append(f @ f.T + n * np.eye(n))
    rhs = [rng.standard_normal((n, nrhs)) * 10.0 ** rng.uniform(-3, 3, (1, nrhs)) for n in ns]
    a_flat = np.concatenate([m.T.ravel() for m in mats])
    b_flat = np.concatenate([b.T.ravel() for b in rhs])
    A, B, X, info, iters, aoff, boff = _mixed(cuda, ns, a_flat, b_flat, nrhs)
    assert np.array_equal(A, a_flat) and np.array_equal(B, b_flat)
    assert np.all(info == 0) and np.all(iters > 0)
    for s, n in enumerate(ns):
        x = X[boff[s]:boff[s] + n * nrhs].reshape(nrhs, n).T
        for c in range(nrhs):
            assert O.backward_error(mats[s], x[:, c:c + 1], rhs[s][:, c:c + 1]) <= n * EPS64
