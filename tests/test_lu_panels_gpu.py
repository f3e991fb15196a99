"""GPU checks of the large LU's register panels: orders around the 32-wide panels,
the 128-wide outer blocks and the cluster sizes, ties, zero columns, NaN, rows
and columns of extreme scale.

Pivots are compared with the oracle's (nalgebra's icamax rule); factors by
||P A - L U||_F / (||A||_F n eps) <= 10 as the other LU tests."""
import numpy as np
import pytest

import oracle as O
from tests.test_getrf_large_gpu import _getrf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [129, 159, 160, 161, 192, 255, 256, 257, 300, 383, 385, 640, 1025])
def test_orders_at_panel_and_block_edges(cuda, n):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    lu, ipiv, info, _, _ = _getrf(cuda, a)
    _, ipiv_o, _ = O.lu(a)
    assert info == 0 and np.array_equal(ipiv, ipiv_o)
    assert O.lu_reconstruction(a, lu, ipiv) <= 10.0


@pytest.mark.parametrize("n", [1030, 2049, 4097])
def test_orders_where_a_row_gets_fewer_threads(cuda, n):
    """8, 4, 2 and 1 threads to a row (up to 1024, 2048, 4096 and 8192 rows below the
    panel's start), zero columns among them; pivots as LAPACK's (the same rule
    where no NaN is in sight)."""
    import warnings

    import scipy.linalg

    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    a[:, [5, 40]] = 0.0
    lu, ipiv, info, _, _ = _getrf(cuda, a)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        _, piv = scipy.linalg.lu_factor(a, check_finite=False)
    assert info == 6 and np.array_equal(ipiv, piv)
    for i, p in enumerate(ipiv):
        if p != i:
            a[[i, p]] = a[[p, i]]
    d = a - (np.tril(lu, -1) + np.eye(n)) @ np.triu(lu)
    assert np.linalg.norm(d) <= 10.0 * np.linalg.norm(a) * n * 2.0 ** -52


def test_least_workspace_updates_on_the_fp64_pipe(cuda, monkeypatch):
    """Without room for the residues: the same pivots, and the mirror does without
    them by itself."""
    import nalgebra_gb300 as ng
    from nalgebra_gb300 import _lib

    n = 300
    rng = np.random.default_rng(8)
    a = rng.standard_normal((n, n))
    _, ipiv_o, _ = O.lu(a)
    full = _lib.load().nacu_getrf_workspace_bytes(n)
    real = ng._work
    sizes = []

    def scarce(nbytes):
        sizes.append(nbytes)
        if nbytes >= full:
            raise _lib.NacuError("out of memory")
        return real(nbytes)

    monkeypatch.setattr(ng, "_work", scarce)
    lu = ng.DeviceMatrix.from_numpy(a).lu()
    x = lu.solve(ng.DeviceMatrix.from_numpy(np.ones((n, 1)))).to_numpy()
    assert sizes[0] == full and max(sizes[1:]) < full
    assert np.array_equal(lu.ipiv.to_numpy()[:n], ipiv_o)
    assert O.lu_reconstruction(a, lu.lu.to_numpy(), ipiv_o) <= 10.0
    assert O.backward_error(a, x, np.ones((n, 1))) <= 10 * n * 2.0 ** -52


@pytest.mark.parametrize("n", [160, 700])
def test_captured_factorization_has_the_same_bits(cuda, n):
    """Two streams, clusters and launches ahead of their predecessors' ends, as a
    CUDA graph replayed on new inputs."""
    import nalgebra_gb300 as ng
    from nalgebra_gb300 import _lib

    rng = np.random.default_rng(n)
    a = [np.asfortranarray(rng.standard_normal((n, n))) for _ in range(3)]
    want = [_getrf(cuda, x)[:2] for x in a]
    W = ng.DeviceMatrix.from_numpy(a[0])
    wsb = _lib.load().nacu_getrf_workspace_bytes(n)
    ws, ipiv, info = (ng.DeviceBuffer.zeros(*x) for x in ((wsb, np.uint8), (n, np.int32), (2, np.int32)))
    g = ng.Graph()
    with g.capture():
        _lib.call("nacu_dgetrf", n, W.data.data_ptr(), n, ipiv.data_ptr(), info.data_ptr(), ws.data_ptr(), wsb,
                  ng.current_stream())
    for x, (lu, piv) in zip(a, want):
        W.data.copy_(x.ravel(order="F"))
        g.replay()
        ng.synchronize()
        assert np.array_equal(ipiv.to_numpy(), piv) and np.array_equal(W.to_numpy(), lu)


def test_ties_take_the_first_position(cuda):
    """Small integers: equal magnitudes in most columns, resolved by the position
    the rows have after the swaps so far.  The eliminations stay exact while the
    entries are dyadic; the first panel is compared in full."""
    rng = np.random.default_rng(4)
    n = 200
    a = rng.choice([-1.0, 1.0], size=(n, n))
    lu, ipiv, info, _, _ = _getrf(cuda, a)
    lu_o, ipiv_o, _ = O.lu(a)
    assert np.array_equal(ipiv[:4], ipiv_o[:4])
    assert O.lu_reconstruction(a, lu, ipiv) <= 10.0
    p = np.eye(n)[:, ::-1] * 3.0  # an exchange matrix: a swap at every step of the first half
    lu, ipiv, info, _, _ = _getrf(cuda, p)
    lu_o, ipiv_o, _ = O.lu(p)
    assert np.array_equal(ipiv, ipiv_o) and np.array_equal(lu, lu_o)


@pytest.mark.parametrize("cols", [[0], [31, 32], [127, 128, 129], [299]])
def test_zero_columns(cuda, cols):
    n = 300
    rng = np.random.default_rng(5)
    a = rng.standard_normal((n, n))
    a[:, cols] = 0.0
    lu, ipiv, info, _, _ = _getrf(cuda, a)
    _, ipiv_o, _ = O.lu(a)
    assert info == cols[0] + 1 and np.array_equal(ipiv, ipiv_o)
    assert O.lu_reconstruction(a, lu, ipiv) <= 10.0


def test_zero_block_and_row_scales(cuda):
    n = 420
    rng = np.random.default_rng(6)
    a = rng.standard_normal((n, n)) * 2.0 ** rng.integers(-200, 201, size=(n, 1))
    lu, ipiv, info, _, _ = _getrf(cuda, a)
    _, ipiv_o, _ = O.lu(a)
    assert info == 0 and np.array_equal(ipiv, ipiv_o)
    b = np.zeros((n, n))
    b[:100, :100] = rng.standard_normal((100, 100))
    lu, ipiv, info, _, _ = _getrf(cuda, b)
    _, ipiv_o, _ = O.lu(b)
    assert info == 101 and np.array_equal(ipiv[:100], ipiv_o[:100])
    assert np.all(lu[:, 100:] == 0.0) and O.lu_reconstruction(b, lu, ipiv) <= 10.0


def test_nan_is_a_pivot_only_in_first_position(cuda):
    n = 180
    rng = np.random.default_rng(7)
    a = rng.standard_normal((n, n))
    a[90, 0] = np.nan  # below the first position: not chosen
    _, ipiv, _, _, _ = _getrf(cuda, a)
    _, ipiv_o, _ = O.lu(a)
    assert ipiv[0] == ipiv_o[0] != 90
    a[90, 0] = 1.0
    a[0, 0] = np.nan  # the first: it wins
    _, ipiv, _, _, _ = _getrf(cuda, a)
    _, ipiv_o, _ = O.lu(a)
    assert ipiv[0] == ipiv_o[0] == 0
