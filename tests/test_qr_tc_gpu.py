"""GPU checks of the batched QR's trailing update on the tensor cores: row blocks
of 32, column groups of 16, the narrow last panel, zero columns, NaN, extreme
scales, against the oracle's QR::new and least squares.

Tolerance: Householder QR's factors are backward stable columnwise; each panel's
products add errors of a few eps64 times the column's norm, so diag and R agree
with the oracle to 32 n eps64 of the column norm times the (small, N(0,1)
matrices with m >= 1.5 n) condition number: 1e-10 relative, as the other QR tests."""
import numpy as np
import pytest

import oracle as O
from nalgebra_gb300 import workloads as W
from tests.test_qr_gpu import _gels

pytestmark = pytest.mark.gpu


def _compare(w, got):
    A, B, X, diag, info = got
    n = w["n"]
    qr_o, diag_o, x_o, info_o = O.gels_batched(w["ms"], n, w["a_offsets"], w["a_flat"], w["b_offsets"], w["b_flat"])
    assert np.array_equal(info, info_o)
    assert np.array_equal(np.signbit(diag), np.signbit(diag_o))
    scale = np.abs(w["a_flat"]).max()
    assert np.allclose(diag, diag_o, rtol=1e-10, atol=1e-12 * scale)
    assert np.allclose(A, qr_o, rtol=1e-10, atol=1e-11 * max(scale, 1.0))
    ok = info == 0
    assert np.allclose(X[ok], x_o[ok], rtol=1e-9, atol=1e-11)
    return qr_o, diag_o


@pytest.mark.parametrize("n,m_lo,m_hi", [(12, 31, 33), (13, 63, 65), (16, 95, 97), (23, 127, 129), (40, 64, 66), (57, 100, 160),
                                         (64, 511, 513), (65, 129, 200), (100, 160, 161), (128, 255, 257), (17, 2047, 2048)])
def test_row_and_column_edges(cuda, n, m_lo, m_hi):
    w = W.ragged_ls(6, m_lo, m_hi, n, seed=n)
    _compare(w, _gels(cuda, w))
    A, _, _, diag, _ = _gels(cuda, w, with_rhs=False)  # the right-hand side is one more column, no more
    A2, _, _, diag2, _ = _gels(cuda, w)
    assert np.allclose(A, A2, rtol=1e-12, atol=1e-13) and np.allclose(diag, diag2, rtol=1e-12)


def test_zero_columns_and_rank_deficiency(cuda):
    n = 40
    w = W.ragged_ls(5, 70, 90, n, seed=1)
    a = w["a_flat"].copy()
    for s, cols in ((1, [0]), (2, [9, 10]), (3, list(range(8, 24)))):
        m, o = int(w["ms"][s]), int(w["a_offsets"][s])
        for c in cols:
            a[o + c * m:o + (c + 1) * m] = 0.0
    w["a_flat"] = a
    A, B, X, diag, info = _gels(cuda, w)
    qr_o, diag_o, x_o, info_o = O.gels_batched(w["ms"], n, w["a_offsets"], a, w["b_offsets"], w["b_flat"])
    assert np.array_equal(info, info_o) and list(info) == [0, 1, 10, 9, 0]
    # after a zero column the rows' common sign (that of its zero diagonal entry) may differ
    assert np.allclose(np.abs(diag), np.abs(diag_o), rtol=1e-10, atol=1e-12)
    assert np.allclose(np.abs(A), np.abs(qr_o), rtol=1e-10, atol=1e-11 * np.abs(a).max())
    assert np.allclose(X[info == 0], x_o[info == 0], rtol=1e-9, atol=1e-11)


def test_scales(cuda):
    """Columns scaled by powers of two scale R's columns and nothing else."""
    n = 48
    w = W.ragged_ls(3, 100, 140, n, seed=2)
    A, _, _, diag, _ = _gels(cuda, w)
    rng = np.random.default_rng(0)
    e = rng.integers(-300, 301, size=n)
    a = w["a_flat"].copy()
    for s in range(3):
        m, o = int(w["ms"][s]), int(w["a_offsets"][s])
        a[o:o + m * n] = np.ldexp(a[o:o + m * n].reshape(n, m), e[:, None]).ravel()
    w2 = dict(w, a_flat=a)
    A2, _, _, diag2, _ = _gels(cuda, w2)
    assert np.array_equal(diag2, np.ldexp(diag, e[None, :]))


def test_nan_stays_in_its_problem(cuda):
    n = 32
    w = W.ragged_ls(4, 64, 80, n, seed=3)
    clean = _gels(cuda, w)
    a = w["a_flat"].copy()
    a[int(w["a_offsets"][1]) + 11 * int(w["ms"][1]) + 20] = np.nan
    A, B, X, diag, info = _gels(cuda, dict(w, a_flat=a))
    assert np.all(np.isnan(diag[1, 11:])) and np.all(np.isfinite(diag[1, :8]))
    for s in (0, 2, 3):
        assert np.array_equal(X[s], clean[2][s]) and np.array_equal(diag[s], clean[3][s])
