"""GPU check of the batched least squares' accuracy against nalgebra's own loop (the
oracle), for rows of one scale and of very different scales: over thirty problems the
geometric mean of the solutions' error, componentwise and against extended precision,
is no larger than the FP64 loop's.  (The trailing update's digit products keep eight
levels: 0.6 to 0.7 of it; with seven 0.8, and 1.3 to 1.4 for scaled rows.)"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _reference(a, b):
    """Householder least squares in extended precision, large rows first."""
    order = np.argsort(-np.abs(a).max(axis=1))
    a, b = a[order].astype(np.longdouble), b[order].astype(np.longdouble)
    n = a.shape[1]
    for j in range(n):
        v = a[j:, j].copy()
        v[0] += np.copysign(np.sqrt(v @ v), v[0])
        t = 2 / (v @ v)
        a[j:, j:] -= np.outer(v, t * (v @ a[j:, j:]))
        b[j:] -= v * (t * (v @ b[j:]))
    x = np.zeros(n, np.longdouble)
    for j in range(n - 1, -1, -1):
        x[j] = (b[j] - a[j, j + 1:] @ x[j + 1:]) / a[j, j]
    return x


@pytest.mark.parametrize("rows", ["one scale", "falling", "rising"])
def test_error_no_larger_than_the_fp64_loop(cuda, rows):
    import nalgebra_gb300 as ng

    m, n, mats, rhs = 160, 48, [], []
    for seed in range(30):
        rng = np.random.default_rng(seed)
        a, b = rng.standard_normal((m, n)), rng.standard_normal((m, 1))
        if rows != "one scale":
            s = np.sort(2.0 ** rng.integers(-20, 21, size=(m, 1)), axis=0)
            s = s[::-1] if rows == "falling" else s
            a, b = a * s, b * s
        mats.append(a)
        rhs.append(b)
    x = ng.DeviceBatch.from_numpy(mats).qr().solve(ng.DeviceBatch.from_numpy(rhs))
    logs = []
    for a, b, got in zip(mats, rhs, x):
        ref = _reference(a, b[:, 0])
        qr, diag = O.qr(a)[:2]
        loop = O.qr_ls_solve(qr, diag, b[:, 0])[0].ravel()
        logs.append(np.log(float(np.max(np.abs((got - ref) / ref)) / np.max(np.abs((loop - ref) / ref)))))
    assert np.mean(logs) <= 0.0, np.exp(np.mean(logs))
