"""GPU checks of nacu_dgemm_ws, the FP64 GEMM by residues on the tensor cores,
against the compensated FP64 oracle (Dot2) at sizes around its tiles, chunks
and blocks.

Tolerance.  The scaled rows a' and b' have 2-norms above 2^60.3 and are rounded
to integers, so an element's error is at most sqrt(k)/2 (|a'| + |b'|), i.e.
sqrt(k) 2^-60.3 |a||b| with |a||b| the product of the 2-norms; converting the
integer product rounds once or twice and the alpha / beta update twice more:
4 eps64 (|alpha| |A||B| + |beta C|) elementwise.  Tiles whose |a|.|b| falls
below 2^-7 |a||b| are the FP64 kernel's, within k eps64 |A||B|."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from nalgebra_gb300 import _lib

pytestmark = pytest.mark.gpu
EPS64 = 2.220446049250313e-16


def _run(torch, a, b, c, alpha, beta, pad=0):
    m, k = a.shape
    n = b.shape[1]

    def col_major(x):  # leading dimension rows + pad
        full = np.full((x.shape[0] + pad, x.shape[1]), 7.0, order="F")
        full[:x.shape[0]] = x
        return torch.from_numpy(full.ravel(order="F")).cuda()

    A, B, Cm = col_major(a), col_major(b), col_major(c)
    wsb = _lib.load().nacu_dgemm_workspace_bytes(m, n, k)
    assert wsb > 0, "the sizes of these tests take the tensor-core path"
    ws = torch.full((wsb,), 0x7f, dtype=torch.uint8, device="cuda")
    _lib.call("nacu_dgemm_ws", m, n, k, alpha, A.data_ptr(), m + pad, B.data_ptr(), k + pad, beta, Cm.data_ptr(),
              m + pad, ws.data_ptr(), wsb, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    flag = C.c_int(0)
    _lib.load().nacu_split_gemm_error(C.byref(flag))
    assert flag.value == 0
    return Cm.cpu().numpy().reshape(n, m + pad).T[:m]


def _check(torch, a, b, c, alpha, beta, pad=0, eps=4.0):
    got = _run(torch, a, b, c, alpha, beta, pad)
    ref = O.gemm_dot2(alpha, a, b, beta, c)
    norms = np.linalg.norm(a, axis=1)[:, None] * np.linalg.norm(b, axis=0)[None, :]
    bound = abs(alpha) * np.sqrt(a.shape[1]) * 2.0 ** -60.3 * norms
    bound += eps * EPS64 * (abs(alpha) * (np.abs(a) @ np.abs(b)) + abs(beta) * np.abs(c))
    assert np.all(np.abs(got - ref) <= bound), np.max(np.abs(got - ref) / bound)


@pytest.mark.parametrize("m,n,k", [(256, 512, 256), (257, 511, 300), (520, 130, 1024), (301, 260, 1025), (150, 200, 3001),
                                   (128, 4100, 200), (1, 1, 64), (64, 64, 64), (1, 300, 700), (4097, 1, 300),
                                   (33, 1000, 130)])
@pytest.mark.parametrize("alpha,beta,spread,pad", [(1.0, 0.0, 0, 0), (-0.7, 1.3, 20, 3)])
def test_products(cuda, m, n, k, alpha, beta, spread, pad):
    rng = np.random.default_rng(m + n + k)
    a, b, c = rng.standard_normal((m, k)), rng.standard_normal((k, n)), rng.standard_normal((m, n))
    a *= 2.0 ** rng.integers(-spread, spread + 1, size=(m, 1))
    b *= 2.0 ** rng.integers(-spread, spread + 1, size=(1, n))
    if beta == 0.0:
        c[:] = np.nan  # never read
        got = _run(cuda, a, b, c, alpha, beta, pad)
        assert np.all(np.isfinite(got))
        c[:] = 0.0
    _check(cuda, a, b, c, alpha, beta, pad)


def test_rule_keeps_short_and_thin_products_native():
    """Where the FP64 kernel is the faster one the workspace query says none."""
    query = _lib.load().nacu_dgemm_workspace_bytes
    assert all(query(*s) == 0 for s in [(64, 64, 32), (500, 500, 32), (8192, 1, 64), (64, 8192, 64), (20000, 4, 64), (1, 1, 1)])


def test_integers_are_exact(cuda):
    """Products of 26-bit integers: exact in 53 bits, and so here (the chunks of
    1024 residue products reach the FP32 accumulator's 2^24)."""
    rng = np.random.default_rng(5)
    a = rng.integers(-2 ** 20, 2 ** 20 + 1, size=(300, 2100)).astype(np.float64)
    b = rng.integers(-2 ** 20, 2 ** 20 + 1, size=(2100, 270)).astype(np.float64)
    got = _run(cuda, a, b, np.zeros((300, 270)), 1.0, 0.0)
    assert np.array_equal(got, (a.astype(np.int64) @ b.astype(np.int64)).astype(np.float64))


def test_residue_extremes(cuda):
    """All-equal entries: every residue product has the same sign, so the sums of
    a chunk are as large as they get."""
    m, n, k = 256, 256, 2048
    for v in (1.0, -1.0, 1.0 + 2.0 ** -52, 128.0 / 257.0):
        a, b = np.full((m, k), v), np.full((k, n), 1.0 - 2.0 ** -53)
        _check(cuda, a, b, np.zeros((m, n)), 1.0, 0.0)


def test_rejected_tiles_and_special_values(cuda):
    """Rows and columns the scaled integers cannot serve: entries that never
    meet, NaN, infinities, extreme exponents; zero rows and columns are exact."""
    rng = np.random.default_rng(8)
    m, n, k = 400, 390, 512
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    a[5, :256] *= 1e12   # against b[256:, 7] the large halves never meet
    b[256:, 7] *= 1e12
    b[:256, 7] *= 1e-12
    a[140] = 0.0
    b[:, 200] = 0.0
    a[300] *= 1e270
    a[301] *= 1e-290
    a[302] *= 2.0 ** -1060  # subnormal entries
    got = _run(cuda, a, b, np.zeros((m, n)), 1.0, 0.0)
    ref = O.gemm_dot2(1.0, a, b)
    assert np.all(np.abs(got - ref) <= 2 * k * EPS64 * (np.abs(a) @ np.abs(b)) + 1e-300)
    assert np.all(got[140] == 0.0) and np.all(got[:, 200] == 0.0)
    a[9, 3], b[500, 310], a[350, 4] = np.nan, np.inf, -np.inf
    with np.errstate(invalid="ignore"):
        ref2 = a @ b
    got2 = _run(cuda, a, b, np.zeros((m, n)), 1.0, 0.0)
    assert np.array_equal(np.isnan(got2), np.isnan(ref2))
    inf = np.isinf(ref2)
    assert np.array_equal(got2[inf], ref2[inf])
    rows = np.isfinite(a).all(axis=1)
    cols = np.isfinite(b).all(axis=0)
    keep = rows[:, None] & cols[None, :]
    assert np.all(np.abs(got2 - ref)[keep] <= (2 * k * EPS64 * (np.abs(a[rows]) @ np.abs(b[:, cols])) + 1e-300).ravel())


def test_blocks_in_every_direction(cuda):
    """More than one block of 4096 rows, 4096 columns or 8192 products, checked
    against torch's FP64 product of the same operands."""
    torch = cuda
    for m, n, k in ((4200, 300, 500), (300, 4200, 500), (260, 270, 8300)):
        g = torch.Generator(device="cuda").manual_seed(m + k)
        A = torch.randn(k, m, dtype=torch.float64, device="cuda", generator=g)
        B = torch.randn(n, k, dtype=torch.float64, device="cuda", generator=g)
        D = torch.randn(n, m, dtype=torch.float64, device="cuda", generator=g)
        want = 0.5 * (B @ A) - 2.0 * D
        wsb = _lib.load().nacu_dgemm_workspace_bytes(m, n, k)
        ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
        _lib.call("nacu_dgemm_ws", m, n, k, 0.5, A.data_ptr(), m, B.data_ptr(), k, -2.0, D.data_ptr(), m,
                  ws.data_ptr(), wsb, torch.cuda.current_stream().cuda_stream)
        scale = B.abs() @ A.abs()
        assert bool(((D - want).abs() <= (0.5 * k + 8) * EPS64 * (scale + 1)).all())


def test_mirror_gemm_eager_and_captured(cuda):
    """gemm() takes its scratch in stream order, also inside a graph capture."""
    import nalgebra_gb300 as ng

    rng = np.random.default_rng(2)
    a, b = rng.standard_normal((400, 500)), rng.standard_normal((500, 300))
    A, B = ng.DeviceMatrix.from_numpy(a), ng.DeviceMatrix.from_numpy(b)
    c1 = ng.gemm(ng.DeviceMatrix.from_numpy(np.zeros((400, 300))), 1.0, A, B, 0.0).to_numpy()
    c = ng.DeviceMatrix.from_numpy(np.zeros((400, 300)))
    g = ng.Graph()
    with g.capture():
        ng.gemm(c, 1.0, A, B, 0.0)
    for _ in range(2):
        g.replay()
    ng.synchronize()
    assert np.array_equal(c.to_numpy(), c1)
    A.data.copy_(np.asfortranarray(2 * a).ravel(order="F"))
    g.replay()
    ng.synchronize()
    assert np.array_equal(c.to_numpy(), 2 * c1)
