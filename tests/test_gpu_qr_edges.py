"""Blocked Householder QR at panel edges, for scales near the ends of FP64's range and degenerate columns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


@pytest.mark.parametrize("scale", [1.0, 1e-155, 1e150])
@pytest.mark.parametrize("m,n", [(1, 1), (2, 3), (31, 31), (33, 32), (64, 65), (65, 33), (300, 97), (97, 300)])
def test_qr_edges(gpu, m, n, scale):
    """Backward error and orthogonality of Householder QR: 8 max(m, n) eps."""
    rng = np.random.default_rng(m * 7 + n)
    A = rng.standard_normal((m, n)) * scale
    if n > 2:
        A[:, 1] = 0.0                      # a zero column
        A[:, 2] = 3.0 * A[:, 0]            # a dependent one
    if m > 4:
        A[3:, n - 1] = 0.0                 # a column that is already reduced
    i, j = gpu.Index(m), gpu.Index(n)
    Q, R = gpu.qr(gpu.cuITensor(A, i, j), i)
    q, r = Q.array(), R.array()
    tol = 8 * max(m, n) * EPS
    assert np.abs(q.T @ q - np.eye(min(m, n))).max() <= tol
    assert np.abs(q @ (r / scale) - A / scale).max() <= tol * max(1.0, np.abs(A / scale).max()) * np.sqrt(min(m, n))
    assert np.all(np.tril(r, -1) == 0) and np.all(np.diag(r) >= 0)
