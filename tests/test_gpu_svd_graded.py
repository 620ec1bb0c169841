"""FP64 SVD of matrices whose columns (rows of a wide one) differ by more than 1 / eps in size.  One-sided rotations keep
their singular values and vectors accurate relative to each one's own size, which neither the QR before the sweeps nor the
single FP64 sweep that follows the FP32 start may spoil."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


def _graded(n, p, order):
    rng = np.random.default_rng(n + p)
    B = rng.standard_normal((n + 6, n))
    d = 10.0 ** (-p * np.arange(n) / n)
    d = {"down": d, "up": d[::-1], "mixed": rng.permutation(d)}[order]
    return B * d


@pytest.mark.parametrize("order", ["down", "up", "mixed"])
@pytest.mark.parametrize("wide", [False, True], ids=["tall", "wide"])
@pytest.mark.parametrize("n,p", [(14, 18), (16, 18), (25, 16), (30, 20), (44, 16), (97, 18), (150, 16), (192, 20)])
def test_factors_of_a_graded_matrix(gpu, n, p, wide, order):
    """Both factors orthonormal to 4 n eps, whatever the singular value; the product to 4 n eps |A|."""
    A = _graded(n, p, order)
    M = A.T.copy() if wide else A
    i, j = gpu.Index(M.shape[0]), gpu.Index(M.shape[1])
    U, S, V, _ = gpu.svd(gpu.cuITensor(M, i, j), i, mindim=n)
    u, s, v = U.array(), S.store.data.cpu().numpy(), V.array()
    tol = 4 * n * EPS
    assert len(s) == n
    assert max(np.abs(q.T @ q - np.eye(n)).max() for q in (u, v)) <= tol
    assert np.linalg.norm((u * s) @ v.T - M) <= tol * np.linalg.norm(M)


@pytest.mark.parametrize("order", ["down", "up", "mixed"])
@pytest.mark.parametrize("n,p", [(20, 16), (30, 16), (30, 20)])
def test_values_of_a_graded_matrix(gpu, n, p, order):
    """Every singular value to 4 n eps of itself (times the condition of the scaled matrix, below 100 here), against 45
    digits."""
    mp = pytest.importorskip("mpmath")
    mp.mp.dps = 45
    A = _graded(n, p, order)
    ref = sorted([float(x) for x in mp.svd_r(mp.matrix(A.tolist()), compute_uv=False)], reverse=True)
    i, j = gpu.Index(n + 6), gpu.Index(n)
    U, S, V, _ = gpu.svd(gpu.cuITensor(A, i, j), i, mindim=n)
    rel = np.abs(S.store.data.cpu().numpy() / ref - 1)
    assert rel.max() <= 100 * 4 * n * EPS
