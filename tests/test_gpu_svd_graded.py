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


@pytest.mark.parametrize("n,p,order", [(16, 40, "down"), (24, 60, "mixed"), (44, 40, "up"), (97, 60, "down"),
                                       (150, 40, "mixed")])
def test_sizes_beyond_fp32(gpu, n, p, order):
    """Squared norms further apart than FP32's range: the sweeps must still see which pairs are orthogonal, and end."""
    test_factors_of_a_graded_matrix(gpu, n, p, False, order)


@pytest.mark.parametrize("n,tiny", [(14, 1e-25), (24, 1e-18), (48, 1e-18), (96, 1e-25), (192, 1e-18)])
def test_one_small_column(gpu, n, tiny):
    """A single column far below the others: a few sweeps more than without it, not as many as are allowed."""
    import ctypes as C
    from itg import _lib
    A = np.random.default_rng(n).standard_normal((n, n))
    A[:, 3] *= tiny
    i, j = gpu.Index(n), gpu.Index(n)
    U, S, V, _ = gpu.svd(gpu.cuITensor(A, i, j), i, mindim=n)
    sweeps = C.c_int()
    _lib.handle(0).call("itg_svd_info", C.byref(sweeps), None, None)
    assert sweeps.value <= 8
    tol = 4 * n * EPS
    u, s, v = U.array(), S.store.data.cpu().numpy(), V.array()
    assert max(np.abs(q.T @ q - np.eye(n)).max() for q in (u, v)) <= tol
    assert np.linalg.norm((u * s) @ v.T - A) <= tol * np.linalg.norm(A)
