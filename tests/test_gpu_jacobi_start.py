"""The FP32 start of the FP64 Jacobi and its refinement: clusters, columns of rounding noise, graded spectra and
scales near the ends of FP32's range, around the smallest size that takes it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


def _spectrum(kind, r):
    k = np.arange(r) / r
    return {"random": None, "graded": np.exp(-32 * k), "cluster": np.where(k < 0.5, 1.0, 1e-6),
            "deficient": np.where(k < 0.4, np.exp(-8 * k), 0.0), "equal": np.ones(r)}[kind]


@pytest.mark.parametrize("kind", ["random", "graded", "cluster", "deficient", "equal"])
@pytest.mark.parametrize("m,n,scale", [(15, 15, 1.0), (16, 16, 1e-120), (40, 17, 1.0), (24, 24, 1e120), (70, 31, 1e-40),
                                       (64, 64, 1e40), (100, 191, 1.0)])
def test_start_leaves_an_accurate_svd(gpu, m, n, scale, kind):
    """sigma and the product to 4 max(m, n) eps |A|, one factor (the product of rotations) orthonormal to it."""
    rng = np.random.default_rng(m * 31 + n)
    r = min(m, n)
    s = _spectrum(kind, r)
    if s is None:
        A = rng.standard_normal((m, n))
    else:
        U, _ = np.linalg.qr(rng.standard_normal((m, r)))
        V, _ = np.linalg.qr(rng.standard_normal((n, r)))
        A = (U * s) @ V.T
    i, j = gpu.Index(m), gpu.Index(n)
    U, S, V, _ = gpu.svd(gpu.cuITensor(A * scale, i, j), i)
    u, s, v = U.array(), S.store.data.cpu().numpy() / scale, V.array()
    tol = 4 * max(m, n) * EPS
    so = np.linalg.svd(A, compute_uv=False)[: len(s)]
    assert np.abs(s - so).max() <= tol * so[0]
    assert np.linalg.norm((u * s) @ v.T - A) <= tol * np.linalg.norm(A)
    assert min(np.abs(q.T @ q - np.eye(len(s))).max() for q in (u, v)) <= tol
