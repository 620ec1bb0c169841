"""Sixteen-column blocks of the FP32 Jacobi steps around the sizes that take them, against LAPACK."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(63, 63), (64, 64), (65, 65), (256, 70), (255, 80), (257, 81), (256, 256), (100, 97)])
def test_svd_at_the_block_edges(gpu, m, n):
    """sigma and the product to 4 max(m, n) eps |A|."""
    rng = np.random.default_rng(m + 7 * n)
    A = rng.standard_normal((m, n)) * np.exp(-10.0 * np.arange(n) / n)
    i, j = gpu.Index(m), gpu.Index(n)
    U, S, V, _ = gpu.svd(gpu.cuITensor(A, i, j), i)
    u, s, v = U.array(), S.store.data.cpu().numpy(), V.array()
    tol = 4 * max(m, n) * 2.0 ** -52
    so = np.linalg.svd(A, compute_uv=False)
    assert np.abs(s - so).max() <= tol * so[0]
    assert np.linalg.norm((u * s) @ v.T - A) <= tol * np.linalg.norm(A)
