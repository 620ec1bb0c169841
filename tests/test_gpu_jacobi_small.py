"""The one-launch FP32 start around its largest sizes (48 columns, 64 and 128 rows), against LAPACK."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("decay", [0.0, 25.0])
@pytest.mark.parametrize("m,n", [(16, 16), (17, 17), (64, 24), (65, 24), (128, 19), (129, 19), (47, 47), (48, 48), (49, 49)])
def test_svd_at_the_edges(gpu, m, n, decay):
    """sigma and the product to 4 max(m, n) eps |A|."""
    rng = np.random.default_rng(m + 7 * n)
    A = rng.standard_normal((m, n)) * np.exp(-decay * np.arange(n) / n)
    i, j = gpu.Index(m), gpu.Index(n)
    U, S, V, _ = gpu.svd(gpu.cuITensor(A, i, j), i)
    u, s, v = U.array(), S.store.data.cpu().numpy(), V.array()
    tol = 4 * max(m, n) * 2.0 ** -52
    so = np.linalg.svd(A, compute_uv=False)
    assert np.abs(s - so).max() <= tol * so[0]
    assert np.linalg.norm((u * s) @ v.T - A) <= tol * np.linalg.norm(A)
