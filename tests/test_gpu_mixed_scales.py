"""The mixed-precision bond split away from FP32's range: its FP32 Jacobi works on squares of the columns, which leave that
range long before the matrix does."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


@pytest.mark.parametrize("p", [-400, -100, -75, -62, -55, -40, 40, 62, 75, 100, 400])
@pytest.mark.parametrize("m,n,precision", [(60, 60, "fp64"), (210, 200, "fp64"), (230, 200, "split")])
def test_mixed_factorize_at_any_scale(gpu, m, n, p, precision):
    """2^p A gives 2^p times what A gives: the same number of values, an isometry, the product; and on the mixed method
    (no fall-back to the FP64 sweeps)."""
    from itg import _lib
    rng = np.random.default_rng(m + n)
    r = min(m, n)
    U, _ = np.linalg.qr(rng.standard_normal((m, r)))
    V, _ = np.linalg.qr(rng.standard_normal((n, r)))
    s = np.exp(-8.0 * np.arange(r) / r)
    A = (U * s) @ V.T
    k = r // 2
    i, j = gpu.Index(m), gpu.Index(n)
    L, R, spec = gpu.factorize(gpu.cuITensor(np.ldexp(A, p), i, j), i, ortho="left", maxdim=k, mindim=k, method=2,
                               precision=precision)
    mixed = C.c_int()
    _lib.handle(0).call("itg_svd_info", None, C.byref(mixed), None)
    assert mixed.value == 1
    l, rr = L.array(), R.array()
    assert l.shape == (m, k)
    assert np.abs(l.T @ l - np.eye(k)).max() <= 1e-12
    lost = np.linalg.norm(s[k:])
    assert np.linalg.norm(np.ldexp(l @ rr, -p) - A) <= lost * (1 + 1e-9) + 1e-12
