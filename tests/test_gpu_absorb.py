"""The batched SVD with its factors put into chain layout, against LAPACK, for both directions and uneven shapes."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("to_left", [0, 1])
@pytest.mark.parametrize("shapes,maxdim", [([(1, 1)], 1), ([(2, 9), (33, 5), (16, 16)], 4), ([(70, 66)] * 3 + [(7, 40)], 64)])
def test_absorbed_factors(gpu, shapes, maxdim, to_left):
    """A B is the truncated SVD and the factor without sigma an isometry, to 4 max(m, n) eps."""
    from itg import _lib
    import torch
    h = _lib.handle(0)
    rng = np.random.default_rng(maxdim)
    mats = [rng.standard_normal(s) for s in shapes]
    cnt = len(shapes)
    dev = lambda *n: torch.empty(int(np.prod(n)), dtype=torch.float64, device="cuda")
    ptrs = lambda ts: (C.c_void_p * cnt)(*[t.data_ptr() for t in ts])
    ms, ns = [s[0] for s in shapes], [s[1] for s in shapes]
    rs = [min(s) for s in shapes]
    A = [torch.from_numpy(np.asfortranarray(x).ravel(order="F").copy()).cuda() for x in mats]
    U, S, V = [dev(m, r) for m, r in zip(ms, rs)], [dev(r) for r in rs], [dev(n, r) for n, r in zip(ns, rs)]
    ks, te = (C.c_int64 * cnt)(), (C.c_double * cnt)()
    i64 = _lib.i64arr
    h.call("itg_svd_trunc_batched", cnt, i64(ms), i64(ns), ptrs(A), i64([maxdim] * cnt), 1, 0.0, 0, 1, 0, ptrs(U),
           ptrs(S), ptrs(V), ks, te)
    assert list(ks) == [min(r, maxdim) for r in rs]
    L, R = [dev(m, k) for m, k in zip(ms, ks)], [dev(k, n) for n, k in zip(ns, ks)]
    h.call("itg_svd_absorb_batched", cnt, i64(ms), i64(ns), ks, ptrs(U), ptrs(S), ptrs(V), to_left, ptrs(L), ptrs(R))
    h.call("itg_synchronize")
    for x, l, r, k in zip(mats, L, R, ks):
        m, n = x.shape
        l, r = l.cpu().numpy().reshape(k, m).T, r.cpu().numpy().reshape(n, k).T
        u, s, vt = np.linalg.svd(x, full_matrices=False)
        tol = 4 * max(m, n) * 2.0 ** -52
        gap = 1.0 if k == len(s) else (s[k - 1] - s[k]) / s[0]
        assert np.linalg.norm(l @ r - (u[:, :k] * s[:k]) @ vt[:k]) <= tol / gap * np.linalg.norm(x)
        q = r.T if to_left else l
        assert np.abs(q.T @ q - np.eye(k)).max() <= tol * s[0] / s[k - 1]
