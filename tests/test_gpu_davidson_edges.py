"""The queued Davidson at its edges: unrolled and general basis sizes, restarts, a start that is already converged (its
queued vector is dropped), a cancelled correction, sizes down to one element per bond, a zero start."""
import ctypes as C

import numpy as np
import pytest

from oracle import itg_oracle as O

pytestmark = pytest.mark.gpu


def _problem(cl, cr, d, w, seed):
    rng = np.random.default_rng(seed)
    sym = lambda t, a, b: t + np.swapaxes(t, a, b)
    L, R = sym(rng.standard_normal((cl, w, cl)), 0, 2), sym(rng.standard_normal((cr, w, cr)), 0, 2)
    W1, W2 = sym(rng.standard_normal((w, d, d, w)), 1, 2), sym(rng.standard_normal((w, d, d, w)), 1, 2)
    n = cl * d * d * cr
    shape = (cl, d, d, cr)
    H = np.stack([O.flat(O.heff_apply(L, W1, W2, R, O.unflat(np.eye(n)[:, q], shape))) for q in range(n)], axis=1)
    return L, R, W1, W2, shape, 0.5 * (H + H.T), rng


def _solve(L, R, W1, W2, shape, x0, kd, mi, tol, prec=0):
    import torch
    from itg import _lib
    h = _lib.handle(0)
    dev = lambda a: torch.from_numpy(O.flat(a).copy()).cuda()
    p = lambda t: C.c_void_p(t.data_ptr())
    ops = [dev(a) for a in (L, W1, W2, R)]
    x = torch.from_numpy(x0.copy()).cuda()
    e, nmv = C.c_double(), C.c_int()
    cl, d, _, cr = shape
    h.call("itg_davidson_heff2", *[C.c_int64(v) for v in (cl, cr, d, W1.shape[0], W1.shape[3], W2.shape[3])],
           *[p(t) for t in ops], p(x), kd, mi, C.c_double(tol), prec, C.byref(e), C.byref(nmv))
    return e.value, x.cpu().numpy(), nmv.value


@pytest.mark.parametrize("cl,cr", [(1, 1), (1, 5), (7, 6)])
@pytest.mark.parametrize("kd,mi", [(2, 1), (3, 2), (4, 3), (6, 2), (9, 1)])
def test_queued_davidson_matches_oracle(gpu, cl, cr, kd, mi):
    L, R, W1, W2, shape, H, rng = _problem(cl, cr, 2, 3, 10 * cl + cr)
    w, V = np.linalg.eigh(H)
    x0 = V[:, 0] + 1e-3 * rng.standard_normal(len(w))
    dg = O.flat(O.heff_diag(L, W1, W2, R))
    th, xr, nr = O.davidson(lambda v: H @ v, x0, dg, kd, mi, 1e-14)
    e, x, nmv = _solve(L, R, W1, W2, shape, x0, kd, mi, 1e-14)
    assert nmv == nr
    # a Ritz value follows its matrix to rounding; the vector to rounding over the gap to the next one
    assert abs(e - th) <= 1e-12 * np.abs(w).max()
    assert np.linalg.norm(x - xr) <= 1e-9
    assert abs(np.linalg.norm(x) - 1) <= 1e-14


@pytest.mark.parametrize("tol,expect", [(1e-3, 1), (1e-30, None)])
def test_converged_start(gpu, tol, expect):
    """An eigenvector as the start: above the tolerance's residual nothing but the first matvec counts; below it the
    correction is rounding noise."""
    L, R, W1, W2, shape, H, rng = _problem(5, 4, 2, 3, 3)
    w, V = np.linalg.eigh(H)
    e, x, nmv = _solve(L, R, W1, W2, shape, 2.5 * V[:, 0], 3, 2, tol)
    if expect is not None:
        assert nmv == expect
    assert abs(e - w[0]) <= 1e-12 * np.abs(w).max()
    assert min(np.linalg.norm(x - V[:, 0]), np.linalg.norm(x + V[:, 0])) <= 1e-10


def test_zero_start_is_refused(gpu):
    from itg import _lib
    L, R, W1, W2, shape, H, rng = _problem(3, 3, 2, 3, 4)
    with pytest.raises(_lib.ITGError, match="zero start vector"):
        _solve(L, R, W1, W2, shape, np.zeros(H.shape[0]), 3, 2, 1e-14)
