"""The batched Davidson after a call that ended early: the staging ring that its kernels read in place belongs to the
next call from the return on, whether that call fits in it or makes it grow."""
import ctypes as C

import numpy as np
import pytest

from oracle import itg_oracle as O

pytestmark = pytest.mark.gpu


def _call(h, probs, x0, kd=4):
    import torch
    from itg import _lib
    dev = lambda a: torch.from_numpy(O.flat(a).copy()).cuda()
    ops = [[dev(p[q]) for p in probs] for q in range(4)]
    x = [torch.from_numpy(v.copy()).cuda() for v in x0]
    n = len(probs)
    ptrs = lambda ts: (C.c_void_p * n)(*[t.data_ptr() for t in ts])
    e, nmv = (C.c_double * n)(), (C.c_int * n)()
    W1, W2 = probs[0][1], probs[0][2]
    h.call("itg_davidson_heff2_batched", n, _lib.i64arr([p[0].shape[0] for p in probs]),
           _lib.i64arr([p[3].shape[0] for p in probs]), C.c_int64(2), C.c_int64(W1.shape[0]), C.c_int64(W1.shape[3]),
           C.c_int64(W2.shape[3]), *[ptrs(t) for t in ops], ptrs(x), kd, 2, C.c_double(1e-14), e, nmv)
    return list(e)


def _problem(cl, cr, seed):
    rng = np.random.default_rng(seed)
    sym = lambda t, a, b: t + np.swapaxes(t, a, b)
    w, d = 3, 2
    return (sym(rng.standard_normal((cl, w, cl)), 0, 2), sym(rng.standard_normal((w, d, d, w)), 1, 2),
            sym(rng.standard_normal((w, d, d, w)), 1, 2), sym(rng.standard_normal((cr, w, cr)), 0, 2))


@pytest.mark.parametrize("count", [4, 150], ids=["same", "grown"])
def test_call_after_one_that_ended_early(gpu, count):
    from itg import _lib
    h = _lib.Handle(0)
    try:
        first = [_problem(6, 5, q) for q in range(4)]
        zero = [np.random.default_rng(q).standard_normal(6 * 4 * 5) for q in range(4)]
        zero[2][:] = 0.0
        with pytest.raises(_lib.ITGError, match="zero start vector 2"):
            _call(h, first, zero)
        probs = [_problem(3 + q % 4, 2 + q % 3, 50 + q) for q in range(count)]
        starts, want = [], []
        for L, W1, W2, R in probs:
            shape = (L.shape[0], 2, 2, R.shape[0])
            n = int(np.prod(shape))
            H = np.stack([O.flat(O.heff_apply(L, W1, W2, R, O.unflat(c, shape))) for c in np.eye(n)], axis=1)
            w, V = np.linalg.eigh(0.5 * (H + H.T))
            x0 = V[:, 0] + 1e-3 * np.random.default_rng(n).standard_normal(n)
            dg = O.flat(O.heff_diag(L, W1, W2, R))
            starts.append(x0)
            want.append((O.davidson(lambda v: H @ v, x0, dg, 4, 2, 1e-14)[0], np.abs(w).max()))
        got = _call(h, probs, starts)
        for e, (th, scale) in zip(got, want):
            assert abs(e - th) <= 1e-12 * scale
    finally:
        h.close()
