"""Permutation and permuted sums at the edges of the tiles, segments and short modes, and for every form of the
scalars: bit for bit what one multiplication and one fused multiply-add of each element give."""
import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _arr(t, xs):
    return (t * max(1, len(xs)))(*xs)


def _fma(b, y, ax):
    """round(b y + ax) for the scalars used here, all with b y exact or b = 1."""
    return b * y + ax


@pytest.mark.parametrize("dims,perm", [
    ((1,), (0,)), ((8193,), (0,)), ((3, 8200), (0, 1)), ((65, 64), (1, 0)), ((63, 129), (1, 0)), ((1, 7, 1), (2, 1, 0)),
    ((2, 2200, 3), (1, 0, 2)), ((2300, 2, 5), (1, 2, 0)), ((5, 33, 3, 17), (3, 2, 1, 0)), ((129, 4, 3, 63), (0, 3, 2, 1)),
    ((31, 5, 4, 3), (0, 2, 1, 3)), ((2, 2, 2, 2, 2, 2), (5, 3, 1, 0, 2, 4)), ((300, 70, 3), (2, 0, 1))])
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-1.0, 0.0), (0.3, 0.0), (1.0, 1.0), (-1.0, 1.0), (0.3, -2.0)])
def test_permute_and_sum_at_the_edges(gpu, dims, perm, alpha, beta):
    import torch
    from itg import _lib
    h = _lib.handle(0)
    rng = np.random.default_rng(math.prod(dims) + 7)
    A = rng.standard_normal(dims)
    A.flat[0] = -0.0
    out = tuple(dims[p] for p in perm)
    B = rng.standard_normal(out)
    a, b = (torch.from_numpy(x.ravel(order="F").copy()).cuda() for x in (A, B))
    ref = alpha * np.transpose(A, perm)
    mA, mB = list(range(len(dims))), list(perm)
    p = lambda t: C.c_void_p(t.data_ptr())
    if beta == 0.0:
        c = torch.full_like(b, float("nan"))
        h.call("itg_permute", 0, C.c_double(alpha), p(a), len(dims), _arr(C.c_int64, dims), _arr(C.c_int32, mA), p(c),
               _arr(C.c_int32, mB))
        outs = [c]
    else:
        ref = _fma(beta, B, ref)
        c = torch.full_like(b, float("nan"))
        inplace = b.clone()
        for src, dst in ((b, c), (inplace, inplace)):
            h.call("itg_axpby_permuted", 0, C.c_double(alpha), p(a), len(dims), _arr(C.c_int64, dims),
                   _arr(C.c_int32, mA), C.c_double(beta), p(src), _arr(C.c_int32, mB), p(dst))
        outs = [c, inplace]
    for o in outs:
        got = o.cpu().numpy().reshape(out, order="F")
        assert np.array_equal(got, ref) and np.array_equal(np.signbit(got), np.signbit(ref))
