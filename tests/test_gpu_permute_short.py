"""Transposes with a short mode on either side, at the lengths where the choice of the tile changes: the bits of the
element-wise form, for copies, sums and general scalars, and over many modes of two."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SHORT = [(2, 2), (8, 9), (9, 8), (16, 17), (17, 16), (24, 25), (32, 2), (32, 32), (33, 32), (32, 33), (16, 65), (64, 16),
         (65, 9), (8, 200), (200, 8), (25, 100), (100, 24)]
CASES = [((a, 7, b), (2, 1, 0)) for a, b in SHORT] + [((2,) * 12, tuple(range(12))[::-1]), ((3, 2, 5, 4, 3), (4, 0, 3, 1, 2))]


@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-1.0, 1.0), (1.5, 0.0), (0.75, -0.5)])
@pytest.mark.parametrize("dims,order", CASES)
def test_short_modes(gpu, dims, order, alpha, beta):
    from itg import _lib
    import torch
    h = _lib.handle(0)
    rng = np.random.default_rng(sum(dims))
    a = rng.standard_normal(dims)
    b = rng.standard_normal([dims[i] for i in order])
    flat = lambda x: torch.from_numpy(x.ravel(order="F").copy()).cuda()
    A, B = flat(a), flat(b)
    out = torch.empty_like(B)
    r = len(dims)
    h.call("itg_axpby_permuted", 0, alpha, A.data_ptr(), r, _lib.i64arr(dims), _lib.i32arr(range(1, r + 1)), beta,
           C.c_void_p(B.data_ptr()), _lib.i32arr([i + 1 for i in order]), out.data_ptr())
    h.call("itg_synchronize")
    got = out.cpu().numpy().reshape(b.shape, order="F")
    pa = alpha * a.transpose(order)
    if beta == 0.0:
        assert np.array_equal(got, pa)
    else:  # beta b is exact, so the fused sum is rounded once like numpy's
        assert np.array_equal(got, pa + beta * b)
