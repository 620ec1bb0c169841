"""Both tile shapes of the transpose on either side of the rule between them, for copies, sums and general scalars:
the bits of the element-wise form."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-1.0, 1.0), (1.5, 0.0), (0.75, -0.5)])
@pytest.mark.parametrize("dims,order", [((96, 96, 3), (1, 0, 2)), ((80, 5, 80), (2, 1, 0)), ((100, 80), (1, 0)),
                                        ((2, 300, 7), (1, 2, 0)), ((33, 65, 4), (2, 1, 0)), ((45, 45, 2), (1, 0, 2))])
def test_transpose_tiles(gpu, dims, order, alpha, beta):
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
    elif beta == 1.0:
        assert np.array_equal(got, pa + b)
    else:  # beta b is exact, so the fused sum is rounded once like numpy's
        assert np.array_equal(got, pa + beta * b)
