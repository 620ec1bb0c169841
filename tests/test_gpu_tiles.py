"""The narrow tiles (32x32, 16x16) of the FP64 gather-GEMM against the wide ones: bit-identical at
tile edges, remainders and in every operand layout."""
import ctypes as C

import numpy as np
import pytest

from oracle import itg_oracle as O

pytestmark = pytest.mark.gpu


def _arr(t, xs):
    return (t * len(xs))(*xs)


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (16, 16, 16), (17, 15, 33), (33, 31, 5), (129, 65, 47)])
def test_narrow_tiles_bit_identical(gpu, m, n, k, ta, tb):
    import torch
    from itg import _lib
    h = _lib.handle(0)
    dA, mA = ((k, m), (2, 1)) if ta else ((m, k), (1, 2))
    dB, mB = ((n, k), (3, 2)) if tb else ((k, n), (2, 3))
    rng = np.random.default_rng(m * 1000 + n * 10 + k)
    A, B, C0 = rng.standard_normal(dA), rng.standard_normal(dB), rng.standard_normal((m, n))
    a, b = (torch.from_numpy(O.flat(x).copy()).cuda() for x in (A, B))
    p = lambda t: C.c_void_p(t.data_ptr())
    shape = (2, _arr(C.c_int64, dA), _arr(C.c_int32, mA), 2, _arr(C.c_int64, dB), _arr(C.c_int32, mB), 2,
             _arr(C.c_int64, (m, n)), _arr(C.c_int32, (1, 3)))
    outs = []
    for tile in range(5):
        h.call("itg_autotune_force", *shape, tile, 0)
        c = torch.from_numpy(O.flat(C0).copy()).cuda()
        h.call("itg_contract", 0, C.c_double(0.5), p(a), *shape[:3], p(b), *shape[3:6], C.c_double(-1.25), p(c),
               *shape[6:], 0)
        outs.append(c.cpu().numpy())
    h.call("itg_autotune_clear")
    assert all(np.array_equal(outs[0], x) for x in outs[1:])
    ref = 0.5 * O.contract(A, mA, B, mB, (1, 3)) - 1.25 * C0
    # one rounding per term of the depth-k sum, of the scaling and of the update
    bound = 2.0 ** -53 * (k + 3) * (0.5 * np.abs(A if not ta else A.T) @ np.abs(B if not tb else B.T)
                                    + 2 * 1.25 * np.abs(C0))
    assert np.all(np.abs(O.unflat(outs[0], (m, n)) - ref) <= 2 * bound)
