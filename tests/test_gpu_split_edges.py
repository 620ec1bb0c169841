"""Split-precision tiles at the edges of their stages and groups: every variant gives the same bits, within the
stated bound of the FP64 product."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (129, 65, 64), (100, 257, 65), (260, 130, 128), (128, 384, 129),
                                   (300, 200, 191), (520, 129, 1025), (140, 300, 4200), (3000, 900, 70)])
def test_variants_agree(gpu, m, n, k):
    from itg import _lib
    import torch
    h = _lib.handle(0)
    g = torch.Generator().manual_seed(m + n + k)
    A = torch.randn(m * k, dtype=torch.float64, generator=g).cuda()
    B = torch.randn(k * n, dtype=torch.float64, generator=g).cuda()
    d = lambda *v: (2, _lib.i64arr(v))
    a, b, c = (*d(m, k), _lib.i32arr([1, 3])), (*d(k, n), _lib.i32arr([3, 2])), (*d(m, n), _lib.i32arr([1, 2]))
    outs = []
    h.call("itg_set_autotune", 0)
    try:
        for force in (0, 128, 128 | 0x1000, 256, 256 | 0x1000):  # 0: the untimed choice
            if force:
                h.call("itg_autotune_force", *a, *b, *c, -1, force)
            out = torch.empty(m * n, dtype=torch.float64, device="cuda")
            h.call("itg_contract", 0, 1.0, A.data_ptr(), *a, B.data_ptr(), *b, 0.0, out.data_ptr(), *c, 1)
            h.call("itg_synchronize")
            outs.append(out.cpu().numpy())
    finally:
        h.call("itg_autotune_clear")
        h.call("itg_set_autotune", 1)
    for o in outs[1:]:
        assert np.array_equal(o, outs[0])
    An, Bn = A.cpu().numpy().reshape(k, m).T, B.cpu().numpy().reshape(n, k).T
    ref = (An.astype(np.longdouble) @ Bn.astype(np.longdouble)) if m * n * k < 2e7 else An @ Bn
    bound = _lib.load_library().itg_split_error_bound(k) + k * 2.0 ** -53
    assert np.linalg.norm((outs[0].reshape(n, m).T - ref).astype(float)) <= bound * np.linalg.norm(An) * np.linalg.norm(Bn)


@pytest.mark.parametrize("m,n,k", [(3, 700, 300), (257, 33, 2100), (900, 260, 64), (40, 5, 9000)])
def test_operand_orders_agree(gpu, m, n, k):
    """Row exponents of operands with contiguous k and with contiguous rows (found in chunks of k): the same bits."""
    from itg import _lib
    import torch
    h = _lib.handle(0)
    g = torch.Generator().manual_seed(m + n + k)
    A = torch.randn(k, m, dtype=torch.float64, generator=g) * torch.exp2(torch.randint(-40, 40, (k, m), generator=g))
    B = torch.randn(n, k, dtype=torch.float64, generator=g)
    c = (2, _lib.i64arr([m, n]), _lib.i32arr([1, 2]))
    outs = []
    for ta in (0, 1):
        for tb in (0, 1):  # column-major, so the first mode is contiguous
            a = (2, _lib.i64arr([k, m] if ta else [m, k]), _lib.i32arr([3, 1] if ta else [1, 3]))
            b = (2, _lib.i64arr([n, k] if tb else [k, n]), _lib.i32arr([2, 3] if tb else [3, 2]))
            x, y = (A.T if ta else A).contiguous().cuda(), (B.T if tb else B).contiguous().cuda()
            out = torch.empty(m * n, dtype=torch.float64, device="cuda")
            h.call("itg_contract", 0, 1.0, x.data_ptr(), *a, y.data_ptr(), *b, 0.0, out.data_ptr(), *c, 1)
            h.call("itg_synchronize")
            outs.append(out.cpu().numpy())
    for o in outs[1:]:
        assert np.array_equal(o, outs[0])
