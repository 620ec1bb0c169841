"""Calls on a caller's stream: behind an event of another stream, with the caller's own work and events between the calls,
and inside a capture.  Kernels that may start while their predecessor drains must still see everything before them."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N = 96


@pytest.fixture
def h(gpu):
    from itg import _lib
    h = _lib.Handle(0)
    yield h
    h.close()


def _p(t):
    return C.c_void_p(t.data_ptr())


def _mul(h, A, B, out, prec):
    from itg import _lib
    d, m = _lib.i64arr([N, N]), _lib.i32arr
    h.call("itg_contract", 0, 1.0, _p(A), 2, d, m([1, 2]), _p(B), 2, d, m([2, 3]), 0.0, _p(out), 2, d, m([1, 3]), prec)


@pytest.mark.parametrize("profile", [0, 1], ids=["", "profiled"])
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "split"])
def test_product_behind_another_streams_event(gpu, h, prec, profile):
    """Each operand is written on a second stream after a long fill; the handle's stream waits for its event only."""
    import torch
    rng = np.random.default_rng(5)
    mats = [torch.from_numpy(rng.standard_normal(N * N)).cuda() for _ in range(6)]
    big = torch.empty(1 << 26, dtype=torch.float64, device="cuda")
    A, out = torch.zeros(N * N, dtype=torch.float64, device="cuda"), torch.empty(N * N, dtype=torch.float64, device="cuda")
    got = [torch.empty_like(out) for _ in mats]
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    h.call("itg_set_stream", C.c_void_p(s1.cuda_stream))
    h.call("itg_profile", profile)
    torch.cuda.synchronize()
    with torch.cuda.stream(s1):
        _mul(h, A, A, out, prec)            # plans, tuning
    torch.cuda.synchronize()
    for X, g in zip(mats, got):
        with torch.cuda.stream(s2):
            s2.wait_stream(s1)              # the last product has read A
            big.fill_(1.0)
            A.copy_(X)
            ev = s2.record_event()
        s1.wait_event(ev)
        _mul(h, A, A, out, prec)
        _mul(h, out, A, g, prec)
        with torch.cuda.stream(s1):
            out.fill_(float("nan"))         # the caller's own kernel, then the next call
    torch.cuda.synchronize()
    h.call("itg_profile", 0)
    for X, g in zip(mats, got):
        a = X.cpu().numpy().reshape(N, N)   # row-major view of the column-major data: (A A) A = A (A A)
        ref = a @ a @ a
        assert np.linalg.norm(g.cpu().numpy().reshape(N, N) - ref) <= 1e-12 * np.linalg.norm(ref)


@pytest.mark.parametrize("m,n", [(65, 33), (97, 300), (300, 97)])
def test_qr_in_a_capture(gpu, h, m, n):
    """The QR forks to a stream of its own and joins it: a captured call, replayed on new data, gives the direct call's
    bits."""
    import torch
    r = min(m, n)
    A = torch.randn(m * n, dtype=torch.float64, device="cuda")
    new = lambda k: torch.empty(k, dtype=torch.float64, device="cuda")
    Q, R, Qd, Rd = new(m * r), new(r * n), new(m * r), new(r * n)
    s = torch.cuda.Stream()
    h.call("itg_set_stream", C.c_void_p(s.cuda_stream))
    torch.cuda.synchronize()
    h.call("itg_qr", m, n, _p(A), m, _p(Q), _p(R))      # sizes the workspace
    h.call("itg_synchronize")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        h.call("itg_qr", m, n, _p(A), m, _p(Q), _p(R))
    for _ in range(3):
        A.normal_()
        Q.zero_()
        R.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        h.call("itg_qr", m, n, _p(A), m, _p(Qd), _p(Rd))
        h.call("itg_synchronize")
        assert torch.equal(Q, Qd) and torch.equal(R, Rd)


def test_products_in_a_capture(gpu, h):
    import torch
    A = torch.randn(N * N, dtype=torch.float64, device="cuda")
    outs = [torch.empty_like(A) for _ in range(4)]
    s = torch.cuda.Stream()
    h.call("itg_set_stream", C.c_void_p(s.cuda_stream))
    torch.cuda.synchronize()

    def chain(o):
        for prec in (0, 1):
            _mul(h, A, A, o[prec], prec)
            _mul(h, o[prec], A, o[2 + prec], prec)
    chain(outs)
    h.call("itg_synchronize")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        chain(outs)
    A.normal_()
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    direct = [torch.empty_like(A) for _ in range(4)]
    chain(direct)
    h.call("itg_synchronize")
    assert all(torch.equal(a, b) for a, b in zip(outs, direct))


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "split"])
def test_mixed_product_behind_another_streams_event(gpu, h, prec):
    """real x complex, whose first launch is the product itself: both operands come from a second stream."""
    import torch
    from itg import _lib
    rng = np.random.default_rng(6)
    reals = [rng.standard_normal((N, N)) for _ in range(4)]
    cplx = [rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N)) for _ in range(4)]
    dev = lambda x: torch.from_numpy(x.ravel(order="F").copy()).cuda()
    dr, dc = [dev(x) for x in reals], [dev(x) for x in cplx]
    big = torch.empty(1 << 26, dtype=torch.float64, device="cuda")
    A, B = torch.zeros_like(dr[0]), torch.zeros_like(dc[0])
    got = [torch.empty_like(B) for _ in dr]
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    h.call("itg_set_stream", C.c_void_p(s1.cuda_stream))
    d, m = _lib.i64arr([N, N]), _lib.i32arr
    one, zero = (C.c_double * 2)(1.0, 0.0), (C.c_double * 2)(0.0, 0.0)

    def mul(out):
        h.call("itg_contract_z", 0, 1, one, _p(A), 2, d, m([1, 2]), _p(B), 2, d, m([2, 3]), zero, _p(out), 2, d,
               m([1, 3]), prec)
    torch.cuda.synchronize()
    mul(got[0])                             # plans, tuning
    torch.cuda.synchronize()
    for x, z, g in zip(dr, dc, got):
        with torch.cuda.stream(s2):
            s2.wait_stream(s1)
            big.fill_(1.0)
            A.copy_(x)
            B.copy_(z)
            ev = s2.record_event()
        s1.wait_event(ev)                   # the last thing that the library put on s1 is a product
        mul(g)
    torch.cuda.synchronize()
    for x, z, g in zip(reals, cplx, got):
        ref = x @ z
        # N eps |x| |z|, with |x| |z| ~ sqrt(N) |x z|, is 2e-13
        got_xz = g.cpu().numpy().reshape(N, N, order="F")
        assert np.linalg.norm(got_xz - ref) <= 1e-12 * np.linalg.norm(ref)
