"""A split product's wait that runs out is reported by the next synchronising call, once, and the handle works on.

The self-test runs the split kernels' own wait on a barrier that nobody arrives on, with a 50 ms limit, and records the
outcome where those kernels do.  Nothing faults or hangs."""
import ctypes as C

import numpy as np
import pytest

from oracle import itg_oracle as O

pytestmark = pytest.mark.gpu

CALLS = ["synchronize", "nrm2", "memcpy_d2h", "svd", "davidson"]


def _sync_call(h, name, A):
    import torch
    p = lambda t: C.c_void_p(t.data_ptr())
    if name == "synchronize":
        h.call("itg_synchronize")
    elif name == "nrm2":
        r = C.c_double()
        h.call("itg_nrm2", A.numel(), p(A), C.byref(r))
    elif name == "memcpy_d2h":
        out = np.empty(A.numel())
        h.call("itg_memcpy_d2h", out.ctypes.data_as(C.c_void_p), p(A), C.c_size_t(8 * A.numel()))
    elif name == "svd":
        U, S, V = (torch.empty(n, dtype=torch.float64, device="cuda") for n in (900, 30, 900))
        k, te, dc = C.c_int64(), C.c_double(), C.c_double()
        h.call("itg_svd_trunc", 30, 30, p(A), 30, 30, 1, 0.0, 0, 1, 0, p(U), p(S), p(V), C.byref(k), C.byref(te),
               C.byref(dc))
    else:
        x = A[:36].clone()
        e, nmv = C.c_double(), C.c_int()
        h.call("itg_davidson_heff2", 3, 3, 2, 3, 3, 3, p(A), p(A), p(A), p(A), p(x), 3, 1, 1e-14, 0, C.byref(e),
               C.byref(nmv))


@pytest.mark.parametrize("name", CALLS)
def test_timeout_is_reported_once(gpu, name):
    import torch
    from itg import _lib
    h = _lib.Handle(0)
    try:
        A = torch.from_numpy(np.random.default_rng(1).standard_normal(900)).cuda()
        h.call("itg_set_wait_limit_ns", C.c_uint64(50_000_000))
        h.call("itg_wait_selftest", 2)
        with pytest.raises(_lib.ITGError, match="ran out") as ei:
            _sync_call(h, name, A)
        assert ei.value.status == _lib.ITG_ERR_TIMEOUT
        h.call("itg_set_wait_limit_ns", C.c_uint64(4_000_000_000))
        _sync_call(h, name, A)
        B = torch.empty(900, dtype=torch.float64, device="cuda")
        p = lambda t: C.c_void_p(t.data_ptr())
        d, m = _lib.i64arr([30, 30]), _lib.i32arr
        h.call("itg_contract", 0, 1.0, p(A), 2, d, m([1, 2]), p(A), 2, d, m([2, 3]), 0.0, p(B), 2, d, m([1, 3]), 1)
        h.call("itg_synchronize")
        a = O.unflat(A.cpu().numpy(), (30, 30))
        assert np.linalg.norm(O.unflat(B.cpu().numpy(), (30, 30)) - a @ a) <= 1e-12 * np.linalg.norm(a @ a)
    finally:
        h.close()
