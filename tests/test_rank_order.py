"""The order of singular values behind every factorisation: a permutation whatever the values are.

The gathers read columns through the ranks, so a rank that two values share leaves a slot unwritten.  The rule
(csrc/itg_rank.cuh) is plain C++ and is run here as the kernels run it; on the GPU, matrices with NaN and infinities go
through each kernel that uses it.
"""
import ctypes as C
import itertools
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "itensorsgpu.jl_gb300" / "csrc"
NAN, INF = float("nan"), float("inf")


@pytest.fixture(scope="module")
def order(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("rank")
    (d / "rank.cpp").write_text(
        '#include "itg_rank.cuh"\n'
        'extern "C" void ranks(const double* s, int n, int* rank) {\n'
        "  for (int j = 0; j < n; ++j) {\n"
        "    rank[j] = 0;\n"
        "    for (int i = 0; i < n; ++i) rank[j] += itg_rank_before(s[i], i, s[j], j);\n"
        "  }\n"
        "}\n")
    subprocess.run([cxx, "-O2", "-shared", "-fPIC", "-I", str(CSRC), str(d / "rank.cpp"), "-o", str(d / "rank.so")],
                   check=True)
    lib = C.CDLL(str(d / "rank.so"))

    def run(vals):
        s = np.ascontiguousarray(vals, dtype=np.float64)
        r = np.empty(len(s), dtype=np.int32)
        lib.ranks(s.ctypes.data_as(C.c_void_p), len(s), r.ctypes.data_as(C.c_void_p))
        return r
    return run


def test_ranks_are_a_permutation(order):
    for vals in itertools.product([NAN, INF, 2.0, 2.0, 0.0, -0.0, -1.0], repeat=4):
        r = order(vals)
        assert sorted(r) == list(range(4)), vals
        s = np.empty(4)
        s[r] = vals
        k = int(np.isnan(vals).sum())
        assert np.isnan(s[:k]).all() and (s[k:-1] >= s[k + 1:]).all()


def test_ranks_of_numbers_are_stable(order):
    rng = np.random.default_rng(0)
    v = rng.integers(0, 9, 200).astype(float)
    r = order(v)
    o = np.empty(200, dtype=int)
    o[r] = np.arange(200)
    assert (o == np.argsort(-v, kind="stable")).all()


def _bad(m, n, x, cplx=False):
    rng = np.random.default_rng(m + n)
    A = rng.standard_normal((m, n))
    if cplx:
        A = A + 1j * rng.standard_normal((m, n))
    A[1, 2] = x
    return A


@pytest.mark.gpu
@pytest.mark.parametrize("x", [NAN, INF], ids=["nan", "inf"])
@pytest.mark.parametrize("m,n,cplx", [(6, 5, False), (20, 18, False), (18, 23, False), (60, 40, False), (9, 7, True)])
def test_svd_of_non_finite_input(gpu, m, n, cplx, x):
    """The first singular value is not a number (or infinite); every column of the factors is one of the rotated ones.
    (Weights that are all NaN are truncated to one value, as all-negative ones are.)"""
    i, j = gpu.Index(m), gpu.Index(n)
    U, S, V, _ = gpu.svd(gpu.cuITensor(_bad(m, n, x, cplx), i, j), i)
    s = S.store.data.cpu().numpy()
    assert 1 <= len(s) <= min(m, n) and not np.isfinite(s[0])
    assert U.array().shape == (m, len(s)) and V.array().shape == (n, len(s))
    if not cplx and 12 <= min(m, n) <= 24 and np.isnan(x):
        # columns with NaN are not rotated: the rotations of the others are whole
        q = V.array() if m >= n else U.array()
        assert np.abs(q.T @ q - np.eye(len(s))).max() <= 1e-13


@pytest.mark.gpu
@pytest.mark.parametrize("cplx", [False, True])
def test_eigen_of_non_finite_input(gpu, cplx):
    A = _bad(14, 14, NAN, cplx)
    A = A + A.conj().T
    i = gpu.Index(14)
    D, U, _ = gpu.eigen(gpu.cuITensor(A, i, i.prime()), [i], [i.prime()])
    assert np.isnan(D.store.data.cpu().numpy()[0])


@pytest.mark.gpu
def test_batched_svd_of_non_finite_input(gpu):
    """A bad instance among good ones: its first value is NaN, the others are untouched."""
    import torch
    from itg import _lib
    h = _lib.handle(0)
    shapes = [(12, 10), (9, 13), (30, 20)]
    mats = [np.random.default_rng(q).standard_normal(s) for q, s in enumerate(shapes)]
    mats[1][2, 3] = NAN
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a.T).reshape(-1).copy()).cuda()
    A = [dev(a) for a in mats]
    r = [min(s) for s in shapes]
    out = [[torch.zeros(x * k, dtype=torch.float64, device="cuda") for x, k in zip(dims, r)]
           for dims in ([s[0] for s in shapes], [1] * 3, [s[1] for s in shapes])]
    ptrs = lambda ts: (C.c_void_p * 3)(*[t.data_ptr() for t in ts])
    k, te = (C.c_int64 * 3)(), (C.c_double * 3)()
    h.call("itg_svd_trunc_batched", 3, _lib.i64arr([s[0] for s in shapes]), _lib.i64arr([s[1] for s in shapes]), ptrs(A),
           _lib.i64arr([0, 0, 0]), C.c_int64(1), C.c_double(0.0), 0, 1, 0, ptrs(out[0]), ptrs(out[1]), ptrs(out[2]), k, te)
    for q in range(3):
        s = out[1][q].cpu().numpy()
        if q == 1:
            assert 1 <= k[q] <= r[q] and np.isnan(s[0])
        else:
            ref = np.linalg.svd(mats[q], compute_uv=False)
            assert np.abs(s[: k[q]] - ref[: k[q]]).max() <= 4 * max(shapes[q]) * 2.0 ** -52 * ref[0]
