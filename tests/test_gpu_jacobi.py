"""The register-resident Jacobi steps at the edges of their block, row and column ranges, FP64 and FP32
(the mixed method's start), against LAPACK."""
import ctypes as C

import numpy as np
import pytest

from oracle import itg_oracle as O

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


def _graded(m, n, seed, decay):
    rng = np.random.default_rng(seed)
    r = min(m, n)
    U, _ = np.linalg.qr(rng.standard_normal((m, r)))
    V, _ = np.linalg.qr(rng.standard_normal((n, r)))
    return (U * np.exp(-decay * np.arange(r) / r)) @ V.T


@pytest.mark.parametrize("m,n", [(11, 11), (12, 12), (13, 13), (24, 24), (25, 25), (33, 26), (40, 64), (128, 128),
                                 (130, 129), (257, 193), (513, 200), (2049, 30)])
def test_fp64_svd_at_the_kernel_edges(gpu, m, n):
    """sigma to the backward error of a stable SVD, 4 max(m, n) eps |A|; both factors orthonormal and the product
    equal to A within the same."""
    A = _graded(m, n, m * 31 + n, 12.0)
    i, j = gpu.Index(m), gpu.Index(n)
    U, S, V, _ = gpu.svd(gpu.cuITensor(A, i, j), i)
    u, s, v = U.array(), S.store.data.cpu().numpy(), V.array()
    tol = 4 * max(m, n) * EPS
    so = np.linalg.svd(A, compute_uv=False)
    assert np.abs(s - so).max() <= tol * so[0]
    assert np.linalg.norm((u * s) @ v.T - A) <= tol * np.linalg.norm(A)
    # one factor is a product of rotations; the other divides by sigma >= e^-12
    for q in (u, v):
        assert np.abs(q.T @ q - np.eye(len(s))).max() <= tol * so[0] / so[-1]
    assert min(np.abs(q.T @ q - np.eye(len(s))).max() for q in (u, v)) <= tol


@pytest.mark.parametrize("m,n", [(200, 200), (203, 197), (1025, 1023), (260, 1000)])
def test_mixed_split_at_the_kernel_edges(gpu, m, n):
    """FP32 start (16-byte and element-wise rows, 4 and 8 rows a thread): isometry 1e-13 as everywhere, and
    L R equal to the truncated SVD to P's accuracy over its gap."""
    r = min(m, n)
    k = r // 2
    rng = np.random.default_rng(m + n)
    U, _ = np.linalg.qr(rng.standard_normal((m, r)))
    V, _ = np.linalg.qr(rng.standard_normal((n, r)))
    s = np.exp(-6.0 * np.arange(r) / r)
    s[k:] *= 0.25
    A = (U * s) @ V.T
    i, j = gpu.Index(m), gpu.Index(n)
    for ortho in ("left", "right"):
        L, R, spec = gpu.factorize(gpu.cuITensor(A, i, j), i, ortho=ortho, maxdim=k, method=2, precision="split")
        Q = L.array() if ortho == "left" else R.array()
        Q = Q.reshape(-1, k)
        assert np.abs(Q.T @ Q - np.eye(k)).max() <= 1e-13
        got = (L * R).array()
        ref = (U[:, :k] * s[:k]) @ V[:, :k].T
        # |dP| <= 1e-13 P_max turns the kept subspace by dP / gap(P), seen in the product times sigma_k
        gap = s[k - 1] ** 2 - s[k] ** 2
        assert np.abs(got - ref).max() <= 1e-13 / gap * s[k - 1] + 1e-12
        assert np.abs(spec.eigs - s[:k] ** 2).max() <= 1e-12


def test_fp64_eigen_of_a_start_in_fp32(gpu):
    """n above the FP32 start's threshold, eigenvalues of both signs and a scale outside FP32's range."""
    n = 210
    rng = np.random.default_rng(3)
    A = rng.standard_normal((n, n)) * 1e60
    A = A + A.T
    i, j = gpu.Index(n), gpu.Index(n)
    D, U, _ = gpu.eigen(gpu.cuITensor(A, i, j), [i], [j])
    w = np.sort(np.linalg.eigvalsh(A))[::-1]
    d = D.store.data.cpu().numpy()
    # |A + c I| <= 2 c with c the largest row sum, at most n max|A|
    assert np.abs(d - w).max() <= 4 * n * EPS * 2 * np.abs(A).sum(axis=0).max()
    u = U.array()
    assert np.abs(u.T @ u - np.eye(n)).max() <= 4 * n * EPS
