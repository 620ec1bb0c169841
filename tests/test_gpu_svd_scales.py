"""FP64 SVD, factorisation and eigendecomposition near the ends of FP64's range, where the columns' squared norms leave
it, through every kernel that takes a part: the one-CTA sweeps, the FP32 start in one launch and in blocks, the QR before
the sweeps (whose column step has a form of its own for these scales) and the blocked steps.  2^p scales: each result is
compared with that of the unscaled matrix in numpy, so nothing but the range is in question.  (mindim: the truncation's
own weights, sigma^2, are zero at the lower end.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52
# 2^-530 (3e-160): the sum of squares is subnormal; 2^-496 (5e-150) and 2^-486: squares of dot products are
POWERS = [-530, -512, -496, -486, -300, 300, 480, 500]
SHAPES = [(8, 8), (14, 13), (20, 20), (40, 25), (60, 60), (130, 97), (90, 150)]


def _matrix(m, n, p):
    rng = np.random.default_rng(m * 31 + n)
    A = rng.standard_normal((m, n))
    A[:, n - 1] = 0.5 * A[:, 0]            # a dependent column
    return A, np.ldexp(A, p)


@pytest.mark.parametrize("p", POWERS)
@pytest.mark.parametrize("m,n", SHAPES)
def test_svd(gpu, m, n, p):
    """sigma and the product to 4 max(m, n) eps |A|, one factor orthonormal to it."""
    A, B = _matrix(m, n, p)
    i, j = gpu.Index(m), gpu.Index(n)
    U, S, V, _ = gpu.svd(gpu.cuITensor(B, i, j), i, maxdim=min(m, n) - 1, mindim=min(m, n) - 1)
    u, s, v = U.array(), np.ldexp(S.store.data.cpu().numpy(), -p), V.array()
    tol = 4 * max(m, n) * EPS
    so = np.linalg.svd(A, compute_uv=False)
    assert len(s) == min(m, n) - 1
    assert np.abs(s - so[: len(s)]).max() <= tol * so[0]
    assert np.linalg.norm((u * s) @ v.T - A) <= tol * np.linalg.norm(A) + so[len(s)]
    assert min(np.abs(q.T @ q - np.eye(len(s))).max() for q in (u, v)) <= tol


@pytest.mark.parametrize("p", [-530, -496, 480])
@pytest.mark.parametrize("m,n", [(20, 20), (90, 60)])
@pytest.mark.parametrize("ortho", ["left", "right"])
def test_factorize(gpu, m, n, p, ortho):
    A, B = _matrix(m, n, p)
    i, j = gpu.Index(m), gpu.Index(n)
    k = min(m, n) - 1
    L, R, _ = gpu.factorize(gpu.cuITensor(B, i, j), i, ortho=ortho, maxdim=k, mindim=k, precision="fp64")
    l, r = L.array(), R.array() if R.inds[0] in L.inds else R.array().T
    q = l if ortho == "left" else r.T
    tol = 8 * max(m, n) * EPS
    assert np.abs(q.T @ q - np.eye(k)).max() <= tol
    so = np.linalg.svd(A, compute_uv=False)
    assert np.linalg.norm(np.ldexp(l @ r, -p) - A) <= tol * np.linalg.norm(A) + so[k]


@pytest.mark.parametrize("p", POWERS)
@pytest.mark.parametrize("n", [8, 14, 40, 130])
def test_eigen(gpu, n, p):
    A, _ = _matrix(n, n, 0)
    A = A + A.T
    i = gpu.Index(n)
    D, U, _ = gpu.eigen(gpu.cuITensor(np.ldexp(A, p), i, i.prime()), [i], [i.prime()])
    d = np.ldexp(D.store.data.cpu().numpy(), -p)
    w = np.linalg.eigvalsh(A)[::-1]
    # |w_j| + c with c up to sqrt(n) |A|_F is what the sweeps see
    assert np.abs(d - w).max() <= 8 * n * EPS * np.sqrt(n) * np.linalg.norm(A)
