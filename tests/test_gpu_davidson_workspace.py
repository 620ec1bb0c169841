"""The queued Davidson at the basis sizes whose projected matrix ends beyond k^2 + 4 k + 8 doubles of its workspace."""
import numpy as np
import pytest

from oracle import itg_oracle as O
from test_gpu_davidson_edges import _problem, _solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kd", [5, 7, 32])
def test_basis_of_general_size(gpu, kd):
    L, R, W1, W2, shape, H, rng = _problem(7, 6, 2, 3, 100 + kd)
    w, V = np.linalg.eigh(H)
    x0 = V[:, 0] + 1e-3 * rng.standard_normal(len(w))
    dg = O.flat(O.heff_diag(L, W1, W2, R))
    th, xr, nr = O.davidson(lambda v: H @ v, x0, dg, kd, 1, 1e-8)
    e, x, nmv = _solve(L, R, W1, W2, shape, x0, kd, 1, 1e-8)
    assert nmv == nr
    # a Ritz value follows its matrix to rounding; the vector to rounding over the gap to the next one
    assert abs(e - th) <= 1e-12 * np.abs(w).max()
    assert np.linalg.norm(x - xr) <= 1e-9
