"""Which form a complex solve takes (csrc/ac.cu, AcSlices::build): one block,
clusters, and the block forms where blocks would fetch more halo rows than they
own or do not fit.  Every form ends at ||r|| < 1e-12 ||b|| of its recurrence,
whose distance from b - A x stays within a few hundred roundings of the
diagonally dominant systems' ||A|| ||x||: 1e-10 ||b||.
"""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

from ohmnivore_b200 import mna  # noqa: E402
from ohmnivore_b200 import solver as S  # noqa: E402


@pytest.mark.parametrize("scattered", [0.0, 0.2, 1.0])
@pytest.mark.parametrize("n,per_row", [(1, 1), (33, 4), (1999, 15), (2100, 6), (4999, 15), (10001, 5), (10001, 40),
                                       (29000, 2), (33000, 4)])
def test_complex_solve(n, per_row, scattered):
    rng = np.random.default_rng(n + per_row)
    rows = np.repeat(np.arange(n), rng.integers(1, 2 * per_row, n))
    near = np.clip(rows + rng.integers(-40, 41, len(rows)), 0, n - 1)
    cols = np.where(rng.random(len(rows)) < scattered, rng.integers(0, n, len(rows)), near)
    key = np.unique(np.concatenate([rows * n + cols, np.arange(n) * (n + 1)]))
    rows, cols = key // n, key % n
    val = rng.uniform(-1.0, 1.0, len(key)) + 1j * rng.uniform(-1.0, 1.0, len(key))
    off = np.bincount(rows, np.where(rows == cols, 0.0, np.abs(val)), n)
    val[rows == cols] = (1.2 * off + 0.1) * np.exp(1j * rng.uniform(0.0, 6.0, n))
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    b = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    x = S.GpuSolver(None, S.BiCgStabParams(tolerance=1e-12, max_iterations=2000)).solve_complex(
        mna.Csr(n, n, rp, cols, val), b)
    a = sp.csr_matrix((val, cols, rp), shape=(n, n))
    assert np.linalg.norm(b - a @ x) <= 1e-10 * np.linalg.norm(b)
