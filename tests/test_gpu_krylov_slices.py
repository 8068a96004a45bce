"""Slice layouts of the single-system Krylov solve (csrc/solver_kernel.cuh,
``krylov_slice``) against the global-memory solve, which runs the same
iteration in the same order: the results must be equal bit for bit.  Sizes at
the edges: one block (up to 1,024 rows), clusters of 2 to 16 blocks (up to
27,200), grids beyond, ragged 32-row slices, rows of uneven length, pairs whose two rows
belong to different blocks, slices too large for shared memory, several lanes
per row.  Small systems are also compared with a dense solve.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from ohmnivore_b200 import _lib, circuits as ck, mna  # noqa: E402
from ohmnivore_b200 import solver as S  # noqa: E402


def _both(a, b, params):
    ctx = S.Context(0)
    try:
        out = []
        for layout in (_lib.KRYLOV_LAYOUT_AUTO, _lib.KRYLOV_LAYOUT_GLOBAL):
            ctx.set_krylov_layout(layout)
            solver = S.GpuSolver(ctx, params)
            out.append((solver.solve_real(a, b), solver.last_info["krylov_iterations"]))
    finally:
        ctx.close()
    (xs, ks), (xg, kg) = out
    np.testing.assert_array_equal(xs, xg)
    assert ks == kg
    return xs


def _random_system(n, per_row, seed, wide_rows=0):
    """Rows of 1 to 2 per_row - 1 random nonzeros (wide_rows of them 100) and
    a dominant diagonal."""
    rng = np.random.default_rng(seed)
    count = rng.integers(1, 2 * per_row, n)
    count[rng.permutation(n)[:wide_rows]] = 100
    rows = np.repeat(np.arange(n), count)
    cols = np.where(rng.random(len(rows)) < 0.8, np.clip(rows + rng.integers(-40, 41, len(rows)), 0, n - 1),
                    rng.integers(0, n, len(rows)))
    key = np.unique(np.concatenate([rows * n + cols, np.arange(n) * (n + 1)]))
    rows, cols = key // n, key % n
    val = rng.uniform(-1.0, 1.0, len(key))
    off = np.bincount(rows, np.where(rows == cols, 0.0, np.abs(val)), n)
    val[rows == cols] = 1.5 * off + 0.1
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    return mna.Csr(n, n, rp, cols, val), rng.standard_normal(n)


@pytest.mark.parametrize("n", [1, 31, 33, 1024, 1025, 2049, 16385, 27200, 27201, 40007])
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "mixed"])
def test_sizes(n, prec):
    a, b = _random_system(n, 2, n, wide_rows=n // 500)
    x = _both(a, b, S.BiCgStabParams(tolerance=1e-12, max_iterations=2000, precision=prec, max_refinements=8))
    r = b - a.spmv(x)
    assert np.linalg.norm(r) <= 1e-11 * np.linalg.norm(b)


@pytest.mark.parametrize("per_row", [4, 8, 16, 40])
@pytest.mark.parametrize("n", [700, 5001, 20011])
def test_lanes_per_row(per_row, n):
    a, b = _random_system(n, per_row, per_row)
    x = _both(a, b, S.BiCgStabParams(tolerance=1e-12, max_iterations=2000))
    assert np.linalg.norm(b - a.spmv(x)) <= 1e-11 * np.linalg.norm(b)


@pytest.mark.parametrize("nodes", [900, 6000, 30000])
def test_pairs_across_blocks(nodes):
    """Voltage sources along a ladder: their branch rows come last, so the
    2x2 pairs join rows of different blocks."""
    rng = np.random.default_rng(nodes)
    c = ck.CircuitBuilder()
    k = np.arange(1, nodes, dtype=np.int64)
    c.resistors(k, k + 1, rng.uniform(1e2, 1e3, nodes - 1))
    c.resistors(np.arange(1, nodes + 1), 0, rng.uniform(1e3, 1e4, nodes))
    for at in rng.permutation(nodes)[:12] + 1:
        c.vsource(int(at), 0, dc=float(rng.uniform(-5, 5)))
    s = mna.compile_circuit(c.build())
    x = _both(s.g, s.b_dc, S.BiCgStabParams(tolerance=1e-13, max_iterations=5000))
    if nodes < 1000:
        ref = np.linalg.solve(s.g.to_dense(), s.b_dc)
        assert np.max(np.abs(x - ref)) <= 1e-9 * np.max(np.abs(ref))


def test_slices_larger_than_shared_memory():
    """2,100 rows a block on 148 SMs: the matrix slices stream from global memory."""
    s = mna.compile_circuit(ck.resistor_ladder(310_000, seed=3))
    _both(s.g, s.b_dc, S.BiCgStabParams(tolerance=1e-12, max_iterations=2000))
