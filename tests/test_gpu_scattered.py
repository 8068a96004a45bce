"""Systems whose blocks reach rows all over the system (csrc/api.cu,
ohm_scatter()): more blocks instead of one cluster, or the global-memory form
with 1,024 threads a block (GlobalTeam), which also runs ISAI(1) and systems
whose gather vector does not fit in shared memory.  Linear solves end at the
FP64 residual; a circuit whose rows are in random order has the solution of the
one numbered along its mesh.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import torch  # noqa: E402

from ohmnivore_b200 import _lib, circuits as ck, mna  # noqa: E402
from ohmnivore_b200 import solver as S  # noqa: E402


def _scattered(n, per_row, seed=0):
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(n), per_row)
    key = np.unique(np.concatenate([rows * n + rng.integers(0, n, len(rows)), np.arange(n) * (n + 1)]))
    rows, cols = key // n, key % n
    val = rng.uniform(-1.0, 1.0, len(key))
    off = np.bincount(rows, np.where(rows == cols, 0.0, np.abs(val)), n)
    val[rows == cols] = 1.2 * off + 0.1
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    return mna.Csr(n, n, rp, cols, val), rng.standard_normal(n)


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n,per_row", [(1025, 4), (9000, 3), (25600, 4), (27201, 2), (60000, 30), (120007, 10),
                                       (250001, 4)])
def test_linear(n, per_row, prec):
    a, b = _scattered(n, per_row)
    params = S.BiCgStabParams(tolerance=1e-11, max_iterations=500, precision=prec, max_refinements=8)
    x = S.GpuSolver(None, params).solve_real(a, b)
    assert np.linalg.norm(b - a.spmv(x)) <= 2e-11 * np.linalg.norm(b)


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n,per_row", [(1500, 4), (9000, 4), (30000, 4)])
def test_isai(n, per_row, prec):
    a, b = _scattered(n, per_row)
    params = S.BiCgStabParams(tolerance=1e-11, max_iterations=500, precision=prec, max_refinements=8,
                              precond=_lib.PRECOND_ISAI1)
    x = S.GpuSolver(None, params).solve_real(a, b)
    assert np.linalg.norm(b - a.spmv(x)) <= 2e-11 * np.linalg.norm(b)


def _mesh(side, shuffled):
    """RC mesh with diodes, fed through 50 ohm, its resistors in mesh order or
    shuffled (rows are numbered by a node's first component); the system and the row of
    every mesh node."""
    rng = np.random.default_rng(side)
    at = np.arange(side * side).reshape(side, side)
    b = ck.CircuitBuilder()
    b.vsource(1, 0, dc=1.0, tran=(ck.TRAN_PULSE, (0.0, 1.0, 0.0, 1e-12, 1e-12, 1.0, 2.0)))
    b.resistors([1], [2], [50.0])
    p = np.concatenate([at[:, :-1].ravel(), at[:-1, :].ravel()])
    q = np.concatenate([at[:, 1:].ravel(), at[1:, :].ravel()])
    r = rng.uniform(1e2, 1e3, p.size)
    k = np.random.default_rng(1).permutation(p.size) if shuffled else np.arange(p.size)
    b.resistors(2 + p[k], 2 + q[k], r[k])
    b.resistors(2 + at.ravel(), 0, rng.uniform(1e3, 1e4, at.size))
    b.diodes(2 + rng.choice(at.size, at.size // 50, replace=False), 0, is_=1e-14, n=1.0)
    b.capacitors(2 + at.ravel(), 0, rng.uniform(1e-15, 1e-14, at.size))
    s = mna.compile_circuit(b.build())
    row = np.zeros(2 + at.size, np.int64)
    row[s.node_labels] = np.arange(s.n_nodes)
    return s, row[2:]


@pytest.mark.parametrize("side", [150, 500])
def test_circuit_in_random_order(side):
    """abs_tol 1e-10 on Newton's last step, inner solves to 1e-8: 1e-7 leaves a
    margin for the mesh's condition."""
    n = side * side
    out = []
    for shuffled in (False, True):
        s, rows = _mesh(side, shuffled)
        far = np.mean(np.abs(np.repeat(np.arange(s.size), np.diff(s.g.row_ptr)) - s.g.col))
        assert (far > n / 10) == shuffled
        plan = S.NewtonPlan(s)
        got = []
        for prec in (0, 1):
            params = S.NewtonParams(max_iterations=60, abs_tol=1e-10, bicgstab_max_iterations=20000,
                                    bicgstab_tolerance=1e-14, inner_rtol=1e-8 if prec == 0 else 1e-4, precision=prec)
            x = torch.zeros(s.size, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            plan.newton_device(x.data_ptr(), params)
            got.append(x.cpu().numpy()[rows])
            tran = S.Transient(plan, [int(rows[0]), int(rows[n // 2])])
            x.zero_()
            torch.cuda.synchronize()
            tran.run(x.data_ptr(), 0.0, 2e-13, 3, params)
            got.append(x.cpu().numpy()[rows])
        x.zero_()
        torch.cuda.synchronize()
        times, wave = tran.run_adaptive(x.data_ptr(), 2e-12, 6e-12, 0.0, params)
        got.append(x.cpu().numpy()[rows])
        out.append(got)
        plan.close()
    for one, other in zip(*out):
        assert np.max(np.abs(one - other)) <= 1e-7
