"""Two threads, each with a context of its own, running the same kernels at
different sizes: a kernel's shared-memory limit is one per process, so a small
call must not lower it under a large one that is being prepared.  Each result
equals the same call's result without the other thread."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import torch  # noqa: E402

from ohmnivore_b200 import circuits as ck, mna  # noqa: E402
from ohmnivore_b200 import solver as S  # noqa: E402


def _ladder(nodes):
    b = ck.CircuitBuilder()
    rng = np.random.default_rng(nodes)
    k = np.arange(1, nodes, dtype=np.int64)
    b.resistors(k, k + 1, rng.uniform(1e2, 1e3, nodes - 1))
    b.resistors(np.arange(1, nodes + 1), 0, rng.uniform(1e3, 1e4, nodes))
    b.capacitors(np.arange(1, nodes + 1), 0, rng.uniform(1e-13, 1e-12, nodes))
    b.vsource(1, 0, dc=1.0, ac=(1.0, 0.0))
    return mna.compile_circuit(b.build())


def _ac(ctx, nodes):
    s = _ladder(nodes)
    params = S.BiCgStabParams(max_iterations=5000, tolerance=1e-12)
    return lambda: S.ac_sweep(s, [1e6, 1e9], params, ctx)[0]


def _linear(ctx, nodes):
    s = _ladder(nodes)
    solver = S.GpuSolver(ctx, S.BiCgStabParams(max_iterations=5000, tolerance=1e-12))
    return lambda: solver.solve_real(s.g, s.b_dc)


def _batch(ctx, size):
    systems = [mna.compile_circuit(ck.diode_mesh(size, size, seed=k)) for k in range(3)]
    batch = S.NewtonBatch(systems, ctx)
    x = torch.zeros(batch.rows, dtype=torch.float64, device="cuda")
    params = S.NewtonParams(max_iterations=100, abs_tol=1e-10, bicgstab_max_iterations=20000, bicgstab_tolerance=1e-14)

    def call():
        x.zero_()
        torch.cuda.synchronize()
        batch.newton_device(x.data_ptr(), params)
        return x.cpu().numpy()
    return call


@pytest.mark.parametrize("make,large,small", [(_ac, 9000, 20), (_linear, 20000, 1500), (_batch, 24, 4)],
                         ids=["ac_sweep", "solve_real", "batch"])
def test_small_calls_beside_large_ones(make, large, small):
    contexts = [S.Context(0), S.Context(0)]
    calls = [make(ctx, size) for ctx, size in zip(contexts, (large, small))]
    want = [call() for call in calls]
    done, errors = threading.Event(), []

    def small_calls():
        try:
            while not done.is_set():
                np.testing.assert_array_equal(calls[1](), want[1])
        except BaseException as e:      # noqa: BLE001
            errors.append(e)

    other = threading.Thread(target=small_calls)
    other.start()
    try:
        for _ in range(100):
            np.testing.assert_array_equal(calls[0](), want[0])
    finally:
        done.set()
        other.join()
    assert not errors
