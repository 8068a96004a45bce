"""Cluster form of the AC sweep (csrc/ac.cu): sizes at the edges of 32-row
slices, of one block and of clusters, 2x2 pairs whose rows belong to different
blocks, more and fewer points than clusters, rows too uneven for padded
slices (the block forms), against the oracle's complex sparse LU.

The solves stop at ||r|| < 1e-14 ||b||; the ladders' admittance matrices have
condition numbers below 1e4, so 1e-9 leaves a margin of ten.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from ohmnivore_b200 import circuits as ck, mna  # noqa: E402
from ohmnivore_b200 import solver as S  # noqa: E402
from oracle import ac_ref  # noqa: E402


def _system(nodes, seed, sources=1, hub=0):
    """RC ladder with voltage sources at random nodes (branch rows last) and
    a node tied to `hub` others."""
    rng = np.random.default_rng(seed)
    b = ck.CircuitBuilder()
    k = np.arange(1, nodes, dtype=np.int64)
    b.resistors(k, k + 1, rng.uniform(1e2, 1e3, nodes - 1))
    b.resistors(np.arange(1, nodes + 1), 0, rng.uniform(1e3, 1e4, nodes))
    b.capacitors(np.arange(1, nodes + 1), 0, rng.uniform(1e-13, 1e-12, nodes))
    if hub:
        other = rng.choice(np.arange(2, nodes + 1), hub, replace=False)
        b.resistors(np.ones(hub, np.int64), other, rng.uniform(1e4, 1e5, hub))
    for j, at in enumerate(rng.choice(nodes, sources, replace=False) + 1):
        b.vsource(int(at), 0, dc=0.0, ac=(1.0 + j, 30.0 * j))
    return mna.compile_circuit(b.build())


@pytest.mark.parametrize("nodes,sources,hub", [(1, 1, 0), (31, 1, 0), (32, 2, 0), (1900, 3, 0), (2100, 9, 0),
                                               (9001, 40, 0), (35000, 5, 0), (3000, 4, 2500)])
def test_sweep_matches_oracle(nodes, sources, hub):
    s = _system(nodes, nodes, sources, hub)
    freqs = [0.0, 1e6, 3e8, 1e10]
    x, info = S.ac_sweep(s, freqs, S.BiCgStabParams(max_iterations=20000, tolerance=1e-14))
    ref = ac_ref.ac_sweep(s, freqs)
    assert all(p["krylov_code"] == 1 for p in info)
    for k in range(len(freqs)):
        assert np.max(np.abs(x[k] - ref[k])) <= 1e-9 * np.max(np.abs(ref[k])), freqs[k]


def test_more_points_than_clusters():
    s = _system(300, 7, 2)
    freqs = np.logspace(3, 11, 400)
    x, _ = S.ac_sweep(s, freqs, S.BiCgStabParams(max_iterations=20000, tolerance=1e-14))
    for k in (0, 147, 148, 149, 399):
        ref = ac_ref.ac_sweep(s, [freqs[k]])[0]
        assert np.max(np.abs(x[k] - ref)) <= 1e-9 * np.max(np.abs(ref))


@pytest.mark.parametrize("precond", [1, 3])
def test_other_preconditioners(precond):
    s = _system(2500, 11, 1)
    s.b_ac[:] = 0.0
    s.b_ac[: s.n_nodes] = np.linspace(1.0, 2.0, s.n_nodes)
    a = mna.Csr(s.n_nodes, s.n_nodes, *_drop_branches(s))
    x = S.GpuSolver(None, S.BiCgStabParams(max_iterations=20000, tolerance=1e-14, precond=precond)).solve_complex(
        a, s.b_ac[: s.n_nodes])
    import scipy.sparse as sp
    import scipy.sparse.linalg as spl
    ref = spl.spsolve(sp.csr_matrix((a.val, a.col, a.row_ptr), shape=(a.nrows, a.nrows)).tocsc(), s.b_ac[: s.n_nodes])
    assert np.max(np.abs(x - ref)) <= 1e-9 * np.max(np.abs(ref))


def _drop_branches(s):
    g, n = s.g, s.n_nodes
    c = S.c_on_g_pattern(s)
    rows = np.repeat(np.arange(g.nrows), np.diff(g.row_ptr))
    keep = (rows < n) & (g.col < n)
    val = (g.val + 1j * 2e9 * c)[keep]
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows[keep], minlength=n))])
    return rp, g.col[keep], val
