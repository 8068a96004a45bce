"""Teams whose blocks run different forms of the Krylov solve
(csrc/solver_kernel.cuh): a block whose nonzeros touch too many rows of other
blocks runs krylov() beside blocks that run krylov_slice().  Both have to meet at the
same barriers, take the same branches and give the global-memory layout's bits.

``_layouts`` restates the rule by which each block chooses, so that a test can
tell that the layout it is about is the one that ran.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import torch  # noqa: E402

from ohmnivore_b200 import _lib, circuits as ck, mna  # noqa: E402
from ohmnivore_b200 import solver as S  # noqa: E402

BLOCK_BYTES = 227 * 1024          # shared memory of one block
STATIC_BYTES = 4096               # at least the kernels' static part and the reserve


def _blocks(n):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if n <= 1024:
        return 1
    want = -(-n // 512)
    return min(want, 16) if n <= 27200 else min(want, sms)


def _up16(b):
    return (b + 15) // 16 * 16


def _layouts(a, room=BLOCK_BYTES - STATIC_BYTES):
    """Per block of a system with one lane per row and no long rows: "chip",
    "stream", "csr" or "none" (slice_map(), slice_offsets())."""
    n, blocks, rp, col = a.nrows, _blocks(a.nrows), np.asarray(a.row_ptr), np.asarray(a.col)
    assert len(col) <= 5.5 * n
    rows = -(-n // blocks) + 1
    nnz_blk = int(len(col) * rows / n * 1.15) + 512
    halo = min(nnz_blk, 4096) if blocks > 1 else 0
    room = min(rows * 9 + rows // 8 + halo * 12 + 256 + rows * 68 + nnz_blk * 10, room) // 16 * 16
    bits = 0
    while 8 << (bits + 1) <= room // 2 and bits < 14:
        bits += 1
    table = 1 << bits if blocks > 1 else 0
    out = []
    for b in range(blocks):
        r0, r1 = n * b // blocks, n * (b + 1) // blocks
        r = r1 - r0
        near = col[rp[r0]:rp[r1]]
        h = len(np.unique(near[(near < r0) | (near >= r1)]))
        width = np.diff(rp[r0:r1 + 1])
        w = int(sum(width[s:s + 32].max() for s in range(0, r, 32)))

        def offsets(w, starts=(r + 31) // 32):
            z = _up16(4 * (starts + 1)) + _up16(4 * h) + _up16(r) + 64 * w
            vec = z + _up16(8 * (r + h + 1))
            return z, vec, vec + 8 * _up16(8 * r) + 256 * w

        z, _, end = offsets(w)
        z0, vec0, _ = offsets(0)
        z1, vec1, _ = offsets(0, r)
        start = lambda k: k + k // 4  # noqa: E731
        if h >= table // 4 * 3 and blocks > 1 or r + h >= 0xFFFF:
            out.append("none")
        elif w <= 0xFFFF and end <= room and z <= room - 8 * table:
            out.append("chip")
        elif (w <= 0xFFFF and vec0 <= room and z0 <= room - 8 * table and
              32 * w <= start(int(rp[r1])) - start(int(rp[r0]))):
            out.append("stream")
        else:
            out.append("csr" if vec1 <= room and z1 <= room - 8 * table else "none")
    return out


def _solve(a, b, params):
    """(x or None, info) in the automatic and in the global-memory layout."""
    ctx = S.Context(0)
    out = []
    try:
        for layout in (_lib.KRYLOV_LAYOUT_AUTO, _lib.KRYLOV_LAYOUT_GLOBAL):
            ctx.set_krylov_layout(layout)
            solver = S.GpuSolver(ctx, params)
            x = None
            try:
                x = solver.solve_real(a, b)
            except S.SolveError:
                pass
            out.append((x, solver.last_info))
    finally:
        ctx.close()
    return out


def _csr(n, rows, cols, vals):
    order = np.lexsort((cols, rows))
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    return mna.Csr(n, n, rp, cols[order], vals[order])


def _skew(n, wide):
    """2x2 skew blocks [[0 1] [-1 0]]; row 0 also has `wide` entries +1, -1,
    +1, ...: (b, A b) = 0 exactly for b = 1, and row 0's block keeps no slice."""
    k = np.arange(n)
    far = 2 + np.arange(wide)
    rows = np.concatenate([k, np.zeros(wide, np.int64)])
    cols = np.concatenate([k ^ 1, far])
    vals = np.concatenate([np.where(k % 2 == 0, 1.0, -1.0), np.where(far % 2 == 0, 1.0, -1.0)])
    return _csr(n, rows, cols, vals)


@pytest.mark.parametrize("max_it,restarts,code", [(1, 1, 2), (3, 3, 2), (100, 50, 4)])
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n", [10000, 30000])
def test_breakdown_at_the_iteration_limit(n, prec, max_it, restarts, code):
    """(r_hat, v) = 0 in every iteration: each one restarts, the last one
    allowed ends the solve (code 2), or the 51st breakdown does (code 4).  A
    block that met one barrier more or less than the others would make the call
    time out, or the FP64 solve after the failed FP32 one read partial sums that
    nobody wrote."""
    a = _skew(n, 8000)
    kinds = _layouts(a)
    assert kinds[0] == "none" and set(kinds[1:]) == {"chip"}
    params = S.BiCgStabParams(tolerance=1e-10, max_iterations=max_it, precond=_lib.PRECOND_NONE, precision=prec)
    for x, info in _solve(a, np.ones(n), params):
        assert x is None and info["status"] == _lib.ERR_SOLVE and info["krylov_code"] == code
        assert info["krylov_restarts"] == (1 + prec) * restarts
        assert info["fp64_fallbacks"] == prec


def _source(n, spread, kind):
    """b = e_0 with row 0 = e_0: the first iteration takes r[0] to exactly 0,
    so (r_hat, r) = 0 and the solve restarts; column 0 (`spread` in every
    fourth row) sets the residual it does so at.  The other rows are a
    diagonally dominant band or 600-column mesh, for "uneven" and "far" with
    one row of up to 1,500 and 8,000 entries, for "wide" with eight entries a row."""
    rng = np.random.default_rng(n)
    steps = {"mesh": (1, 600), "wide": (1, 2, 5, 9)}.get(kind, (1,))
    k = np.arange(1, n)
    rows, cols = [], []
    for s in steps:
        rows += [k[k + s < n], k[k - s > 0]]
        cols += [k[k + s < n] + s, k[k - s > 0] - s]
    if kind in ("uneven", "far"):
        count = min(n - 20, 1500 if kind == "uneven" else 8000)
        rows.append(np.full(count, 5))
        cols.append(10 + np.arange(count))
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    vals = rng.uniform(-1.0, 1.0, len(rows))
    diag = 1.5 * np.bincount(rows, np.abs(vals), n) + 0.5
    diag[0] = 1.0
    far = np.arange(4, n, 4)
    a = _csr(n, np.concatenate([rows, np.arange(n), far]), np.concatenate([cols, np.arange(n), 0 * far]),
             np.concatenate([vals, diag, spread * diag[far]]))
    return a, np.concatenate([[1.0], np.zeros(n - 1)])


@pytest.mark.parametrize("spread", [0.01, 100.0], ids=["from_r", "from_start"])
@pytest.mark.parametrize("n,kind,layouts", [(900, "band", {"chip"}), (5000, "band", {"chip"}), (40000, "band", {"chip"}),
                                            (900, "uneven", {"csr"}), (5000, "uneven", {"chip", "csr"}),
                                            (40000, "uneven", {"chip", "csr"}), (10000, "far", {"chip", "none"}),
                                            (40000, "far", {"chip", "none"}),
                                            (360000, "mesh", {"stream"}), (5000, "wide", None)])
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "mixed"])
def test_restart(n, kind, layouts, spread, prec):
    """The restart from the current residual, and the one from the solve's
    start where that residual is more than ten times the initial one.  The
    sweeps end at ||b - A x|| < 1e-9 in FP64; x_i <= 200 puts the rounding of
    that residual below 200 * 2^-50 * sqrt(n) = 1.1e-10."""
    a, b = _source(n, spread, kind)
    if layouts:
        assert set(_layouts(a)) == layouts
    (xs, s), (xg, g) = _solve(a, b, S.BiCgStabParams(tolerance=1e-9, max_iterations=2000, precision=prec,
                                                     max_refinements=8))
    assert xs is not None and s["krylov_restarts"] >= 1
    np.testing.assert_array_equal(xs, xg)
    assert {k: s[k] for k in ("krylov_iterations", "krylov_restarts", "fp64_fallbacks")} == \
           {k: g[k] for k in ("krylov_iterations", "krylov_restarts", "fp64_fallbacks")}
    assert np.linalg.norm(b - a.spmv(xs)) <= 1.2e-9


def _spilled(a, vectors, room=BLOCK_BYTES - 1024):
    """Whether the stream layout keeps `vectors` of its eight vectors or fewer
    in shared memory (every block)."""
    n, blocks = a.nrows, _blocks(a.nrows)
    r = n // blocks
    return _up16(4 * (r // 32)) + r + 8 * r + vectors * 8 * r + 8 * r > room


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "mixed"])
def test_vectors_in_global_memory_beside_the_global_solve(prec):
    """3,600 rows a block: d (the seventh vector) and the weights leave shared
    memory, beside one block (a row of 10,000 entries) that runs krylov(): in
    FP32 both keep their own rows of d apart."""
    n = 3600 * _blocks(10**6)
    rng = np.random.default_rng(1)
    k = np.arange(n)
    near = [(k[k + s < n], k[k + s < n] + s) for s in (1, 600)]
    row = n // 2 + 7
    rows = np.concatenate([near[0][0], near[0][1], near[1][0], near[1][1], np.full(10000, row)])
    cols = np.concatenate([near[0][1], near[0][0], near[1][1], near[1][0], row + 700 + np.arange(10000)])
    vals = rng.uniform(-1.0, 1.0, len(rows))
    a = _csr(n, np.concatenate([rows, k]), np.concatenate([cols, k]),
             np.concatenate([vals, 1.2 * np.bincount(rows, np.abs(vals), n) + 0.1]))
    kinds = _layouts(a)
    assert kinds.count("none") == 1 and kinds.count("stream") == len(kinds) - 1 and _spilled(a, 6)
    (xs, s), (xg, g) = _solve(a, rng.standard_normal(n), S.BiCgStabParams(tolerance=1e-12, max_iterations=500,
                                                                          precision=prec, max_refinements=8))
    assert xs is not None and s["krylov_iterations"] == g["krylov_iterations"]
    np.testing.assert_array_equal(xs, xg)


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "mixed"])
def test_long_row_in_a_team_of_one(prec):
    """A 702-row circuit whose hub row stores each off-diagonal entry as eight
    equal parts (5,616 entries, a long row, in one block): the same solution as
    with each entry once, and the global-memory layout's bits."""
    rng = np.random.default_rng(2)
    leaves = 700
    c = ck.CircuitBuilder()
    c.vsource(1, 0, dc=1.0)
    c.resistors([1], [2], [10.0])
    leaf = 3 + np.arange(leaves)
    c.resistors(np.full(leaves, 2), leaf, rng.uniform(1e3, 1e4, leaves))
    c.diodes(leaf, 0, is_=1e-14, n=1.0)
    s = mna.compile_circuit(c.build())
    rp, hub = np.asarray(s.g.row_ptr, np.int64), s.node_index(2)
    rows = np.repeat(np.arange(s.size), np.diff(rp))
    parts = np.where((rows == hub) & (s.g.col != hub), 8, 1)
    first = np.concatenate([[0], np.cumsum(parts)])
    count = np.bincount(rows, parts, s.size).astype(np.int64)
    many = mna.Csr(s.size, s.size, np.concatenate([[0], np.cumsum(count)]), np.repeat(s.g.col, parts),
                   np.repeat(s.g.val / parts, parts))
    assert count[hub] > 4096 and s.size <= 1024
    diodes = s.diode_descriptors.copy()
    at = diodes["g_row_col"]
    diodes["g_row_col"] = np.where(at == mna.SENTINEL, at, first[np.minimum(at, len(parts) - 1)])
    params = S.NewtonParams(max_iterations=100, abs_tol=1e-10, bicgstab_max_iterations=20000, bicgstab_tolerance=1e-14,
                            precision=prec, inner_rtol=1e-4)
    out = []
    ctx = S.Context(0)
    try:
        for a, dd, layout in ((s.g, s.diode_descriptors, _lib.KRYLOV_LAYOUT_GLOBAL),
                              (many, diodes, _lib.KRYLOV_LAYOUT_GLOBAL), (many, diodes, _lib.KRYLOV_LAYOUT_AUTO)):
            ctx.set_krylov_layout(layout)
            out.append(S.newton_solve(ctx, a.val, a.col, a.row_ptr, s.b_dc, dd, s.bjt_descriptors,
                                      s.mosfet_descriptors, s.size, a.nnz, params))
    finally:
        ctx.close()
    np.testing.assert_array_equal(out[1], out[2])
    assert np.max(np.abs(out[2] - out[0])) <= 1e-9
