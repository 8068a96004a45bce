"""The work a user of this framework has it do, as cases of stated sizes.

Every case goes through a public entry point of ``ohmnivore_b200.solver``:

  newton   newton_solve: host arrays in, host solution out, the drop-in call
  dc       NewtonPlan.newton_device: DC operating point on a resident plan
  linear   GpuSolver.solve_real: linear solve from host arrays
  spmv     SolverBackend.spmv on a resident matrix
  tran     Transient.run: fixed-step backward Euler
  adaptive Transient.run_adaptive: BE / TRAP with step control, CMOS chain
  batch    NewtonBatch.newton_device: many circuits of mixed sizes
  ac       ac_sweep: frequency sweep from host arrays
  adjoint  Transient.adjoint: forward run and reverse sweep, all gradients

Circuits are the seeded families of the benchmark: resistor meshes with
diodes, RC meshes, resistor ladders, CMOS inverter chains and BJT
differential-pair meshes.  ``exact`` solves the linear and diode circuits by
direct elimination in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from ohmnivore_b200 import circuits, mna, solver

GMIN, VT = 1e-12, 0.02585        # node conductance to ground and thermal voltage of the circuit model
IS = 1e-14                       # diode saturation current


def listed():
    return [
        # a small rectifier-sized circuit through the drop-in host call: set-up and latency
        {"name": "newton_mesh_24", "kind": "newton", "rows": 24, "cols": 24},
        # a block-level circuit solved again and again on a resident plan (sweeps, optimisers)
        {"name": "dc_mesh_100", "kind": "dc", "rows": 100, "cols": 100, "diodes": 0.10, "volts": 5.0},
        # the benchmark's headline: DC operating point of a 250k-node diode mesh
        {"name": "dc_mesh_500", "kind": "dc", "rows": 500, "cols": 500, "diodes": 0.10, "volts": 5.0},
        # a power-grid-sized mesh, beyond what on-chip memory holds
        {"name": "dc_grid_600", "kind": "dc", "rows": 600, "cols": 600, "diodes": 0.05, "volts": 1.0},
        # linear DC of the benchmark's 10,000-node resistor ladder, host arrays in and out
        {"name": "linear_ladder_10k", "kind": "linear", "nodes": 10000},
        # one matrix-vector product of a host-driven solver, larger than L2
        {"name": "spmv_mesh_2048", "kind": "spmv", "rows": 2048, "cols": 2048},
        # step response of a small RC-diode network, many cheap steps
        {"name": "tran_mesh_20", "kind": "tran", "circuit": "mesh", "size": 20, "steps": 200, "mixed": False},
        # the benchmark's digital transient: 100k CMOS stages, the first 100 steps
        {"name": "tran_chain_100k", "kind": "tran", "circuit": "chain", "size": 100000, "steps": 100, "mixed": True},
        # the reference's adaptive transient on a mid-sized CMOS chain
        {"name": "adaptive_chain_5k", "kind": "adaptive", "stages": 5000, "tstop_ps": 400.0},
        # a Monte Carlo batch of analog circuits of mixed sizes
        {"name": "batch_mc_512", "kind": "batch", "circuits": 512, "lo": 50, "hi": 1500},
        # the benchmark's AC sweep: a 10k-row RC mesh, 10 points per decade from 1 kHz to 1 THz
        {"name": "ac_mesh_100", "kind": "ac", "rows": 100, "cols": 100, "points": 10, "decades": 9},
        # gradients of one output with respect to every R, C and Is over a transient
        {"name": "adjoint_mesh_64", "kind": "adjoint", "rows": 64, "cols": 64, "steps": 40},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["newton", "dc", "dc", "linear", "spmv", "tran", "tran", "adaptive", "batch", "ac", "adjoint"])
    if kind == "newton":
        r = _log_int(rng, 5, 120)
        return {"kind": kind, "rows": r, "cols": max(3, int(r * rng.uniform(0.6, 1.6)))}
    if kind == "dc":
        r = _log_int(rng, 16, 450)
        return {"kind": kind, "rows": r, "cols": max(3, int(r * rng.uniform(0.6, 1.25))),
                "diodes": round(rng.uniform(0.05, 0.10), 3), "volts": rng.choice([1.0, 5.0])}
    if kind == "linear":
        return {"kind": kind, "nodes": _log_int(rng, 100, 100000)}
    if kind == "spmv":
        return {"kind": kind, "rows": _log_int(rng, 300, 2048), "cols": _log_int(rng, 300, 2048)}
    if kind == "tran":
        circuit = rng.choice(["mesh", "chain"])
        size = _log_int(rng, 8, 80) if circuit == "mesh" else _log_int(rng, 50, 100000)
        return {"kind": kind, "circuit": circuit, "size": size, "steps": rng.randrange(20, 100),
                "mixed": circuit == "chain" and rng.random() < 0.5}
    if kind == "adaptive":
        return {"kind": kind, "stages": _log_int(rng, 50, 5000), "tstop_ps": float(rng.randrange(100, 400))}
    if kind == "batch":
        lo = rng.choice([50, 100, 200])
        return {"kind": kind, "circuits": _log_int(rng, 8, 512), "lo": lo, "hi": _log_int(rng, 500, 1500)}
    if kind == "ac":
        r = _log_int(rng, 8, 100)
        return {"kind": kind, "rows": r, "cols": max(3, int(r * rng.uniform(0.6, 1.0))),
                "points": rng.randrange(2, 11), "decades": rng.randrange(3, 10)}
    r = _log_int(rng, 8, 64)
    return {"kind": kind, "rows": r, "cols": max(3, int(r * rng.uniform(0.6, 1.0))), "steps": rng.randrange(10, 40)}


# ------------------------------------------------------------------ circuits --

class _Mesh:
    """Component values of a rows x cols resistor mesh: a source node feeds
    corner (0, 0) through ``r_src``; mesh node (i, j) is row 1 + i cols + j of
    the compiled system, the source node row 0, the source current last."""

    def __init__(self, rows, cols, seed, diodes, caps=False, r_src=100.0, r_lo=10.0):
        rng = np.random.default_rng(seed)
        self.rows, self.cols, self.n = rows, cols, rows * cols
        self.r_src = r_src
        self.rh = np.exp(rng.uniform(math.log(r_lo), math.log(1e4), (rows, cols - 1)))
        self.rv = np.exp(rng.uniform(math.log(r_lo), math.log(1e4), (rows - 1, cols)))
        self.sites = np.sort(rng.choice(self.n, size=int(round(diodes * self.n)), replace=False))
        self.caps = np.exp(rng.uniform(math.log(1e-15), math.log(1e-12), self.n)) if caps else None
        at = np.arange(self.n).reshape(rows, cols)
        self.a = np.concatenate([at[:, :-1].ravel(), at[:-1, :].ravel()])
        self.b = np.concatenate([at[:, 1:].ravel(), at[1:, :].ravel()])
        self.r = np.concatenate([self.rh.ravel(), self.rv.ravel()])

    def circuit(self, dc, ac=None, tran=None):
        b = circuits.CircuitBuilder()
        b.vsource(1, 0, dc=dc, ac=ac, tran=tran, name="V1")
        b.resistors([1], [2], [self.r_src], names=["RSRC"])
        b.resistors(2 + self.a, 2 + self.b, self.r)
        if len(self.sites):
            b.diodes(2 + self.sites, 0, is_=IS, n=1.0)
        if self.caps is not None:
            b.capacitors(2 + np.arange(self.n), 0, self.caps)
        return b.build()

    def conductance(self, dev):
        """The mesh nodes' conductance matrix, dense, the source node eliminated."""
        g = torch.zeros(self.n, self.n, dtype=torch.float64, device=dev)
        a, b = torch.from_numpy(self.a).to(dev), torch.from_numpy(self.b).to(dev)
        y = torch.from_numpy(1.0 / self.r).to(dev)
        g.index_put_((a, b), -y, accumulate=True)
        g.index_put_((b, a), -y, accumulate=True)
        d = torch.full((self.n,), GMIN, dtype=torch.float64, device=dev)
        d.index_add_(0, a, y)
        d.index_add_(0, b, y)
        d[0] += 1.0 / self.r_src
        g.diagonal().add_(d)
        return g

    def with_source(self, v_src, mesh):
        """[source node, mesh nodes, source current] from the mesh voltages."""
        i = -(v_src - mesh[..., :1]) / self.r_src - GMIN * v_src
        return torch.cat([torch.zeros_like(i) + v_src, mesh, i], dim=-1)


def _nvt():
    return float(np.float32(VT)), float(np.float32(IS))     # descriptors hold 32-bit parameters


def _amplifiers(n, rng, r_lo=300.0, r_hi=3e3):
    """A w x w resistor mesh fed by 5 V at a corner, with one NPN differential
    pair and one diode per 100 nodes, every value off its nominal by 5 %."""
    w = max(4, int(math.ceil(math.sqrt(n))))
    off = lambda v: v * (1.0 + 0.05 * rng.standard_normal(np.shape(v)))  # noqa: E731
    edge = lambda m: off(np.exp(rng.uniform(math.log(r_lo), math.log(r_hi), m)))  # noqa: E731
    at = np.arange(w * w).reshape(w, w)
    pairs = max(1, w * w // 100)
    site = np.sort(rng.choice(w * w - 3 * w, size=pairs, replace=False))
    tail = 2 + w * w + np.arange(pairs)
    b = circuits.CircuitBuilder()
    b.vsource(1, 0, dc=5.0, name="VCC")
    b.resistors([1], [2], [off(100.0)], names=["RSRC"])
    b.resistors(2 + at[:, :-1].ravel(), 2 + at[:, 1:].ravel(), edge(w * (w - 1)))
    b.resistors(2 + at[:-1, :].ravel(), 2 + at[1:, :].ravel(), edge(w * (w - 1)))
    b.resistors(tail, 0, off(np.full(pairs, 4300.0)))
    for side in (0, 1):
        b.bjts(2 + site + side, 2 + site + w + side, tail, is_=off(np.full(pairs, 1e-16)),
               bf=off(np.full(pairs, 100.0)), vaf=100.0)
    b.diodes(2 + site + 2 * w, 0, is_=off(np.full(pairs, IS)))
    return b.build()


class _Ladder:
    def __init__(self, nodes, seed):
        rng = np.random.default_rng(seed)
        self.nodes, self.volts = nodes, 10.0
        self.series = np.exp(rng.uniform(math.log(100.0), math.log(1e5), nodes - 1))
        self.shunt = np.exp(rng.uniform(math.log(1e3), math.log(1e6), nodes))

    def circuit(self):
        k = np.arange(1, self.nodes, dtype=np.int64)
        b = circuits.CircuitBuilder()
        b.vsource(1, 0, dc=self.volts, name="V1")
        b.resistors(k, k + 1, self.series)
        b.resistors(np.arange(1, self.nodes + 1), 0, self.shunt)
        return b.build()


# ------------------------------------------------------------------- prepare --

_CTX = None


def _context():
    """One context and its stream, as a program keeps them."""
    global _CTX
    if _CTX is None:
        ctx = solver.Context(0)
        _CTX = ctx, torch.cuda.ExternalStream(ctx.lib.ohm_ctx_stream(ctx.handle))
    return _CTX


def _dc_params():
    return solver.NewtonParams(max_iterations=200, abs_tol=1e-9, bicgstab_max_iterations=20000,
                               bicgstab_tolerance=1e-15, inner_rtol=1e-6, forcing=1, eta_max=0.7)


def _start_params(guess=None):
    return solver.NewtonParams(max_iterations=100, abs_tol=1e-10, bicgstab_max_iterations=20000,
                               bicgstab_tolerance=1e-14, inner_rtol=1e-4, continuation=True, initial_guess=guess)


def _step_params(mixed):
    return solver.NewtonParams(max_iterations=50, abs_tol=1e-10, bicgstab_max_iterations=20000,
                               bicgstab_tolerance=1e-14, inner_rtol=1e-6, precision=1 if mixed else 0)


def _device(array):
    return torch.from_numpy(np.ascontiguousarray(array)).cuda()


class _Buffer:
    """A library buffer as a tensor (no copy)."""

    def __init__(self, buf):
        ptr = buf.ctx.lib.ohm_buf_device_ptr(buf._h)
        self.__cuda_array_interface__ = {"shape": (buf.n,), "typestr": "<f8", "data": (int(ptr), False), "version": 3}


def _pulse():
    return circuits.TRAN_PULSE, (0.0, 1.0, 0.0, 1e-12, 1e-12, 1.0, 2.0)


def _mesh_matrix(rows, cols, seed):
    """CSR of a five-point mesh: columns sorted, values random."""
    rng = np.random.default_rng(seed)
    n = rows * cols
    at = np.arange(n, dtype=np.int64)
    i, j = at // cols, at % cols
    near = np.stack([at - cols, at - 1, at, at + 1, at + cols], axis=1)
    ok = np.stack([i > 0, j > 0, np.ones(n, bool), j < cols - 1, i < rows - 1], axis=1)
    rp = np.concatenate([[0], np.cumsum(ok.sum(axis=1))])
    return mna.Csr(n, n, rp, near[ok], rng.standard_normal(int(rp[-1])) + 2.0), ok


def prepare(case, seed):
    kind = case["kind"]
    ctx, stream = _context()
    s = {"kind": kind, "ctx": ctx, "stream": stream}
    if kind == "newton":
        s["sys"] = mna.compile_circuit(_Mesh(case["rows"], case["cols"], seed, 0.10).circuit(5.0))
        s["params"] = _dc_params()
    elif kind == "dc":
        mesh = _Mesh(case["rows"], case["cols"], seed, case["diodes"])
        sysm = mna.compile_circuit(mesh.circuit(case["volts"]))
        s["plan"], s["params"] = solver.NewtonPlan(sysm, ctx), _dc_params()
        s["x"] = torch.zeros(sysm.size, dtype=torch.float64, device="cuda")
    elif kind == "linear":
        sysm = mna.compile_circuit(_Ladder(case["nodes"], seed).circuit())
        s["a"], s["b"] = sysm.g, sysm.b_dc
        s["solver"] = solver.GpuSolver(ctx, solver.BiCgStabParams(tolerance=1e-14, max_iterations=50000))
    elif kind == "spmv":
        a, _ = _mesh_matrix(case["rows"], case["cols"], seed)
        be = solver.SolverBackend(ctx)
        s["be"], s["a"], s["x"], s["y"] = be, be.upload_matrix(a), be.new_buffer(a.nrows), be.new_buffer(a.nrows)
        s["x"].upload(np.random.default_rng(seed + 1).standard_normal(a.nrows))
        s["out"] = torch.as_tensor(_Buffer(s["y"]), device="cuda")
    elif kind == "tran" and case["circuit"] == "mesh":
        mesh = _Mesh(case["size"], case["size"], seed, 0.05, caps=True, r_src=50.0)
        sysm = mna.compile_circuit(mesh.circuit(0.0, tran=_pulse()))
        s["plan"] = solver.NewtonPlan(sysm, ctx)
        s["tran"] = solver.Transient(s["plan"], list(range(sysm.n_nodes)))
        s["x0"] = torch.zeros(sysm.size, dtype=torch.float64, device="cuda")
        s["h"], s["steps"], s["params"] = 2e-12, case["steps"], _step_params(case["mixed"])
    elif kind in ("tran", "adaptive"):
        stages = case["size"] if kind == "tran" else case["stages"]
        sysm = mna.compile_circuit(circuits.inverter_chain(stages, seed=seed))
        s["plan"] = solver.NewtonPlan(sysm, ctx)
        probes = [k for k in (2, 3, 4, 5, 12, 102, 1002, 2 + stages) if k <= 2 + stages]
        s["tran"] = solver.Transient(s["plan"], [sysm.node_index(k) for k in sorted(set(probes))])
        s["x0"] = torch.zeros(sysm.size, dtype=torch.float64, device="cuda")
        rails = np.zeros(sysm.size)                          # node set: supply, input low, outputs alternating
        rails[:sysm.n_nodes] = np.where(sysm.node_labels % 2 == 1, 1.8, 0.0)
        torch.cuda.synchronize()
        s["plan"].newton_device(s["x0"].data_ptr(), _start_params(rails))
        s["h"] = 5e-12
        if kind == "tran":
            s["tran"].set_predictor(2)
            s["steps"], s["params"] = case["steps"], _step_params(case["mixed"])
        else:
            s["tstop"], s["points"] = case["tstop_ps"] * 1e-12, 8 * int(case["tstop_ps"] / 5.0) + 16
            s["times"], s["wave"] = np.empty(s["points"]), np.empty((s["points"], len(s["tran"].probes)))
            s["params"] = solver.NewtonParams(max_iterations=100, abs_tol=1e-12, bicgstab_tolerance=1e-15,
                                              inner_rtol=1e-8, bicgstab_max_iterations=20000)
    elif kind == "batch":
        rng = np.random.default_rng(seed)
        sizes = np.geomspace(case["lo"], case["hi"], case["circuits"])    # the sizes are the case's, the values the seed's
        systems = [mna.compile_circuit(_amplifiers(n, rng)) for n in sizes]
        s["batch"], s["params"] = solver.NewtonBatch(systems, ctx), _start_params()
        s["x"] = torch.zeros(s["batch"].rows, dtype=torch.float64, device="cuda")
    elif kind == "ac":
        mesh = _Mesh(case["rows"], case["cols"], seed, 0.0, caps=True, r_src=50.0, r_lo=100.0)
        s["sys"] = mna.compile_circuit(mesh.circuit(0.0, ac=(1.0, 0.0)))
        s["freqs"] = _frequencies(case)
        s["params"] = solver.BiCgStabParams(max_iterations=50000, tolerance=1e-14)
    else:
        mesh = _Mesh(case["rows"], case["cols"], seed, 0.05, caps=True, r_src=50.0)
        ckt = mesh.circuit(0.0, tran=_pulse())
        sysm = mna.compile_circuit(ckt)
        s["plan"] = solver.NewtonPlan(sysm, ctx)
        s["tran"] = solver.Transient(s["plan"])
        s["comps"] = solver.ComponentTable(ckt, sysm)
        s["x0"] = torch.zeros(sysm.size, dtype=torch.float64, device="cuda")
        s["w"] = np.zeros(sysm.size)
        s["w"][1 + _output_node(case)] = 1.0
        s["h"], s["steps"], s["params"] = 2e-12, case["steps"], _step_params(False)
    if "x0" in s:
        s["x"] = s["x0"].clone()
    torch.cuda.synchronize()
    return s


def _frequencies(case):
    return 1e3 * 10.0 ** (np.arange(case["points"] * case["decades"]) / case["points"])


def _output_node(case):
    return min(3, case["rows"] - 1) * case["cols"] + min(3, case["cols"] - 1)


# ----------------------------------------------------------------------- run --

def run(s):
    kind = s["kind"]
    if kind == "newton":
        y = s["sys"]
        return solver.newton_solve(s["ctx"], y.g.val, y.g.col, y.g.row_ptr, y.b_dc, y.diode_descriptors,
                                   y.bjt_descriptors, y.mosfet_descriptors, y.size, y.g.nnz, s["params"])
    if kind == "dc":
        with torch.cuda.stream(s["stream"]):
            s["x"].zero_()
        s["plan"].newton_device(s["x"].data_ptr(), s["params"])
        return s["x"]
    if kind == "linear":
        return s["solver"].solve_real(s["a"], s["b"])
    if kind == "spmv":
        s["be"].spmv(s["a"], s["x"], s["y"])
        return s["out"]
    if kind == "tran":
        with torch.cuda.stream(s["stream"]):
            s["x"].copy_(s["x0"])
        wave = s["tran"].run(s["x"].data_ptr(), 0.0, s["h"], s["steps"], s["params"])
        return {"wave": wave, "x": s["x"]}
    if kind == "adaptive":
        with torch.cuda.stream(s["stream"]):
            s["x"].copy_(s["x0"])
        times, wave = s["tran"].run_adaptive(s["x"].data_ptr(), s["h"], s["tstop"], 0.0, s["params"], s["points"])
        s["times"][:] = np.nan                               # the number of steps is the run's own
        s["wave"][:] = np.nan
        s["times"][:len(times)], s["wave"][:len(times)] = times, wave
        return {"times": s["times"], "wave": s["wave"], "x": s["x"]}
    if kind == "batch":
        with torch.cuda.stream(s["stream"]):
            s["x"].zero_()
        s["batch"].newton_device(s["x"].data_ptr(), s["params"])
        return s["x"]
    if kind == "ac":
        return solver.ac_sweep(s["sys"], s["freqs"], s["params"], s["ctx"])[0]
    g, info = s["tran"].adjoint(s["x0"].data_ptr(), 0.0, s["h"], s["steps"], s["w"], s["comps"], s["params"], 0)
    return {"R": g["R"], "C": g["C"], "Is": g["Is"], "output": info["output"]}


# ---------------------------------------------------------------------- work --

def work(case):
    """Each input read once and each output written once; two operations per
    matrix entry and product that cannot be avoided."""
    kind = case["kind"]
    if kind == "linear":
        n = case["nodes"] + 1
        return _csr_work(n, 3 * n, 1)
    if kind == "spmv":
        n = case["rows"] * case["cols"]
        return _csr_work(n, 5 * n - 2 * (case["rows"] + case["cols"]), 1)
    if kind in ("tran", "adaptive"):
        steps = case["steps"] if kind == "tran" else int(case["tstop_ps"] / 5.0)
        if case.get("circuit") == "mesh":
            n = case["size"] ** 2
            w = _csr_work(n, 5 * n, steps)
            w["bytes"] += 8 * n * steps
            return w
        n = case["size"] if kind == "tran" else case["stages"]
        w = _csr_work(n, 5 * n, steps)
        w["bytes"] += 2 * 64 * n + 8 * 8 * steps
        return w
    if kind == "batch":
        n = case["circuits"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        return _csr_work(n, 5 * n, 1)
    n = case["rows"] * case["cols"]
    if kind == "ac":
        points = case["points"] * case["decades"]
        return {"bytes": 5 * n * 20 + 16 * n * (1 + points), "flops": 8 * 5 * n * points}
    if kind == "adjoint":
        w = _csr_work(n, 5 * n, 2 * case["steps"])
        w["bytes"] += 2 * 16 * 3 * n
        return w
    return _csr_work(n, 5 * n, 1)


def _csr_work(n, nnz, products):
    return {"bytes": 12 * nnz + 4 * n + 16 * n, "flops": 2 * nnz * products}


# --------------------------------------------------------------------- exact --

def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    if kind in ("newton", "dc") and case["rows"] * case["cols"] <= 11000:
        volts = 5.0 if kind == "newton" else case["volts"]
        mesh = _Mesh(case["rows"], case["cols"], seed, 0.10 if kind == "newton" else case["diodes"])
        b = torch.zeros(mesh.n, dtype=torch.float64, device=dev)
        b[0] = volts / mesh.r_src
        return mesh.with_source(volts, _diode_newton(mesh, mesh.conductance(dev), b, 0.0 * b)).cpu().numpy()
    if kind == "linear":
        return _ladder_exact(_Ladder(case["nodes"], seed))
    if kind == "spmv":
        a, ok = _mesh_matrix(case["rows"], case["cols"], seed)
        x = np.random.default_rng(seed + 1).standard_normal(a.nrows)
        v, near = np.zeros(ok.shape), np.zeros(ok.shape, dtype=np.int64)
        v[ok], near[ok] = a.val, a.col
        return (v * x[near]).sum(axis=1)
    if kind == "ac":
        return _ac_exact(case, seed, dev)
    if kind == "tran" and case["circuit"] == "mesh" and case["size"] <= 32:
        mesh = _Mesh(case["size"], case["size"], seed, 0.05, caps=True, r_src=50.0)
        v, _ = _be_run(mesh, 2e-12, case["steps"], dev)
        wave = mesh.with_source(1.0, torch.stack(v[1:])).cpu().numpy()
        return {"wave": wave[:, :-1], "x": wave[-1]}
    if kind == "adjoint":
        return _adjoint_exact(case, seed, dev)
    return None


def _diode_newton(mesh, g, b, x):
    """G x + diode currents = b on the mesh nodes: Newton with the junction
    voltages limited, dense elimination."""
    nvt, is_ = _nvt()
    sites = torch.from_numpy(mesh.sites).to(g.device)
    if not len(sites):
        return torch.linalg.solve(g, b)
    vcrit = nvt * math.log(nvt / (math.sqrt(2.0) * is_))
    v = x[sites]
    left = 2
    for _ in range(300):
        e = torch.exp(torch.clamp(v / nvt, -80.0, 80.0))
        a, rhs = g.clone(), b.clone()
        a.diagonal()[sites] += is_ * e / nvt
        rhs[sites] -= is_ * (e - 1.0) - is_ * e / nvt * v
        x = torch.linalg.solve(a, rhs)
        new = x[sites]
        far = (new > vcrit) & ((new - v).abs() > 2.0 * nvt)
        up = torch.where(v > 0, v + nvt * torch.log(torch.clamp(1.0 + (new - v) / nvt, min=1e-3)),
                         nvt * torch.log(torch.clamp(new / nvt, min=1e-3)))
        step = float((new - v).abs().max())
        v = torch.where(far, up, new)
        if step < 1e-9:
            left -= 1
            if left == 0:
                return x
    raise RuntimeError("no operating point")


def _be_run(mesh, h, steps, dev):
    """Backward Euler from rest with the source at 1 V from the first step on:
    the voltages after each step, and the matrix without diodes."""
    a = mesh.conductance(dev)
    ch = torch.from_numpy(mesh.caps).to(dev) / h
    a.diagonal().add_(ch)
    v = [torch.zeros(mesh.n, dtype=torch.float64, device=dev)]
    for _ in range(steps):
        b = ch * v[-1]
        b[0] += 1.0 / mesh.r_src
        v.append(_diode_newton(mesh, a, b, v[-1]))
    return v, a


def _adjoint_exact(case, seed, dev):
    h, steps = 2e-12, case["steps"]
    mesh = _Mesh(case["rows"], case["cols"], seed, 0.05, caps=True, r_src=50.0)
    nvt, is_ = _nvt()
    v, a = _be_run(mesh, h, steps, dev)
    ch = torch.from_numpy(mesh.caps).to(dev) / h
    sites = torch.from_numpy(mesh.sites).to(dev)
    ra, rb = torch.from_numpy(mesh.a).to(dev), torch.from_numpy(mesh.b).to(dev)
    r = torch.from_numpy(mesh.r).to(dev)
    rhs = torch.zeros(mesh.n, dtype=torch.float64, device=dev)
    rhs[_output_node(case)] = 1.0
    g_src, g_r, g_c = torch.zeros_like(r[:1]), torch.zeros_like(r), torch.zeros_like(ch)
    g_is = torch.zeros(len(sites), dtype=torch.float64, device=dev)
    for n in range(steps, 0, -1):
        e = torch.exp(torch.clamp(v[n][sites] / nvt, -80.0, 80.0))
        j = a.clone()
        j.diagonal()[sites] += is_ * e / nvt
        lam = torch.linalg.solve(j, rhs)                     # J is symmetric
        g_src += (1.0 - v[n][0]) * (0.0 - lam[0]) / mesh.r_src ** 2
        g_r += (v[n][ra] - v[n][rb]) * (lam[ra] - lam[rb]) / (r * r)
        g_c -= (v[n] - v[n - 1]) / h * lam
        g_is -= lam[sites] * (e - 1.0)
        rhs = ch * lam
    return {"R": torch.cat([g_src, g_r]).cpu().numpy(), "C": g_c.cpu().numpy(), "Is": g_is.cpu().numpy(),
            "output": float(v[steps][_output_node(case)])}


def _ladder_exact(lad):
    """Elimination of the tridiagonal system of nodes 2..n, node 1 at the source voltage."""
    n = lad.nodes
    gs, gp = 1.0 / lad.series, 1.0 / lad.shunt + GMIN
    d = gp[1:] + gs
    d[:-1] += gs[1:]
    rhs = np.zeros(n - 1)
    rhs[0] = gs[0] * lad.volts
    for k in range(1, n - 1):
        m = gs[k] / d[k - 1]
        d[k] -= m * gs[k]
        rhs[k] += m * rhs[k - 1]
    v = np.zeros(n - 1)
    v[-1] = rhs[-1] / d[-1]
    for k in range(n - 3, -1, -1):
        v[k] = (rhs[k] + gs[k + 1] * v[k + 1]) / d[k]
    i = -(lad.volts - v[0]) * gs[0] - gp[0] * lad.volts
    return np.concatenate([[lad.volts], v, [i]])


def _ac_exact(case, seed, dev):
    """Block elimination over the mesh rows, all frequencies at once."""
    mesh = _Mesh(case["rows"], case["cols"], seed, 0.0, caps=True, r_src=50.0, r_lo=100.0)
    rows, cols = mesh.rows, mesh.cols
    w = torch.from_numpy(2.0 * math.pi * _frequencies(case)).to(dev)
    gh = torch.from_numpy(1.0 / mesh.rh).to(dev)
    gv = torch.from_numpy(1.0 / mesh.rv).to(dev)
    c = torch.from_numpy(mesh.caps).to(dev).view(rows, cols)
    diag = torch.full((rows, cols), GMIN, dtype=torch.float64, device=dev)
    diag[:, :-1] += gh
    diag[:, 1:] += gh
    diag[:-1] += gv
    diag[1:] += gv
    diag[0, 0] += 1.0 / mesh.r_src
    inv, y = [], []
    rhs = torch.zeros(len(w), cols, dtype=torch.complex128, device=dev)
    rhs[:, 0] = 1.0 / mesh.r_src
    for i in range(rows):
        block = torch.zeros(len(w), cols, cols, dtype=torch.complex128, device=dev)
        block.diagonal(dim1=1, dim2=2).copy_(torch.complex(diag[i].expand(len(w), cols), w[:, None] * c[i]))
        block.diagonal(1, 1, 2).sub_(gh[i])
        block.diagonal(-1, 1, 2).sub_(gh[i])
        if i:
            block -= gv[i - 1][:, None] * inv[-1] * gv[i - 1]
            rhs = gv[i - 1] * (inv[-1] @ y[-1][..., None])[..., 0]
        inv.append(torch.linalg.inv(block))
        y.append(rhs)
    v = [None] * rows
    for i in range(rows - 1, -1, -1):
        t = y[i] if i == rows - 1 else y[i] + gv[i] * v[i + 1]
        v[i] = (inv[i] @ t[..., None])[..., 0]
    return mesh.with_source(1.0, torch.cat(v, dim=1)).cpu().numpy()
