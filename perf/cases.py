"""Performance cases: the work a user of this framework has it do, through its
public entry points, on the GPU.

Kinds of case (each a plain dict; sizes vary within the ranges of ``draw``):

  simulate      one ``Simulator.simulate`` call from |0...0> with the amplitudes
                and <Z> read back: compile, run and read-out of one circuit.
  program       a compiled ``GateProgram`` replayed on a state in hand.
  manager       the drop-in kernel manager: queued gate kernels and one sync.
  density       a noisy circuit as superoperators on the vectorised density
                matrix, then the populations.
  trajectories  a batch of Monte-Carlo quantum-jump trajectories.
  batch         many independent small circuits in one launch.
  measure       read-out of a state in hand: marginals, populations, norm,
                overlap with a second state, and shots.

Outputs are device views of the states and the host results of the calls.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cast_simulator_b200.cuda import CudaKernelGenSpec, CudaKernelManager, CudaPrecision, CudaStatevector
from cast_simulator_b200.fusion import CircuitGraph, FusionConfig, optimize, optimize_native
from cast_simulator_b200.simulator import (
    CircuitBatch,
    QuantumState,
    Representation,
    Simulator,
    inner_product,
    marginal_probabilities,
    qubit_populations,
    sample,
)
from cast_simulator_b200.trajectory import TrajectoryProgram
from cast_simulator_b200.types import QuantumCircuit


# ── cases ────────────────────────────────────────────────────────────────────


def listed():
    return [
        # one small circuit end to end: what a test, a notebook or an optimiser's
        # inner loop does; compile, launches and read-back count
        dict(name="simulate-12q-f64", kind="simulate", n=12, f64=True, depth=10, k=4),
        # a small register replayed: launches and their gaps count
        dict(name="program-17q-f32", kind="program", circuit="brickwork", n=17, f64=False,
             depth=20, k=4, split=False),
        # the 22-qubit QFT (CX form) at the default fusion width: sparse wide gates
        dict(name="qft-22q-f64", kind="program", circuit="qft", n=22, f64=True, depth=0, k=6,
             split=False),
        # single precision at a register larger than the L2 cache
        dict(name="program-26q-f32", kind="program", circuit="brickwork", n=26, f64=False,
             depth=20, k=4, split=False),
        # the headline: 30 qubits, depth 20, complex128
        dict(name="program-30q-f64", kind="program", circuit="brickwork", n=30, f64=True, depth=20,
             k=4, split=False),
        # a dense circuit at the default fusion width in double precision
        dict(name="fused6-24q-f64", kind="program", circuit="brickwork", n=24, f64=True, depth=12,
             k=6, split=False),
        # split precision on the tensor cores
        dict(name="split-28q-f32", kind="program", circuit="brickwork", n=28, f64=False, depth=20,
             k=6, split=True),
        # the drop-in ABI: one launch a gate, per-kernel timing on (its default)
        dict(name="manager-23q-f64", kind="manager", circuit="brickwork", n=23, f64=True, depth=12,
             k=4),
        # an exact noisy simulation: 12 qubits are a 24-qubit vector
        dict(name="density-12q-f64", kind="density", n=12, f64=True, depth=8, k=4),
        # the noisy-trajectory configuration: 16 qubits, depth 30
        dict(name="trajectories-16q", kind="trajectories", n=16, depth=30, k=3, count=2048),
        # a burst of small circuits, both precisions
        dict(name="batch-256", kind="batch", n_min=8, n_max=13, depth=16, k=3, count=256),
        # read-out of a 27-qubit state
        dict(name="measure-27q-f32", kind="measure", n=27, f64=False, measured=5, shots=100000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["simulate", "program", "program", "program", "program", "split", "manager",
                       "density", "trajectories", "batch", "measure", "measure"])
    f64 = rng.random() < 0.5
    if kind == "simulate":
        return dict(kind=kind, n=rng.randint(3, 18), f64=f64, depth=rng.randint(2, 20),
                    k=rng.randint(2, 5))
    if kind == "program":
        qft = rng.random() < 0.3
        n = rng.randint(10, 28)
        return dict(kind=kind, circuit="qft" if qft else "brickwork", n=n, f64=f64,
                    depth=rng.randint(0, 6) if qft else rng.randint(4, 24),
                    k=rng.choice([2, 3, 4, 4, 5, 6] if n <= 26 else [3, 4, 4]), split=False)
    if kind == "split":
        return dict(kind="program", circuit="brickwork", n=rng.randint(16, 29), f64=False,
                    depth=rng.randint(4, 24), k=rng.choice([5, 6]), split=True)
    if kind == "manager":
        return dict(kind=kind, circuit=rng.choice(["brickwork", "qft"]), n=rng.randint(10, 25),
                    f64=f64, depth=rng.randint(3, 16), k=rng.randint(2, 6))
    if kind == "density":
        return dict(kind=kind, n=rng.randint(4, 12), f64=f64, depth=rng.randint(2, 10),
                    k=rng.choice([2, 4]))
    if kind == "trajectories":
        return dict(kind=kind, n=rng.randint(4, 18), depth=rng.randint(4, 24), k=rng.randint(2, 4),
                    count=_log_int(rng, 32, 1024))
    if kind == "batch":
        lo = rng.randint(2, 10)
        return dict(kind=kind, n_min=lo, n_max=lo + rng.randint(0, 4), depth=rng.randint(4, 24),
                    k=rng.randint(2, 4), count=_log_int(rng, 16, 300))
    return dict(kind=kind, n=rng.randint(10, 29), f64=f64, measured=rng.randint(1, 12),
                shots=_log_int(rng, 100, 1000000))


# ── helpers ──────────────────────────────────────────────────────────────────


class _DeviceArray:
    """A device statevector's memory for torch (kept alive by the tensor)."""

    def __init__(self, owner, sv):
        self.owner = owner
        self.__cuda_array_interface__ = {
            "shape": (len(sv),), "typestr": "<f8" if sv.precision() == CudaPrecision.F64 else "<f4",
            "data": (sv.dptr, False), "version": 2}


def _view(sv, owner=None):
    """The statevector's scalars (interleaved re/im) as a torch tensor, no copy."""
    return torch.as_tensor(_DeviceArray(owner or sv, sv), device="cuda")


class _Slot:
    """A statevector inside a larger buffer, as the batch API takes it."""

    def __init__(self, buf, offset, n, f64):
        self._n, self._prec = n, CudaPrecision.F64 if f64 else CudaPrecision.F32
        self.dptr = buf.data_ptr() + offset * (8 if f64 else 4)

    def n_qubits(self):
        return self._n

    def precision(self):
        return self._prec


_SIMS: dict = {}


def _sim(f64, split=False):
    """One simulator (and so one stream) a precision, as a program keeps it."""
    key = (bool(f64), bool(split))
    if key not in _SIMS:
        _SIMS[key] = Simulator(CudaKernelGenSpec.f64() if f64 else CudaKernelGenSpec.f32(),
                               split_precision=split)
    return _SIMS[key]


def _circuit(case, seed):
    if case.get("circuit") == "qft":
        circ = QuantumCircuit.qft_cx(case["n"])
        if case["depth"]:  # the transform inside a larger circuit
            for g in QuantumCircuit.brickwork(case["n"], case["depth"], seed).gates():
                circ.add(g)
        return circ
    return QuantumCircuit.brickwork(case["n"], case["depth"], seed)


def _noisy(case, seed):
    return QuantumCircuit.brickwork(case["n"], case["depth"], seed, 1e-3, 5e-4)


def _fused_gates(case, seed):
    return optimize_native(case["n"], _circuit(case, seed).gates(),
                           FusionConfig.size_only(case["k"])).gates()


def _superoperators(case, seed):
    n = case["n"]
    ops = [g.to_density_matrix_gate(n) for g in _noisy(case, seed).gates()]
    return optimize_native(2 * n, ops, FusionConfig.size_only(case["k"])).gates()


def _graph(case, seed):
    graph = CircuitGraph.from_circuit(_circuit(case, seed))
    optimize(graph, FusionConfig.size_only(case["k"]))
    return graph


def _random_state(n, f64, seed):
    """A normalised complex Gaussian state as 2^(n+1) scalars on the GPU."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    x = torch.empty(2 << n, dtype=torch.float64 if f64 else torch.float32, device="cuda")
    x.normal_(generator=gen)
    return x.div_(float(torch.linalg.vector_norm(x)))


def _statevector(n, f64, seed):
    sv = CudaStatevector(n, CudaPrecision.F64 if f64 else CudaPrecision.F32)
    _view(sv).copy_(_random_state(n, f64, seed))
    return sv


def _batch_members(case, seed):
    """(n, f64, fused gates) of every circuit of a batch, sizes cycling over the range."""
    out = []
    for i in range(case["count"]):
        n = case["n_min"] + i % (case["n_max"] - case["n_min"] + 1)
        circ = QuantumCircuit.brickwork(n, 1 + (i * 7) % case["depth"], seed * 1000 + i)
        out.append((n, i % 4 >= 2, optimize_native(n, circ.gates(),
                                                   FusionConfig.size_only(case["k"])).gates()))
    return out


def _measured(case):
    n, m = case["n"], min(case["measured"], case["n"])
    return [(j * n) // m for j in range(m)]


# ── the calls ────────────────────────────────────────────────────────────────


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "simulate":
        st["sim"], st["graph"] = _sim(case["f64"]), _graph(case, seed)
    elif kind == "program":
        sim = _sim(case["f64"], case["split"])
        st["prog"] = sim.compile_batch(_fused_gates(case, seed), case["n"])
        st["stream"] = sim.stream
        st["sv"] = _statevector(case["n"], case["f64"], seed)
        st["out"] = _view(st["sv"])
    elif kind == "manager":
        mgr = CudaKernelManager(CudaKernelGenSpec.f64() if case["f64"] else CudaKernelGenSpec.f32())
        st["mgr"], st["ids"] = mgr, [mgr.generate(g) for g in _fused_gates(case, seed)]
        st["sv"] = _statevector(case["n"], case["f64"], seed)
        st["out"] = _view(st["sv"])
    elif kind == "density":
        sim = _sim(case["f64"])
        st["prog"] = sim.compile_batch(_superoperators(case, seed), 2 * case["n"])
        st["stream"] = sim.stream
        sv = CudaStatevector(2 * case["n"], CudaPrecision.F64 if case["f64"] else CudaPrecision.F32)
        st["state"] = QuantumState(sv, case["n"], Representation.DensityMatrix)
        st["out"] = _view(sv)
    elif kind == "trajectories":
        st["prog"] = TrajectoryProgram(_noisy(case, seed), case["k"])
        st["stream"], st["seed"] = _sim(False).stream, seed
    elif kind == "batch":
        members = _batch_members(case, seed)
        total = {f64: sum(2 << n for n, p, _ in members if p == f64) for f64 in (False, True)}
        st["buf"] = {f64: torch.zeros(max(2, total[f64]), device="cuda",
                                      dtype=torch.float64 if f64 else torch.float32)
                     for f64 in (False, True)}
        st["batch"], at = CircuitBatch(), {False: 0, True: 0}
        for n, f64, gates in members:
            st["batch"].add(_Slot(st["buf"][f64], at[f64], n, f64), gates)
            at[f64] += 2 << n
        st["stream"] = _sim(True).stream
    else:
        st["a"] = _statevector(case["n"], case["f64"], seed)
        st["b"] = _statevector(case["n"], case["f64"], seed + 1000003)
        st["stream"], st["seed"], st["measured"] = _sim(case["f64"]).stream, seed, _measured(case)
        st["keys"] = np.empty(case["shots"], dtype=np.uint64)
    torch.cuda.synchronize()
    return st


def run(st):
    kind = st["kind"]
    if kind == "simulate":
        state = st["sim"].simulate(st["graph"])
        return {"amplitudes": state.download_amplitudes(), "z": state.expectation_z()}
    if kind == "program":
        st["prog"].run(st["sv"], st["stream"])
        return st["out"]
    if kind == "manager":
        for i in st["ids"]:
            st["mgr"].apply(i, st["sv"])
        st["mgr"].sync()
        return st["out"]
    if kind == "density":
        st["state"].sv.zero(st["stream"])
        st["prog"].run(st["state"].sv, st["stream"])
        st["stream"].sync()
        return {"rho": st["out"], "populations": st["state"].populations()}
    if kind == "trajectories":
        z, samples = st["prog"].run(st["case"]["count"], st["seed"], st["stream"])
        return {"z": z, "samples": samples.view(np.int32)}
    if kind == "batch":
        z = st["batch"].run(st["stream"])
        return {"z": np.concatenate(z), "f32": st["buf"][False], "f64": st["buf"][True]}
    a, s = st["a"], st["stream"]
    p1, norm = qubit_populations(a, s)
    overlap = inner_product(a, st["b"], s)
    keys = sample(a, st["case"]["shots"], st["seed"], None, s, out=st["keys"])
    return {"marginals": marginal_probabilities(a, st["measured"], s), "p1": p1,
            "norm": norm, "norm_squared": a.norm_squared(),
            "overlap": np.array([overlap.real, overlap.imag]), "keys": keys.view(np.int64)}


# ── what a pass cannot do without ────────────────────────────────────────────


def _gate_flops(gates, n):
    """8 operations a nonzero matrix entry and group."""
    return sum(8.0 * np.count_nonzero(np.abs(g.matrix()) > 1e-12) * 2.0 ** (n - g.n_qubits())
               for g in gates)


def work(case):
    kind, amp = case["kind"], 16 if case.get("f64", False) else 8
    if kind == "simulate":
        gates = _graph(case, 1).gates_in_row_order()
        return {"bytes": sum(16.0 * g.matrix().size for g in gates) + (16.0 + amp) * 2 ** case["n"],
                "flops": _gate_flops(gates, case["n"])}
    if kind in ("program", "manager"):
        return {"bytes": 2.0 * amp * 2 ** case["n"],
                "flops": _gate_flops(_fused_gates(case, 1), case["n"])}
    if kind == "density":  # the state is written, not read: it starts from |0><0|
        return {"bytes": 1.0 * amp * 4 ** case["n"] + 8.0 * 2 ** case["n"],
                "flops": _gate_flops(_superoperators(case, 1), 2 * case["n"])}
    if kind == "trajectories":
        ops = TrajectoryProgram(_noisy(case, 1), case["k"]).ops()
        per = sum(8.0 * np.count_nonzero(np.abs(m) > 1e-12) * 2.0 ** (case["n"] - k)
                  for op, k, _, _, _, mats in ops if op == "gate" for m in mats)
        return {"bytes": case["count"] * (8.0 * case["n"] + 4), "flops": case["count"] * per}
    if kind == "batch":
        members = _batch_members(case, 1)
        return {"bytes": sum((16.0 if f64 else 8.0) * 2 ** n + 8 * n for n, f64, _ in members),
                "flops": sum(_gate_flops(g, n) for n, _, g in members)}
    # populations, norm, marginals and shots read the state once each, the overlap two
    return {"bytes": 6.0 * amp * 2 ** case["n"] + 8.0 * case["shots"],
            "flops": 30.0 * 2 ** case["n"]}


def tolerance(case):
    kind = case["kind"]
    if kind == "trajectories":
        # FP32 amplitudes move <Z> by about 1e-6 of itself; a shot flips where its
        # uniform falls within that of a step of the CDF
        return {"rel": 2e-5, "max": 2e-3, "differ": 0.005}
    if kind == "batch":  # both precisions: the FP32 states measured 3e-7 from 64 bits
        return {"rel": 2e-6, "max": 1e-4}
    if kind == "measure":  # FP64 sums of the same terms; whole keys stay the same
        return {"rel": 1e-13, "max": 1e-12}
    # at least four times the distance from 64 bits seen at the listed depths, with
    # room for the deepest drawn ones (error grows as the root of the gate count):
    # 2.8e-5 split, 2.4e-15
    # FP64, 9e-7 FP32
    if case.get("split"):
        return {"rel": 1.2e-4, "max": 2.4e-3}
    return {"rel": 3e-14, "max": 1.2e-12} if case["f64"] else {"rel": 6e-6, "max": 2.4e-4}


# ── the results in 64 bits, in plain torch ───────────────────────────────────


def _apply(psi, matrix, qubits):
    """The gate (ascending qubits, qubits[b] = bit b of the matrix index) on psi."""
    n, k = int(psi.numel()).bit_length() - 1, len(qubits)
    shape, hi = [], n
    for q in reversed(qubits):
        shape += [1 << (hi - q - 1), 2]
        hi = q
    shape.append(1 << hi)
    targets, rest = list(range(1, 2 * k, 2)), list(range(0, 2 * k + 1, 2))
    order = targets + rest
    x = psi.view(shape).permute(order)
    y = torch.as_tensor(matrix, device=psi.device) @ x.reshape(1 << k, -1)
    back = [order.index(i) for i in range(len(order))]
    return y.view(x.shape).permute(back).reshape(-1)


def _exact_state(gates, n, psi=None):
    if psi is None:
        psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
        psi[0] = 1
    for g in gates:
        psi = _apply(psi, np.ascontiguousarray(g.matrix()), list(g.qubits()))
    return psi


def _exact_z(psi):
    n = int(psi.numel()).bit_length() - 1
    p = psi.abs().square()
    p1 = [float(p.view(-1, 2, 1 << q)[:, 1].sum()) for q in range(n)]
    total = float(p.sum())
    return np.array([(total - 2 * x) / total for x in p1])


def exact(case, seed):
    kind = case["kind"]
    if kind == "simulate":
        psi = _exact_state(_graph(case, seed).gates_in_row_order(), case["n"])
        return {"amplitudes": psi.cpu().numpy(), "z": _exact_z(psi)}
    if kind in ("program", "manager"):
        x = _random_state(case["n"], case["f64"], seed).double()
        psi = _exact_state(_fused_gates(case, seed), case["n"], torch.view_as_complex(x.view(-1, 2)))
        return torch.view_as_real(psi).reshape(-1)
    if kind == "density":
        rho = _exact_state(_superoperators(case, seed), 2 * case["n"])
        diag = rho.view(1 << case["n"], 1 << case["n"]).diagonal().real
        return {"rho": torch.view_as_real(rho).reshape(-1), "populations": diag.cpu().numpy()}
    if kind == "trajectories":
        return None
    if kind == "batch":
        z, states = [], {False: [], True: []}
        for n, f64, gates in _batch_members(case, seed):
            psi = _exact_state(gates, n)
            z.append(_exact_z(psi))
            states[f64].append(torch.view_as_real(psi).reshape(-1))
        pad = torch.zeros(2, dtype=torch.float64, device="cuda")
        return {"z": np.concatenate(z), "f32": torch.cat(states[False]) if states[False] else pad,
                "f64": torch.cat(states[True]) if states[True] else pad}
    a, b = (_random_state(case["n"], case["f64"], s).double().view(-1, 2)
            for s in (seed, seed + 1000003))
    p = a.square().sum(1)
    marg = p
    n, measured = case["n"], _measured(case)
    # sum out the qubits that are not measured, from the highest down
    for q in range(n - 1, -1, -1):
        if q not in measured:
            marg = marg.view(-1, 2, 1 << q).sum(1).reshape(-1)
    p1 = np.array([float(p.view(-1, 2, 1 << q)[:, 1].sum()) for q in range(n)])
    re = float((a * b).sum())
    im = float((a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]).sum())
    total = float(p.sum())
    return {"marginals": marg.cpu().numpy(), "p1": p1, "norm": total, "norm_squared": total,
            "overlap": np.array([re, im]), "keys": None}
