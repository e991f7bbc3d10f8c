"""Merged gate passes (several gates of a program for one read and one write of
the state) against the oracle, at the edges of their tiles."""
import numpy as np
import pytest

from cast_simulator_b200 import types as T
from cast_simulator_b200.cuda import CudaPrecision, CudaStatevector
from cast_simulator_b200.simulator import GateProgram, Stream
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _random_gates(n, count, widths, seed):
    rng = np.random.default_rng(seed)
    out = []
    for i in range(count):
        k = min(n, widths[i % len(widths)])
        qs = rng.choice(n, size=k, replace=False)
        if i % 3 == 0:  # neighbouring targets, the common shape of fused circuits
            q0 = int(rng.integers(0, n - k + 1))
            qs = np.arange(q0, q0 + k)
        out.append(T.QuantumGate.random_unitary([int(q) for q in qs], rng))
    return out


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("n,widths", [
    (6, (2, 3)),           # below the smallest tile: one kernel a gate
    (7, (1, 2, 3, 4)),     # one tile, one block a gate
    (8, (4,)), (9, (1, 2)), (11, (3,)),
    (12, (1, 2, 3, 4)), (13, (4, 3)), (16, (2, 4)), (19, (4, 3, 1)), (20, (1, 2, 3, 4)),
    (22, (4, 3)),          # complex64: 4-qubit gates alone, 3-qubit ones merged
])
@pytest.mark.parametrize("prec", [CudaPrecision.F64, CudaPrecision.F32])
def test_program_matches_oracle(n, widths, graph, prec):
    rng = np.random.default_rng(n)
    psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    psi /= np.linalg.norm(psi)
    gates = _random_gates(n, 24, widths, 100 + n)
    tol = 1e-12 if prec == CudaPrecision.F64 else 1e-6
    prog = GateProgram(prec, n, tol, tol)
    want = psi.copy()
    for g in gates:
        prog.add(g.matrix(), g.qubits())
        O.apply_gate(want, g.matrix(), g.qubits())
    sv, st = CudaStatevector(n, prec), Stream()
    # 24 unitary gates: each adds at most a few units of 2^k roundings
    bound = 24 * 16 * (2.3e-16 if prec == CudaPrecision.F64 else 1.2e-7)
    for _ in range(3 if graph else 1):  # a direct run, the captured one, a replay
        sv.upload(psi)
        prog.run(sv, st, use_graph=graph)
        st.sync()
        assert np.abs(sv.download() - want).max() <= bound * np.abs(want).max()


def _sparse_gate(n, k, per_row, rng):
    """A unitary of 2^k with per_row nonzeros a row: blocks times a permutation."""
    d = 1 << k
    m = np.zeros((d, d), dtype=np.complex128)
    for b in range(0, d, per_row):
        q, _ = np.linalg.qr(rng.standard_normal((per_row, per_row)) + 1j * rng.standard_normal((per_row, per_row)))
        m[b:b + per_row, b:b + per_row] = q
    m = m[rng.permutation(d)][:, rng.permutation(d)]
    qs = np.sort(rng.choice(n, size=k, replace=False))
    if rng.random() < 0.5:
        q0 = int(rng.integers(0, n - k + 1))
        qs = np.arange(q0, q0 + k)
    return T.QuantumGate(m, [int(q) for q in qs])


@pytest.mark.parametrize("n", [7, 9, 10, 12, 13, 16, 19, 21])
@pytest.mark.parametrize("prec", [CudaPrecision.F64, CudaPrecision.F32])
def test_sparse_gates_in_passes(n, prec):
    rng = np.random.default_rng(n)
    psi = O.random_state(n, n)
    tol = 1e-12 if prec == CudaPrecision.F64 else 1e-6
    prog, want = GateProgram(prec, n, tol, tol), psi.copy()
    for i in range(18):
        # 5 to 7 qubits with 1 to 8 nonzeros a row (7 qubits: up to 2 merge, more run alone)
        k = 5 + i % 3
        g = (T.QuantumGate.random_unitary([int(q) for q in rng.choice(n, size=3, replace=False)], rng)
             if i % 6 == 5 else _sparse_gate(n, min(k, n), (1, 2, 1, 4, 8)[i % 5], rng))
        prog.add(g.matrix(), g.qubits())
        O.apply_gate(want, g.matrix(), g.qubits())
    sv, st = CudaStatevector(n, prec), Stream()
    bound = 18 * 8 * (2.3e-16 if prec == CudaPrecision.F64 else 1.2e-7)
    for _ in range(3):  # a direct run, the captured one, a replay
        sv.upload(psi)
        prog.run(sv, st)
        st.sync()
        assert np.abs(sv.download() - want).max() <= bound * np.abs(want).max()


def test_a_changed_choice_replaces_plan_and_graphs():
    """A program that has a graph runs the grouping its plan() reports after a kernel
    choice changes, and the old one again after it is taken back."""
    from cast_simulator_b200.simulator import set_kernel_choice

    n, prec = 12, CudaPrecision.F64
    psi, gates = O.random_state(n, 4), _random_gates(n, 20, (3,), 5)
    st, sv = Stream(), CudaStatevector(n, prec)

    def program():
        prog = GateProgram(prec, n, 1e-12, 1e-12)
        for g in gates:
            prog.add(g.matrix(), g.qubits())
        return prog

    def state(prog):
        sv.upload(psi)
        prog.run(sv, st)
        st.sync()
        return sv.download()

    prog = program()
    merged = [state(prog) for _ in range(3)]  # direct, captured, replayed
    assert all(np.array_equal(m, merged[0]) for m in merged)
    masks = {sum(1 << q for q in g.qubits() if q < 5) for g in gates} - {0}
    for m in masks:
        set_kernel_choice(prec, 3, m, "register")
    try:
        alone = state(program())
        assert not np.array_equal(alone, merged[0])  # other roundings: the test can tell them apart
        for _ in range(3):
            assert np.array_equal(state(prog), alone)
    finally:
        for m in masks:
            set_kernel_choice(prec, 3, m, None)
    for _ in range(3):
        assert np.array_equal(state(prog), merged[0])
    want = psi.copy()
    for g in gates:
        O.apply_gate(want, g.matrix(), g.qubits())
    for got in (merged[0], alone):
        assert np.abs(got - want).max() <= 20 * 16 * 2.3e-16


@pytest.mark.parametrize("bad", [np.inf, np.nan])
@pytest.mark.parametrize("widths", [(1,), (2,), (1, 2, 3, 4)])
@pytest.mark.parametrize("prec", [CudaPrecision.F64, CudaPrecision.F32])
@pytest.mark.parametrize("path", ["program", "batch"])
def test_an_infinity_stays_in_its_groups(path, prec, widths, bad):
    """An amplitude that is not finite reaches the amplitudes that gates on its qubits
    mix it with, and no others."""
    from cast_simulator_b200.simulator import CircuitBatch

    n, acted, at = 10, [1, 4, 5, 8], 0b1011010110
    rng = np.random.default_rng(len(widths))
    gates = [T.QuantumGate.random_unitary(sorted(int(q) for q in rng.choice(acted, size=widths[i % len(widths)],
                                                                             replace=False)), rng)
             for i in range(12)]
    psi = O.random_state(n, 6)
    want = psi.copy()
    want[at] = 0
    for g in gates:
        O.apply_gate(want, g.matrix(), g.qubits())
    psi[at] = bad
    sv, st = CudaStatevector(n, prec), Stream()
    sv.upload(psi)
    if path == "program":
        prog = GateProgram(prec, n, 0.0, 0.0)
        for g in gates:
            prog.add(g.matrix(), g.qubits())
        assert len(set(prog.plan()[0].tolist())) < len(gates)
        prog.run(sv, st)
        st.sync()
    else:
        batch = CircuitBatch()
        batch.add(sv, gates, init_zero=False)
        batch.run(st)
    mask = sum(1 << q for q in acted)
    apart = (np.arange(1 << n) ^ at) & ~mask != 0  # never in a group with the bad one
    got = sv.download()[apart]
    assert np.isfinite(got).all()
    bound = 12 * 16 * (2.3e-16 if prec == CudaPrecision.F64 else 1.2e-7)
    assert np.abs(got - want[apart]).max() <= bound


@pytest.mark.parametrize("prec", [CudaPrecision.F64, CudaPrecision.F32])
def test_under_a_callers_capture(prec):
    """On a stream that the caller captures, a program enqueues gate after gate and
    allocates nothing; the caller's graph replays it."""
    import torch

    n = 12
    psi, gates = O.random_state(n, 8), _random_gates(n, 20, (1, 2, 3, 4), 9)
    prog, want = GateProgram(prec, n, 0.0, 0.0), psi.copy()
    for g in gates:
        prog.add(g.matrix(), g.qubits())
        O.apply_gate(want, g.matrix(), g.qubits())
    sv, graph, side = CudaStatevector(n, prec), torch.cuda.CUDAGraph(), torch.cuda.Stream()

    class Captured:
        handle = side.cuda_stream

    bound = 20 * 16 * (2.3e-16 if prec == CudaPrecision.F64 else 1.2e-7)
    with torch.cuda.graph(graph, stream=side):
        prog.run(sv, Captured, use_graph=False)
    for _ in range(2):
        sv.upload(psi)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert np.abs(sv.download() - want).max() <= bound * np.abs(want).max()
    sv.upload(psi)  # and in passes again outside the capture
    prog.run(sv, Captured, use_graph=False)
    torch.cuda.synchronize()
    assert np.abs(sv.download() - want).max() <= bound * np.abs(want).max()


@pytest.mark.parametrize("graph", [False, True])
def test_a_dropped_programs_matrices_stay_until_its_launches_end(graph):
    """Programs dropped with their launches queued, each followed by another that could
    take its buffer."""
    n, prec = 22, CudaPrecision.F64
    st, other = Stream(), Stream()
    a, b = CudaStatevector(n, prec), CudaStatevector(n, prec)
    psi = O.random_state(n, 2)
    a.upload(psi)
    b.upload(psi)
    want_a, want_b = psi.copy(), psi.copy()
    for j in range(4):
        for sv, stream, want, runs in ((a, st, want_a, 3), (b, other, want_b, 1)):
            gates = _random_gates(n, 6, (3, 4), 10 * j + runs)
            prog = GateProgram(prec, n, 1e-12, 1e-12)
            for g in gates:
                prog.add(g.matrix(), g.qubits())
            for _ in range(runs):
                prog.run(sv, stream, use_graph=graph)
                for g in gates:
                    O.apply_gate(want, g.matrix(), g.qubits())
            del prog  # its launches are still queued
    st.sync()
    other.sync()
    bound = 4 * 3 * 6 * 16 * 2.3e-16
    assert np.abs(a.download() - want_a).max() <= bound
    assert np.abs(b.download() - want_b).max() <= bound
