"""How a gate program is grouped into merged passes (no GPU): every grouping is a
legal order of the program, within the kernel's limits."""
import numpy as np
import pytest

from cast_simulator_b200 import types as T
from cast_simulator_b200.cuda import CudaPrecision
from cast_simulator_b200.simulator import GateProgram, set_kernel_choice
from oracle import oracle as O

TILE = 13  # qubits of the largest tile


def _program(n, prec, gates):
    prog = GateProgram(prec, n, 0.0, 0.0)
    for g in gates:
        prog.add(g.matrix(), g.qubits())
    return prog


def _gates(n, count, widths, seed, spread):
    rng = np.random.default_rng(seed)
    out = []
    for i in range(count):
        k = min(n, widths[i % len(widths)])
        q0 = int(rng.integers(0, n - k + 1))
        qs = rng.choice(n, size=k, replace=False) if spread else np.arange(q0, q0 + k)
        out.append(T.QuantumGate.random_unitary([int(q) for q in qs], rng))
    return out


@pytest.mark.parametrize("prec", [CudaPrecision.F64, CudaPrecision.F32])
@pytest.mark.parametrize("spread", [False, True])
@pytest.mark.parametrize("n,widths", [(5, (1, 2)), (8, (2, 3)), (14, (4,)), (17, (1, 2, 3, 4)),
                                      (22, (4, 2)), (30, (4, 3)), (33, (2,))])
def test_plan_is_a_legal_order(n, widths, spread, prec):
    gates = _gates(n, 150, widths, n, spread)
    which, place = _program(n, prec, gates).plan()
    order = sorted(range(len(gates)), key=lambda i: (which[i], place[i]))
    assert len({(int(a), int(b)) for a, b in zip(which, place)}) == len(gates)
    for p in set(which.tolist()):
        members = [i for i in order if which[i] == p]
        assert [int(place[i]) for i in members] == list(range(len(members)))
        assert len(members) <= 16
        if len(members) > 1:
            assert len({q for i in members for q in gates[i].qubits()}) <= min(n, TILE)
    at = {g: i for i, g in enumerate(order)}
    for q in range(n):  # gates that share a qubit keep their order
        chain = [i for i, g in enumerate(gates) if q in g.qubits()]
        assert all(at[a] < at[b] for a, b in zip(chain, chain[1:]))


def test_plan_order_gives_the_same_state():
    n, gates = 9, _gates(9, 40, (1, 2, 3, 4), 3, True)
    which, place = _program(n, CudaPrecision.F64, gates).plan()
    assert len(set(which.tolist())) < len(gates)  # something was merged
    a, b = O.random_state(n, 5), O.random_state(n, 5)
    for g in gates:
        O.apply_gate(a, g.matrix(), g.qubits())
    for i in sorted(range(len(gates)), key=lambda i: (which[i], place[i])):
        O.apply_gate(b, gates[i].matrix(), gates[i].qubits())
    # 40 unitary gates in FP64, in another order of commuting ones
    assert np.abs(a - b).max() <= 40 * 16 * 2.3e-16


def test_forced_kernel_choices_are_not_merged():
    gates = _gates(12, 30, (3,), 1, False)
    prog = _program(12, CudaPrecision.F64, gates)
    merged = len(set(prog.plan()[0].tolist()))
    low = [i for i, g in enumerate(gates) if tuple(g.qubits()) == (0, 1, 2)]
    assert low and merged < len(gates)
    set_kernel_choice(CudaPrecision.F64, 3, 0b111, "register")
    try:
        which = prog.plan()[0].tolist()
        assert all(which.count(which[i]) == 1 for i in low)
    finally:
        set_kernel_choice(CudaPrecision.F64, 3, 0b111, None)
    assert len(set(prog.plan()[0].tolist())) == merged
