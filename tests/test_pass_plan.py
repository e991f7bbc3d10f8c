"""How a gate program is grouped into merged passes (no GPU): every grouping is a
legal order of the program, within the kernel's limits."""
import numpy as np
import pytest

from cast_simulator_b200 import types as T
from cast_simulator_b200.cuda import CudaPrecision
from cast_simulator_b200.simulator import GateProgram, gate_engine, set_kernel_choice
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


def _greedy(masks, n, tb, low, most):
    """The grouping as a plain restatement: every seed grown to the end, every count a
    walk over the whole window."""
    out, pending = [], list(range(len(masks)))
    low_mask = (1 << min(low, n)) - 1

    def scan(q):
        taken, ready, blocked = [], [], 0
        for i in pending[:128]:
            if not masks[i] & blocked:
                if not masks[i] & ~q and len(taken) < most:
                    taken.append(i)
                    continue
                if masks[i] & ~q:
                    ready.append(masks[i])
            blocked |= masks[i]
        return taken, ready

    while pending:
        taken, ready = scan(low_mask)
        best, tile = [], 0
        for seed in ready + ([low_mask] if taken else []):
            q = low_mask | seed
            if q.bit_count() > tb:
                continue
            taken, around = scan(q)
            while True:
                grow, gain, added = 0, 0, 1
                for x in around:
                    if (q | x).bit_count() <= tb:
                        more = len(scan(q | x)[0]) - len(taken)
                        add = (q | x).bit_count() - q.bit_count()
                        if more > 0 and (not grow or more * added > gain * add):
                            grow, gain, added = q | x, more, add
                if not grow:
                    break
                q = grow
                taken, around = scan(q)
            if len(taken) > len(best):
                best, tile = taken, q
        if len(best) < 2:
            best = pending[:1]
        out.append(best)
        pending = [i for i in pending if i not in set(best)]
    return out


@pytest.mark.parametrize("n,widths,spread", [(9, (1,), True), (12, (1, 2), False), (14, (1, 2, 3, 4), True),
                                             (17, (2, 1), True), (20, (1, 1, 2), False)])
def test_plan_is_the_greedy_grouping(n, widths, spread):
    gates = _gates(n, 160, widths, n, spread)
    which, place = _program(n, CudaPrecision.F64, gates).plan()
    masks = [sum(1 << q for q in g.qubits()) for g in gates]
    tile = min(n, 11, max(9, n - 8))  # of complex128 states below 22 qubits
    want = _greedy(masks, n, tile, 3, 16)
    got = [[] for _ in range(int(which.max()) + 1)]
    for i in np.lexsort((place, which)):
        got[which[i]].append(int(i))
    assert got == want


def test_long_programs_are_planned_quickly():
    """Planning is paid in a program's first run: it grows with the gates, not with
    their number times what waits behind them (50000 took 0.9 s)."""
    import time

    n, x = 20, T.QuantumGate.random_unitary([0], np.random.default_rng(1)).matrix()
    prog = GateProgram(CudaPrecision.F64, n, 0.0, 0.0)
    for i in range(50000):
        prog.add(x, [i % n])
    best = min(_timed(prog.plan, time.perf_counter) for _ in range(3))
    assert best < 0.3


def _timed(f, clock):
    t = clock()
    f()
    return clock() - t


def test_tuned_choices_leave_merging_alone():
    from cast_simulator_b200 import autotune as A

    n = 24
    for prec, name in ((CudaPrecision.F64, "f64"), (CudaPrecision.F32, "f32")):
        prog = _program(n, prec, T.QuantumCircuit.brickwork(n, 6, 1).gates())
        plan = prog.plan()
        recs = [{"precision": name, "k": k, "low_mask": m, "engine": e, "tile_bits": tb}
                for (k, m), (e, tb) in zip(A.kernel_classes(), 99 * A.KERNEL_CANDIDATES)]
        try:
            assert A.apply_kernel_choices(recs) == len(recs)
            assert np.array_equal(prog.plan(), plan)
            # they do decide the kernel of a gate that runs alone
            r = next(r for r in recs if r["k"] == 2 and r["engine"] == "tile")
            q = A.class_targets(n, 2, r["low_mask"])
            assert gate_engine(A.haar(2, np.random.default_rng(0)), q, n, prec) == "tile"
        finally:
            for r in recs:
                set_kernel_choice(prec, r["k"], r["low_mask"], None)


def test_a_chosen_tile_size_is_not_merged():
    gates = _gates(12, 30, (3,), 1, False)
    prog = _program(12, CudaPrecision.F64, gates)
    low = [i for i, g in enumerate(gates) if tuple(g.qubits()) == (0, 1, 2)]
    set_kernel_choice(CudaPrecision.F64, 3, 0b111, None, 12)  # the built-in kernel, another tile
    try:
        which = prog.plan()[0].tolist()
        assert all(which.count(which[i]) == 1 for i in low)
    finally:
        set_kernel_choice(CudaPrecision.F64, 3, 0b111, None)
