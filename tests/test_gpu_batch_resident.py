"""Batched circuits whose state is held in shared memory (and their neighbours
that stream it), at the edges of the sizes that fit, against the oracle."""
import numpy as np
import pytest

from cast_simulator_b200 import types as T
from cast_simulator_b200.cuda import CudaPrecision, CudaStatevector
from cast_simulator_b200.simulator import CircuitBatch, Stream
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _circuit(n, count, seed):
    rng = np.random.default_rng(seed)
    out = []
    for i in range(count):
        k = min(n, 1 + i % 4)
        out.append(T.QuantumGate.random_unitary([int(q) for q in rng.choice(n, size=k, replace=False)], rng))
    return out


@pytest.mark.parametrize("prec", [CudaPrecision.F64, CudaPrecision.F32])
@pytest.mark.parametrize("sizes", [(1, 2, 3, 4), (5, 6, 7, 8), (3, 4, 7, 9), (10, 11, 12), (13,), (13, 14), (14, 15)])
def test_batch_matches_oracle(sizes, prec):
    st, batch, want, svs = Stream(), CircuitBatch(), [], []
    for j, n in enumerate(sizes):
        for zero in (True, False):
            gates = _circuit(n, 0 if j == 1 and zero else 13, 7 * n + zero)
            psi = O.zero_state(n) if zero else O.random_state(n, n)
            sv = CudaStatevector(n, prec)
            sv.upload(psi)
            batch.add(sv, gates, init_zero=zero)
            for g in gates:
                O.apply_gate(psi, g.matrix(), g.qubits())
            svs.append(sv)
            want.append(psi)
    z = batch.run(st)
    # 13 unitary gates, at most 16 products and sums each
    bound = 13 * 16 * (2.3e-16 if prec == CudaPrecision.F64 else 1.2e-7)
    for got_z, sv, psi in zip(z, svs, want):
        n = sv.n_qubits()
        assert np.abs(sv.download() - psi).max() <= bound
        p = np.abs(psi) ** 2
        idx = np.arange(1 << n)
        want_z = [1 - 2 * p[(idx >> q) & 1 == 1].sum() / p.sum() for q in range(n)]
        assert np.abs(got_z - want_z).max() <= 4 * bound


@pytest.mark.parametrize("prec", [CudaPrecision.F64, CudaPrecision.F32])
def test_a_refused_circuit_leaves_the_batch_as_it_was(prec):
    st, batch = Stream(), CircuitBatch()
    svs = [CudaStatevector(n, prec) for n in (9, 8, 12)]
    gates = [_circuit(n, 9, n) for n in (9, 8, 12)]
    batch.add(svs[0], gates[0])
    wide = T.QuantumGate.random_unitary([0, 1, 2, 3, 4], np.random.default_rng(0))
    outside = T.QuantumGate.random_unitary([7, 8], np.random.default_rng(0))
    for bad in (wide, outside):
        with pytest.raises(RuntimeError):
            batch.add(svs[1], gates[1] + [bad])
        assert len(batch) == 1
    batch.run(st)
    batch.add(svs[2], gates[2])  # after a run: the tables go up again
    z = batch.run(st)
    assert [len(x) for x in z] == [9, 12]
    bound = 9 * 16 * (2.3e-16 if prec == CudaPrecision.F64 else 1.2e-7)
    for sv, gs in ((svs[0], gates[0]), (svs[2], gates[2])):
        psi = O.zero_state(sv.n_qubits())
        for g in gs:
            O.apply_gate(psi, g.matrix(), g.qubits())
        assert np.abs(sv.download() - psi).max() <= bound
