"""Calls that follow a refused one: its status never becomes that of a later launch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _brickwork(n, seed, **noise):
    from cast_simulator_b200.types import QuantumCircuit

    return QuantumCircuit.brickwork(n, 4, seed, **noise)


def _refused(cblib):
    """A device allocation that no GPU can give (16 TiB)."""
    from cast_simulator_b200.cuda import CudaPrecision, CudaStatevector

    with pytest.raises(RuntimeError):
        CudaStatevector(40, CudaPrecision.F64)


@pytest.mark.parametrize("call", ["norm", "populations", "marginal", "overlap", "program", "batch",
                                  "sample", "trajectories"])
def test_a_refused_allocation_leaves_later_calls_alone(cblib, call):
    from cast_simulator_b200 import simulator as S
    from cast_simulator_b200.cuda import CudaPrecision, CudaStatevector
    from cast_simulator_b200.trajectory import TrajectoryProgram

    n, st = 10, S.Stream()
    sv = CudaStatevector(n, CudaPrecision.F64)
    sv.zero()
    gates = _brickwork(n, 3).gates()
    prog, batch = S.GateProgram(CudaPrecision.F64, n, 1e-12, 1e-12), S.CircuitBatch()
    for g in gates:
        prog.add(g.matrix(), g.qubits())
    batch.add(sv, gates)
    traj = TrajectoryProgram(_brickwork(n, 3, depolarizing=1e-3), 3)
    want = traj.run(3, 5)[0]
    _refused(cblib)
    if call == "norm":
        assert abs(sv.norm_squared() - 1) < 1e-12
    elif call == "populations":
        assert np.allclose(S.qubit_populations(sv, st)[0], 0)
    elif call == "marginal":
        assert np.allclose(S.marginal_probabilities(sv, [1, 4], st), [1, 0, 0, 0])
    elif call == "overlap":
        assert abs(S.inner_product(sv, sv, st) - 1) < 1e-12
    elif call == "program":
        prog.run(sv, st)
        st.sync()
        assert abs(sv.norm_squared() - 1) < 1e-12
    elif call == "batch":
        assert len(batch.run(st)[0]) == n
    elif call == "sample":
        assert (S.sample(sv, 16, 1, stream=st) == 0).all()
    else:
        assert np.array_equal(traj.run(3, 5, st)[0], want)


def test_reductions_on_many_streams_between_refusals(cblib):
    """Threads share one scratch and one count of finished blocks: every result stays
    that of its own state while other threads' allocations are refused."""
    import threading

    from cast_simulator_b200 import simulator as S
    from cast_simulator_b200.cuda import CudaPrecision, CudaStatevector

    wrong = []

    def work(j):
        n, st = 12 + 3 * j, S.Stream()
        sv = CudaStatevector(n, CudaPrecision.F64 if j % 2 else CudaPrecision.F32)
        sv.zero()
        try:
            for i in range(30):
                if i % 5 == j % 5:
                    _refused(cblib)
                p, norm = S.qubit_populations(sv, st)
                m = S.marginal_probabilities(sv, [0, n - 1], st)
                if norm != 1 or p.any() or m.tolist() != [1, 0, 0, 0] or S.inner_product(sv, sv, st) != 1:
                    wrong.append((j, i))
        except Exception as e:
            wrong.append((j, str(e)))

    threads = [threading.Thread(target=work, args=(j,)) for j in range(5)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:4]


def test_a_reduction_refuses_a_stream_under_capture(cblib):
    """Refused before anything is enqueued: the capture goes on and later reductions
    keep their scratch."""
    import torch

    from cast_simulator_b200 import simulator as S
    from cast_simulator_b200.cuda import CudaPrecision, CudaStatevector

    sv = CudaStatevector(14, CudaPrecision.F64)
    sv.zero()
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    x = torch.zeros(8, device="cuda")

    class Captured:
        handle = side.cuda_stream

    with torch.cuda.graph(graph, stream=side):
        x += 1
        with pytest.raises(RuntimeError, match="captured"):
            S.qubit_populations(sv, Captured)
        x += 1
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [2.0] * 8
    p, norm = S.qubit_populations(sv, S.Stream())
    assert norm == 1 and not p.any()


def test_dropping_a_large_program_leaves_a_capture_valid(cblib):
    """A plan's buffer beyond what the pool keeps is freed at once, also while a stream
    is being captured."""
    import torch

    from cast_simulator_b200 import simulator as S
    from cast_simulator_b200.cuda import CudaPrecision, CudaStatevector
    from cast_simulator_b200.types import QuantumGate

    n, st = 12, S.Stream()
    m = QuantumGate.random_unitary([0, 1, 2, 3], np.random.default_rng(0)).matrix()
    prog = S.GateProgram(CudaPrecision.F64, n, 0.0, 0.0)
    for i in range(11500):  # 6 KB of matrix each in the plan: more than 64 MB
        prog.add(m, [i % 8, i % 8 + 1, i % 8 + 2, i % 8 + 3])
    sv = CudaStatevector(n, CudaPrecision.F64)
    sv.zero()
    prog.run(sv, st)
    st.sync()
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    x = torch.zeros(8, device="cuda")
    with torch.cuda.graph(graph, stream=side):
        x += 1
        del prog
        x += 1
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [2.0] * 8
