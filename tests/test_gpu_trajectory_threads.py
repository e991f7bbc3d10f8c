"""Trajectory programs of different sizes run from several host threads at once:
each thread's results are those of the same program run alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [False, True])
def test_programs_of_different_sizes_run_in_threads(cblib, graph):
    from cast_simulator_b200.simulator import Stream
    from cast_simulator_b200.trajectory import TrajectoryProgram
    from cast_simulator_b200.types import QuantumCircuit

    # from one small tile to two of 2^13 amplitudes and the most matrices a pass takes
    shapes = [(8, 3, 2), (10, 4, 3), (13, 4, 4), (14, 6, 4)]
    circuits = [QuantumCircuit.brickwork(n, depth, n, depolarizing=1e-3, damping=5e-4)
                for n, depth, _ in shapes]
    alone = [TrajectoryProgram(c, k).run(4, 11)[0] for c, (_, _, k) in zip(circuits, shapes)]
    wrong = []

    def work(j):
        st = Stream()
        try:
            for _ in range(60):
                prog = TrajectoryProgram(circuits[j], shapes[j][2])
                for _ in range(4):
                    z, _s = prog.run(4, 11, st, use_graph=graph)
                    if not np.array_equal(z, alone[j]):
                        wrong.append((shapes[j], "differs from the run alone"))
        except RuntimeError as e:
            wrong.append((shapes[j], str(e)))

    threads = [threading.Thread(target=work, args=(j,)) for j in range(len(shapes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:4]


@pytest.mark.parametrize("n,k,p", [(8, 2, 3e-2), (12, 3, 1e-2), (13, 4, 3e-3), (14, 2, 1e-2), (16, 3, 1e-2),
                                   (17, 2, 3e-3)])
def test_fired_pieces_match_the_plain_kernel(cblib, n, k, p):
    """The same draws (depolarizing: they do not depend on the state) in passes where a
    piece stays quiet, block by block where it fires, and block by block throughout."""
    from cast_simulator_b200.trajectory import TrajectoryProgram
    from cast_simulator_b200.types import QuantumCircuit

    prog = TrajectoryProgram(QuantumCircuit.brickwork(n, 8, n, depolarizing=p), k)
    blocks = sum(op[0] == "gate" for op in prog.ops())
    z, _ = prog.run(24, 3)
    prog.set_launch(1024, 0)  # the kernel without segments
    plain, _ = prog.run(24, 3)
    # a block is at most 16 FP32 products and sums an amplitude; fired sites add as many
    assert np.abs(z - plain).max() <= 4 * blocks * 16 * 1.2e-7
