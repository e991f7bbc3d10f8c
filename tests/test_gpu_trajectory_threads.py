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
