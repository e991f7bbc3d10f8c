"""Which blocks of a trajectory program share passes (seg_plan.cpp, no GPU): pieces
that often fire are short or none, and a program where none pays has none."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "cast_simulator_b200", "csrc")


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    exe = tmp_path_factory.mktemp("seg_plan") / "main"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC,
                    os.path.join(HERE, "seg_plan_main.cpp"), os.path.join(CSRC, "seg_plan.cpp"),
                    os.path.join(CSRC, "pass_plan.cpp"), "-o", str(exe)], check=True)

    def run(n, layers, p, damping):
        # a block of two qubits has four error sites
        r = subprocess.run([str(exe), str(n), str(layers), repr((1 - p) ** 4), str(int(damping))],
                           capture_output=True, text=True, check=True, timeout=60)
        rows = [tuple(map(int, x.split())) for x in r.stdout.split("\n") if x]
        return rows[:-1], rows[-1][0], rows[-1][1]

    return run


@pytest.mark.parametrize("n", [8, 12, 13, 14, 15, 16, 17, 18])
@pytest.mark.parametrize("damping", [False, True])
def test_pieces_follow_the_error_rate(plan, n, damping):
    lengths = []
    for p in (1e-4, 1e-3, 1e-2):
        segs, blocks, _ = plan(n, 30, p, damping)
        assert segs and all(passes < count for _, count, passes in segs)
        ends = [first + count for first, count, _ in segs]
        assert all(e <= first for e, (first, _, _) in zip(ends, segs[1:])) and ends[-1] <= blocks
        lengths.append(max(count for _, count, _ in segs))
        if damping:  # no piece reaches over a damping layer
            assert lengths[-1] <= n // 2
        else:  # not the whole circuit, however quiet its blocks
            assert lengths[-1] < blocks
    assert lengths == sorted(lengths, reverse=True)
    assert damping or lengths[0] > 2 * lengths[-1]


@pytest.mark.parametrize("n", [8, 12, 13, 14, 17])
@pytest.mark.parametrize("damping", [False, True])
def test_strong_noise_has_no_segments(plan, n, damping):
    segs, _, threads = plan(n, 30, 0.1, damping)
    assert not segs and threads == (1024 if n == 17 else 512)
