"""The waiting rule of the grid barrier (csrc/grid_barrier.cuh) on the host: a
block that waits while another works on for many times the poll limit does not
give up, one whose peers have stopped does, after a bounded number of polls."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "lightgraphs.jl_gb300", "csrc")


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path_factory.mktemp("barrier") / "barrier_check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-w", "-I", CSRC, "-o", exe,
                    os.path.join(ROOT, "tests", "barrier_check.cpp")], check=True)
    return exe


def play(exe, games):
    text = "".join("%d %d %d\n" % g for g in games)
    out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout.split()
    return [int(x) for x in out[:3]], [int(x) for x in out[3:-1]], int(out[-1])


def test_waits_while_work_goes_on(harness):
    limit = play(harness, [])[0][0]
    # a beat every thousand polls, one a stretch, and one just inside a stretch
    gave_up = play(harness, [(40 * limit, gap, 40 * limit) for gap in (1000, limit // 2, limit)])[1]
    assert gave_up == [0, 0, 0]


def test_gives_up_when_nothing_moves(harness):
    limit = play(harness, [])[0][0]
    never, stopped = play(harness, [(10 * limit, 0, 0), (20 * limit, 1000, 7 * limit)])[1]
    assert never == limit + 1
    assert 7 * limit < stopped <= 9 * limit + 9


def test_beats_come_in_time(harness):
    (limit, turns, entries), _, beats = play(harness, [])
    assert beats == 20 + 10 * turns // 8
    # a poll takes about as long as the loads that an entry waits for, and a
    # turn waits for 32 rows of 16 loads at most
    assert 100 * entries < limit and 50 * turns * 32 * 16 < limit


def test_loops_between_barriers_beat():
    # every row walk between two barriers reports its turns
    bfs = open(os.path.join(CSRC, "bfs.cu")).read()
    run = bfs[bfs.index("k_bfs_run(DevGraph g, BfsRun r)"):]
    run = run[:run.index("\n}\n")]
    assert run.count("beat_turn(") >= 2 and "entry_due()) beat_now(" in run
    core = open(os.path.join(CSRC, "learned.cu")).read()
    assert core.count("beat_turn(") >= 5 and core.count("work_due(core_units(g, v))") == 2
