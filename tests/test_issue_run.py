"""How a run is issued (lbm_issue.h), on the host with a stand-in for the CUDA
runtime whose calls can be made to fail: a graph that cannot be built or
launched costs nothing but launches, a launch that is refused leaves the domain
saying what its lattices hold and no incomplete graph behind, and run lengths
that alternate do not build a graph again and again."""
import os
import re
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "nflow-red-poplar_b200", "csrc")
CREATE, BEGIN, END, INSTANTIATE, GRAPH_LAUNCH, IS_CAPTURING, KERNEL = range(7)
RUNS = [5, 5, 5, 6, 6, 6, 6, 70, 70, 70, 70, 300, 300, 1, 1, 1, 1, 97, 97, 97, 97]


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("issue") / "driver")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", os.path.join(HERE, "native", "fake_cuda"),
                    "-I", CSRC, "-o", exe, os.path.join(HERE, "native", "issue_run_driver.cpp")],
                   check=True)

    def run(call, n, runs, breaks=0):
        r = subprocess.run([exe, str(call), str(n), str(breaks)] + [str(v) for v in runs],
                           capture_output=True, text=True, timeout=60)
        assert r.returncode == 0, (call, n, r.stdout)
        return tuple(map(int, re.findall(r"=(\d+)", r.stdout)))

    return run


@pytest.mark.parametrize("call", [CREATE, BEGIN, END, INSTANTIATE, GRAPH_LAUNCH])
def test_graph_failures_cost_launches_only(driver, call):
    for n in list(range(0, 30)) + [-1, -2, -5, -9]:
        failed, _ = driver(call, n, RUNS)
        assert failed == 0, n


@pytest.mark.parametrize("breaks", [0, 1])
def test_refused_launches_leave_a_consistent_domain(driver, breaks):
    for n in range(1, 400):
        failed, _ = driver(KERNEL, n, RUNS, breaks)
        assert failed <= 1, n
    for n in (-1, -7, -40, -200):
        failed, _ = driver(KERNEL, n, RUNS, breaks)
        assert failed > 0, n


def test_refused_capture_query(driver):
    assert driver(IS_CAPTURING, 3, RUNS)[0] == 1


def test_graphs_built(driver):
    assert driver(CREATE, 0, [6])[1] == 0
    assert driver(CREATE, 0, [6] * 5)[1] == 1
    # lengths that alternate from one lattice, with and without a graph of one
    assert driver(CREATE, 0, [6, 8] * 40)[1] == 0
    assert driver(CREATE, 0, [6] * 3 + [8, 6] * 40)[1] == 1
    assert driver(CREATE, 0, [6] * 3 + [6, 6, 8] * 40)[1] == 1
    # a new length for good: its graph takes the place of the old one
    assert driver(CREATE, 0, [6] * 3 + [8] * 30)[1] == 2
