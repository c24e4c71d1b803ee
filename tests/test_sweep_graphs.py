"""CUDA graphs of queued sweeps: what is captured, and that it is replayed."""
import os
import subprocess

import pytest

import graphs

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
@pytest.mark.parametrize("variant,N,B", [("LL", 1000, 11), ("HH", 5000, 24)])
def test_one_capture_a_step(sbp, variant, N, B):
    # in the dense form a step's ticks of three sweeps have the same launches:
    # the first is captured (or found from an earlier call), the others replay it
    # (99: a step that runs to its limit does so in ticks of three too)
    g = graphs.dcsbm(variant, N, B, 3)
    rep = sbp.partition(g, seed=1, dense_max=N, max_nodal_itr=99)
    ticks = rep["graph_captures"] + rep["graph_replays"]
    assert rep["graph_captures"] <= rep["outer_steps"]
    assert 3 * ticks >= rep["nodal_itrs"]
    lab = g.partitions.copy()
    off = sbp.partition(g, seed=1, dense_max=N, max_nodal_itr=99, use_graphs=0)
    assert (lab == g.partitions).all() and off["S"] == rep["S"]
    assert off["graph_captures"] == off["graph_replays"] == 0


@pytest.mark.gpu
def test_graphs_of_sweeps_only_calls(sbp, tmp_path):
    # captured where the graph is replayed in the same call, otherwise issued
    # directly: a call does not pay for a graph that only a later call with the
    # same buffers could replay
    from gsap_b200 import build
    exe = tmp_path / "sweep_graphs"
    lib = os.path.join(ROOT, "gsap_b200")
    cuda = os.path.dirname(os.path.dirname(build.nvcc()))
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(lib, "csrc"),
                    "-I", os.path.join(cuda, "include"),
                    os.path.join(ROOT, "tests", "sweep_graphs_main.cpp"),
                    os.path.join(lib, "libsbp.so"), f"-Wl,-rpath,{lib}",
                    "-L", os.path.join(cuda, "lib64"), "-lcudart",
                    f"-Wl,-rpath,{os.path.join(cuda, 'lib64')}", "-o", str(exe)], check=True)
    # ticks of three sweeps, the last one of the rest
    counts = ["1", "3", "5", "6", "7", "9", "10", "30"]
    r = subprocess.run([str(exe), *counts], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    got = [tuple(int(x) for x in line.split()) for line in r.stdout.splitlines()]
    assert [x[0] for x in got] == [int(c) for c in counts]
    for sweeps, captures, replays, same, moved in got:
        assert same and moved, sweeps
        ticks = sweeps // 3  # equal ones
        assert captures <= (1 if ticks > 2 else 0), sweeps
        # a graph of the same launches, from an earlier call, may serve sooner
        assert captures + replays <= ticks and (replays >= ticks - 2 or ticks < 3), sweeps
