"""CUDA graphs of queued sweeps: what is captured, and that it is replayed."""
import pytest

import graphs


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
