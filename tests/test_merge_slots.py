"""Merge slots past GSAP's grid keep targets and dS of earlier steps, and so
targets of larger block counts.  They take part in a block's best proposal, but
the blockmodel of the present step has no rows of such blocks."""
import pytest

pytestmark = pytest.mark.gpu


def outcome(sbp, g, seed, dense_max):
    try:
        rep = sbp.partition(g, seed=seed, dense_max=dense_max, ref_grid=1, verbose=1)
    except sbp.SbpError as e:  # a kept target past B that wins ends the run
        return str(e)
    return g.partitions.tobytes(), rep["S"], rep["B"], rep["nodal_itrs"]


# Sparse graphs: at the merge steps from these B the grid (entries of M, at
# most E) ends before slot 10 B, and the dense form of the step's sweeps holds
# the labels.  In the oracle's runs 70 to 160 of the kept targets lie past B.
@pytest.mark.parametrize("N,blocks,hi,seed,dense_max,B", [
    (1500, 8, 6, 0, 700, 634), (1500, 8, 6, 1, 700, 634), (2000, 10, 8, 2, 900, 845)])
def test_kept_targets_of_a_larger_block_count(sbp, capfd, N, blocks, hi, seed, dense_max, B):
    g = sbp.dcsbm(N, blocks, 1.0, 0.9, seed=seed, deg_min=2, deg_max=hi)
    assert g.E + 256 < 10 * B and B <= dense_max
    capfd.readouterr()
    got = outcome(sbp, g, seed, dense_max)
    assert f" B={B} " in capfd.readouterr().err
    assert got == outcome(sbp, g, seed, 0)  # the CSR form, whose rows are searched
