"""The two CSR directions of a graph handed in as arrays need not carry the same
weights (each is checked by itself): unit weights in one say nothing about the
other, and each direction of the blockmodel counts its own entries."""
import numpy as np
import pytest

import graphs

pytestmark = pytest.mark.gpu


def one_direction_weighted(which):
    g = graphs.dcsbm("HH", 3000, seed=9)
    w = np.random.default_rng(2).integers(1, 6, g.E).astype(np.uint32)
    ptr = g.in_ptr if which == "in" else g.out_ptr
    total = np.concatenate([[0], np.cumsum(w.astype(np.int64))])
    deg = (total[ptr[1:]] - total[ptr[:-1]]).astype(np.uint32)
    if which == "in":
        g.in_w, g.deg_in = w, deg
    else:
        g.out_w, g.deg_out = w, deg
    return g


@pytest.mark.parametrize("which", ["in", "out"])
def test_weights_in_one_direction(sbp, which):
    g = one_direction_weighted(which)
    B = 60
    p = np.random.default_rng(4).integers(0, B, g.N).astype(np.int32)
    p[:B] = np.arange(B)
    a = sbp.build_blockmodel(g, p, B)
    for side, ptr, idx, w in (("o", g.out_ptr, g.out_idx, g.out_w),
                              ("i", g.in_ptr, g.in_idx, g.in_w)):
        M = np.zeros((B, B), np.uint32)
        np.add.at(M, (np.repeat(p, np.diff(ptr)), p[idx]), w)
        row, col = np.nonzero(M)
        assert np.array_equal(np.diff(a[side + "ptr"]), np.bincount(row, minlength=B)), side
        assert np.array_equal(a[side + "col"], col), side
        assert np.array_equal(a[side + "cnt"], M[row, col]), side
        assert np.array_equal(a["d_out" if side == "o" else "d_in"], M.sum(1)), side
