"""Nodal dS, proposals and accepted moves at the edges of the kernel paths: a
vertex goes to 8, 16 or 32 lanes, to a CTA or to the heavy-vertex CTA by its
entry counts; each edge of each path, unit and mixed weights, both forms of
the blockmodel, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL = 1e-9  # the FP64 tolerance of the entropy terms, floor of 1 bit
N = 12000
# (out-entries, in-entries) of vertices 0, 1, ...
SHAPES = [(0, 0), (1, 0), (0, 1), (7, 1), (8, 8), (16, 0), (0, 16), (9, 8), (17, 0), (16, 16),
          (32, 0), (0, 32), (32, 1), (1, 32), (32, 32), (33, 0), (0, 33), (33, 31), (31, 33),
          (64, 0), (0, 64), (33, 32), (65, 0), (0, 65), (64, 64), (128, 0), (0, 128), (65, 64),
          (128, 1), (1, 128), (127, 127), (128, 128), (129, 0), (0, 129), (129, 129),
          (0, 2048), (2048, 2048), (1, 2049), (2047, 2050), (5, 4091), (5, 4092), (3, 5000),
          (4100, 4100)]


def shaped_graph(sbp, weighted):
    rng = np.random.default_rng(8)
    K = len(SHAPES)
    src, dst = [], []
    for v, (no, ni) in enumerate(SHAPES):
        src += [np.full(no, v), rng.integers(K, N, ni)]
        dst += [rng.integers(K, N, no), np.full(ni, v)]
    src, dst = np.concatenate(src), np.concatenate(dst)
    w = rng.integers(1, 6, src.size).astype(np.uint32) if weighted else None
    return sbp.Graph.from_edges(N, src, dst, w)


def close(a, b):
    with np.errstate(invalid="ignore"):
        return (a == b) | (np.abs(a - b) <= REL * np.maximum(np.abs(b), 1.0))


@pytest.mark.parametrize("weighted", [False, True], ids=["unit", "weighted"])
@pytest.mark.parametrize("dmax", ["0", "4096"], ids=["csr", "dense"])
@pytest.mark.parametrize("B", [2, 300, 3000, N])
def test_path_edges(sbp, orc, monkeypatch, weighted, dmax, B):
    monkeypatch.setenv("SBP_DENSE_MAX", dmax)
    g = shaped_graph(sbp, weighted)
    rng = np.random.default_rng(B)
    p = rng.integers(0, B, N).astype(np.int32)
    p[-B:] = np.arange(B, dtype=np.int32)
    # every shape, to random blocks, to its own and to neighbours' blocks
    K = len(SHAPES)
    verts = np.tile(np.arange(K, dtype=np.int32), 12)
    props = rng.integers(0, B, verts.size).astype(np.int32)
    src, dst, _ = g.edges()
    for i, v in enumerate(verts):
        near = dst[src == v] if i % 3 == 0 else src[dst == v]
        if i % 3 < 2 and near.size:
            props[i] = p[near[rng.integers(near.size)]]
    got = sbp.delta_mdl_nodal(g, p, B, verts, props)
    want, _ = orc.nodal_delta(g, p, B, verts, props)
    ok = close(got, want)
    assert ok.all(), (verts[~ok], props[~ok], got[~ok], want[~ok])
    for seq in range(3):
        pa, da, xa, _ = sbp.nodal_batch(g, p, B, 21, seq, 0, K)
        pb, db, xb, _ = orc.nodal_batch(g, p, B, 21, seq, 0, K)
        assert np.array_equal(xa, xb), "proposals differ"
        assert close(da, db).all()
        # a dS within its tolerance of 0 (0 before rounding, as of the vertex
        # without edges) may round to either sign: all other moves agree
        moves = (np.abs(da) > REL) | (np.abs(db) > REL)
        assert np.array_equal(pa[:K][moves], pb[:K][moves]), "accepted moves differ"
        assert np.array_equal(pa[:K] != p[:K], da < 0.0)


# hubs: the edge to them (1024 entries in all), more than one hash class of
# blocks, lists longer than a thread's share
HUBS = [(1000, 24), (1000, 25), (200, 824), (200, 825), (3, 2100), (4100, 60), (3, 17000),
        (20000, 9)]


# cells of a few thousand counts at most, whose x log2 x rounds by less than
# 1e-11 each: REL holds with room
@pytest.mark.parametrize("dmax", ["0", "4096"], ids=["csr", "dense"])
@pytest.mark.parametrize("B,weighted", [(300, False), (3000, False), (3000, True), (N, True)])
def test_hub_edges(sbp, orc, monkeypatch, dmax, B, weighted):
    monkeypatch.setenv("SBP_DENSE_MAX", dmax)
    monkeypatch.setattr("test_nodal_paths.SHAPES", HUBS)
    g = shaped_graph(sbp, weighted)
    rng = np.random.default_rng(B + 1)
    p = rng.integers(0, B, N).astype(np.int32)
    p[-B:] = np.arange(B, dtype=np.int32)
    K = len(HUBS)
    verts = np.tile(np.arange(K, dtype=np.int32), 8)
    props = rng.integers(0, B, verts.size).astype(np.int32)
    got = sbp.delta_mdl_nodal(g, p, B, verts, props)
    want, _ = orc.nodal_delta(g, p, B, verts, props)
    assert close(got, want).all()
    for seq in range(4):
        _, da, xa, _ = sbp.nodal_batch(g, p, B, 21, seq, 0, K)
        _, db, xb, _ = orc.nodal_batch(g, p, B, 21, seq, 0, K)
        assert np.array_equal(xa, xb), "proposals differ"
        assert close(da, db).all()


@pytest.mark.parametrize("weighted", [False, True], ids=["unit", "weighted"])
@pytest.mark.parametrize("B", [2, 33, 300])
@pytest.mark.parametrize("batches", [1, 7, N // 40])
def test_dense_update_edges(sbp, weighted, B, batches):
    # the dense form updated from the moves of vertices of every size, batches
    # of 40 to 12,000 vertices, against the CSR form rebuilt after each batch
    g = shaped_graph(sbp, weighted)
    p = np.random.default_rng(B).integers(0, B, N).astype(np.int32)
    p[-B:] = np.arange(B, dtype=np.int32)
    sweeps = 1 if batches > 7 else 3
    a, b = (sbp.nodal_sweeps(g, p, B, 3, 5, num_batches=batches, sweeps=sweeps, dense_max=d)
            for d in (0, N))
    assert (a[0] != p).any()
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


# log of a ratio of two FP64 sums of positive terms
LOGH_TOL = 1e-9


@pytest.mark.parametrize("B", [2, 40, 3000])
@pytest.mark.parametrize("dmax", ["0", "4096"], ids=["csr", "dense"])
def test_path_edges_general_mode(sbp, orc, monkeypatch, dmax, B):
    # every path's edges with mixed weights, exact dS and Hastings ratio: long
    # runs of one block (B = 2) and blocks met once
    monkeypatch.setenv("SBP_DENSE_MAX", dmax)
    g = shaped_graph(sbp, True)
    rng = np.random.default_rng(B)
    p = rng.integers(0, B, N).astype(np.int32)
    p[-B:] = np.arange(B, dtype=np.int32)
    K = len(SHAPES)
    verts = np.tile(np.arange(K, dtype=np.int32), 8)
    props = rng.integers(0, B, verts.size).astype(np.int32)
    src, dst, _ = g.edges()
    for i, v in enumerate(verts):
        near = dst[src == v] if i % 3 == 0 else src[dst == v]
        if i % 3 < 2 and near.size:
            props[i] = p[near[rng.integers(near.size)]]
    got, lh = sbp.delta_mdl_nodal_mode(g, p, B, verts, props, exact=1)
    want, lh_o = orc.nodal_delta_exact(g, p, B, verts, props)
    assert close(got, want).all() and (np.abs(lh - lh_o) <= LOGH_TOL).all()


@pytest.mark.parametrize("weighted", [False, True], ids=["unit", "weighted"])
@pytest.mark.parametrize("B", [3, 200, 5000])
@pytest.mark.parametrize("dmax", ["0", "4096"], ids=["csr", "dense"])
def test_many_wide_vertices(sbp, orc, monkeypatch, dmax, B, weighted):
    # more vertices of 65 to 128 entries in a batch than take a CTA each: a warp
    # each, every count of entries, all out, all in and mixed, few blocks (many
    # entries of one block) and many
    monkeypatch.setenv("SBP_DENSE_MAX", dmax)
    total = np.resize(np.arange(65, 129), 1600)
    out = np.where(np.arange(1600) % 4 == 0, total,
                   np.where(np.arange(1600) % 4 == 1, 0, total * (np.arange(1600) % 7) // 6))
    monkeypatch.setattr("test_nodal_paths.SHAPES", list(zip(out, total - out)))
    g = shaped_graph(sbp, weighted)
    rng = np.random.default_rng(B)
    p = rng.integers(0, B, N).astype(np.int32)
    p[-B:] = np.arange(B, dtype=np.int32)
    verts = np.arange(1600, dtype=np.int32)
    props = rng.integers(0, B, 1600).astype(np.int32)
    props[::3] = p[g.out_idx[g.out_ptr[verts[::3]] % g.E]]  # blocks of some neighbours
    got = sbp.delta_mdl_nodal(g, p, B, verts, props)
    want, mag = orc.nodal_delta_scale(g, p, B, verts, props)
    # at B = 3 cells of 17,000: FP64 rounding of the row sums (mag) passes REL
    ok = close(got, want) | (np.abs(got - want) <= 1e-12 * mag)
    assert ok.all(), (verts[~ok], got[~ok], want[~ok], mag[~ok])
    # the same bits as on a CTA each: the batch in parts below the limit
    parts = [sbp.delta_mdl_nodal(g, p, B, verts[i:i + 400], props[i:i + 400])
             for i in range(0, 1600, 400)]
    assert np.array_equal(got.view(np.int64), np.concatenate(parts).view(np.int64))
    pa, da, xa, _ = sbp.nodal_batch(g, p, B, 21, 4, 0, 1600)
    pb, db, xb, _ = orc.nodal_batch(g, p, B, 21, 4, 0, 1600)
    assert np.array_equal(xa, xb), "proposals differ"
    _, mag = orc.nodal_delta_scale(g, p, B, verts, xb)
    assert (close(da, db) | (np.abs(da - db) <= 1e-12 * mag)).all()


@pytest.mark.parametrize("weighted", [False, True], ids=["unit", "weighted"])
@pytest.mark.parametrize("B", [31, 32, 64, 65, 512, 513])
def test_dense_update_in_few_blocks(sbp, weighted, B):
    # the chunk sums of the dense form added up over a warp (large batches, up to
    # 512 blocks) or entry by entry: draws read them, so the labels would differ
    g = shaped_graph(sbp, weighted)
    p = np.random.default_rng(B).integers(0, B, N).astype(np.int32)
    p[-B:] = np.arange(B, dtype=np.int32)
    a, b = (sbp.nodal_sweeps(g, p, B, 7, 2, num_batches=2, sweeps=4, dense_max=d) for d in (0, N))
    assert (a[0] != p).sum() > 10
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
