"""The blockmodel rebuild and the per-block draws at the edges of their
paths: segments of the lengths where a row goes from the comparison tile to a
warp, a CTA and a cluster, columns across bitmap windows, unit and mixed
weights, every launch shape, against the oracle (exact)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# entries of blocks 0, 1, ... (one vertex each)
LENGTHS = [0, 1, 2, 8, 9, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 257, 511, 512, 513, 1023,
           1024, 1025, 1985, 2048, 2049, 12287, 12288, 12289, 40000]


def long_rows(sbp, N, weighted):
    """Vertex k has LENGTHS[k] out-entries and vertex N-1-k as many
    in-entries (repeated neighbours among them), the others a few."""
    rng = np.random.default_rng(N)
    src, dst = [np.arange(100, N - 100)], [rng.integers(0, N, N - 200)]
    for k, n in enumerate(LENGTHS):
        other = rng.integers(0, N, n)
        src += [np.full(n, k), other]
        dst += [rng.permutation(other), np.full(n, N - 1 - k)]
    src, dst = np.concatenate(src), np.concatenate(dst)
    w = rng.integers(1, 6, src.size).astype(np.uint32) if weighted else None
    return sbp.Graph.from_edges(N, src, dst, w)


@pytest.mark.parametrize("N", [16385, 140000])
@pytest.mark.parametrize("weighted", [False, True], ids=["unit", "weighted"])
@pytest.mark.parametrize("cap,entries", [(32, 512), (64, 1024), (128, 1024)])
def test_rebuild_edges(sbp, orc, monkeypatch, N, weighted, cap, entries):
    monkeypatch.setenv("SBP_DENSE_MAX", "0")
    monkeypatch.setenv("SBP_REBUILD_WARP_CAP", str(cap))
    monkeypatch.setenv("SBP_REBUILD_BIG_ENTRIES", str(entries))
    g = long_rows(sbp, N, weighted)
    rng = np.random.default_rng(1)
    own = np.arange(N, dtype=np.int32)
    few = rng.integers(0, 300, N).astype(np.int32)  # every row long
    few[:300] = np.arange(300)
    for p, B in ((own, N), (few, 300)):
        a = sbp.build_blockmodel(g, p, B)
        b = orc.build_blockmodel(g, p, B)
        for k in ("optr", "ocol", "ocnt", "iptr", "icol", "icnt", "d_out", "d_in"):
            assert np.array_equal(a[k], b[k]), (B, k)
        # draws from rows of every length: vertices next to the long ones
        _, _, xa, _ = sbp.nodal_batch(g, p, B, 5, 3, 100, 1500)
        _, _, xb, _ = orc.nodal_batch(g, p, B, 5, 3, 100, 1500)
        assert np.array_equal(xa, xb), B


# short segments side by side, so that a tile of consecutive rows takes several
# rounds of its 1920-entry window (segments padded to fours)
GROUP, WINDOW = 400, 1920


def crowded_tiles(sbp, weighted):
    """Vertices 0, 1, ... have runs of segments of 20 to 128 out-entries,
    vertices N-1, N-2, ... as many in-entries; the others a few."""
    N = 60000
    rng = np.random.default_rng(11)
    lens = np.concatenate([
        rng.integers(20, 33, GROUP), np.full(GROUP, 32), rng.integers(20, 65, GROUP),
        np.full(GROUP, 64), rng.integers(20, 129, GROUP), np.full(GROUP, 128),
        np.sort(rng.integers(20, 51, GROUP))[::-1], rng.integers(0, 41, GROUP)])
    K = lens.size
    mid = np.arange(K, N - K)
    own = np.repeat(np.arange(K), lens)
    base = rng.integers(K, N - K - 30, K)
    # neighbours near a base of the vertex's own, so that columns repeat
    other = base[own] + rng.integers(0, 30, own.size)
    src = np.concatenate([own, rng.permutation(mid), rng.permutation(other)])
    dst = np.concatenate([other, mid, N - 1 - own])
    w = rng.integers(1, 6, src.size).astype(np.uint32) if weighted else None
    return sbp.Graph.from_edges(N, src.astype(np.int32), dst.astype(np.int32), w)


@pytest.mark.parametrize("weighted", [False, True], ids=["unit", "weighted"])
@pytest.mark.parametrize("cap", [32, 64, 128])
def test_rebuild_tiles_of_several_rounds(sbp, orc, monkeypatch, weighted, cap):
    monkeypatch.setenv("SBP_DENSE_MAX", "0")
    monkeypatch.setenv("SBP_REBUILD_WARP_CAP", str(cap))
    g = crowded_tiles(sbp, weighted)
    N, p = g.N, np.arange(g.N, dtype=np.int32)
    rows = max(8, min(256, 1024 * N // g.E))
    for ptr in (g.out_ptr, g.in_ptr):
        n = np.diff(ptr)
        padded = np.where(n <= cap, (n + 3) & ~3, 0)
        tiles = np.pad(padded, (0, -N % rows)).reshape(-1, rows)
        at = np.cumsum(tiles, axis=1) - tiles
        assert (tiles.sum(1) > 2 * WINDOW).any()
        assert ((at < WINDOW) & (at + tiles > WINDOW)).any() and (at == WINDOW).any()
    a = sbp.build_blockmodel(g, p, N)
    b = orc.build_blockmodel(g, p, N)
    for k in ("optr", "ocol", "ocnt", "iptr", "icol", "icnt", "d_out", "d_in"):
        assert np.array_equal(a[k], b[k]), k


def by_degree(sbp, variant, N, B, seed):
    """A DCSBM graph with its vertices numbered by falling degree."""
    g = sbp.dcsbm_variant(variant, N, B, seed=seed)
    new = np.empty(N, np.int32)
    new[np.argsort(-(g.deg_out.astype(np.int64) + g.deg_in), kind="stable")] = np.arange(N)
    src, dst, w = g.edges()
    truth = np.empty(N, np.int32)
    truth[new] = g.true_partitions
    return sbp.Graph.from_edges(N, new[src], new[dst], w, truth)


@pytest.mark.parametrize("per_block", [1, 3])
def test_batches_of_a_graph_numbered_by_degree(sbp, orc, monkeypatch, per_block):
    monkeypatch.setenv("SBP_DENSE_MAX", "0")
    g = by_degree(sbp, "HH", 20000, 32, 4)
    q = np.arange(g.N, dtype=np.int32) // per_block
    B = int(q[-1]) + 1
    for b in range(4):
        lo, hi = b * 5000, (b + 1) * 5000
        pa, da, xa, _ = sbp.nodal_batch(g, q, B, 13, 40 + b, lo, hi)
        pb, db, xb, _ = orc.nodal_batch(g, q, B, 13, 40 + b, lo, hi)
        assert np.array_equal(xa, xb), "proposals differ"
        with np.errstate(invalid="ignore"):  # -inf on both sides (a block of degree 0)
            assert ((da == db) | (np.abs(da - db) <= 1e-9 * np.maximum(np.abs(db), 1.0))).all()
        # a dS within its tolerance of 0 may round to either sign
        moves = (np.abs(da) > 1e-9) | (np.abs(db) > 1e-9)
        assert np.array_equal(pa[lo:hi][moves], pb[lo:hi][moves]), "accepted moves differ"
        q = pb


def test_partition_of_a_graph_numbered_by_degree(sbp, orc):
    g = by_degree(sbp, "LL", 1000, 11, 0)
    rep = sbp.partition(g, seed=0, dense_max=0)
    lab, rep_o, _ = orc.partition(g, seed=0)
    assert rep["B"] == rep_o["B"] and abs(rep["S"] - rep_o["S"]) <= 1e-9 * abs(rep_o["S"])
    assert sbp.evaluate(lab, g.partitions)[2] > 0.999


def test_tile_word_of_the_last_block(sbp, monkeypatch):
    # at 2^25 blocks the last column at the last place of the longest segment a
    # tile takes would be the word of ones that pads a tile
    monkeypatch.setenv("SBP_DENSE_MAX", "0")
    monkeypatch.setenv("SBP_REBUILD_WARP_CAP", "128")
    N = 1 << 25
    dst = np.concatenate([np.arange(1, 128), [N - 1]]).astype(np.int32)
    g = sbp.Graph.from_edges(N, np.zeros(128, np.int32), dst, None)
    a = sbp.build_blockmodel(g, np.arange(N, dtype=np.int32), N)
    assert np.array_equal(a["ocol"], dst) and (a["ocnt"] == 1).all()
    assert a["optr"][0] == 0 and (a["optr"][1:] == 128).all()
    assert np.array_equal(a["icol"], np.zeros(128)) and (a["icnt"] == 1).all()
    assert np.array_equal(np.flatnonzero(np.diff(a["iptr"])), dst)
    assert a["d_out"][0] == 128 and a["d_out"].sum() == 128 and (a["d_in"][dst] == 1).all()


@pytest.mark.parametrize("weighted", [False, True], ids=["unit", "weighted"])
@pytest.mark.parametrize("B", [300, 9000, 12288, 12289])
def test_many_long_segments(sbp, orc, monkeypatch, B, weighted):
    # twenty blocks of some 15k entries (a CTA each up to 12288 blocks, else a
    # cluster), one of 30k (a cluster); their columns few, and about and above
    # the 8192 whose totals a cluster adds up in shared memory
    monkeypatch.setenv("SBP_DENSE_MAX", "0")
    rng = np.random.default_rng(B)
    size = np.concatenate([np.full(20, 2000), [4300], np.ones(B - 21, np.int64)])
    size[21:] += np.bincount(rng.integers(0, B - 21, 13000 - (B - 21)), minlength=B - 21)
    N = int(size.sum())
    p = np.repeat(np.arange(B, dtype=np.int32), size)
    first = np.cumsum(size) - size
    b = rng.integers(0, B, 7 * N)
    u, v = np.repeat(np.arange(N), 7), first[b] + rng.integers(0, size[b])
    src, dst = np.concatenate([u, v]).astype(np.int32), np.concatenate([v, u]).astype(np.int32)
    order = rng.permutation(N).astype(np.int32)  # a block's vertices lie apart
    w = rng.integers(1, 6, src.size).astype(np.uint32) if weighted else None
    g = sbp.Graph.from_edges(N, order[src], order[dst], w)
    lab = np.empty(N, np.int32)
    lab[order] = p
    n = np.bincount(lab, weights=np.diff(g.out_ptr), minlength=B)
    giants = int((n > 12288).sum())
    assert giants >= 21 and n.max() > 1024 * giants > np.sort(n)[-2]
    a, o = sbp.build_blockmodel(g, lab, B), orc.build_blockmodel(g, lab, B)
    for k in ("optr", "ocol", "ocnt", "iptr", "icol", "icnt", "d_out", "d_in"):
        assert np.array_equal(a[k], o[k]), k
