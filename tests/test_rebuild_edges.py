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
