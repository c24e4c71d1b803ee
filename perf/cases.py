"""The partitioner's workloads, as a user's program runs them.

Graphs are directed DCSBM graphs in the four GraphChallenge-style variants
(p_in 0.8 or 0.5, Dirichlet concentration of the block sizes 20 or 1,
power-law out-degrees of exponent 2.5 on [5, 50]), made here with numpy.

``listed()`` are the fixed cases, ``draw(rng)`` one more of the same ranges,
``prepare`` makes what a program has in hand before the call, ``run`` is one
pass through the public entry points, ``work`` the bytes and operations a
pass cannot do without, ``exact`` the 64-bit value where the outputs are
computed numbers.
"""
import numpy as np
import torch

from gsap_b200 import sbp

# (p_in, Dirichlet alpha) of a variant
VARIANTS = {"LL": (0.8, 20.0), "LH": (0.8, 1.0), "HL": (0.5, 20.0), "HH": (0.5, 1.0)}


def listed():
    return [
        # The smallest whole job: a 1k graph from host memory (a served
        # request's most frequent size). Latency and launches count.
        dict(name="plain-1k-LL", kind="partition", variant="LL", N=1000, B=11, weighted=False),
        # A small graph of odd size with edge weights 1-4 (multigraph input).
        dict(name="plain-5k-weighted", kind="partition", variant="HL", N=5003, B=23,
             weighted=True),
        # The ordinary whole job of one graph from host memory: upload,
        # partition, labels back.
        dict(name="plain-20k-HH", kind="partition", variant="HH", N=20000, B=32, weighted=False),
        # A graph kept in device memory and partitioned; detectable blocks of
        # uneven sizes, odd vertex count.
        dict(name="resident-50k-LH", kind="resident", variant="LH", N=49999, B=45),
        # The headline: 200k vertices, graph resident.
        dict(name="resident-200k-HH", kind="resident", variant="HH", N=200000, B=71),
        # The exact-MDL scoring with Metropolis-Hastings acceptance, the
        # option for users who want the standard objective.
        dict(name="exactmh-20k-HL", kind="exactmh", variant="HL", N=20000, B=32),
        # Many graphs in one call: N log-uniform on [1k, 50k], all variants.
        dict(name="batch-48", kind="batch", count=48, N_min=1000, N_max=50000),
        # Requests to a running server, all in flight together, in the
        # served mix of sizes (1k/5k/20k/50k at 0.4/0.3/0.2/0.1).
        dict(name="served-24", kind="served", count=24),
        # Refinement of given labels at a fixed block count: the nodal phase
        # alone, from host arrays.
        dict(name="sweeps-200k", kind="sweeps", variant="HH", N=200000, B=450, sweeps=5),
        # Scoring of a given partition by the standard description length.
        dict(name="mdl-200k", kind="mdl", variant="LH", N=199999, B=431, exact=1),
        # The objective of a blockmodel that a host program keeps in device
        # memory, written to device memory without allocation.
        dict(name="mdl-device-B350", kind="mdl_device", variant="HH", N=50000, B=350),
        # Device edge lists into a resident graph, and its CSR pair back on
        # the host (the load generator of the batched and served modes).
        dict(name="ingest-200k", kind="ingest", variant="HH", N=200000, B=71),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["partition", "partition", "partition", "resident", "exactmh", "batch",
                       "served", "sweeps", "mdl", "mdl_device", "ingest"])
    variant = rng.choice(sorted(VARIANTS))
    if kind == "batch":
        hi = _log_int(rng, 2000, 50000)
        return dict(kind=kind, count=rng.randint(2, 40), N_min=1000, N_max=hi)
    if kind == "served":
        return dict(kind=kind, count=rng.randint(2, 24))
    if kind == "exactmh":
        N = _log_int(rng, 1000, 20000)
        return dict(kind=kind, variant=variant, N=N, B=rng.randint(8, 40))
    N = _log_int(rng, 1000, 200000 if kind in ("sweeps", "mdl", "ingest") else 100000)
    if kind in ("partition", "resident"):
        c = dict(kind=kind, variant=variant, N=N, B=rng.randint(8, 71))
        if kind == "partition":
            c["weighted"] = rng.random() < 0.3
        return c
    if kind == "ingest":
        return dict(kind=kind, variant=variant, N=N, B=rng.randint(8, 71))
    B = _log_int(rng, 8, max(16, N // 4))
    if kind == "mdl_device":
        B = min(B, 65536)
    c = dict(kind=kind, variant=variant, N=N, B=B)
    if kind == "mdl":
        c["exact"] = rng.randint(0, 1)
    if kind == "sweeps":
        c["sweeps"] = rng.randint(1, 5)
    return c


# ------------------------------------------------------------------ inputs --
def _distinct(key):
    """The distinct values of key, ascending, and how often each occurs."""
    key = np.sort(key)
    at = np.flatnonzero(np.concatenate([[True], key[1:] != key[:-1]]))
    return key[at], np.diff(np.concatenate([at, [key.size]]))


def _edges(variant, N, B, seed, weighted=False):
    """(src, dst, w or None), source-major, without self loops or repeats."""
    p_in, alpha = VARIANTS[variant]
    rng = np.random.default_rng(seed)
    label = rng.choice(B, N, p=rng.dirichlet(np.full(B, alpha)))
    _, label = np.unique(label, return_inverse=True)  # no empty blocks
    nb = int(label.max()) + 1
    k = np.arange(5, 51)
    pk = k ** -2.5
    deg = rng.choice(k, N, p=pk / pk.sum())
    src = np.repeat(np.arange(N), deg)
    E = src.size
    own = label[src]
    other = (own + 1 + rng.integers(0, max(nb - 1, 1), E)) % nb
    blk = np.where(rng.random(E) < p_in, own, other)
    # destination within the block in proportion to degree
    order = np.argsort(label, kind="stable")
    cum = np.cumsum(deg[order]).astype(np.float64)
    size = np.bincount(label, minlength=nb)
    last = np.cumsum(size)
    hi = cum[last - 1]
    lo = hi - np.bincount(label, weights=deg, minlength=nb)
    x = lo[blk] + rng.random(E) * (hi - lo)[blk]
    at = np.minimum(np.searchsorted(cum, x, side="right"), last[blk] - 1)
    dst = order[at]
    key, _ = _distinct((src * np.int64(N) + dst)[src != dst])
    src, dst = (key // N).astype(np.int32), (key % N).astype(np.int32)
    w = rng.integers(1, 5, src.size).astype(np.uint32) if weighted else None
    return src, dst, w


def _graph(variant, N, B, seed, weighted=False):
    src, dst, w = _edges(variant, N, B, seed, weighted)
    return sbp.Graph.from_edges(N, src, dst, w)


def _labels(N, B, seed):
    """Labels in [0, B), block sizes uneven, no empty block."""
    rng = np.random.default_rng(seed + 1)
    p = rng.choice(B, N, p=rng.dirichlet(np.full(B, 2.0))).astype(np.int32)
    p[:B] = np.arange(B, dtype=np.int32)
    return p


def _cells(case, seed):
    """The blockmodel of a case's labels: rows, columns, counts (ascending),
    weighted block degrees, and the edge count."""
    N, B = case["N"], case["B"]
    src, dst, _ = _edges(case["variant"], N, B_PLANTED, seed)
    part = _labels(N, B, seed)
    key, cnt = _distinct(part[src].astype(np.int64) * B + part[dst])
    d_out = np.bincount(part[src], minlength=B)
    d_in = np.bincount(part[dst], minlength=B)
    return key // B, key % B, cnt, d_out, d_in, src.size


# planted blocks of the graphs that are scored under other labels
B_PLANTED = 71


def _many(case, seed):
    """(variant, N, B, seed) of each graph of a batched or served case: the
    same sizes for every seed, other graphs."""
    rng = np.random.default_rng(2)
    out = []
    for i in range(case["count"]):
        v = str(rng.choice(sorted(VARIANTS)))
        if case["kind"] == "batch":
            N = int(round(case["N_min"] * (case["N_max"] / case["N_min"]) ** rng.random()))
        else:
            N = int(rng.choice([1000, 5000, 20000, 50000], p=[0.4, 0.3, 0.2, 0.1]))
        out.append((v, N, int(round(2.6 * N ** 0.34)), seed * 1000 + i))
    return out


class _Server:
    """A running server that is closed with the state that holds it."""

    def __init__(self):
        self.s = sbp.Server()

    def __del__(self):
        self.s.close()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("batch", "served"):
        gs = [_graph(*spec) for spec in _many(case, seed)]
        st = dict(kind=kind, graphs=gs, seeds=[seed + i for i in range(len(gs))])
        if kind == "served":
            st["server"] = _Server()
        return st
    st = dict(kind=kind, seed=seed)
    if kind in ("partition", "exactmh"):
        st["g"] = _graph(case["variant"], case["N"], case["B"], seed, case.get("weighted", False))
    elif kind == "resident":
        st["g"] = _graph(case["variant"], case["N"], case["B"], seed)
        st["rg"] = sbp.ResidentGraph(st["g"])
    elif kind in ("sweeps", "mdl"):
        st["g"] = _graph(case["variant"], case["N"], B_PLANTED, seed)
        st["part"] = _labels(case["N"], case["B"], seed)
        st["B"] = case["B"]
        st["exact"] = case.get("exact", 0)
        st["sweeps"] = case.get("sweeps", 0)
    elif kind == "mdl_device":
        r, c, cnt, d_out, d_in, E = _cells(case, seed)
        ptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=case["B"]))])
        st["arrays"] = [torch.as_tensor(a.astype(np.int32)).cuda()
                        for a in (ptr, c, cnt, d_out, d_in)]
        st["out"] = torch.zeros(2, dtype=torch.float64, device="cuda")
        st.update(N=case["N"], E=E, B=case["B"])
    elif kind == "ingest":
        src, dst, _ = _edges(case["variant"], case["N"], case["B"], seed)
        # the same number of edges for every seed, in no order
        E = min(8 * case["N"], src.size)
        keep = np.random.default_rng(seed + 3).permutation(src.size)[:E]
        src, dst = src[keep], dst[keep]
        st["src"], st["dst"] = torch.as_tensor(src).cuda(), torch.as_tensor(dst).cuda()
        st["N"] = case["N"]
    return st


# --------------------------------------------------------------------- run --
def run(state):
    kind = state["kind"]
    if kind in ("partition", "exactmh"):
        opt = dict(exact=1, mh=1) if kind == "exactmh" else {}
        rep = sbp.partition(state["g"], seed=state["seed"], **opt)
        return dict(labels=state["g"].partitions, B=rep["B"], S=rep["S"])
    if kind == "resident":
        lab, rep = state["rg"].partition(seed=state["seed"])
        return dict(labels=lab, B=rep["B"], S=rep["S"])
    if kind == "batch":
        labs, reps, _ = sbp.partition_batch(state["graphs"], seeds=state["seeds"])
        return _pack(labs, reps)
    if kind == "served":
        srv = state["server"].s
        ids = [srv.submit(g, seed=k) for g, k in zip(state["graphs"], state["seeds"])]
        res = [srv.poll(j) for j in ids]
        return _pack([r[0] for r in res], [r[1] for r in res])
    if kind == "sweeps":
        return list(sbp.nodal_sweeps(state["g"], state["part"], state["B"], state["seed"], 1,
                                     sweeps=state["sweeps"]))
    if kind == "mdl":
        return list(sbp.mdl(state["g"], state["part"], state["B"], exact=state["exact"]))
    if kind == "mdl_device":
        out = state["out"]
        sbp.mdl_device_static(state["N"], state["E"], state["B"],
                              *[a.data_ptr() for a in state["arrays"]], out.data_ptr(),
                              out.data_ptr() + 8,
                              stream=torch.cuda.current_stream().cuda_stream)
        return out
    dg = sbp.DeviceGraph.from_edges(state["N"], state["src"].data_ptr(), state["dst"].data_ptr(),
                                    state["src"].numel())
    g = dg.download()
    dg.close()
    return [g.out_ptr, g.out_idx, g.out_w, g.in_ptr, g.in_idx, g.in_w, g.deg_out, g.deg_in]


def _pack(labs, reps):
    return dict(labels=np.concatenate(labs), B=np.array([r["B"] for r in reps]),
                S=np.array([r["S"] for r in reps]))


# -------------------------------------------------------------------- work --
def work(case):
    """Each input read once and each output written once; operations of one
    evaluation of the objective over the edges (2 a graph entry) for whole
    partitions, which cannot end without one."""
    kind = case["kind"]
    mean_deg = 9.78  # of the power law, less its repeated edges

    def graph_bytes(N, E):  # both CSR directions with weights, both degrees
        return 16.0 * E + 16.0 * N

    if kind in ("batch", "served"):
        if kind == "batch":
            ratio = case["N_max"] / case["N_min"]
            mean_N = case["N_min"] * (ratio - 1.0) / np.log(ratio) if ratio > 1 else case["N_min"]
        else:
            mean_N = 0.4 * 1000 + 0.3 * 5000 + 0.2 * 20000 + 0.1 * 50000
        N = case["count"] * float(mean_N)
        E = mean_deg * N
        return dict(bytes=graph_bytes(N, E) + 4.0 * N, flops=4.0 * E)
    N, B = float(case["N"]), float(case["B"])
    E = mean_deg * N
    nnz = min(E, B * B)
    if kind in ("partition", "resident", "exactmh"):
        return dict(bytes=graph_bytes(N, E) + 4.0 * N, flops=4.0 * E)
    if kind == "sweeps":
        n = case["sweeps"]
        return dict(bytes=graph_bytes(N, E) + 8.0 * N + 32.0 * n, flops=4.0 * E * n)
    if kind == "mdl":
        return dict(bytes=graph_bytes(N, E) + 4.0 * N, flops=2.0 * E + 4.0 * nnz)
    if kind == "mdl_device":
        return dict(bytes=8.0 * nnz + 12.0 * B, flops=4.0 * nnz)
    E = 8.0 * N
    return dict(bytes=8.0 * E + graph_bytes(N, E), flops=2.0 * E)


# ------------------------------------------------------------------- exact --
def exact(case, seed):
    kind = case["kind"]
    if kind not in ("mdl", "mdl_device"):
        return None
    _, _, cnt, d_out, d_in, E = _cells(case, seed)
    N, B = float(case["N"]), float(case["B"])

    def xlx(a):
        a = a[a > 0].astype(np.longdouble)
        return (a * np.log2(a)).sum()

    data = xlx(cnt) - xlx(d_out) - xlx(d_in)
    x = np.longdouble(B) * B / E
    if case.get("exact", 0):
        model = (E * ((1 + x) * np.log1p(x) - x * np.log(x)) + N * np.log(np.longdouble(B))) \
            / np.log(np.longdouble(2))
    else:
        model = E * (1 + x) * np.log1p(x) - x * np.log(x) + N * np.log(np.longdouble(B))
    out = [float(model - data), float(data)]
    return out if kind == "mdl" else torch.tensor(out, dtype=torch.float64)
