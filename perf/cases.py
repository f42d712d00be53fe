"""Timed cases of the library's main path: loading a graph (CPBT, CSR, CSC) and running the
toolkits, the batched operators and the differentiable PageRank on it, through `endgraph_gb300.Graph`.

A case names what a program does (`kind`) and its sizes.  Graphs are R-MAT (a=0.57, b=0.19, c=0.19,
d=0.05) with randomly permuted ids, as in bench.py, generated here with torch so that `exact` can
rebuild them.  Inputs and outputs are CUDA tensors, except where a program's data is on the host.

  load_pagerank  load_directed of device records, then PageRank: the reference's pagerank toolkit
  load_bfs       load_directed of device records, then one BFS: preprocessing at scale
  load_cc        load_undirected_from_directed, then CC: the reference's cc toolkit
  load_host      load_directed of records in pinned host memory: ingest
  pagerank, bfs, sssp, msbfs   one call on a graph that is already built
  graph_batch    many uneven small graphs: one load, 64-root BFS and 64-source SSSP per graph
  ppr_step       a training step on edge weights: personalised PageRank, L2 loss, adjoint
"""
import ctypes
import math

import numpy as np
import torch

import endgraph_gb300 as eg

A, B, C = 0.57, 0.19, 0.19
DAMPING = 0.85
TELEPORT = 0.15
UNREACHED = 1e9  # distance of an unreached vertex
CHUNK = 1 << 26  # edges generated or reduced together


# ---- cases --------------------------------------------------------------------------------------
def listed():
    return [
        # the plain configuration: 2^16 vertices, edge factor 16, 20 iterations, build included;
        # all of it is launches and latency
        dict(name="load_pagerank_2p16", kind="load_pagerank", V=1 << 16, E=1 << 20, iterations=20, weighted=False),
        # a service answering BFS queries on a small graph of an odd size
        dict(name="bfs_100k", kind="bfs", V=100_003, E=1_000_003),
        # single-source shortest paths on a small weighted graph: many short levels
        dict(name="sssp_50k", kind="sssp", V=50_021, E=800_017),
        # preprocessing at scale, then the first traversal of the new graph
        dict(name="load_bfs_2p25", kind="load_bfs", V=1 << 25, E=1 << 29, weighted=False),
        # analytics at scale on a built graph
        dict(name="pagerank_2p25", kind="pagerank", V=1 << 25, E=1 << 29, iterations=20),
        dict(name="bfs_2p25", kind="bfs", V=1 << 25, E=1 << 29),
        dict(name="sssp_2p22", kind="sssp", V=1 << 22, E=1 << 26),
        # a power-law graph a quarter the size of the 41,652,230-vertex one, symmetrised for CC
        dict(name="load_cc_10m", kind="load_cc", V=10_413_058, E=367_091_295, weighted=False),
        # 64 BFS roots in one bit-parallel traversal
        dict(name="msbfs_2p23", kind="msbfs", V=1 << 23, E=1 << 27, roots=64),
        # independent graphs of 1k to 500k vertices, edge factor 4 to 32, weights in [0, 1)
        dict(name="graph_batch_64", kind="graph_batch", graphs=64, roots=64, layout=1),
        # learnable edge weights: forward, loss and adjoint of 50 unrolled iterations, 64 seeds
        dict(name="ppr_step_1m", kind="ppr_step", V=1_000_003, E=16_000_037, seeds=64, iterations=50),
        # ingest of host records: the copy and the build behind it
        dict(name="load_host_2p24", kind="load_host", V=1 << 24, E=1 << 28, weighted=False),
    ]


def draw(rng):
    def size(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    def graph(vlo, vhi, emax):
        V = size(vlo, vhi)
        if rng.random() < 0.4:  # powers of two are as common as odd sizes
            V = 1 << max(1, round(math.log2(V)))
        return V, min(emax, max(1, int(V * rng.uniform(4, 32))))

    kind = rng.choice(["load_pagerank", "load_bfs", "load_cc", "load_host", "pagerank", "bfs", "bfs", "sssp", "sssp",
                       "msbfs", "graph_batch", "ppr_step"])
    if kind == "load_pagerank":
        V, E = graph(1 << 12, 1 << 24, 1 << 28)
        return dict(kind=kind, V=V, E=E, iterations=rng.randint(5, 30), weighted=rng.random() < 0.3)
    if kind == "load_bfs":
        V, E = graph(1 << 14, 1 << 25, 1 << 28)
        return dict(kind=kind, V=V, E=E, weighted=rng.random() < 0.3)
    if kind == "load_cc":
        V, E = graph(1 << 12, 1 << 23, 1 << 27)
        return dict(kind=kind, V=V, E=E, weighted=rng.random() < 0.2)
    if kind == "load_host":
        V, E = graph(1 << 16, 1 << 24, 1 << 27)
        return dict(kind=kind, V=V, E=E, weighted=rng.random() < 0.3)
    if kind == "pagerank":
        V, E = graph(1 << 12, 1 << 25, 1 << 28)
        return dict(kind=kind, V=V, E=E, iterations=rng.randint(5, 30))
    if kind == "bfs":
        V, E = graph(1 << 10, 1 << 25, 1 << 28)
        return dict(kind=kind, V=V, E=E)
    if kind == "sssp":
        V, E = graph(1 << 10, 1 << 22, 1 << 26)
        return dict(kind=kind, V=V, E=E)
    if kind == "msbfs":
        V, E = graph(1 << 14, 1 << 23, 1 << 27)
        return dict(kind=kind, V=V, E=E, roots=rng.choice([rng.randint(1, 63), 64]))
    if kind == "graph_batch":
        return dict(kind=kind, graphs=rng.randint(2, 80), roots=rng.choice([rng.randint(1, 63), 64]),
                    layout=rng.randint(2, 1 << 20))
    V, E = graph(1 << 12, 1 << 20, 1 << 24)
    return dict(kind=kind, V=V, E=E, seeds=rng.choice([1, rng.randint(2, 63), 64]), iterations=rng.randint(8, 50))


# ---- inputs -------------------------------------------------------------------------------------
def generator(seed):
    return torch.Generator("cuda").manual_seed(seed)


def rmat(gen, V, E, records, permute=True):
    """R-MAT pairs into records[:, 0] and records[:, 1] (int32 CUDA tensor), ids permuted."""
    scale = max(1, (V - 1).bit_length())
    perm = torch.randperm(V, generator=gen, device="cuda", dtype=torch.int32) if permute else None
    for e0 in range(0, E, CHUNK):
        n = min(CHUNK, E - e0)
        src = torch.zeros(n, dtype=torch.int32, device="cuda")
        dst = torch.zeros(n, dtype=torch.int32, device="cuda")
        for _ in range(scale):
            r = torch.rand(n, generator=gen, device="cuda")
            s = r >= A + B
            d = ((r >= A) & ~s) | (r >= A + B + C)
            src.mul_(2).add_(s)
            dst.mul_(2).add_(d)
        for k, x in ((0, src), (1, dst)):
            if V != 1 << scale:  # fold the 2^scale ids onto V
                x = ((x.to(torch.int64) * V) >> scale).to(torch.int32)
            records[e0:e0 + n, k] = perm[x] if permute else x


def records_of(case, seed, weighted):
    """The case's edge list: (E, 2) int32 {src, dst}, or (E, 3) with a float weight in [0, 1)."""
    gen = generator(seed)
    rec = torch.empty((case["E"], 3 if weighted else 2), dtype=torch.int32, device="cuda")
    rmat(gen, case["V"], case["E"], rec)
    if weighted:
        rec[:, 2] = torch.rand(case["E"], generator=gen, device="cuda").view(torch.int32)
    return rec, gen


def some_sources(rec, gen, n):
    """n sources of random edges: vertices with out-edges."""
    at = torch.randint(0, rec.shape[0], (n,), generator=gen, device="cuda")
    return rec[at, 0].cpu().numpy().astype(np.uint32)


def batch_shapes(case):
    """Vertex and edge counts of a graph batch: 1k to 500k vertices, 4 to 32 edges each."""
    rng = np.random.default_rng(case["layout"])
    V = np.exp(rng.uniform(np.log(1_000), np.log(500_000), case["graphs"])).astype(np.uint32)
    E = (V * rng.uniform(4, 32, case["graphs"])).astype(np.uint64)
    return V, E


def prepare(case, seed):
    kind = case["kind"]
    st = dict(kind=kind, graph=eg.Graph(eta=1, max_iterations=20), **{k: v for k, v in case.items() if k != "kind"})
    g = st["graph"]
    if kind == "graph_batch":
        nv, ne = batch_shapes(case)
        gen = generator(seed)
        off = np.concatenate([[0], np.cumsum(ne)]).astype(np.uint64)
        rec = torch.empty((int(off[-1]), 3), dtype=torch.int32, device="cuda")
        for v, a, z in zip(nv, off[:-1], off[1:]):
            rmat(gen, int(v), int(z - a), rec[int(a):int(z)], permute=False)
        rec[:, 2] = torch.rand(len(rec), generator=gen, device="cuda").view(torch.int32)
        rng = np.random.default_rng(seed + 1)
        roots = np.concatenate([rng.integers(0, v, case["roots"]) for v in nv]).astype(np.uint32)
        total = int(nv.astype(np.int64).sum())
        st.update(records=rec, graph_edges=off, graph_vertices=nv, root_list=roots,
                  levels=torch.empty((total, 64), dtype=torch.uint8, device="cuda"),
                  dist=torch.empty((total, 64), dtype=torch.float32, device="cuda"))
        return st
    V, E = case["V"], case["E"]
    weighted = case.get("weighted", False) or kind == "sssp"
    rec, gen = records_of(case, seed, weighted)
    st["records"] = rec
    if kind in ("load_bfs", "bfs", "sssp"):
        st["root"] = int(some_sources(rec, gen, 1)[0])
    if kind in ("load_bfs", "load_cc", "load_host"):  # cvert and cidx: one entry per list and a sentinel
        st["index"] = {k: torch.zeros(n, dtype=t, device="cuda") for k, n, t in (
            ("csr_off", V + 1, torch.int64), ("bitmap", V // 64 + 1, torch.int64), ("csc_off", V + 1, torch.int64),
            ("cvert", V + 1, torch.int32), ("cidx", V + 1, torch.int64))}
    if kind in ("load_bfs", "bfs"):
        st["level"] = torch.empty(V, dtype=torch.int32, device="cuda")
        st["parent"] = torch.empty(V, dtype=torch.int32, device="cuda")
    elif kind == "load_cc":
        st["label"] = torch.empty(V, dtype=torch.int32, device="cuda")
    elif kind in ("load_pagerank", "pagerank"):
        st["rank"] = torch.empty(V, dtype=torch.float32, device="cuda")
    elif kind == "sssp":
        st["dist"] = torch.empty(V, dtype=torch.float32, device="cuda")
    elif kind == "msbfs":
        st["root_list"] = some_sources(rec, gen, case["roots"])
        st["levels"] = torch.empty((case["roots"], V), dtype=torch.uint8, device="cuda")
    elif kind == "load_host":
        st["records"] = torch.empty(rec.shape, dtype=rec.dtype, pin_memory=True)
        st["records"].copy_(rec)
    elif kind == "ppr_step":
        st["seed_list"] = some_sources(rec, gen, case["seeds"])
        st["weights"] = torch.rand(E, generator=gen, device="cuda") + 0.5
        st["target"] = torch.rand((case["seeds"], V), generator=gen, device="cuda") / V
        st["x"] = torch.empty((case["seeds"], V), dtype=torch.float32, device="cuda")
        st["grad"] = torch.empty(E, dtype=torch.float32, device="cuda")
        g.load_directed_with_ids(rec, V)
        del st["records"]
    if kind in ("pagerank", "bfs", "sssp", "msbfs"):  # a program keeps the built graph
        g.load_directed(rec, V)
        del st["records"]
    return st


# ---- one pass -----------------------------------------------------------------------------------
def index_arrays(st):
    """The index arrays of the built CSR and CSC.  Neighbours inside a list are in no set order, so
    the adjacency shows in what is computed from it."""
    lib, g = eg.load_library(), st["graph"]
    p = {k: ctypes.c_void_p(x.data_ptr()) for k, x in st["index"].items()}
    for status in (lib.eg_copy_csr(g.h, p["csr_off"], None, None, p["bitmap"], eg.EG_DEVICE),
                   lib.eg_copy_csc(g.h, p["csc_off"], None, None, p["cvert"], p["cidx"], eg.EG_DEVICE)):
        if status:
            raise RuntimeError(lib.eg_last_error().decode())
    return st["index"]


def run(st):
    g, kind = st["graph"], st["kind"]
    if kind == "load_pagerank":
        g.load_directed(st["records"], st["V"])
        return dict(rank=g.pagerank(st["iterations"], DAMPING, out=st["rank"]))
    if kind == "load_bfs":
        g.load_directed(st["records"], st["V"])
        # any in-neighbour one level up may be a vertex's parent: the parents differ from run to run
        level, _ = g.bfs(st["root"], level=st["level"], parent=st["parent"])
        return dict(level=level, **index_arrays(st))
    if kind == "load_cc":
        g.load_undirected_from_directed(st["records"], st["V"])
        return dict(label=g.cc(label=st["label"]), **index_arrays(st))
    if kind == "load_host":
        g.load_directed(st["records"], st["V"])
        return index_arrays(st)
    if kind == "pagerank":
        return g.pagerank(st["iterations"], DAMPING, out=st["rank"])
    if kind == "bfs":
        return g.bfs(st["root"], level=st["level"], parent=st["parent"])[0]
    if kind == "sssp":
        return g.sssp(st["root"], dist=st["dist"])
    if kind == "msbfs":
        levels, edges = g.msbfs(st["root_list"], levels=st["levels"])
        return dict(levels=levels, edges=edges)
    if kind == "graph_batch":
        g.load_graph_batch(st["records"], st["graph_edges"], st["graph_vertices"])
        levels, edges = g.msbfs_graphs(st["root_list"], st["roots"], levels=st["levels"])
        dist = g.sssp_graphs(st["root_list"], st["roots"], dist=st["dist"])
        return dict(levels=levels[:, :st["roots"]], edges=edges, dist=dist[:, :st["roots"]])
    x = g.ppr(st["weights"], st["seed_list"], TELEPORT, st["iterations"], out=st["x"])
    grad = g.ppr_backward(st["weights"], st["seed_list"], x - st["target"], TELEPORT, st["iterations"],
                          dl_dw=st["grad"])
    return dict(x=x, grad=grad)


# ---- the work of a pass -------------------------------------------------------------------------
def work(case):
    """Bytes: inputs read once, outputs written once; an operator on a built graph reads the lists
    that it has to (4 bytes an edge, 8 with a weight) once per iteration, or once where it could."""
    kind = case["kind"]
    if kind == "graph_batch":
        nv, ne = batch_shapes(case)
        V, E = int(nv.astype(np.int64).sum()), int(ne.sum())
        return dict(bytes=12 * E + 16 * E + 32 * V + 4 * E + 8 * E + V * case["roots"] * 5, flops=E * case["roots"])
    V, E = case["V"], case["E"]
    rec = 12 if case.get("weighted", False) else 8
    load = rec * E + 2 * (rec - 4) * E + 32 * V  # records in; two adjacencies, offsets, degrees, index out
    if kind == "load_pagerank":
        return dict(bytes=load + case["iterations"] * (4 * E + 16 * V), flops=case["iterations"] * E)
    if kind == "load_bfs":
        return dict(bytes=load + 4 * E + 8 * V, flops=0)
    if kind == "load_cc":
        return dict(bytes=rec * E + 4 * (rec - 4) * E + 32 * V + 8 * E + 4 * V, flops=0)
    if kind == "load_host":
        return dict(bytes=load, flops=0)
    if kind == "pagerank":
        return dict(bytes=case["iterations"] * (4 * E + 16 * V), flops=case["iterations"] * E)
    if kind == "bfs":
        return dict(bytes=4 * E + 16 * V, flops=0)
    if kind == "sssp":
        return dict(bytes=8 * E + 12 * V, flops=E)
    if kind == "msbfs":
        return dict(bytes=4 * E + 8 * V + V * case["roots"], flops=0)
    n, K = case["seeds"], case["iterations"]
    # forward and adjoint each read ids, weights and one row in and one row out per iteration, the
    # adjoint the forward's rows too; the gradient is accumulated over the iterations
    return dict(bytes=K * (2 * 8 * E + 5 * 4 * n * V) + 12 * E + 8 * n * V, flops=K * 6 * n * E)


# ---- 64-bit values ------------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind in ("load_pagerank", "pagerank"):
        rec, _ = records_of(case, seed, case.get("weighted", False))
        x = exact_pagerank(rec, case["V"], case["iterations"])
        return dict(rank=x) if kind == "load_pagerank" else x
    if kind == "sssp":
        rec, gen = records_of(case, seed, True)
        return exact_sssp(rec, case["V"], int(some_sources(rec, gen, 1)[0]))
    if kind == "ppr_step":
        return exact_ppr(case, seed)
    return None  # whole numbers; a graph batch's distances would take minutes


def exact_pagerank(rec, V, iterations):
    E = rec.shape[0]
    deg = torch.zeros(V, dtype=torch.float64, device="cuda")
    for e0 in range(0, E, CHUNK):
        s = rec[e0:e0 + CHUNK, 0]
        deg.index_add_(0, s, torch.ones(len(s), dtype=torch.float64, device="cuda"))
    deg.clamp_(min=1)
    curr = 1 / deg
    for it in range(iterations):
        nxt = torch.zeros(V, dtype=torch.float64, device="cuda")
        for e0 in range(0, E, CHUNK):
            r = rec[e0:e0 + CHUNK]
            nxt.index_add_(0, r[:, 1], curr[r[:, 0]])
        curr = (1 - DAMPING) + DAMPING * nxt
        if it < iterations - 1:
            curr = curr / deg
    return curr


def exact_sssp(rec, V, root):
    src, dst = rec[:, 0].to(torch.int64), rec[:, 1].to(torch.int64)
    w = rec[:, 2].contiguous().view(torch.float32).to(torch.float64)
    dist = torch.full((V,), UNREACHED, dtype=torch.float64, device="cuda")
    dist[root] = 0
    while True:
        new = dist.scatter_reduce(0, dst, dist[src] + w, "amin")
        if torch.equal(new, dist):
            return dist
        dist = new


def exact_ppr(case, seed):
    V, E, n, K = case["V"], case["E"], case["seeds"], case["iterations"]
    rec, gen = records_of(case, seed, False)
    seeds = torch.from_numpy(some_sources(rec, gen, n).astype(np.int64)).cuda()
    w = (torch.rand(E, generator=gen, device="cuda") + 0.5).double()
    target = (torch.rand((n, V), generator=gen, device="cuda") / V).double()
    src, dst = rec[:, 0].to(torch.int64), rec[:, 1].to(torch.int64)
    total = torch.zeros(V, dtype=torch.float64, device="cuda").index_add_(0, src, w)
    a = w / total[src]
    # A^T by destination for the forward sweeps, A by source for the adjoint's
    by_dst, by_src = torch.argsort(dst), torch.argsort(src)

    def sweep(order, rows, cols):
        off = torch.zeros(V + 1, dtype=torch.int64, device="cuda")
        off[1:] = torch.cumsum(torch.bincount(rows, minlength=V), 0)
        m = torch.sparse_csr_tensor(off, cols[order], a[order], (V, V))
        return lambda x: m @ x

    forward, backward = sweep(by_dst, dst, src), sweep(by_src, src, dst)
    cols = torch.arange(n, device="cuda")
    x = torch.zeros((V, n), dtype=torch.float64, device="cuda")
    x[seeds, cols] = 1
    kept = [x]
    for _ in range(K):
        x = (1 - TELEPORT) * forward(x)
        x[seeds, cols] += TELEPORT
        kept.append(x)
    out = kept[K].t().contiguous()
    lam = (out.float().double() - target).t().contiguous()  # the loss gradient of a float32 x
    ga = torch.zeros(E, dtype=torch.float64, device="cuda")
    step = max(1, CHUNK // n)
    for k in range(K - 1, -1, -1):
        for e0 in range(0, E, step):
            s, d = src[e0:e0 + step], dst[e0:e0 + step]
            ga[e0:e0 + step] += (1 - TELEPORT) * (kept[k][s] * lam[d]).sum(1)
        lam = (1 - TELEPORT) * backward(lam)
    dot = torch.zeros(V, dtype=torch.float64, device="cuda").index_add_(0, src, a * ga)
    return dict(x=out, grad=(ga - dot[src]) / total[src])
