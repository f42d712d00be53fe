"""GPU: the 64-column row engine (batched SSSP, personalised PageRank and its adjoint) on lists whose
lengths sit at the edges of its blocking: rows gathered together, edges per warp step, edges per
task, and lists cut into several tasks."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 40, 63, 64, 65, 96, 511, 512, 513, 1024, 1025, 3000]


def _fans(seed, V=4096):
    """Destination i < len(LENGTHS) has LENGTHS[i] in-edges and source 1000 + i as many out-edges;
    a random sparse graph connects the rest.  Vertices from 4000 on have no edges at all."""
    rng = np.random.default_rng(seed)
    src, dst = [], []
    for i, n in enumerate(LENGTHS):
        src += [rng.integers(100, 4000, n), np.full(n, 1000 + i)]
        dst += [np.full(n, i), rng.integers(0, 4000, n)]
    src.append(rng.integers(0, 4000, 6000))
    dst.append(rng.integers(0, 4000, 6000))
    src, dst = (np.concatenate(x).astype(np.uint32) for x in (src, dst))
    p = rng.permutation(len(src))
    return src[p], dst[p], V


@pytest.mark.parametrize("P", [1, 2])
@pytest.mark.parametrize("n", [1, 5, 64])
def test_sssp_batch_list_lengths(eg_lib, P, n):
    import endgraph_gb300 as eg
    src, dst, V = _fans(n)
    w = np.random.default_rng(n + 1).random(len(src)).astype(np.float32)
    csr = oracle.build_csr(src, dst, w, V, np.array([0, V], np.uint32))
    sources = np.concatenate([[1000 + len(LENGTHS) - 1, 4050], src[:62]]).astype(np.uint32)[:n]
    with eg.Graph(partitions=P) as g:
        g.load_directed(eg.pack_edges(src, dst, w), V)
        dist = g.sssp_batch(sources)
    for s in range(n):
        ref = oracle.sssp(csr["off"][0], csr["adj"], csr["w"], V, int(sources[s]))
        assert np.array_equal(dist[s].view(np.uint32), ref.view(np.uint32)), s


def _ppr64(src, dst, w, V, seeds, alpha, K):
    """K unrolled iterations in FP64, differentiable in w (torch, CPU)."""
    import torch
    s, d = torch.from_numpy(src.astype(np.int64)), torch.from_numpy(dst.astype(np.int64))
    a = w / torch.zeros(V, dtype=torch.float64).index_add(0, s, w)[s]
    e = torch.zeros((V, len(seeds)), dtype=torch.float64)
    e[torch.from_numpy(seeds.astype(np.int64)), torch.arange(len(seeds))] = 1.0
    x = e
    for _ in range(K):
        x = alpha * e + (1 - alpha) * torch.zeros_like(x).index_add(0, d, a[:, None] * x[s])
    return x.t()


@pytest.mark.parametrize("n,K", [(2, 1), (2, 2), (7, 5), (64, 9)])
def test_ppr_and_adjoint_list_lengths(eg_lib, n, K):
    """Seeds include a vertex without in-edges, one without any edges, and the longest lists; the
    tolerances are those of the other FP64 comparisons of these operators: 1e-6 (relative L1) for
    the scores, 1e-4 (relative L2) for the gradient."""
    import torch

    import endgraph_gb300 as eg
    src, dst, V = _fans(n + K)
    no_in = np.setdiff1d(src, dst)
    assert len(no_in)
    seeds = np.concatenate([[no_in[0], 4050, len(LENGTHS) - 1, 1000 + len(LENGTHS) - 1], src[:60]]).astype(np.uint32)[:n]
    rng = np.random.default_rng(K)
    w = rng.uniform(0.5, 1.5, len(src)).astype(np.float32)
    tgt = rng.random((n, V)).astype(np.float32) / V
    alpha = 0.15
    with eg.Graph() as g:
        g.load_directed_with_ids(eg.pack_edges(src, dst), V)
        for _ in range(2):  # a second call reuses the buffers
            x = g.ppr(w, seeds, alpha, K)
            dw = g.ppr_backward(w, seeds, 2 * (x - tgt), alpha, K)
        other = np.roll(seeds, 1) if n > 2 else seeds[::-1].copy()  # other seeds on the same buffers
        x2 = g.ppr(w, other, alpha, K)
        dw2 = g.ppr_backward(w, other, 2 * (x2 - tgt), alpha, K)
    for sd, xg, dg in ((seeds, x, dw), (other, x2, dw2)):
        wt = torch.tensor(w, dtype=torch.float64, requires_grad=True)
        ref = _ppr64(src, dst, wt, V, sd, alpha, K)
        ref.backward(torch.from_numpy((2 * (xg - tgt)).astype(np.float64)))
        r = ref.detach().numpy()
        assert np.abs(xg - r).sum() / np.abs(r).sum() <= 1e-6
        gr = wt.grad.numpy()
        assert np.linalg.norm(dg - gr) / np.linalg.norm(gr) <= 1e-4


def test_ppr_adjoint_checkpoint_stride(eg_lib):
    """Iterates that do not fit an eighth of the GPU's memory (80 of 512 MiB) are kept at a stride and
    recomputed in between."""
    import torch

    import endgraph_gb300 as eg
    V, E, n, K, alpha = 1 << 21, 1 << 20, 2, 80, 0.15
    gen = torch.Generator("cuda").manual_seed(3)
    # edges among the first 2^17 vertices only: in-lists and iterates that differ from one step to the next
    rec = torch.randint(0, 1 << 17, (E, 2), generator=gen, device="cuda", dtype=torch.int32)
    seeds = rec[:n, 0].cpu().numpy().astype(np.uint32)
    w = torch.rand(E, generator=gen, device="cuda") + 0.5
    dl = torch.rand((n, V), generator=gen, device="cuda")
    with eg.Graph() as g:
        g.load_directed_with_ids(rec, V)
        dw = torch.empty(E, device="cuda")
        g.ppr_backward(w, seeds, dl, alpha, K, dl_dw=dw)
    s, d, wt = rec[:, 0].long(), rec[:, 1].long(), w.double()
    tot = torch.zeros(V, dtype=torch.float64, device="cuda").index_add(0, s, wt)
    a = wt / tot[s]
    e = torch.zeros((V, n), dtype=torch.float64, device="cuda")
    e[torch.from_numpy(seeds.astype(np.int64)).cuda(), torch.arange(n, device="cuda")] = 1.0
    xs = [e]
    for _ in range(K - 1):
        xs.append(alpha * e + (1 - alpha) * torch.zeros_like(e).index_add(0, d, a[:, None] * xs[-1][s]))
    lam = dl.double().t().contiguous()
    ga = torch.zeros(E, dtype=torch.float64, device="cuda")
    for k in range(K - 1, -1, -1):
        ga += (1 - alpha) * (xs[k][s] * lam[d]).sum(1)
        lam = (1 - alpha) * torch.zeros_like(lam).index_add(0, s, a[:, None] * lam[d])
    dot = torch.zeros(V, dtype=torch.float64, device="cuda").index_add(0, s, a * ga)
    ref = (ga - dot[s]) / tot[s]
    assert float((dw.double() - ref).norm() / ref.norm()) <= 1e-4


@pytest.mark.parametrize("V,E,longest", [(50, 1, 1), (3000, 31, 1), (40_000, 70_001, 1), (3_000_000, 2_900_003, 2),
                                         (1_500_000, 4_000_037, 700)])
def test_ppr_walk_over_lists(eg_lib, V, E, longest):
    """Batches from one edge to a full one, with up to a few hundred lists of one or two edges in each (task
    records and source rows come in groups of 8 and 32), and with lists longer than a batch.  Seeds
    repeat and include vertices with and without in-edges."""
    import torch

    import endgraph_gb300 as eg
    K, alpha, n = 4, 0.15, 5
    gen = torch.Generator("cuda").manual_seed(V)
    if longest == 1:      # a matching: every list has one edge
        src, dst = torch.randperm(V, generator=gen, device="cuda")[:E], torch.randperm(V, generator=gen, device="cuda")[:E]
        if E > V:
            src, dst = torch.cat([src, src[: E - V]]), torch.cat([dst, dst[: E - V].flip(0)])
    elif longest == 2:
        src, dst = (torch.randperm(V, generator=gen, device="cuda")[torch.arange(E, device="cuda") // 2] for _ in range(2))
        dst = dst[torch.randperm(E, generator=gen, device="cuda")]
    else:
        src, dst = (torch.randint(0, V, (E,), generator=gen, device="cuda") for _ in range(2))
        src[: 700 * 30] = torch.arange(30, device="cuda").repeat(700)
        dst[E - 700 * 30:] = torch.arange(40, 70, device="cuda").repeat(700)
    src, dst = src[:E], dst[:E]
    E = len(src)
    rec = torch.stack([src, dst], 1).to(torch.int32).contiguous()
    seeds = torch.stack([src[0], dst[0], dst[-1], dst[0], torch.tensor(V - 1, device="cuda")])
    w = torch.rand(E, generator=gen, device="cuda") + 0.5
    dl = torch.rand((n, V), generator=gen, device="cuda")
    with eg.Graph() as g:
        g.load_directed_with_ids(rec, V)
        x = torch.empty((n, V), device="cuda")
        dw = torch.empty(E, device="cuda")
        sd = seeds.cpu().numpy().astype(np.uint32)
        g.ppr(w, sd, alpha, K, out=x)
        g.ppr_backward(w, sd, dl, alpha, K, dl_dw=dw)
    s, d, wt = src.long(), dst.long(), w.double()
    tot = torch.zeros(V, dtype=torch.float64, device="cuda").index_add(0, s, wt)
    a = wt / tot[s]
    e = torch.zeros((V, n), dtype=torch.float64, device="cuda")
    e[seeds.long(), torch.arange(n, device="cuda")] = 1.0
    xs = [e]
    for _ in range(K):
        xs.append(alpha * e + (1 - alpha) * torch.zeros_like(e).index_add(0, d, a[:, None] * xs[-1][s]))
    lam = dl.double().t().contiguous()
    ga = torch.zeros(E, dtype=torch.float64, device="cuda")
    for k in range(K - 1, -1, -1):
        ga += (1 - alpha) * (xs[k][s] * lam[d]).sum(1)
        lam = (1 - alpha) * torch.zeros_like(lam).index_add(0, s, a[:, None] * lam[d])
    dot = torch.zeros(V, dtype=torch.float64, device="cuda").index_add(0, s, a * ga)
    ref = (ga - dot[s]) / tot[s]
    assert float((x.double() - xs[K].t()).abs().sum() / xs[K].abs().sum()) <= 1e-6
    # lists of one edge have no gradient: what is left are the roundings of terms of size |gA| / s
    assert float((dw.double() - ref).norm()) <= 1e-4 * float(ref.norm()) + 1e-6 * float((ga / tot[s]).norm())


@pytest.mark.parametrize("V,E,shape", [(40, 1, "one"), (5000, 5000, "one"), (3_000_000, 2_950_003, "two"),
                                       (200_000, 3_000_001, "hubs")])
def test_sssp_batch_walk_over_lists(eg_lib, V, E, shape):
    """Batches of up to 512 lists, of which a few, all or none have a changed source in a sweep; chains, so
    that a handful of sources changes at a time; lists longer than a batch between short ones."""
    import endgraph_gb300 as eg
    rng = np.random.default_rng(V)
    perm = rng.permutation(V)
    if shape == "one":      # a cycle: every list has one source
        src, dst = perm[:E], np.roll(perm, 1)[:E]
    elif shape == "two":    # up to two sources per list, a long chain among them
        src, dst = perm[np.arange(E) // 2 % V], perm[(np.arange(E) + 1) % V]
        src[:300], dst[:300] = perm[:300], perm[1:301]
    else:
        src, dst = rng.integers(0, V, E), rng.integers(0, V, E)
        dst[: 40 * 1500] = np.repeat(np.arange(40) * 7, 1500)
    src, dst = src.astype(np.uint32), dst.astype(np.uint32)
    w = rng.random(E).astype(np.float32)
    csr = oracle.build_csr(src, dst, w, V, np.array([0, V], np.uint32))
    sources = np.array([src[0], src[E // 2], src[-1], dst[0]], np.uint32)
    with eg.Graph() as g:
        g.load_directed(eg.pack_edges(src, dst, w), V)
        dist = g.sssp_batch(sources)
    for s in range(len(sources)):
        ref = oracle.sssp(csr["off"][0], csr["adj"], csr["w"], V, int(sources[s]))
        assert np.array_equal(dist[s].view(np.uint32), ref.view(np.uint32)), s


@pytest.mark.parametrize("n", [31, 32, 33])
def test_ppr_row_widths(eg_lib, n):
    """Rows of 32 columns for up to 32 seeds, of 64 for more."""
    test_ppr_and_adjoint_list_lengths(eg_lib, n, 3)


@pytest.mark.parametrize("per", [1, 31, 32, 33])
def test_sssp_graphs_row_widths(eg_lib, per):
    """Distances of a batch come as rows of 64 columns whatever width the sweeps used, on the host and on the
    device; columns past the last source are unreached."""
    import torch

    import endgraph_gb300 as eg
    rng = np.random.default_rng(per)
    sizes, edges = [700, 33, 2000], [5000, 40, 30_000]
    graphs = [(rng.integers(0, v, e).astype(np.uint32), rng.integers(0, v, e).astype(np.uint32),
               rng.random(e).astype(np.float32)) for v, e in zip(sizes, edges)]
    rec = np.concatenate([eg.pack_edges(s, d, w) for s, d, w in graphs])
    eoff = np.cumsum([0] + edges).astype(np.uint64)
    V = sum(sizes)
    sources = np.concatenate([rng.integers(0, v, per) for v in sizes]).astype(np.uint32)
    want = np.full((V, 64), 1e9, np.float32)
    at = 0
    for k, (s, d, w) in enumerate(graphs):
        csr = oracle.build_csr(s, d, w, sizes[k], np.array([0, sizes[k]], np.uint32))
        for j in range(per):
            want[at:at + sizes[k], j] = oracle.sssp(csr["off"][0], csr["adj"], csr["w"], sizes[k], int(sources[k * per + j]))
        at += sizes[k]
    with eg.Graph() as g:
        g.load_graph_batch(rec, eoff, np.array(sizes, np.uint32))
        assert np.array_equal(g.sssp_graphs(sources, per), want)
        buf = torch.zeros(64 * V + 3, device="cuda")
        for skip in (0, 1, 3):
            out = buf[skip:skip + 64 * V].view(V, 64)
            g.sssp_graphs(sources, per, dist=out)
            assert np.array_equal(out.cpu().numpy(), want), skip


@pytest.mark.parametrize("deg", [1, 2, 3, 23, 24, 25, 31, 32, 33, 511, 512, 513, 0])
def test_ppr_weights_by_list_length(eg_lib, deg):
    """Out-lists of `deg` edges (0: of every length from 1 to 1,100, and many of one): those that a lane takes by
    itself, those that a warp takes, and those cut into tasks, alone and next to each other."""
    import torch

    import endgraph_gb300 as eg
    rng = np.random.default_rng(deg)
    lens = np.full(max(3, 60_000 // deg), deg) if deg else rng.permutation(np.concatenate([np.arange(1, 1101), np.ones(5000, int)]))
    V, K, alpha = len(lens) + 7, 3, 0.15
    src = np.repeat(np.arange(len(lens)), lens).astype(np.uint32)
    dst = rng.integers(0, V, len(src)).astype(np.uint32)
    p = rng.permutation(len(src))
    src, dst = src[p], dst[p]
    w = rng.uniform(0.5, 1.5, len(src)).astype(np.float32)
    for n in (1, 5):
        seeds = src[:n].copy()
        dl = rng.random((n, V)).astype(np.float32)
        with eg.Graph() as g:
            g.load_directed_with_ids(eg.pack_edges(src, dst), V)
            x = g.ppr(w, seeds, alpha, K)
            dw = g.ppr_backward(w, seeds, dl, alpha, K)
        wt = torch.tensor(w, dtype=torch.float64, requires_grad=True)
        ref = _ppr64(src, dst, wt, V, seeds, alpha, K)
        ref.backward(torch.from_numpy(dl.astype(np.float64)))
        r, gr = ref.detach().numpy(), wt.grad.numpy()
        assert np.abs(x - r).sum() / np.abs(r).sum() <= 1e-6
        # lists of one edge have no gradient: what is left of the roundings is small against the longest ones'
        assert np.linalg.norm(dw - gr) <= 1e-4 * max(np.linalg.norm(gr), 1e-2 * np.linalg.norm(dl))


def test_ppr_weights_of_short_lists_in_time(eg_lib):
    """Normalising 8 M weights of 8 M sources is 8 M random reads and 0.2 GB besides, less than 0.1 ms at 5 TB/s
    and 0.25 measured.  With a warp for each list it took 2.8 ms, its gradient 3.6."""
    import torch

    import endgraph_gb300 as eg
    V = E = 1 << 23
    gen = torch.Generator("cuda").manual_seed(1)
    rec = torch.randint(0, V, (E, 2), generator=gen, device="cuda", dtype=torch.int32)
    w = torch.rand(E, generator=gen, device="cuda") + 0.5
    dw, dl = torch.empty(E, device="cuda"), torch.rand((1, V), generator=gen, device="cuda")
    seeds = rec[:1, 0].cpu().numpy().astype(np.uint32)
    best = {}
    with eg.Graph() as g:
        g.load_directed_with_ids(rec, V)
        g.profile(True)
        for _ in range(4):
            g.profile_reset()
            g.ppr_backward(w, seeds, dl, 0.15, 1, dl_dw=dw)
            for k, (_, ms) in g.profile_read().items():
                best[k] = min(best.get(k, 1e9), ms)
    assert best["ppr_weights"] <= 1.0 and best["ppr_weight_grad"] <= 1.2, best


def _spmm_launches(K, C):
    """Forward sweeps of an adjoint of K steps at stride C: up to the last checkpoint, then in each segment."""
    return K - 1 if C == 1 else (K - 1) // C * C + sum(min(C, K - k) - 1 for k in range(0, K, C))


@pytest.mark.parametrize("n", [5, 32, 33, 64])
@pytest.mark.parametrize("K", [1, 2, 23])
def test_ppr_adjoint_strides(eg_lib, n, K):
    """The adjoint with all iterates kept and with checkpoints every 2, 3, 4 and ceil(sqrt(K)) steps (the last segment
    full or not), chosen by the memory it may keep; the stride shows in the number of forward sweeps.  Rows of
    both widths, seeds without in-edges and without any; the tolerance is that of the other comparisons."""
    import torch

    import endgraph_gb300 as eg
    src, dst, V0 = _fans(n + K)
    V = 8192  # a row array is 1 MiB (32 columns) or 2 (64)
    assert V0 <= V
    no_in = np.setdiff1d(src, dst)
    seeds = np.concatenate([[no_in[0], V - 1, 0, 1000], src[:60]]).astype(np.uint32)[:n]
    rng = np.random.default_rng(K)
    w = rng.uniform(0.5, 1.5, len(src)).astype(np.float32)
    dl = rng.random((n, V)).astype(np.float32) / V
    alpha, mib = 0.15, 1 if n <= 32 else 2
    wt = torch.tensor(w, dtype=torch.float64, requires_grad=True)
    _ppr64(src, dst, wt, V, seeds, alpha, K).backward(torch.from_numpy(dl.astype(np.float64)))
    ref = wt.grad.numpy()
    # rows kept at each stride for K = 23: 23, 12 + 2, 8 + 3, 6 + 4, 5 + 5
    strides = {-1: 1, 23 * mib: 1, 14 * mib: 2, 11 * mib: 3, 10 * mib: 4, 0: 5} if K == 23 else {-1: 1, 2 * mib: 1, 0: min(K, 2)}
    with eg.Graph() as g:
        g.load_directed_with_ids(eg.pack_edges(src, dst), V)
        g.profile(True)
        for keep in list(strides) + list(strides)[::-1]:
            g.set_option(eg.EG_OPT_PPR_KEEP_MIB, keep)
            g.profile_reset()
            dw = g.ppr_backward(w, seeds, dl, alpha, K)
            assert g.profile_read().get("ppr_spmm", (0, 0))[0] == _spmm_launches(K, strides[keep]), keep
            assert np.linalg.norm(dw - ref) / np.linalg.norm(ref) <= 1e-4, keep


def test_ppr_adjoint_gives_memory_back(eg_lib):
    """Iterates kept by an earlier call are freed when less is allowed."""
    import torch

    import endgraph_gb300 as eg
    V, E, K = 1 << 20, 1 << 20, 20  # 128 MiB a row array: 2.5 GiB of iterates, 9 arrays at the widest stride
    gen = torch.Generator("cuda").manual_seed(4)
    rec = torch.randint(0, V, (E, 2), generator=gen, device="cuda", dtype=torch.int32)
    w, dl = torch.rand(E, generator=gen, device="cuda") + 0.5, torch.rand((2, V), generator=gen, device="cuda")
    seeds = rec[:2, 0].cpu().numpy().astype(np.uint32)
    with eg.Graph() as g:
        g.load_directed_with_ids(rec, V)
        out = []
        for keep in (-1, 0, 1 << 20):
            g.set_option(eg.EG_OPT_PPR_KEEP_MIB, keep)
            dw = torch.empty(E, device="cuda")
            g.ppr_backward(w, seeds, dl, 0.15, K, dl_dw=dw)
            torch.cuda.synchronize()
            out.append((torch.cuda.mem_get_info()[0], dw))
    assert out[1][0] - out[0][0] >= 1 << 30 and out[1][0] - out[2][0] >= 1 << 30
    for _, dw in out[1:]:
        assert float((dw - out[0][1]).norm() / out[0][1].norm()) <= 1e-5
