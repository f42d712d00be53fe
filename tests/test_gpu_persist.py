"""GPU: the single-source traversals that run every step inside one persistent launch, on the shapes
their queues and barriers are cut by: lists at the edges of a queue piece, hubs of many pieces,
traversals deeper than one launch, and thresholds that a step cannot move."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _sssp_ref(src, dst, w, V, root):
    csr = oracle.build_csr(src, dst, w, V, np.array([0, V], np.uint32))
    return oracle.sssp(csr["off"][0], csr["adj"], csr["w"], V, root)


def _check_sssp(src, dst, w, V, roots, deltas=(-1,)):
    import endgraph_gb300 as eg
    src, dst, w = src.astype(np.uint32), dst.astype(np.uint32), w.astype(np.float32)
    refs = {r: _sssp_ref(src, dst, w, V, r) for r in roots}
    with eg.Graph() as g:
        g.load_directed(eg.pack_edges(src, dst, w), V)
        for delta in deltas:
            g.set_option(eg.EG_OPT_SSSP_DELTA, delta)
            for r in roots:
                d = g.sssp(r)
                assert np.array_equal(d.view(np.uint32), refs[r].view(np.uint32)), (delta, r)


@pytest.mark.parametrize("deg", [1, 31, 32, 33, 127, 128, 129, 255, 256, 257, 511, 512, 513, 8193, 70000])
def test_sssp_piece_edges(eg_lib, deg):
    """A root of `deg` out-edges whose neighbours fan out again, over a small random graph."""
    V = 80_000
    rng = np.random.default_rng(deg)
    nbr = rng.choice(V - 1, deg, replace=False) + 1
    src = np.concatenate([np.zeros(deg, np.int64), rng.integers(0, V, 200_000)])
    dst = np.concatenate([nbr, rng.integers(0, V, 200_000)])
    _check_sssp(src, dst, rng.random(len(src)), V, [0, int(nbr[0])], deltas=(-1, 0, 3000))


def test_sssp_deeper_than_one_launch(eg_lib):
    """A chain of 10,000 vertices: more steps than one launch makes; and a root without edges."""
    n = 10_000
    rng = np.random.default_rng(1)
    perm = rng.permutation(n)
    _check_sssp(perm[:-1], perm[1:], rng.random(n - 1), n + 1, [int(perm[0]), n], deltas=(-1, 0))


def test_sssp_threshold_below_float_resolution(eg_lib):
    """Distances so large that adding the threshold step changes nothing: phases still advance.
    Zero weights, equal weights and weights of very different sizes."""
    V = 3000
    rng = np.random.default_rng(2)
    src, dst = rng.integers(0, V, 20_000), rng.integers(0, V, 20_000)
    w = rng.choice(np.array([0.0, 1e-6, 1.0, 3e7]), 20_000)
    _check_sssp(src, dst, w, V, [int(src[0]), int(src[1])], deltas=(-1, 0, 1))


@pytest.mark.parametrize("V,E", [(1, 1), (2, 5), (33, 64), (1025, 8191), (4097, 8193), (40_000, 1_300_000)])
def test_sssp_grid_sizes(eg_lib, V, E):
    """From one CTA to the whole GPU."""
    rng = np.random.default_rng(V)
    src, dst = rng.integers(0, V, E), rng.integers(0, V, E)
    _check_sssp(src, dst, rng.random(E), V, [int(src[0])], deltas=(-1, 0, 20_000))


def _check_bfs(src, dst, V, roots, directions=(0, 1, 2), divisors=(20,)):
    import endgraph_gb300 as eg
    src, dst = src.astype(np.uint32), dst.astype(np.uint32)
    csr = oracle.build_csr(src, dst, None, V, np.array([0, V], np.uint32))
    deg = np.diff(csr["off"][0].astype(np.int64))
    with eg.Graph() as g:
        g.load_directed(eg.pack_edges(src, dst), V)
        for root in roots:
            ref = oracle.bfs_levels(csr["off"][0], csr["adj"], V, root)
            for direction in directions:
                g.set_option(eg.EG_OPT_BFS_DIRECTION, direction)
                for div in divisors:
                    g.set_option(eg.EG_OPT_DENSE_DIVISOR, div)
                    lv, par = g.bfs(root)
                    assert np.array_equal(lv, ref), (root, direction, div)
                    assert oracle.bfs_check_parents(csr["off"][0], csr["adj"], V, root, lv, par) == 0
                    run = g.last_run()
                    assert run["edges"] == int(deg[ref != oracle.UNREACHED].sum())
                    assert run["iterations"] == int(ref[ref != oracle.UNREACHED].max()) + 1
                    assert run["iterations"] == run["push"] + run["pull"]


@pytest.mark.parametrize("deg", [1, 4, 5, 31, 33, 127, 129, 255, 256, 257, 1027, 1028, 1029, 5000, 70000])
def test_bfs_list_edges(eg_lib, deg):
    """A vertex whose out-list and in-list have `deg` entries: pieces of the queue, the dense level's
    first in-edges, the warp's walk and the segments.  Its in-neighbours are reached late or not at
    all, so that whole lists are read in vain."""
    V = 80_000
    rng = np.random.default_rng(deg)
    hub, nbr = 7, rng.choice(V - 10, deg, replace=False) + 10
    back = rng.choice(V - 10, deg, replace=False) + 10
    src = np.concatenate([np.full(deg, hub), back, rng.integers(10, V // 2, 120_000)])
    dst = np.concatenate([nbr, np.full(deg, hub), rng.integers(10, V // 2, 120_000)])
    _check_bfs(src, dst, V, [hub, int(back[0]), int(src[-1])], divisors=(1, 20, 1 << 30))


def test_bfs_deeper_than_one_launch(eg_lib):
    """A chain of 9,000 vertices in every direction mode, and a root without edges."""
    n = 9_000
    perm = np.random.default_rng(4).permutation(n)
    _check_bfs(perm[:-1], perm[1:], n + 1, [int(perm[0]), int(perm[n // 2])], directions=(0, 1))
    _check_bfs(perm[:-1], perm[1:], n + 1, [int(perm[n - 300]), n])


@pytest.mark.parametrize("V,E", [(1, 1), (2, 5), (33, 64), (1025, 8191), (4097, 8193), (40_000, 1_300_000)])
def test_bfs_grid_sizes(eg_lib, V, E):
    rng = np.random.default_rng(V)
    src, dst = rng.integers(0, V, E), rng.integers(0, V, E)
    _check_bfs(src, dst, V, [int(src[0]), 0])


def test_bfs_outputs_on_the_device(eg_lib):
    """Level and parent arrays of the caller are written in place; either may be left out."""
    import torch

    import endgraph_gb300 as eg
    V, E = 5000, 40_000
    rng = np.random.default_rng(8)
    src, dst = rng.integers(0, V, E).astype(np.uint32), rng.integers(0, V, E).astype(np.uint32)
    csr = oracle.build_csr(src, dst, None, V, np.array([0, V], np.uint32))
    root = int(src[0])
    ref = oracle.bfs_levels(csr["off"][0], csr["adj"], V, root)
    with eg.Graph() as g:
        g.load_directed(eg.pack_edges(src, dst), V)
        level = torch.full((V + 16,), 77, dtype=torch.int32, device="cuda")
        parent = torch.full((V + 16,), 78, dtype=torch.int32, device="cuda")
        g.bfs(root, level=level[5:5 + V], parent=parent[3:3 + V])
        lv, par = level.cpu().numpy(), parent.cpu().numpy()
        assert (lv[:5] == 77).all() and (lv[5 + V:] == 77).all() and (par[:3] == 78).all() and (par[3 + V:] == 78).all()
        assert np.array_equal(lv[5:5 + V].view(np.uint32), ref)
        assert oracle.bfs_check_parents(csr["off"][0], csr["adj"], V, root, lv[5:5 + V].view(np.uint32).copy(),
                                        par[3:3 + V].view(np.uint32).copy()) == 0
        level.fill_(0)
        g.bfs(root, level=level[:V], want_parent=False)
        assert np.array_equal(level[:V].cpu().numpy().view(np.uint32), ref)


def _check_cc(src, dst, V, w=None):
    import endgraph_gb300 as eg
    src, dst = src.astype(np.uint32), dst.astype(np.uint32)
    ref = oracle.cc_labels(src, dst, V)
    with eg.Graph() as g:
        g.load_undirected_from_directed(eg.pack_edges(src, dst, w), V)
        assert np.array_equal(g.cc(), ref)


def test_cc_chain_and_components(eg_lib):
    """Paths whose parents form long chains, several components of similar size beside a large one,
    and vertices without edges."""
    n = 30_000
    _check_cc(np.arange(n - 1), np.arange(1, n), n + 5)
    _check_cc(np.arange(1, n), np.arange(n - 1), n)
    perm = np.random.default_rng(1).permutation(n)
    _check_cc(perm[:-1], perm[1:], n)
    _check_cc(perm[:-2], perm[2:], n)          # two interleaved paths
    rng = np.random.default_rng(2)
    part = rng.integers(0, 7, 60_000)          # seven random graphs over one id space
    ids = [np.flatnonzero(part == k) for k in range(7)]
    src = np.concatenate([rng.choice(i, 12_000) for i in ids])
    dst = np.concatenate([rng.choice(i, 12_000) for i in ids])
    _check_cc(src, dst, 60_000)


@pytest.mark.parametrize("deg", [1, 2, 3, 255, 257, 258, 259, 514, 20_000])
def test_cc_lists_outside_the_common_component(eg_lib, deg):
    """A star whose hub is outside the largest component: its list goes through the queue."""
    V = 120_000
    rng = np.random.default_rng(deg)
    big = rng.permutation(V - 30_000) + 30_000
    leaves = rng.choice(29_990, deg, replace=False) + 10
    src = np.concatenate([big[:-1], np.full(deg, 5), leaves[: deg // 2]])
    dst = np.concatenate([big[1:], leaves, rng.permutation(leaves)[: deg // 2]])
    _check_cc(src, dst, V)


@pytest.mark.parametrize("V,E", [(1, 1), (2, 1), (5, 3), (1025, 700), (4097, 4096), (40_000, 900_000)])
def test_cc_grid_sizes(eg_lib, V, E):
    rng = np.random.default_rng(V)
    src, dst = rng.integers(0, V, E), rng.integers(0, V, E)
    _check_cc(src, dst, V, rng.random(E).astype(np.float32))


def test_launches_in_turn_on_one_handle(eg_lib):
    """Every launch finds its state words zeroed by the launch before it, whichever traversal that was,
    also across launches that continue (a chain deeper than one) and across loads."""
    import torch

    import endgraph_gb300 as eg
    n = 4_500
    rng = np.random.default_rng(11)
    chain = np.arange(n, dtype=np.uint32)
    src, dst = rng.integers(0, n, 30_000).astype(np.uint32), rng.integers(0, n, 30_000).astype(np.uint32)
    with eg.Graph() as g:
        for src, dst in ((chain[:-1], chain[1:]), (src, dst)):
            w = rng.random(len(src)).astype(np.float32)
            csr = oracle.build_csr(src, dst, w, n, np.array([0, n], np.uint32))
            level = oracle.bfs_levels(csr["off"][0], csr["adj"], n, 0)
            dist = oracle.sssp(csr["off"][0], csr["adj"], csr["w"], n, 0)
            labels = oracle.cc_labels(src, dst, n)
            lv = torch.empty(n, dtype=torch.int32, device="cuda")
            for _ in range(2):
                g.load_directed(eg.pack_edges(src, dst, w), n)
                ranks = g.pagerank(3)
                for call in (0, 1, 0, 0, 2, 1, 1, 2, 0):
                    if call == 0:
                        lv.fill_(-2)  # pending on torch's stream when the call is made
                        g.bfs(0, level=lv, want_parent=False)
                        assert np.array_equal(lv.cpu().numpy().view(np.uint32), level)
                    elif call == 1:
                        assert np.array_equal(g.sssp(0).view(np.uint32), dist.view(np.uint32))
                    else:
                        assert np.array_equal(g.pagerank(3), ranks)
                g.load_undirected_from_directed(eg.pack_edges(src, dst, w), n)
                assert np.array_equal(g.cc(), labels)
                assert np.array_equal(g.cc(), labels)


@pytest.mark.parametrize("spin_cap", [1, 200, 20_000])
def test_barrier_given_up_as_it_completes(eg_lib, spin_cap):
    """A CTA that gives up at a barrier which then completes for the others (the self-test's first launch) makes
    the call fail, and the state words are clean for the launches after it."""
    import endgraph_gb300 as eg
    n = 600
    i = np.arange(n - 1, dtype=np.uint32)
    with eg.Graph() as g:
        g.load_undirected_from_directed(eg.pack_edges(i, i + 1, np.ones(n - 1, np.float32)), n)
        for _ in range(2):
            assert g.selftest_grid_barrier(spin_cap) == 5  # EG_ERR_TIMEOUT
            assert np.array_equal(g.bfs(0)[0], np.arange(n))
            assert np.array_equal(g.sssp(0), np.arange(n, dtype=np.float32))
            assert not g.cc().any()


def _spread(src, dst, n, V, seed):
    """A graph over n vertices moved to random ids of V."""
    ids = np.random.default_rng(seed).choice(V, n, replace=False)
    return ids[src], ids[dst], ids


@pytest.mark.parametrize("deg", [1, 13, 257, 1036, 1037, 5000])
def test_bfs_bits_list_edges(eg_lib, deg):
    """More vertices than the traversal keeps levels alone for: reached vertices are bits as well, copied before
    each dense level.  Lists at the edges of a dense level's phases, half of them read in vain."""
    V, n = (1 << 23) + 1, 40_000
    rng = np.random.default_rng(deg)
    nbr, back = rng.choice(n - 10, deg, replace=False) + 10, rng.choice(n - 10, deg, replace=False) + 10
    src = np.concatenate([np.full(deg, 7), back, rng.integers(10, n // 2, 60_000)])
    dst = np.concatenate([nbr, np.full(deg, 7), rng.integers(10, n // 2, 60_000)])
    s, d, ids = _spread(src, dst, n, V, deg)
    _check_bfs(s, d, V, [int(ids[7]), int(s[-1])], divisors=(1, 20))


def test_bfs_bits_sizes(eg_lib):
    """On both sides of the switch, and a vertex count that fills its last word of bits."""
    rng = np.random.default_rng(3)
    src, dst = rng.integers(0, 30_000, 200_000), rng.integers(0, 30_000, 200_000)
    for V in (1 << 23, (1 << 23) + 1, (1 << 23) + 63, (1 << 23) + 64):
        s, d, ids = _spread(src, dst, 30_000, V, V & 7)
        s[0], d[0], s[1], d[1] = ids[0], V - 1, V - 1, 0
        _check_bfs(s, d, V, [int(ids[0]), V - 1, 0])


def test_bfs_bits_deeper_than_one_launch(eg_lib):
    n, V = 9_000, (1 << 23) + 100
    i = np.arange(n - 1)
    s, d, ids = _spread(i, i + 1, n, V, 8)
    _check_bfs(s, d, V, [int(ids[0])], directions=(0, 1))
    _check_bfs(s, d, V, [int(ids[n - 300])])


@pytest.mark.parametrize("V", [(1 << 20) + 1, 1 << 22, 1 << 23])
def test_sssp_automatic_step_on_sparse_graphs(eg_lib, V):
    """A star: nothing is relaxed twice however wide the step, so that an automatic step narrower than 0.7 of the mean
    weight only adds phases, which walk the far bits.  At 2^22 ten phases took 0.57 ms, two 0.17."""
    import time

    import torch

    import endgraph_gb300 as eg
    i = torch.arange(1, V, device="cuda", dtype=torch.int32)
    gen = torch.Generator("cuda").manual_seed(V)
    w = torch.rand(V - 1, generator=gen, device="cuda")
    rec = torch.stack([torch.zeros_like(i), i, w.view(torch.int32)], 1).contiguous()
    dist = torch.empty(V, device="cuda")
    with eg.Graph() as g:
        g.load_directed(rec, V)
        t = {}
        for delta in (-1, 350_000):  # automatic; 0.7 of the mean weight
            g.set_option(eg.EG_OPT_SSSP_DELTA, delta)
            t[delta] = 1e9
            for _ in range(6):
                torch.cuda.synchronize()
                a = time.perf_counter()
                g.sssp(0, dist=dist)
                t[delta] = min(t[delta], time.perf_counter() - a)
            assert float(dist[0]) == 0 and bool((dist[1:] == w).all())
    assert t[-1] <= 1.5 * t[350_000], t
