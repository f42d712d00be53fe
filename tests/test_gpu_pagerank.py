"""GPU: the one-partition PageRank sweep on lists that end, begin and stay open at every edge of its
blocking (lanes, blocks of 512 edges, runs of blocks), in the persistent launch and with one launch
per sweep, with and without renumbered gathers."""
import numpy as np
import pytest

import oracle
from helpers import rel_l1

pytestmark = pytest.mark.gpu


def _check(src, dst, V, iterations, relabels=(0, 1)):
    """Relative L1 error against FP64 within 1e-6, the bound of the other PageRank comparisons."""
    import endgraph_gb300 as eg
    src, dst = src.astype(np.uint32), dst.astype(np.uint32)
    out, _ = oracle.degrees(src, dst, V)
    csc = oracle.build_csc(src, dst, None, V, np.array([0, V], np.uint32))
    with eg.Graph() as g:
        g.load_directed(eg.pack_edges(src, dst), V)
        for relabel in relabels:
            g.set_option(eg.EG_OPT_PR_RELABEL, relabel)
            for it in iterations:
                ref = oracle.pagerank(csc["off"][0], csc["adj"], out, V, it, 0.85)
                for _ in range(2):
                    assert rel_l1(g.pagerank(it, 0.85), ref) <= 1e-6, (relabel, it)


@pytest.mark.parametrize("length", [1, 2, 7, 8, 9, 16, 255, 256, 257, 511, 512, 513, 1024, 1025, 4096, 4097, 40_000])
def test_pagerank_list_lengths(eg_lib, length):
    """Every list has `length` in-edges (after one shorter list that shifts the others)."""
    V = 50_000
    rng = np.random.default_rng(length)
    lists = max(2, min(V, 120_000 // length))
    dst = np.concatenate([np.full(3, 0), np.repeat(np.arange(1, lists), length)])
    src = rng.integers(0, V, len(dst))
    _check(src, dst, V, (1, 2, 5))
    _check(src[3:], dst[3:], V, (2,))  # not shifted: lists end on block edges


@pytest.mark.parametrize("E", [1, 7, 8, 9, 31, 255, 256, 511, 512, 513, 1023, 1024, 1025, 16_384, 100_003])
def test_pagerank_edge_counts(eg_lib, E):
    rng = np.random.default_rng(E)
    V = 777
    _check(rng.integers(0, V, E), rng.integers(0, V, E), V, (1, 3))


@pytest.mark.parametrize("E", [(1 << 22) + 1, 5_000_003, 13_000_001])
def test_pagerank_one_launch_per_sweep(eg_lib, E):
    """More edges than the persistent launch takes; a hub of a quarter of them, and short lists."""
    V = 600_011
    rng = np.random.default_rng(E)
    dst = rng.integers(0, V, E)
    dst[: E // 4] = 12_345
    _check(rng.integers(0, V, E), dst, V, (1, 4))


@pytest.mark.parametrize("V,E", [(40, (1 << 24) + 5), (700_001, (1 << 24) + 1), (1_500_000, 17_000_003), (5_000_000, 17_000_000)])
def test_pagerank_sweeps_with_hot_sources(eg_lib, V, E):
    """Sweeps with a launch each, sources of very different out-degree (those of the first ranks are read from
    shared memory: one, all that the first lines hold, a full table), hubs, lists of one edge and none."""
    rng = np.random.default_rng(V)
    src = (V * rng.random(E) ** 4).astype(np.int64)
    dst = rng.integers(0, V, E)
    dst[: E // 8] = V // 3
    dst[E // 8: E // 4] //= 50
    _check(src, dst, V, (1, 4), relabels=(-1, 0, 1))


def test_list_starts_made_once(eg_lib):
    """Sweeps with and without renumbered sources in turn, and batched BFS between them, share one table of list
    starts: it is made anew only when the first sweep that wants places comes."""
    import endgraph_gb300 as eg
    V, E = 30_000, 400_000
    rng = np.random.default_rng(3)
    src, dst = rng.integers(0, V, E), rng.integers(0, V, E)
    src, dst = src.astype(np.uint32), dst.astype(np.uint32)
    out, _ = oracle.degrees(src, dst, V)
    csc = oracle.build_csc(src, dst, None, V, np.array([0, V], np.uint32))
    ref = oracle.pagerank(csc["off"][0], csc["adj"], out, V, 5, 0.85)
    csr = oracle.build_csr(src, dst, None, V, np.array([0, V], np.uint32))
    roots = src[:40]
    levels = [oracle.bfs_levels(csr["off"][0], csr["adj"], V, int(r)) for r in roots]
    with eg.Graph() as g:
        for load in range(2):
            g.load_directed(eg.pack_edges(src, dst), V)
            g.profile(True)
            g.profile_reset()
            for relabel in (0, 1, 0, 1, 1, 0):
                g.set_option(eg.EG_OPT_PR_RELABEL, relabel)
                assert rel_l1(g.pagerank(5), ref) <= 1e-6
                lv, _ = g.msbfs(roots)
                for s in range(len(roots)):
                    assert np.array_equal(lv[s], np.where(levels[s] == oracle.UNREACHED, 255, levels[s]).astype(np.uint8))
            assert g.profile_read()["pr_setup"][0] == 2


@pytest.mark.parametrize("E", [5_000_011, 12_000_003, (1 << 24) + 1, 60_000_001])
def test_pagerank_of_a_hub(eg_lib, E):
    """One list of nearly all edges, summed over up to tens of thousands of runs: its vertex's value has the roundings
    of a single sum and of the formula, each at most half a unit in the last place (2^-24, relative):
    the sum, damping times it, what is added, and the division; the terms' own roundings are independent
    and average out.  In FP32 throughout it was 1e-6 and more off."""
    import torch

    import endgraph_gb300 as eg
    V = 3001
    gen = torch.Generator("cuda").manual_seed(E)
    rec = torch.randint(0, V, (E, 2), generator=gen, device="cuda", dtype=torch.int32)
    rec[: E - 4 * V, 1] = 1234
    s, d = rec[:, 0].long(), rec[:, 1].long()
    deg = torch.bincount(s, minlength=V).double()
    with eg.Graph() as g:
        g.load_directed(rec, V)
        for it in (1, 2):
            cur = 1 / deg
            for k in range(it):
                nxt = 0.15 + 0.85 * torch.zeros_like(cur).index_add(0, d, cur[s])
                cur = nxt if k == it - 1 else nxt / deg
            for relabel in (0, 1):
                g.set_option(eg.EG_OPT_PR_RELABEL, relabel)
                got = g.pagerank(it, 0.85)
                assert abs(float(got[1234]) - float(cur[1234])) <= 4 * 2.0**-24 * float(cur[1234]), (it, relabel)


def test_pagerank_that_overflows(eg_lib):
    """Values past the largest float become infinite, as in a plain sum, and not NaN."""
    import endgraph_gb300 as eg
    V, E = 2000, 300_000
    rng = np.random.default_rng(4)
    src, dst = rng.integers(0, V, E).astype(np.uint32), rng.integers(0, V, E).astype(np.uint32)
    dst[:100_000] = 7
    with eg.Graph() as g:
        g.load_directed(eg.pack_edges(src, dst), V)
        x = g.pagerank(2, -1e35)  # the second sweep sums values of 1e33 and more
        assert not np.isnan(x).any() and np.isinf(x[7])
