"""GPU: the warp sweeps of PageRank and batched BFS on graphs whose runs hold several blocks of 512 edges (2, 4 and
8 of them), against the same steps in torch (PageRank in FP64)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# edges for runs of 2, 4 and 8 blocks (list_run_shift: (E >> (10 + s)) >= 24000), an odd number each
SIZES = [(24_000 << 10) + 12_345, (24_000 << 11) + 777, (24_000 << 12) + 5]
V = 600_011


def _graph(E):
    """Lists of every kind: a hub of a quarter of the edges (it crosses thousands of runs), lists of 512 and 4,096
    edges, lists of one, and what is left at random."""
    import torch
    gen = torch.Generator("cuda").manual_seed(E)
    rec = torch.empty((E, 2), dtype=torch.int32, device="cuda")
    rec[:, 0] = (V * torch.rand(E, generator=gen, device="cuda", dtype=torch.float64) ** 3).int().clamp(max=V - 1)
    dst = torch.randint(0, V // 2, (E,), generator=gen, device="cuda", dtype=torch.int32)
    dst[: E // 4] = 12_345
    at = E // 4
    for length, first in ((512, V // 2), (4096, V // 2 + 1000), (513, V // 2 + 2000)):
        n = 200
        dst[at: at + n * length] = first + torch.arange(n, device="cuda", dtype=torch.int32).repeat_interleave(length)
        at += n * length
    n = V // 4
    dst[at: at + n] = 3 * V // 4 + torch.arange(n, device="cuda", dtype=torch.int32)
    rec[:, 1] = dst
    return rec


@pytest.mark.parametrize("E", SIZES)
def test_pagerank_runs_of_several_blocks(eg_lib, E):
    import torch

    import endgraph_gb300 as eg
    rec = _graph(E)
    s, d = rec[:, 0].long(), rec[:, 1].long()
    deg = torch.bincount(s, minlength=V).double()
    has = deg > 0
    out = torch.empty(V, device="cuda")
    with eg.Graph() as g:
        g.load_directed(rec, V)
        g.profile(True)
        for it in (1, 4):
            cur = torch.where(has, 1.0 / deg.clamp(min=1), torch.ones_like(deg))
            for k in range(it):
                nxt = 0.15 + 0.85 * torch.zeros_like(cur).index_add(0, d, cur[s])
                cur = nxt if k == it - 1 else torch.where(has, nxt / deg.clamp(min=1), nxt)
            for relabel in (-1, 0, 1):
                g.set_option(eg.EG_OPT_PR_RELABEL, relabel)
                g.profile_reset()
                for _ in range(2):
                    g.pagerank(it, 0.85, out=out)
                    assert float((out.double() - cur).abs().sum() / cur.sum()) <= 1e-6, (it, relabel)
                ran = g.profile_read()
                assert ran["pr_pull"][0] == 2 * it and "pr_persistent" not in ran  # a launch per sweep


@pytest.mark.parametrize("E", SIZES)
def test_msbfs_runs_of_several_blocks(eg_lib, E):
    import torch

    import endgraph_gb300 as eg
    rec = _graph(E)
    s, d = rec[:, 0].long(), rec[:, 1].long()
    roots = np.array([12_345, 0, int(rec[-1, 0]), V - 1, 7], np.uint32)
    ref = torch.full((len(roots), V), 255, dtype=torch.uint8, device="cuda")
    for i, r in enumerate(roots):
        front = torch.zeros(V, dtype=torch.bool, device="cuda")
        front[int(r)] = True
        ref[i, int(r)] = 0
        for level in range(1, 255):
            nxt = torch.zeros(V, dtype=torch.bool, device="cuda")
            nxt[d[front[s]]] = True
            nxt &= ref[i] == 255
            if not bool(nxt.any()):
                break
            ref[i][nxt] = level
            front = nxt
    levels = torch.empty((len(roots), V), dtype=torch.uint8, device="cuda")
    with eg.Graph() as g:
        g.load_directed(rec, V)
        g.profile(True)
        for relabel in (0, 1):
            for div in (1 << 30, 20):  # every level swept; levels pushed and swept
                g.set_option(eg.EG_OPT_PR_RELABEL, relabel)
                g.set_option(eg.EG_OPT_BATCH_DIVISOR, div)
                g.profile_reset()
                g.msbfs(roots, levels=levels)
                assert g.profile_read()["msbfs_pull"][0] >= 1
                assert bool((levels == ref).all()), (relabel, div)
