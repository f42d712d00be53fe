"""GPU: output arrays that kernels cannot or should not work on in place (odd addresses, pinned host memory)
are filled as any other."""
import ctypes

import numpy as np
import pytest

import oracle
from helpers import graph_batch

pytestmark = pytest.mark.gpu

V, E = 3001, 20_000


class _Out:
    """`n` bytes at `offset` bytes past an aligned address, on the device or in pinned host memory."""

    def __init__(self, n, kind):
        import torch
        self.kind, self.n = kind, n
        self.off = 16 if kind == "pinned" else kind
        if kind == "pinned":
            self.buf = torch.full((n + 64,), 0x5A, dtype=torch.uint8).pin_memory()
        else:
            self.buf = torch.full((n + 64,), 0x5A, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
        self.ptr = ctypes.c_void_p(self.buf.data_ptr() + self.off)

    def get(self, dtype):
        b = self.buf.cpu().numpy()
        assert (b[: self.off] == 0x5A).all() and (b[self.off + self.n:] == 0x5A).all()
        return b[self.off: self.off + self.n].copy().view(dtype)


KINDS = ["pinned", 0, 1, 2, 3, 4, 8]


@pytest.fixture(scope="module")
def case():
    rng = np.random.default_rng(5)
    src, dst = rng.integers(0, V, E).astype(np.uint32), rng.integers(0, V, E).astype(np.uint32)
    w = rng.random(E).astype(np.float32)
    csr = oracle.build_csr(src, dst, w, V, np.array([0, V], np.uint32))
    return src, dst, w, csr


@pytest.mark.parametrize("kind", KINDS)
def test_traversals(eg_lib, case, kind):
    import endgraph_gb300 as eg
    src, dst, w, csr = case
    L, root, reached = eg_lib, int(src[0]), ctypes.c_uint64()
    ref = oracle.bfs_levels(csr["off"][0], csr["adj"], V, root)
    with eg.Graph() as g:
        g.load_directed(eg.pack_edges(src, dst, w), V)
        level, parent = _Out(4 * V, kind), _Out(4 * V, kind)
        assert L.eg_bfs(g.h, root, level.ptr, parent.ptr, eg.EG_DEVICE, ctypes.byref(reached)) == 0
        lv = level.get(np.uint32)
        assert np.array_equal(lv, ref)
        assert oracle.bfs_check_parents(csr["off"][0], csr["adj"], V, root, lv, parent.get(np.uint32)) == 0
        only = _Out(4 * V, kind)
        assert L.eg_bfs(g.h, root, None, only.ptr, eg.EG_DEVICE, None) == 0
        assert oracle.bfs_check_parents(csr["off"][0], csr["adj"], V, root, lv, only.get(np.uint32)) == 0
        dist = _Out(4 * V, kind)
        assert L.eg_sssp(g.h, root, dist.ptr, eg.EG_DEVICE) == 0
        d = oracle.sssp(csr["off"][0], csr["adj"], csr["w"], V, root)
        assert np.array_equal(dist.get(np.uint32), d.view(np.uint32))
        for it in (1, 4):
            rank = _Out(4 * V, kind)
            assert L.eg_pagerank(g.h, it, 0.85, rank.ptr, eg.EG_DEVICE) == 0
            assert np.abs(rank.get(np.float32) - g.pagerank(it, 0.85)).max() <= 1e-5
        g.load_undirected_from_directed(eg.pack_edges(src, dst), V)
        label = _Out(4 * V, kind)
        assert L.eg_cc(g.h, label.ptr, eg.EG_DEVICE) == 0
        assert np.array_equal(label.get(np.uint32), oracle.cc_labels(src, dst, V))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("nper", [3, 40])
def test_graph_batch_rows(eg_lib, kind, nper):
    import torch

    import endgraph_gb300 as eg
    Vs, eoff, parts, src, dst, w = graph_batch(6, 9, weighted=True)
    rng = np.random.default_rng(nper)
    roots = np.concatenate([rng.integers(0, v, nper) for v in Vs]).astype(np.uint32)
    with eg.Graph() as g:
        g.load_graph_batch(eg.pack_edges(src, dst, w), eoff, Vs)
        n = int(Vs.sum())
        levels, _ = g.msbfs_graphs(roots, nper)
        dist = g.sssp_graphs(roots, nper)
        rd = torch.from_numpy(roots.view(np.int32)).cuda()
        torch.cuda.synchronize()
        rp = ctypes.c_void_p(rd.data_ptr())
        out = _Out(64 * n, kind)
        assert eg_lib.eg_msbfs_graphs(g.h, rp, nper, out.ptr, eg.EG_DEVICE, None) == 0
        assert np.array_equal(out.get(np.uint8).reshape(n, 64), levels)
        out = _Out(256 * n, kind)
        assert eg_lib.eg_sssp_graphs(g.h, rp, nper, out.ptr, eg.EG_DEVICE) == 0
        assert np.array_equal(out.get(np.uint32).reshape(n, 64), dist.view(np.uint32))
