"""GPU: levels that fill the queues of the persistent traversals past the CTAs' shared parts."""
import pytest

from test_queue_bound import HUBS, ONES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("direction", [0, 1, 2])
def test_dense_level_of_two_phases(eg_lib, direction):
    """The level of test_queue_bound.py: both phases of a dense level overflow the shared queues.  Every vertex
    is the root's child, and the next level's queue is walked whole."""
    import torch

    import endgraph_gb300 as eg
    V = 1 + ONES + HUBS
    hub0 = 1 + ONES
    i32 = dict(device="cuda", dtype=torch.int32)
    E = (V - 1) + ONES + HUBS * 2048
    rec = torch.empty((E, 2), **i32)
    rec[: V - 1, 0] = 0
    rec[: V - 1, 1] = torch.arange(1, V, **i32)
    ones = rec[V - 1: V - 1 + ONES]
    ones[:, 0] = torch.arange(1, hub0, **i32)
    ones[:, 1] = 0
    hubs = rec[V - 1 + ONES:].view(HUBS, 2048, 2)
    h = torch.arange(HUBS, **i32)
    hubs[:, :, 0] = (hub0 + h)[:, None]
    hubs[:, :, 1] = hub0 + (h[:, None] + 1 + torch.arange(2048, **i32)[None, :]) % HUBS
    level, parent = torch.empty(V, **i32), torch.empty(V, **i32)
    with eg.Graph() as g:
        g.load_directed(rec, V)
        g.set_option(eg.EG_OPT_BFS_DIRECTION, direction)
        for _ in range(2):
            g.bfs(0, level=level, parent=parent)
            assert int(level[0]) == 0 and bool((level[1:] == 1).all())
            assert bool((parent == 0).all())
            assert g.last_run()["edges"] == E
