"""CPU: the queues of the persistent traversals hold what a step can append to them.  The entries are
counted on the host with the kernels' own block arithmetic (eg_queue.cuh)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def count(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("queue") / "queue_bound")
    r = subprocess.run(["g++", "-x", "c++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "endgraph_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "queue", "queue_bound.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def run(V, E, phases, ctas=304, seed=1, keep=1, few=0):
        args = [V, E, ctas, seed, keep, few, *phases]
        r = subprocess.run([exe, *map(str, args)], capture_output=True, text=True)
        assert r.returncode == 0
        return [int(x) for x in r.stdout.split()]
    return run


# A root with an edge to every other vertex; ONES vertices of one out-edge, found by the first in-edges or
# the warps' walk (32 to an append); HUBS vertices whose in-lists (2,048 edges from each other's 2,048
# out-edges) are walked by segments in the level's second phase: 8 pieces to an append.
ONES, HUBS = 933_888, 91_200


def _two_phase_level():
    V = 1 + ONES + HUBS
    return V, (V - 1) + ONES + HUBS * 2048, [f"{ONES // 32}:32", f"{HUBS}:8"]


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_dense_level_of_two_phases(count, seed):
    V, E, phases = _two_phase_level()
    used, reserved, pieces = count(V, E, phases, seed=seed)
    assert pieces == ONES + 8 * HUBS and pieces <= used <= reserved
    # with a block left open per warp and phase the same level would not fit
    used, reserved, _ = count(V, E, phases, seed=seed, keep=0)
    assert used > reserved


@pytest.mark.parametrize("few", [0, 1])
@pytest.mark.parametrize("ctas", [1, 2, 9, 50, 304])
@pytest.mark.parametrize("per", [1, 3, 32, 100, 257, 2048, 2049])
@pytest.mark.parametrize("vertices", [100, 2049, 5000, 40_000, 300_000])
def test_levels_of_any_size(count, few, ctas, per, vertices):
    """Levels that reach every vertex, in one phase and in two, appended in equal parts: from queues that no CTA's
    shared part overflows to ones where all do."""
    appends = -(-vertices // per)
    for phases in ([f"{appends}:{per}"], [f"{appends // 2}:{per}", f"{appends - appends // 2}:{per}"]):
        used, reserved, pieces = count(appends * per, appends * per, phases, ctas=ctas, seed=per, few=few)
        assert pieces == appends * per and pieces <= used <= reserved


def test_small_graphs_reserve_what_they_can_use(count):
    """1,000 vertices and 8,000 edges fit one CTA's shared part: nothing for unfinished blocks (1.2 M entries, 19 MB a
    queue, when every warp of the GPU counted)."""
    assert count(1000, 8000, ["1000:1"], ctas=3)[1] <= 1000 + 8000 // 256 + 64
    assert count(100_003, 1_000_003, ["103909:1"], ctas=304)[1] <= 310_000
