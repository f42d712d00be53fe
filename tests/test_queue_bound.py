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

    def run(V, E, phases, sms=152, ctas=None, seed=1, keep=1):
        args = [V, E, sms, ctas if ctas is not None else 2 * sms, seed, keep, *phases]
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
