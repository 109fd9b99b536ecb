"""Calls near the smallest device budget that holds them: a budget that once
sufficed keeps sufficing."""
import functools

import pytest

import subgraphmatchgpu_b200 as sme

pytestmark = pytest.mark.gpu
MB = 1 << 20


@functools.lru_cache(maxsize=None)
def graph(name):
    return {"rmat12": lambda: sme.Graph.rmat(12, 8, seed=3), "rmat14": lambda: sme.Graph.rmat(14, 6, seed=6),
            "ba": lambda: sme.Graph.ba(6000, 5, seed=4), "er": lambda: sme.Graph.er(20000, 8.0, seed=5)}[name]()


# each level's frontier leaves room for the next one's although the budget's
# share is far below the 1 MiB that a batch may cost in a larger arena
@pytest.mark.parametrize("name,query,budget", [("ba", 2, 3.0), ("rmat12", 3, 3.5), ("ba", 3, 4.0), ("ba", 7, 4.0),
                                               ("rmat14", 2, 4.0), ("er", 2, 5.0), ("er", 7, 5.5), ("rmat14", 3, 6.0),
                                               ("rmat12", 7, 8.0), ("rmat14", 7, 10.0)])
def test_external_frontiers_leave_room_for_the_next_level(name, query, budget):
    g = graph(name)
    want = g.count(query, warp_granularity=3)
    assert g.count(query, mode=sme.EXTERNAL_GPU, mem_limit_bytes=int(budget * MB)) == want
