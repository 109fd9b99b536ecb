"""Calls near the smallest device budget that holds them: a budget that once
sufficed keeps sufficing."""
import ctypes as C
import functools

import numpy as np
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


# paths that share next to no lists: a batch sized for 32 times the list cache
# (3 of 12.8 MB) does not fit it and is halved until it does, again and again
@pytest.mark.parametrize("query", [0, 3])
def test_external_batches_whose_lists_do_not_fit_are_halved(query):
    g = sme.Graph.er(200000, 16.0, seed=9)
    want = g.count(query, warp_granularity=3)
    assert g.count(query, mode=sme.EXTERNAL_GPU, mem_limit_bytes=8 * MB) == want
    s = sme.last_stats()
    assert s.batches > 8 and s.h2d_bytes > 8 * (g.n + 1) + 4 * g.m  # lists came more than once


# the buffer for the instances lies beside the budget, not in it: 480 KB of it
# would be missing from the 4 MiB that these frontiers need
def test_enumeration_buffers_do_not_take_from_the_budget():
    g = graph("rmat12")
    g.to_device(0)
    want, cap = g.count(3), 30000
    out, n, o = np.zeros((cap, 4), np.uint32), C.c_uint64(), sme.opts(3, mem_limit_bytes=4 * MB)
    st = sme.lib().sme_enumerate(g.handle, C.byref(o), out.ctypes.data, cap, C.byref(n))
    assert (st, n.value) == (8, want), sme.lib().sme_last_error()  # more instances than the buffer holds
    assert len(np.unique(out, axis=0)) == cap
    g.release_device()


# a materialising step whose frontiers never fit at once counts their children
# once per batch, not once more per frontier
def test_frontiers_that_never_fit_are_not_counted_twice():
    g = graph("rmat14")
    g.to_device(0)
    want = g.count(2, warp_granularity=3)
    assert g.count(2, sme.GPU_GPSM_REUSE, mem_limit_bytes=4 * MB) == want
    s = sme.last_stats()
    assert s.batches > 50
    assert s.kernel_launches < 5 * s.batches  # 366 for 78 batches; 394 with a count per frontier
    g.release_device()
