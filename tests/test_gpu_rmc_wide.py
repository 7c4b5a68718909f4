"""RMC and g(r) with cutoffs near half the cell's width: the eight cells of the
neighbour rows then hold thousands of atoms each, and the rows most of all pairs.

The counts are integers and have to be equal to those over all pairs, also without
memory for the rows.  g(r) is timed against the same call just past half the width,
which takes all pairs: a factor of 30 when one thread sorted each cell, of 1 without."""
import time

import numpy as np
import pytest

import mdff_b200
from mdff_b200 import systems

from gpu_memory import memory_left
from test_gpu_rmc import rmc_params

pytestmark = pytest.mark.gpu


def best(f, k=3):
    t = []
    for _ in range(k):
        a = time.perf_counter()
        f()
        t.append(time.perf_counter() - a)
    return min(t)


def test_chain():
    s = systems.mgo_pim(grid=(34, 34, 34), rc=8.0, alpha=0.4, kmax=3, seed=2)   # 4 913 ions a cell
    half = 0.5 * s["cell"][0, 0]
    e = mdff_b200.Engine(s["params"], s["itype"], s["pos"], s["cell"])
    for cut in (half - 1.3, half + 0.2):
        gexp = e.gr(cut, 0.05) * 1.01
        res, g = e.rmc(rmc_params(10 ** 9, 40, cut, 0.05), gexp, seed=1)
        assert res["kacc"] > 1 and np.array_equal(g, e.gr(cut, 0.05))


def liquid(m):
    s = systems.mgo_pim(grid=(m, m, m), rc=8.0, alpha=0.4, kmax=3, seed=2, jitter=0.1)
    return mdff_b200.Engine(s["params"], s["itype"], s["pos"], s["cell"]), s["cell"][0, 0]


def test_gr_time():
    e, edge = liquid(32)
    t = {f: best(lambda: e.gr(f * edge, 0.05)) for f in (0.24, 0.49, 0.51)}
    assert max(t[0.24], t[0.49]) < 10.0 * t[0.51], t


@pytest.mark.parametrize("m,left", [(32, 100), (40, 1000)])
def test_gr_without_memory(m, left):
    """Rows of 161 MB in 100 MB, and of 630 MB where they are more than a quarter of what is free."""
    e, edge = liquid(m)
    g = e.gr(0.19 * edge, 0.05)
    with memory_left(left << 20):
        assert np.array_equal(g, e.gr(0.19 * edge, 0.05))
    assert np.array_equal(g, e.gr(0.19 * edge, 0.05))
