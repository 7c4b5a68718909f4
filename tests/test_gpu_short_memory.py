"""The FP64 polarisable path where device memory is short: the tables that make it
faster are left out, and the values are those of a context that has them.

Tolerances: the same sums in another order, as in test_gpu_pair.py; the dipoles
are solved to 1e-12."""
import numpy as np
import pytest
import torch

import mdff_b200
from mdff_b200 import systems

from gpu_memory import memory_left
from helpers import rel

pytestmark = pytest.mark.gpu


def ions(m, rc=10.0):
    s = systems.mgo_pim(grid=(m, m, m), rc=rc, alpha=0.3, kmax=8, seed=4)
    s["params"].conv_tol_ind = 1e-12
    return s


def evaluate(s, eng, steps=2):
    a = eng.engforce()
    eng.md_start(s["vel"])
    return a, eng.step(steps)


def compare(a, b):
    for k in ("f", "mu", "tau_coul"):
        assert rel(a[0][k], b[0][k]) < 1e-10, k
    assert abs(a[0]["e"]["u_coul"] - b[0]["e"]["u_coul"]) <= 1e-11 * abs(b[0]["e"]["u_coul"])
    assert rel(a[1]["f"], b[1]["f"]) < 1e-9
    assert a[1]["thermo"][-1]["scf_iter"] == b[1]["thermo"][-1]["scf_iter"]


@pytest.mark.parametrize("m,left", [(20, 60), (28, 1000)])
def test_pair_table(m, left):
    """Tables of about 105 MB in 60 MB, and of 290 MB where that is more than a quarter of
    what is free: then it stays free."""
    s = ions(m)
    want = evaluate(s, mdff_b200.Engine(s["params"], s["itype"], s["pos"], s["cell"]))
    eng = mdff_b200.Engine(s["params"], s["itype"], s["pos"], s["cell"])
    with memory_left(left << 20):
        got = evaluate(s, eng)
        free = torch.cuda.mem_get_info()[0]
    compare(got, want)
    assert left < 256 or free > 0.8 * (left << 20)


def test_creation():
    """The reciprocal space's buffers are the first evaluation's: a context that evaluates no
    force does without them."""
    s = systems.mgo_pim(grid=(48, 48, 48), rc=5.0, alpha=0.6, kmax=8, seed=4)
    args = [s[k] for k in ("params", "itype", "pos", "cell")]
    free = torch.cuda.mem_get_info()[0]
    eng = mdff_b200.Engine(*args)
    made = torch.cuda.mem_get_info()[0]
    eng.gr(4.0, 0.1)
    torch.cuda.synchronize()
    eng.engforce()
    assert free - made < 240 << 20 and made - torch.cuda.mem_get_info()[0] > 100 << 20
