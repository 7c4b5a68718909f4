"""A neighbour-list build that finds no memory: the call fails with MDFF_E_NOMEM, and
the context goes on from the next positions as if it had not been made."""
import numpy as np
import pytest

import mdff_b200
from mdff_b200 import abi, systems

from gpu_memory import memory_left

pytestmark = pytest.mark.gpu


def liquid():
    s = systems.lj_argon(ncell=30)
    s["pos"] = s["pos"] + np.random.default_rng(0).normal(0.0, 0.03, s["pos"].shape)
    e = mdff_b200.Engine(s["params"], s["itype"], s["pos"], s["cell"])
    e.set_positions(s["pos"])
    return s, e.engforce()


def failed_step(s):
    """An engine after a step whose list build failed: 3 000 of 108 000 atoms in one
    place need rows of 1.6 GB."""
    e = mdff_b200.Engine(s["params"], s["itype"], s["pos"], s["cell"])
    e.md_start(s["vel"])
    crowd = s["pos"].copy()
    crowd[:3000] = 0.5 * np.diag(s["cell"]) + np.random.default_rng(1).uniform(-0.2, 0.2, (3000, 3))
    e.set_positions(crowd)
    with memory_left(600 << 20), pytest.raises(mdff_b200.EngineError) as err:
        e.step(1)
    assert err.value.code == abi.E_NOMEM
    return e


def test_next_evaluation():
    s, f = liquid()
    e = failed_step(s)
    e.set_positions(s["pos"])
    g = e.engforce()
    assert np.array_equal(f["f"], g["f"]) and f["e"] == g["e"]


def test_positions_after_a_failed_step():
    """The evaluation is one of the positions set last, not of the failed step's."""
    s, f = liquid()
    e = failed_step(s)
    e.set_positions(s["pos"])
    e.nlist_build()
    g = e.engforce()
    assert np.array_equal(f["f"], g["f"]) and f["e"] == g["e"]
