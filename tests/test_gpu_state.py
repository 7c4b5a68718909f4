"""Reading a state back, and the captured step's kernels against the plain ones.

Exact: a copied state is the same bytes through either entry point; a captured step does
the arithmetic of the plain one, in the same order."""
import ctypes as C

import numpy as np
import pytest

import mdff_b200
from mdff_b200 import abi, systems

pytestmark = pytest.mark.gpu


def argon(n, integrator=abi.NVE_VV, seed=0):
    m = int(np.ceil((n / 4) ** (1.0 / 3.0)))
    s = systems.lj_argon(ncell=max(m, 4), seed=seed)
    s["params"].integrator = integrator
    if integrator != abi.NVE_VV:
        s["params"].nhc_n = 2
        s["params"].timesca_thermo = 0.5
    keep = np.sort(np.random.default_rng(seed).permutation(len(s["pos"]))[:n])
    return dict(s, pos=s["pos"][keep], vel=s["vel"][keep], itype=s["itype"][keep])


def engine(s):
    e = mdff_b200.Engine(s["params"], s["itype"], s["pos"], s["cell"])
    e.md_start(s["vel"])
    return e


@pytest.mark.parametrize("n", [1, 255, 256, 257, 60000])
def test_state(n):
    e = engine(argon(n))
    r = e.step(1)
    xyz = [np.empty(n) for _ in range(3)]
    f = [np.empty(n) for _ in range(3)]
    dp = C.POINTER(C.c_double)
    p = [a.ctypes.data_as(dp) for a in xyz + f]
    assert mdff_b200.lib().mdff_get_positions(e._h, *p[:3]) == 0
    assert mdff_b200.lib().mdff_step(e._h, 0, None, None, None, None, None, None, *p[3:], None) == 0
    assert np.array_equal(r["pos"], np.stack(xyz, axis=1)) and np.array_equal(r["f"], np.stack(f, axis=1))
    assert np.array_equal(e.positions(), r["pos"])
    assert r["pos"].flags.c_contiguous and r["f"].flags.c_contiguous


@pytest.mark.parametrize("integrator", [abi.NVE_VV, abi.NVT_NHCN])
@pytest.mark.parametrize("n", [200, 500, 30000])
def test_captured_step_is_the_plain_one(n, integrator):
    s = argon(n, integrator)
    a, b = engine(s), engine(s)
    b.enable_profile(True)   # profiled steps run as plain launches
    ra, rb = a.step(12), b.step(12)
    assert np.array_equal(ra["pos"], rb["pos"]) and np.array_equal(ra["f"], rb["f"])
    assert ra["thermo"] == rb["thermo"]
    assert any(t["nlist_rebuilt"] for t in a.step(40)["thermo"])
