"""The real-space kernels against the oracle where their routes change: each
short-range potential with a kernel of its own (12-6, BMH, BMHFTD) and those of
the general one, the atom counts around the switch from a warp an atom to eight
lanes, and the three minimum images (diagonal cell, sheared cell, and a cutoff of
half the cell, where the exact one decides).

Tolerance: a pair's force is a few dozen roundings (2^-53) off, its short-range
and damping terms cancel to no less than 1e-3 of their size at these distances,
and a row adds up to a thousand pairs: 53 * 2^-53 * 1e3 * sqrt(1e3) < 1e-9 for the
worst pair and far less in the norm; 1e-10 of the norm asserted, energies and
stresses 1e-11 and 1e-10, as in the other force tests."""
import numpy as np
import pytest

import mdff_b200
import oracle
from mdff_b200 import abi, systems

from helpers import rel

pytestmark = pytest.mark.gpu

H = 2.106


def atoms(n, shape="diagonal", rc=5.0, seed=0):
    m = max(2, int(np.ceil(n ** (1.0 / 3.0))))
    m += m & 1
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
    keep = np.sort(np.random.default_rng(seed).permutation(len(g))[:n])
    t = 1 + (g.sum(1) % 2)[keep]
    o = np.argsort(t, kind="stable")
    edge = np.array([m * H, m * H * 1.03, m * H * 0.98])
    if shape != "half":
        edge = np.maximum(edge, 2.0 * rc + 1.5)
    cell = np.diag(edge)
    if shape == "sheared":
        cell = np.diag(np.maximum(edge, 2.0 * rc + 4.0)) + np.array([[0, 0, 0], [1.3, 0, 0], [-0.9, 1.1, 0]])
    pos = (g[keep][o] + 0.25 + np.random.default_rng(seed + 1).normal(0, 0.04, (n, 3))) * H
    return t[o].astype(np.int32), pos, cell


def params(kind, rc, trunc=abi.TRUNC_LINEAR):
    p = systems.mgo_params(rc, 0.45, 5)
    p.lbmhftd = kind in ("bmhftd", "lj+bmhftd", "pim")
    p.lbmhft = kind == "bmh"
    p.lnmlj = kind in ("lj", "lj9-7", "lj+bmhftd")
    p.lmorse = kind == "morse"
    p.trunc = trunc
    for a in (0, 1):
        for b in (0, 1):
            p.epslj[a][b], p.sigmalj[a][b] = 0.02 * (1 + a + b), 1.7 + 0.1 * (a + b)
            p.epsmor[a][b], p.rhomor[a][b], p.sigmamor[a][b] = 0.05 * (1 + a + b), 1.1, 2.2
            if kind == "lj9-7":
                p.plj[a][b], p.qlj[a][b] = 7.0, 9.0
    if kind != "pim":
        p.lcoulomb = 0
        p.ldip_polar[0] = 0
    return p


def compare(p, itype, pos, cell, coul=False):
    a = mdff_b200.Engine(p, itype, pos, cell).engforce()
    b = oracle.Oracle(p, itype, pos, cell).engforce()
    for k in ("f", "tau_nonb") + (("mu", "ef", "efg", "tau_coul") if coul else ()):
        assert rel(a[k], b[k]) < 1e-10 or np.linalg.norm(np.asarray(a[k]) - b[k]) < 1e-12, k
    for k in ("u_lj", "vir_lj", "u_bmhft", "vir_bmhft", "u_morse", "vir_morse") + (("u_dir", "u_pol") if coul else ()):
        assert abs(a["e"][k] - b["e"][k]) <= 1e-11 * max(1.0, abs(b["e"][k])), k


@pytest.mark.parametrize("kind", ["lj", "lj9-7", "bmh", "bmhftd", "lj+bmhftd", "morse"])
@pytest.mark.parametrize("shape", ["diagonal", "sheared", "half"])
def test_potentials_and_images(kind, shape):
    n = 216
    t, pos, cell = atoms(n, shape)
    rc = 5.0 if shape != "half" else 0.5 * min(np.diag(cell))
    for trunc in (abi.TRUNC_NONE, abi.TRUNC_LINEAR, abi.TRUNC_QUADRATIC) if kind == "lj" else (abi.TRUNC_LINEAR,):
        compare(params(kind, rc, trunc), t, pos, cell)


@pytest.mark.parametrize("kind", ["lj", "bmh", "bmhftd"])
@pytest.mark.parametrize("n", [1, 7, 33, 257, 23999, 24000])
def test_atom_counts(kind, n):
    t, pos, cell = atoms(n)
    compare(params(kind, 5.0), t, pos, cell)


@pytest.mark.parametrize("shape", ["diagonal", "sheared", "half"])
def test_charges_and_dipoles(shape):
    t, pos, cell = atoms(216, shape)
    rc = 5.0 if shape != "half" else 0.5 * min(np.diag(cell))
    p = params("pim", rc)
    p.conv_tol_ind = 1e-13
    compare(p, t, pos, cell, coul=True)
