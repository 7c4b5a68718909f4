"""Pairs whose two nearest images are equally far (a fractional difference of
exactly 1/2), where d - rint(d) and the reference's d - NINT(d) take different
ones: ions on a grid of binary fractions in cells of half the grid's powers of
two, so that every coordinate, distance and cutoff is exact, with the cutoff at or
beyond half the cell's narrowest width and the types drawn at random, so that
no symmetry hides the image that was taken.

Tolerances: those of test_gpu_pair.py and test_gpu_batch_edges.py, which compare the
same kernels; a pair with the wrong image is off by its whole contribution."""
import numpy as np
import pytest

import mdff_b200
import oracle
from mdff_b200 import fit

from test_gpu_batch import _base, _cfg_params
from test_gpu_pair import compare, params

pytestmark = pytest.mark.gpu

CELLS = {"diagonal": np.diag([8.0, 16.0, 16.0]),
         "sheared": np.array([[8.0, 0.0, 0.0], [4.0, 16.0, 0.0], [0.0, 0.0, 16.0]])}   # columns: a = (8, 4, 0)


def grid_ions(seed):
    g = np.stack(np.meshgrid(np.arange(4), np.arange(8), np.arange(8), indexing="ij"), -1).reshape(-1, 3)
    return np.repeat([1, 2], 128).astype(np.int32), 2.0 * g[np.random.default_rng(seed).permutation(256)]


def ties(pos, cell, rc):
    """Pairs within rc by the NINT image that rint takes from another one."""
    s = pos @ np.linalg.inv(cell).T
    d = (s[:, None] - s[None])[~np.eye(len(s), dtype=bool)]
    a, b = d - np.copysign(np.floor(np.abs(d) + 0.5), d), d - np.rint(d)
    r = a @ cell.T
    return ((r ** 2).sum(-1) <= rc * rc) & (np.abs((a - b) @ cell.T).max(-1) > 0)


@pytest.mark.parametrize("kind", ["lj", "lj9-7", "bmh", "bmhftd", "morse"])
@pytest.mark.parametrize("shape", ["diagonal", "sheared"])
def test_pairs(kind, shape):
    t, pos = grid_ions(0)
    assert ties(pos, CELLS[shape], 5.0).any()
    compare(params(kind, 5.0), t, pos, CELLS[shape])


@pytest.mark.parametrize("shape", ["diagonal", "sheared"])
def test_charges_and_dipoles(shape):
    t, pos = grid_ions(1)
    assert ties(pos, CELLS[shape], 4.0).any()
    p = params("pim", 4.0)
    p.poldip_iso[0] = 0.5   # (random neighbours: the table's value has no solution)
    p.conv_tol_ind = 1e-13
    compare(p, t, pos, CELLS[shape], coul=True)


@pytest.mark.parametrize("shape", ["diagonal", "sheared"])
def test_batch(shape):
    t, pos = grid_ions(2)
    conf = dict(itype=t, pos=pos, cell=CELLS[shape], rc=4.0, alpha=0.6, kmax=[5, 7, 7])
    base = _base()
    base.poldip_iso[0] = 0.5
    space = fit.mgo_space(base)
    theta0 = space.get(base)
    b = mdff_b200.Batch(base, [conf])
    out = b.forces()
    o = oracle.Oracle(_cfg_params(base, conf), t, pos, conf["cell"])
    r = o.engforce()
    f, tau = np.asarray(r["f"]), r["tau_nonb"] + r["tau_coul"]
    assert np.linalg.norm(out["f"][0] - f) <= 1e-10 * np.linalg.norm(f)
    assert np.linalg.norm(out["tau"][0] - tau) <= 1e-10 * np.linalg.norm(tau)
    ft, tt = f + np.random.default_rng(3).normal(0.0, 0.1, f.shape), tau + 0.1 * np.eye(3)
    b.set_targets([ft], [tt], 1.0, 0.01)
    loss, g, _ = b.loss_grad()
    (cf, cs), = fit.batch_constants([len(t)], 1.0, 0.01)
    lo, go, _ = o.loss_grad(ft, tt, cf, cs)
    assert abs(loss - lo) <= 1e-9 * abs(lo)
    ge, gr = space.project(g, theta0), space.project(go, theta0)
    assert (np.abs(ge - gr) * np.abs(theta0)).max() <= 1e-8 * np.abs(gr * theta0).max()
