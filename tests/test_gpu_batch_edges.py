"""A batch of configurations at the edges of its kernels' tiles against the
oracle: atom counts around the 16-atom table blocks, the 64-atom field blocks and
the 128-atom chunks; k ranges with every number of m = |nz| values an item can
take, odd counts of column pairs, dimensions without wave vectors, a long one;
diagonal and sheared cells, and cutoffs of just half the cell's width.

Tolerances: the other batch tests' (a different order of summation in FP64):
forces and stress 1e-10, energy 1e-11, loss 1e-9, gradient 1e-8 of its largest
parameter-scaled component."""
import numpy as np
import pytest

import oracle
import mdff_b200
from mdff_b200 import abi, fit

from test_gpu_batch import _base, _cfg_params

pytestmark = pytest.mark.gpu

CASES = [(3, (3, 3, 3)), (2, (4, 2, 4)), (15, (0, 5, 5)), (16, (5, 0, 6)), (17, (4, 5, 0)), (33, (0, 0, 7)), (63, (6, 4, 8)),
         (64, (4, 6, 9)), (65, (5, 5, 10)), (127, (2, 3, 11)), (128, (7, 8, 12)), (129, (6, 7, 13)), (257, (4, 4, 20)),
         (40, (2, 3, 40)), (20, (9, 9, 5))]


def confs_of(shape):
    out = []
    for k, (n, kmax) in enumerate(CASES):
        m = max(2, int(np.ceil(n ** (1.0 / 3.0))))
        m += m & 1
        rng = np.random.default_rng(k)
        g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
        keep = np.sort(rng.permutation(len(g))[:n])
        t = 1 + (g.sum(1) % 2)[keep]
        o = np.argsort(t, kind="stable")
        edge = 2.2 * m * np.array([1.0, 1.04, 1.02])
        cell = np.diag(edge)
        if shape == "sheared":
            cell = cell + np.array([[0, 0, 0], [0.4, 0, 0], [-0.3, 0.5, 0]])
        inv = np.linalg.inv(cell)
        width = 1.0 / np.linalg.norm(inv, axis=0).max()
        rc = 0.5 * width if shape == "half" else 0.45 * width
        out.append(dict(itype=t[o].astype(np.int32), pos=(g[keep][o] + 0.3 + rng.normal(0, 0.04, (n, 3))) * 2.2, cell=cell, rc=rc,
                        alpha=2.6 / rc, kmax=list(kmax)))
    return out


@pytest.mark.parametrize("shape", ["diagonal", "sheared", "half"])
def test_against_oracle(shape):
    confs, base = confs_of(shape), _base()
    space = fit.mgo_space(base)
    theta0 = space.get(base)
    b = mdff_b200.Batch(base, confs)
    out = b.forces()
    rng = np.random.default_rng(5)
    ft = [f + rng.normal(0.0, 0.1, f.shape) for f in out["f"]]
    tt = [t + np.eye(3) * 0.1 for t in out["tau"]]
    for c, conf in enumerate(confs):
        r = oracle.Oracle(_cfg_params(base, conf), conf["itype"], conf["pos"], conf["cell"]).engforce()
        tau_o = r["tau_nonb"] + r["tau_coul"]
        u_o = r["e"]["u_bmhft"] + r["e"]["u_coul"]
        fo = np.asarray(r["f"])
        assert np.linalg.norm(out["f"][c] - fo) <= 1e-10 * max(1.0, np.linalg.norm(fo)), CASES[c]
        assert np.linalg.norm(out["tau"][c] - tau_o) <= 1e-10 * max(1.0, np.linalg.norm(tau_o)), CASES[c]
        assert abs(out["energy"][c] - u_o) <= 1e-11 * max(1.0, abs(u_o)), CASES[c]
    b.set_targets(ft, tt, 1.0, 0.01)
    loss, g, _ = b.loss_grad()
    go, lo = abi.ParamGrad(), 0.0
    for conf, f, t, (cf, cs) in zip(confs, ft, tt, fit.batch_constants([len(c["itype"]) for c in confs], 1.0, 0.01)):
        l, go, _ = oracle.Oracle(_cfg_params(base, conf), conf["itype"], conf["pos"], conf["cell"]).loss_grad(f, t, cf, cs, go)
        lo += l
    assert abs(loss - lo) <= 1e-9 * abs(lo)
    ge, gr = space.project(g, theta0), space.project(go, theta0)
    assert (np.abs(ge - gr) * np.abs(theta0)).max() <= 1e-8 * np.abs(gr * theta0).max()
