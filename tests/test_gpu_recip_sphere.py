"""The FP64 path's reciprocal space with the k sphere of fp64_keps (gaps between the
columns, columns whose mirror in ny is left out, runs of columns shorter and
longer than a column block), against a direct sum: what the sphere leaves out of the
full half space, which test_gpu_recip_fp64.py holds to the oracle, in plain numpy.

Tolerance: 1e-12 of the full value's norm, as there; the direct sum is a sum of
fewer terms of at most the same size."""
import numpy as np
import pytest

import mdff_b200

from test_gpu_recip_fp64 import ions

pytestmark = pytest.mark.gpu

COUL = 14.3996441494161   # eV A; the field is without it


def left_out(p, itype, pos, cell, keps):
    """How many of the half space's vectors are past the sphere, and their field, field
    gradient and energy (src/field.f90:2646-2873)."""
    n1, n2, n3 = np.meshgrid(np.arange(p.kES[0] + 1), np.arange(-p.kES[1], p.kES[1] + 1), np.arange(-p.kES[2], p.kES[2] + 1),
                             indexing="ij")
    n = np.stack([n1, n2, n3], -1).reshape(-1, 3)
    n = n[(n[:, 0] > 0) | ((n[:, 0] == 0) & ((n[:, 1] > 0) | ((n[:, 1] == 0) & (n[:, 2] > 0))))]
    k = 2.0 * np.pi * n @ np.linalg.inv(cell)   # (columns: the cell vectors)
    k2 = (k ** 2).sum(1)
    k = k[k2 > -4.0 * p.alphaES ** 2 * np.log(keps)]
    k2 = (k ** 2).sum(1)
    a = np.exp(-0.25 * k2 / p.alphaES ** 2) / k2
    q = np.array([p.qch[t - 1] for t in itype])
    mu = np.array([list(p.dip[t - 1]) for t in itype])
    e = np.exp(1j * pos @ k.T)
    s = ((q[:, None] + 1j * (mu @ k.T)) * e).sum(0)
    w = 8.0 * np.pi / abs(np.linalg.det(cell)) * a
    c = e * (w * np.conj(s))
    ef = c.imag @ k
    g = np.einsum("ik,ka,kb->iab", c.real, k, k)
    return len(k), ef, COUL * g, COUL * 0.5 * (w * abs(s) ** 2).sum()


@pytest.mark.parametrize("keps", [0.3, 0.05, 1e-3, 1e-6])
@pytest.mark.parametrize("n,kmax,tilt", [(130, (8, 9, 10), 1.1), (129, (5, 2, 12), 0.0), (40, (7, 3, 9), 0.7),
                                         (257, (3, 17, 6), 1.1), (33, (9, 8, 31), 0.3)])
def test_sphere(n, kmax, tilt, keps):
    p, itype, pos, cell = ions(n, kmax, "both", tilt=tilt)
    full = mdff_b200.Engine(p, itype, pos, cell).engforce()
    half = mdff_b200.Engine(p, itype, pos, cell).kspace_info()["half"]
    p.fp64_keps = keps
    eng = mdff_b200.Engine(p, itype, pos, cell)
    part = eng.engforce()
    nk, ef, g, u = left_out(p, itype, pos, cell, keps)
    assert eng.kspace_info()["main"] == half - nk   # (1e-6 holds most of these sets whole)
    assert np.linalg.norm(full["ef"] - part["ef"] - ef) <= 1e-12 * np.linalg.norm(full["ef"])
    six = np.stack([g[:, 0, 0], g[:, 1, 1], g[:, 2, 2], g[:, 0, 1], g[:, 0, 2], g[:, 1, 2]], 1)
    assert np.linalg.norm(full["efg"] - part["efg"] - six) <= 1e-12 * np.linalg.norm(full["efg"])
    assert abs(full["e"]["u_rec"] - part["e"]["u_rec"] - u) <= 1e-12 * abs(full["e"]["u_rec"])
