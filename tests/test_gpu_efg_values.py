"""Principal values of tensors where a closed form can go wrong: exactly and nearly
axial ones, rank one, a zero determinant of the deviator, a large isotropic part,
diagonal ones (exact), one off-diagonal element, zero, and scales at which the
iteration takes over.

Tolerance, relative to the largest value: the kernel's construction is backward stable, some ten
roundings of the tensor (2^-53 each), and so is LAPACK's: 4e-15 asserted; the
diagonal tensors exact."""
import numpy as np
import pytest

import mdff_b200
from mdff_b200 import systems

pytestmark = pytest.mark.gpu

N = 512


def rotated(values, rng):
    q = np.linalg.qr(rng.normal(size=(N, 3, 3)))[0]
    a = np.einsum("nij,nj,nkj->nik", q, np.broadcast_to(values, (N, 3)), q)
    return 0.5 * (a + a.transpose(0, 2, 1))


def tensors(kind, rng):
    if kind == "random":
        a = rng.normal(size=(N, 3, 3))
        return 0.5 * (a + a.transpose(0, 2, 1))
    if kind == "one":
        a = np.zeros((N, 3, 3))
        for i in range(N):
            a[i][np.diag_indices(3)] = rng.normal(size=3)
            p, q = [(0, 1), (0, 2), (1, 2)][i % 3]
            a[i, p, q] = a[i, q, p] = rng.normal() * 10.0 ** rng.integers(-18, 2)
        return a
    v = {"axial": [-1.0, -1.0, 2.0], "oblate": [-2.0, 1.0, 1.0], "near": [-1.0, -1.0 + 1e-9, 2.0 - 1e-9], "rank1": [0.0, 0.0, 3.0],
         "symmetric": [1.0, 0.0, -1.0], "shifted": [1000.0, 1000.0 + 1e-4, 1000.0 - 2e-4], "identity": [1.0, 1.0, 1.0]}[kind]
    return rotated(np.array(v), rng)


@pytest.mark.parametrize("kind", ["random", "one", "axial", "oblate", "near", "rank1", "symmetric", "shifted", "identity"])
@pytest.mark.parametrize("scale", [1.0, 1e-90, 1e-120, 1e90, 1e120])
def test_values(kind, scale):
    s = systems.mgo_pim(grid=(8, 8, 8), rc=6.0, alpha=0.5, kmax=7)
    e = mdff_b200.Engine(s["params"], s["itype"], s["pos"], s["cell"])
    a = tensors(kind, np.random.default_rng(len(kind))) * scale
    t = np.stack([a[:, 0, 0], a[:, 1, 1], a[:, 2, 2], a[:, 0, 1], a[:, 0, 2], a[:, 1, 2]], axis=1)
    got = np.sort(e.efg_nmr(t)[0][:, :3], axis=1) / scale
    ref = np.linalg.eigvalsh(a / scale)
    assert np.max(np.abs(got - ref) / np.abs(ref).max(axis=1)[:, None]) < 4e-15


def test_diagonal_and_zero():
    s = systems.mgo_pim(grid=(8, 8, 8), rc=6.0, alpha=0.5, kmax=7)
    e = mdff_b200.Engine(s["params"], s["itype"], s["pos"], s["cell"])
    t = np.zeros((N, 6))
    t[: N // 2, :3] = np.random.default_rng(1).normal(size=(N // 2, 3))
    nmr = e.efg_nmr(t)[0]
    assert np.array_equal(np.sort(nmr[:, :3], axis=1), np.sort(t[:, :3], axis=1))
    assert np.all(nmr[N // 2:, 3] == 0.0)
