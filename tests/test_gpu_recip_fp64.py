"""The FP64 path's reciprocal space (int8-digit GEMMs on the tensor cores)
against the oracle at the edges of its tiles: nz ranges around the 32-byte K
steps and the widest one (kz = 31), the first one past it (kz = 32, the CUDA-core
kernels), a single column, atom counts around the 16-atom blocks and the
128-atom tiles, sources with and without dipoles, a triclinic cell and a k
sphere.  The ions stand further apart than the real-space cutoff, so that the
reciprocal part is what is compared.

Tolerance: the digit sums are exact, so a structure factor or a field differs
from the oracle's by a few roundings of its operands (2^-53 each, and the phases'
kmax 2^-53 relative to 2 pi) and by the oracle's own summation error, sqrt(terms)
2^-53 with fewer than 1e6 terms: 1e-13 of the norm; 1e-12 asserted."""
import numpy as np
import pytest

import mdff_b200
import oracle
from mdff_b200 import abi

from helpers import rel

pytestmark = pytest.mark.gpu


def ions(n, kmax, dipoles, tilt=0.0, keps=0.0):
    m = int(np.ceil(n ** (1.0 / 3.0)))
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * 3.0
    rng = np.random.default_rng(100 * n + sum(kmax))
    cell = np.eye(3) * 3.0 * max(m, 2) + tilt * np.array([[0, 0, 0], [1, 0, 0], [0.5, -0.7, 0]])
    p = abi.default_params()
    p.ntype = 2
    p.lcoulomb = 1
    p.cutlongrange = 2.0
    p.alphaES = 0.9
    for d in range(3):
        p.kES[d] = kmax[d]
    p.qch[0], p.qch[1] = 1.3, -1.3
    if dipoles:
        p.dip[0][0], p.dip[0][1], p.dip[0][2] = 0.3, -0.1, 0.2
        p.dip[1][2] = -0.4
    p.doefield = p.doefg = 1
    p.fp64_keps = keps
    itype = np.where(np.arange(n) % 2 == 0, 1, 2).astype(np.int32)
    itype = np.sort(itype)
    return p, itype, g + rng.uniform(-0.4, 0.4, g.shape), cell


@pytest.mark.parametrize("n,kmax", [(1, (3, 3, 3)), (15, (2, 5, 7)), (16, (5, 2, 15)), (17, (4, 4, 16)),
                                    (127, (0, 9, 8)), (128, (9, 0, 23)), (129, (7, 8, 9)), (700, (6, 7, 31)),
                                    (60, (3, 4, 32)), (33, (0, 0, 5)), (257, (16, 3, 0))])
@pytest.mark.parametrize("dipoles", ["", "both"])
def test_against_oracle(n, kmax, dipoles):
    p, itype, pos, cell = ions(n, kmax, dipoles)
    a = mdff_b200.Engine(p, itype, pos, cell).engforce()
    b = oracle.Oracle(p, itype, pos, cell).engforce()
    for k in ("f", "ef", "efg", "tau_coul"):
        assert rel(a[k], b[k]) < 1e-12 or np.linalg.norm(np.asarray(a[k]) - b[k]) < 1e-13, k
    assert abs(a["e"]["u_rec"] - b["e"]["u_rec"]) <= 1e-12 * max(1.0, abs(b["e"]["u_rec"]))


@pytest.mark.parametrize("keps", [0.0, 1e-3])
def test_triclinic_and_sphere(keps):
    p, itype, pos, cell = ions(130, (8, 9, 10), "both", tilt=1.1, keps=keps)
    a = mdff_b200.Engine(p, itype, pos, cell)
    r = a.engforce()
    if keps == 0.0:
        b = oracle.Oracle(p, itype, pos, cell).engforce()
        for k in ("f", "ef", "efg", "tau_coul"):
            assert rel(r[k], b[k]) < 1e-12, k
        return
    # the sphere: what it leaves out is below its Gaussian factor
    p.fp64_keps = 0.0
    full = mdff_b200.Engine(p, itype, pos, cell)
    f = full.engforce()
    assert a.kspace_info()["main"] < full.kspace_info()["main"]
    assert rel(r["ef"], f["ef"]) < 3e-2 and rel(r["ef"], f["ef"]) > 0.0


def test_repeated_and_many_contexts():
    """Two contexts of different sizes, evaluated in turn, keep their values."""
    cases = [ions(129, (7, 8, 9), "both"), ions(700, (6, 7, 31), "both"), ions(40, (2, 2, 2), "")]
    eng = [mdff_b200.Engine(*c) for c in cases]
    first = [e.engforce() for e in eng]
    for e, f in list(zip(eng, first))[::-1]:
        g = e.engforce()
        assert np.array_equal(f["f"], g["f"]) and np.array_equal(f["efg"], g["efg"])
