"""The workloads whose speed this framework is judged by, and their values in plain 64-bit torch.

Every case goes through the public Python binding (mdff_b200.Engine, Batch,
fit) as a user's program calls it.  The kinds:

  lj      Lennard-Jones argon, NVE velocity Verlet: Engine.step
  silica  a rigid-ion Ewald silica melt, one whole evaluation: Engine.engforce
  pim     polarisable-ion MgO molecular dynamics (NVE, Nose-Hoover chains or
          constant pressure; FP64 and mixed precision): Engine.step
  efg     the electric field gradients of a trajectory's frames, each with its
          own dipole solve: Engine.efgcalc
  fit     force matching, loss and adjoint gradient over a ragged batch:
          fit.force_match_loss and backward
  stat    EFG post-processing of many configurations: Engine.efg_dist_ptr
  rmc     reverse Monte Carlo on g(r): Engine.rmc

`exact` gives the same outputs by direct summation (pair list, whole k set,
conjugate gradients to round-off) in torch.float64, without the engine.
"""
import math

import numpy as np
import torch

import mdff_b200
from mdff_b200 import abi, fit, systems

PRESS, TIME, COUL = 0.00624150964712042, 98.2269514139276, 14.3996441494161
MIX, F64 = "mixed", "fp64"


def listed():
    pim = dict(kind="pim", rc=10.0, alpha=0.3, ext=5)
    return [
        # the smallest calls: a 500-atom argon box between two outputs of its
        # trajectory (launches and host round trips per step count)
        dict(name="lj-500-nve", kind="lj", ncell=5, steps=20),
        # the same path with the GPU full
        dict(name="lj-108000-nve", kind="lj", ncell=30, steps=4),
        # one evaluation of a rigid-ion melt with its field gradients, as a
        # single-point calculation makes it
        dict(name="silica-1536-point", kind="silica", n_si=512),
        # a small polarisable cell at constant pressure (the host takes part in each step)
        dict(pim, name="pim-512-npt-fp64", gx=8, gy=8, gz=8, rc=8.0, alpha=0.4, kmax=9, vac=0.0, ens="npt", prec=F64,
             steps=4, ext=0),
        # the elongated 3000-ion cell in NVE
        dict(pim, name="pim-3000-nve-fp64", gx=10, gy=10, gz=30, kmax=10, vac=0.0, ens="nve", prec=F64, steps=4, ext=0),
        # a ragged cell with vacancies, mixed precision, thermostatted
        dict(pim, name="pim-4056-nvt-mixed", gx=16, gy=16, gz=16, kmax=12, vac=0.01, ens="nvt", prec=MIX, steps=4),
        # the 32 440-ion production run in both precisions
        dict(pim, name="pim-32440-nvt-mixed", gx=32, gy=32, gz=32, kmax=23, vac=0.01, ens="nvt", prec=MIX, steps=4),
        dict(pim, name="pim-32440-nvt-fp64", gx=32, gy=32, gz=32, kmax=23, vac=0.01, ens="nvt", prec=F64, steps=2),
        # field gradients along a trajectory: every frame is new to the solver
        dict(pim, name="efg-4056x2-fp64", kind="efg", gx=16, gy=16, gz=16, kmax=12, vac=0.01, prec=F64, frames=2),
        # force matching over 64 ragged configurations of 200 to 2000 ions
        dict(name="fit-64-fp64", kind="fit", nconf=64, nmin=200, nmax=2000, prec=F64),
        # distributions over a trajectory's field gradients, held on the GPU
        dict(name="stat-32440x32", kind="stat", natm=32440, nconf=32),
        # a stretch of a reverse Monte Carlo chain
        dict(name="rmc-32440", kind="rmc", grid=32, vac=0.01, moves=2000),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["lj", "silica", "pim", "pim", "pim", "pim", "efg", "fit", "fit", "stat", "rmc"])
    if kind == "lj":
        n = log_int(4, 30)
        return dict(kind=kind, ncell=n, steps=rng.randint(1, 20 if n < 12 else 4))
    if kind == "silica":
        return dict(kind=kind, n_si=log_int(120, 700))
    if kind in ("pim", "efg"):
        prec = rng.choice([F64, MIX])
        # even site counts per edge: the rock-salt occupation is periodic
        g = [2 * log_int(4, 16 if kind == "pim" else 9) for _ in range(3)]
        L = [4.212 / 2 * v for v in g]
        rc = round(min(10.0, 0.5 * min(L) - 0.01) * rng.uniform(0.85, 1.0), 2)
        alpha = round(3.0 / rc, 3)
        kmax = systems.ewald_kmax_for(alpha, max(L), 1e-7, rc)
        c = dict(kind=kind, gx=g[0], gy=g[1], gz=g[2], rc=rc, alpha=alpha, kmax=max(3, min(kmax, 23)),
                 vac=rng.choice([0.0, 0.01, 0.02]), prec=prec, ext=rng.choice([0, 3, 5]))
        if kind == "efg":
            return dict(c, frames=rng.randint(1, 2))
        return dict(c, ens=rng.choice(["nve", "nvt", "nvt", "npt"]), steps=rng.randint(1, 3))
    if kind == "fit":
        lo = log_int(60, 400)
        return dict(kind=kind, nconf=log_int(3, 48), nmin=lo, nmax=rng.randint(lo + 20, 1600), prec=rng.choice([F64, MIX]))
    if kind == "stat":
        return dict(kind=kind, natm=log_int(301, 32440), nconf=log_int(1, 32))
    return dict(kind=kind, grid=2 * log_int(6, 16), vac=rng.choice([0.0, 0.01]), moves=log_int(200, 2000))


# ---- inputs ------------------------------------------------------------------


def _system(case, seed):
    """The system of a case, with the parameters a run of its kind is given."""
    kind = case["kind"]
    if kind == "lj":
        s = systems.lj_argon(ncell=case["ncell"], seed=seed)
        s["pos"] = s["pos"] + np.random.default_rng(seed).normal(0.0, 0.03, s["pos"].shape)
    elif kind == "silica":
        s = systems.silica_bmh(n_si=case["n_si"], seed=seed)
        s["params"].doefield = s["params"].doefg = 1
    else:
        ens = {"nve": abi.NVE_VV, "nvt": abi.NVT_NHCN, "npt": abi.NPT_NHCNP}[case.get("ens", "nve")]
        s = systems.mgo_pim(grid=(case["gx"], case["gy"], case["gz"]), rc=case["rc"], alpha=case["alpha"],
                            kmax=case["kmax"], vacancy_frac=case["vac"], temp=1500.0 if ens == abi.NPT_NHCNP else 2000.0,
                            seed=seed, integrator=ens)
        p = s["params"]
        p.precision = abi.PREC_MIXED if case["prec"] == MIX else abi.PREC_FP64
        p.kspace_reuse = 1 if case["prec"] == MIX else 0
        p.algo_ext_dipole = abi.EXT_ASPC if case["ext"] else abi.EXT_POLY
        p.extrapolate_order = case["ext"]
        p.efg_period = 10
        p.doefield = 1 if kind == "efg" else 0
        p.autotune = 1
        if ens == abi.NPT_NHCNP:
            p.timesca_baro = 1.0
    return s


def _frames(case, s, seed):
    rng = np.random.default_rng(seed + 1)
    return [dict(natm=len(s["itype"]), cell=s["cell"], r=s["pos"] + rng.normal(0.0, 0.08, s["pos"].shape))
            for _ in range(case["frames"])]


def _fit_inputs(case, seed):
    """Configurations, the force field the targets come from, the starting
    parameters of the fit, and the noise of the targets."""
    # the sizes and densities are the data set's; the seed moves the atoms and the targets
    confs = systems.mgo_batch(nconf=case["nconf"], nmin=case["nmin"], nmax=case["nmax"])
    rng = np.random.default_rng(seed)
    for c in confs:
        c["pos"] = c["pos"] + rng.normal(0.0, 0.05, c["pos"].shape)
    base = systems.mgo_params(6.0, 0.5, 6)
    base.precision = abi.PREC_MIXED if case["prec"] == MIX else abi.PREC_FP64
    rng = np.random.default_rng(seed + 1)
    space = fit.mgo_space(base)
    theta = space.get(base) * (1.0 + rng.uniform(-0.02, 0.02, len(space)))
    noise = [rng.normal(0.0, 0.05, (len(c["itype"]), 3)) for c in confs]
    tau = [np.eye(3) * rng.normal(0.0, 0.2) for _ in confs]
    return confs, base, space, theta, noise, tau


def _stat_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    nc, n = case["nconf"], case["natm"]
    e = torch.randn((nc, 6, n), dtype=torch.float64, device="cuda", generator=g) * 2.0
    e[:, 2] = -(e[:, 0] + e[:, 1])
    d = abi.EfgDistParams()
    d.vzzmin, d.resvzz, d.reseta, d.umin, d.resu, d.smax = -40.0, 40.0 / 150, 0.01, -40.0, 40.0 / 150, 80.0
    itype = np.where(np.arange(n) < n // 2, 1, 2).astype(np.int32)
    return e, d, itype


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fit":
        confs, base, space, theta, noise, tau = _fit_inputs(case, seed)
        b = mdff_b200.Batch(base, confs)
        ref = b.forces()
        b.set_targets([f + e for f, e in zip(ref["f"], noise)], [t + e for t, e in zip(ref["tau"], tau)], 1.0, 0.01)
        return dict(kind=kind, batch=b, base=base, space=space, theta=theta)
    if kind == "stat":
        efg, dist, itype = _stat_inputs(case, seed)
        p = systems.mgo_params(6.0, 0.5, 3)
        pos = np.random.default_rng(seed).random((case["natm"], 3)) * 80.0
        eng = mdff_b200.Engine(p, itype, pos, np.eye(3) * 80.0)
        return dict(kind=kind, eng=eng, efg=efg, dist=dist)
    if kind == "rmc":
        g = case["grid"]
        s = systems.mgo_pim(grid=(g, g, g), rc=10.0, alpha=0.3, kmax=3, vacancy_frac=case["vac"], seed=seed)
        eng = mdff_b200.Engine(s["params"], s["itype"], s["pos"], s["cell"])
        eng.set_positions(s["pos"] + np.random.default_rng(seed + 1).normal(0.0, 0.12, s["pos"].shape))
        gexp = eng.gr(10.0, 0.05)
        eng.set_positions(s["pos"])
        rp = abi.RmcParams()
        rp.max_displacement, rp.resolution_gr, rp.cut_rmc = 0.1, 0.05, 10.0
        for k in range(6):
            rp.temp_rmc[k] = 1e-4
        rp.acceptance_max, rp.max_trials = 10 ** 12, case["moves"] + 1
        return dict(kind=kind, eng=eng, rp=rp, gexp=gexp, seed=seed)
    s = _system(case, seed)
    eng = mdff_b200.Engine(s["params"], s["itype"], s["pos"], s["cell"])
    if kind == "efg":
        return dict(kind=kind, eng=eng, frames=_frames(case, s, seed))
    if kind != "silica":
        eng.md_start(s["vel"])
    return dict(kind=kind, eng=eng, steps=case.get("steps", 0))


THERMO = ("e_kin", "temp_r", "u_tot", "e_tot", "h_tot", "u_lj", "u_bmhft", "u_coul", "u_pol", "pressure_tot")


def run(state):
    kind = state["kind"]
    if kind in ("lj", "pim"):
        out = state["eng"].step(state["steps"])
        th = {k: np.array([t[k] for t in out["thermo"]]) for k in THERMO}
        return dict(pos=out["pos"], vel=state["eng"].velocities(), f=out["f"], **th)
    if kind == "silica":
        out = state["eng"].engforce()
        return dict(f=out["f"], ef=out["ef"], efg=out["efg"], tau_nonb=out["tau_nonb"], tau_coul=out["tau_coul"],
                    u_coul=out["e"]["u_coul"], u_bmhft=out["e"]["u_bmhft"])
    if kind == "efg":
        return dict(efg=state["eng"].efgcalc(state["frames"])[0])
    if kind == "fit":
        theta = torch.tensor(state["theta"], requires_grad=True)
        loss = fit.force_match_loss(theta, state["batch"], state["space"], state["base"])
        loss.backward()
        return dict(loss=loss.detach(), grad=theta.grad)
    if kind == "stat":
        return state["eng"].efg_dist_ptr(state["dist"], state["efg"].data_ptr(), state["efg"].shape[0])
    state["seed"] += 1   # the chain goes on with new random numbers
    res, g = state["eng"].rmc(state["rp"], state["gexp"], seed=state["seed"])
    return dict(kall=res["kall"], kacc=res["kacc"], chisq=np.array(res["chisq"]), g=g, pos=state["eng"].positions())


# ---- what a pass cannot do without ----------------------------------------------


def _neighbours(n, vol, rc):
    return n / vol * 4.0 / 3.0 * math.pi * rc ** 3


def _ewald_work(n, vol, rc, alpha, kmax, evals):
    """Operations of `evals` dipole-field evaluations and the two force passes:
    real space ~50 per unordered pair and field (~150 for forces), reciprocal
    space 15 + 18 per (atom, k) with the vectors exp(-k^2/4 alpha^2) >= 1e-7."""
    pairs = 0.5 * n * _neighbours(n, vol, rc)
    kc = 2.0 * alpha * math.sqrt(-math.log(1e-7))
    k = min(0.5 * vol / (2 * math.pi) ** 3 * 4.0 / 3.0 * math.pi * kc ** 3, 0.5 * (2 * kmax + 1) ** 3)
    return pairs * (50.0 * evals + 200.0) + n * k * 33.0 * (evals + 1.0)


def work(case):
    kind = case["kind"]
    if kind == "lj":
        n = 4 * case["ncell"] ** 3
        return dict(bytes=case["steps"] * n * 8.0 * 18, flops=case["steps"] * n * 0.5 * _neighbours(n, n / 0.844, 2.5) * 40)
    if kind == "silica":
        n = 3 * case["n_si"]
        vol = n / 3 * (systems.MASS_SI + 2 * systems.MASS_O) * systems.AMU_G / 2.2 * 1e24
        return dict(bytes=n * 8.0 * 20, flops=_ewald_work(n, vol, 8.0, 0.35, 8, 0))
    if kind in ("pim", "efg"):
        sites = case["gx"] * case["gy"] * case["gz"]
        vol, n = sites * 2.106 ** 3, sites * (1.0 - case["vac"])
        passes, evals = (case["frames"], 11) if kind == "efg" else (case["steps"], 8)
        return dict(bytes=passes * n * 8.0 * 30, flops=passes * _ewald_work(n, vol, case["rc"], case["alpha"], case["kmax"], evals))
    if kind == "fit":
        n = 0.5 * (case["nmin"] + case["nmax"])
        vol = n / 2 * (systems.MASS_O + systems.MASS_MG) * systems.AMU_G / 3.55 * 1e24
        rc = min(10.0, 0.45 * vol ** (1.0 / 3.0))
        return dict(bytes=case["nconf"] * n * 8.0 * 40, flops=case["nconf"] * _ewald_work(n, vol, rc, 3.2 / rc, 20, 26))
    if kind == "stat":
        return dict(bytes=case["natm"] * (48.0 * case["nconf"] + 4.0), flops=case["natm"] * case["nconf"] * 400.0)
    n = case["grid"] ** 3 * (1.0 - case["vac"])
    return dict(bytes=n * 48.0, flops=case["moves"] * 2.0 * _neighbours(n, n * 2.106 ** 3, 10.0) * 12.0)


# ---- the same outputs in plain 64-bit torch ---------------------------------------


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device=_dev())


def _pair_list(x, box, rc):
    """Ordered pairs (i, j) within rc of one another (minimum image, orthorhombic box)."""
    n, found = len(x), []
    step = max(1, 60_000_000 // n)
    for a in range(0, n, step):
        d2 = torch.zeros((min(step, n - a), n), dtype=torch.float64, device=x.device)
        for k in range(3):
            d = x[a:a + step, k, None] - x[None, :, k]
            d -= box[k] * torch.round(d / box[k])
            d2 += d * d
        i, j = torch.nonzero(d2 <= rc * rc, as_tuple=True)
        keep = i + a != j
        found.append(torch.stack([i[keep] + a, j[keep]]))
    return torch.cat(found, dim=1)


def _image(x, box, ij):
    d = x[ij[0]] - x[ij[1]]
    return d - box * torch.round(d / box)


class _Ionic:
    """Charges and induced dipoles with BMHFTD pairs, by direct summation."""

    def __init__(self, p, itype, x, box, rc, alpha, kmax):
        self.p, self.box, self.rc, self.a, self.kmax = p, _t(box), rc, alpha, list(kmax)
        self.t = torch.as_tensor(np.asarray(itype) - 1, device=_dev(), dtype=torch.int64)
        nt = p.ntype
        self.tab = {k: _t(np.ctypeslib.as_array(getattr(p, k)))[:nt, :nt] for k in
                    ("Abmhftd", "Bbmhftd", "Cbmhftd", "Dbmhftd", "BDbmhftd")}
        self.db, self.dc = (_t(np.ctypeslib.as_array(getattr(p, k)))[:nt, :nt, :nt].clone()
                            for k in ("dip_pol_damp_b", "dip_pol_damp_c"))
        self.dk = torch.as_tensor(np.ctypeslib.as_array(p.dip_pol_damp_k)[:nt, :nt, :nt].copy(), device=_dev())
        for a in range(nt):   # pair tables are given for i <= j
            for b in range(a):
                for tab in self.tab.values():
                    tab[a, b] = tab[b, a]
                for q in range(nt):
                    self.db[q, a, b], self.dc[q, a, b], self.dk[q, a, b] = self.db[q, b, a], self.dc[q, b, a], self.dk[q, b, a]
        self.alpha_t = _t(np.ctypeslib.as_array(p.poldip_iso))[:nt] * _t(np.ctypeslib.as_array(p.ldip_polar))[:nt]
        self.q = _t(np.ctypeslib.as_array(p.qch))[self.t]
        self.damped = p.lbmhftd != 0
        self.selfa2 = 2.0 * alpha ** 3 / math.sqrt(math.pi) / 3.0
        self.move(x)

    def move(self, x, box=None):
        self.x = x
        self.ij = _pair_list(x, self.box, self.rc)
        self.r = _image(x, self.box, self.ij)
        self.mu = torch.zeros_like(x)

    @staticmethod
    def _tt(y, k):
        """sum_{m <= k} y^m / m!, k a tensor of orders."""
        s, term = torch.ones_like(y), torch.ones_like(y)
        for m in range(1, int(k.max()) + 1 if k.numel() else 1):
            term = term * y / m
            s = s + torch.where(k >= m, term, torch.zeros_like(term))
        return s

    def _radial(self, d):
        a, e = self.a, torch.exp(-(self.a * d) ** 2) / math.sqrt(math.pi)
        f0 = torch.erfc(a * d)
        f1 = f0 + 2 * a * d * e
        f2 = f1 + 4.0 / 3.0 * (a * d) ** 3 * e
        f3 = f2 + 8.0 / 15.0 * (a * d) ** 5 * e
        return f0 / d, f1 / d ** 3, 3 * f2 / d ** 5, 15 * f3 / d ** 7

    def _damping(self, d):
        """1 - f of the field of j's charge at i, and of i's at j."""
        ti, tj = self.t[self.ij[0]], self.t[self.ij[1]]
        out = []
        for own in (ti, tj):
            b, c, k = self.db[own, ti, tj], self.dc[own, ti, tj], self.dk[own, ti, tj]
            out.append(c * torch.exp(-b * d) * self._tt(b * d, k))
        return out

    def _pair_u(self, d):
        ti, tj = self.t[self.ij[0]], self.t[self.ij[1]]
        A, B, C, D, BD = (self.tab[k][ti, tj] for k in ("Abmhftd", "Bbmhftd", "Cbmhftd", "Dbmhftd", "BDbmhftd"))
        f6 = f8 = 1.0
        if self.damped:
            e = torch.exp(-BD * d)
            f6, f8 = (1.0 - e * self._tt(BD * d, torch.full_like(ti, k)) for k in (6, 8))
        u = A * torch.exp(-B * d) - C * f6 / d ** 6 - D * f8 / d ** 8
        return torch.where(A != 0.0, u, torch.zeros_like(u))

    def rec(self, q, mu):
        """Reciprocal field and field gradient (xx yy zz xy xz yz), sum A_k |S|^2 and its stress sums."""
        b = 2 * math.pi / self.box
        ph = self.x * b
        kx, ky, kz = self.kmax
        ny, nz = (torch.arange(-k, k + 1, device=self.x.device, dtype=torch.float64) for k in (ky, kz))
        Z = torch.exp(1j * nz[:, None] * ph[:, 2])
        Y = torch.exp(1j * ny[:, None] * ph[:, 1])
        E, G, U, T = 0.0, 0.0, 0.0, 0.0
        K1, K2 = torch.meshgrid(ny * b[1], nz * b[2], indexing="ij")
        for nx in range(kx + 1):
            k0 = nx * b[0]
            kk = k0 ** 2 + K1 ** 2 + K2 ** 2
            keep = torch.ones_like(kk) if nx else ((ny[:, None] > 0) | ((ny[:, None] == 0) & (nz > 0))).double()
            ak = keep * torch.exp(-kk / (4 * self.a ** 2)) / torch.where(kk > 0, kk, torch.ones_like(kk))
            XY = Y * torch.exp(1j * nx * ph[:, 0])
            amp = (q + 1j * (k0 * mu[:, 0])) + 1j * (ny * b[1])[:, None] * mu[:, 1]
            S = (XY * amp) @ Z.T + (XY * (1j * mu[:, 2])) @ (Z * (nz * b[2])[:, None]).T
            W = ak * S.conj()
            kc = 2.0 * (1.0 / torch.where(kk > 0, kk, torch.ones_like(kk)) + 0.25 / self.a ** 2)
            str_ = ak * (S.real ** 2 + S.imag ** 2)
            U = U + str_.sum()
            kv = (k0.expand_as(K1), K1, K2)
            T = T + torch.stack([((1.0 if a == c else 0.0) * str_ - kc * kv[a] * kv[c] * str_).sum()
                                 for a, c in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))])
            m = [XY * ((W * K2 ** j) @ Z) for j in range(3)]
            k1 = (ny * b[1])[:, None]
            E = E + torch.stack([k0 * m[0].imag.sum(0), (k1 * m[0].imag).sum(0), m[1].imag.sum(0)], 1)
            G = G + torch.stack([k0 * k0 * m[0].real.sum(0), (k1 * k1 * m[0].real).sum(0), m[2].real.sum(0),
                                 (k0 * k1 * m[0].real).sum(0), k0 * m[1].real.sum(0), (k1 * m[1].real).sum(0)], 1)
        vol = self.box.prod()
        sc = 8 * math.pi / vol
        return E * sc, G * sc, U * 4 * math.pi / vol, T * 4 * math.pi / vol ** 2

    def _gather(self, v):
        return torch.zeros((len(self.x),) + v.shape[1:], dtype=v.dtype, device=v.device).index_add(0, self.ij[0], v)

    def dip_field(self, mu, A1, B2):
        mj = mu[self.ij[1]]
        e = self.r * ((self.r * mj).sum(1) * B2)[:, None] - mj * A1[:, None]
        return self._gather(e) + self.rec(torch.zeros_like(self.q), mu)[0] + 2 * self.selfa2 * mu

    def charge_field(self):
        d = self.r.norm(dim=1)
        A1 = self._radial(d)[1]
        gi = self._damping(d)[0]
        e = self.r * (self.q[self.ij[1]] * (A1 - gi / d ** 3))[:, None]
        return self._gather(e) + self.rec(self.q, torch.zeros_like(self.x))[0]

    def cg(self, b, x):
        al = self.alpha_t.detach()[self.t][:, None]
        pol = al > 0
        ial = torch.where(pol, 1.0 / torch.where(pol, al, torch.ones_like(al)), torch.zeros_like(al))
        _, A1, B2, _ = self._radial(self.r.norm(dim=1))

        def op(v):
            return torch.where(pol, v * ial - self.dip_field(v, A1, B2), torch.zeros_like(v))

        b = torch.where(pol, b, torch.zeros_like(b))
        res = b - op(x)
        z = al * res
        d, rz = z.clone(), (res * z).sum()
        for _ in range(100):
            if res.norm() <= 1e-13 * b.norm():
                break
            Ad = op(d)
            s = rz / (d * Ad).sum()
            x, res = x + s * d, res - s * Ad
            z = al * res
            rz, old = (res * z).sum(), rz
            d = z + rz / old * d
        return x

    def solve(self):
        if float(self.alpha_t.max()) > 0:
            with torch.no_grad():
                self.mu = self.cg(self.charge_field(), self.mu)
        return self.mu

    def forces(self, mu, graph=False):
        """Forces, energies and stress sums at given dipoles."""
        r = self.r.detach().clone().requires_grad_(True)
        i, j = self.ij
        d = r.norm(dim=1)
        f0, A1, B2, _ = self._radial(d)
        rmi, rmj, mimj = (r * mu[i]).sum(1), (r * mu[j]).sum(1), (mu[i] * mu[j]).sum(1)
        qi, qj = self.q[i], self.q[j]
        gi, gj = self._damping(d)
        ud = 0.5 * (qi * qj * f0 - (rmi * rmj * B2 - mimj * A1) + (qi * rmj - qj * rmi) * A1
                    - qi * gj * rmj / d ** 3 + qj * gi * rmi / d ** 3).sum()
        up = 0.5 * self._pair_u(d).sum()
        gd, gp = (torch.autograd.grad(u, r, create_graph=graph, retain_graph=True)[0] for u in (ud, up))
        E, G, ur, tr = self.rec(self.q, mu)
        Gm = torch.stack([(G[:, [0, 3, 4]] * mu).sum(1), (G[:, [3, 1, 5]] * mu).sum(1), (G[:, [4, 5, 2]] * mu).sum(1)], 1)
        f = self._gather(-2 * gp) + COUL * (self._gather(-2 * gd) + self.q[:, None] * E + Gm)
        vol = self.box.prod()

        def stress(g):
            return torch.stack([(r.detach()[:, a] * -g[:, b] + r.detach()[:, b] * -g[:, a]).sum()
                                for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))]) * 0.5 / vol

        tn, tc = stress(gp) / PRESS, (stress(gd) + tr) * COUL / PRESS
        al = self.alpha_t[self.t]
        upol = 0.5 * ((mu * mu).sum(1)[al > 0] / al[al > 0]).sum()
        us = -self.a / math.sqrt(math.pi) * (self.q ** 2).sum() - self.selfa2 * (mu ** 2).sum()
        return dict(f=f, tn=tn, tc=tc, u_pair=up, u_coul=COUL * (ud + ur + us + upol), u_pol=COUL * upol, E=E, G=G)

    def efg(self, mu, out):
        """Field and field gradient (energy units for the gradient) from forces()'s reciprocal part."""
        r, (i, j) = self.r, self.ij
        _, A1, B2, C3 = self._radial(r.norm(dim=1))
        gi = self._damping(r.norm(dim=1))[0]
        qj, mj = self.q[j], mu[j]
        rm = (r * mj).sum(1)
        e = r * (qj * (A1 - gi / r.norm(dim=1) ** 3) + rm * B2)[:, None] - mj * A1[:, None]
        g = []
        for a, c in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)):
            v = -(qj * B2 + rm * C3) * r[:, a] * r[:, c] + (r[:, a] * mj[:, c] + r[:, c] * mj[:, a]) * B2
            g.append(v + (qj * A1 + rm * B2 if a == c else 0.0))
        G = self._gather(torch.stack(g, 1)) + out["G"]
        G[:, :3] -= 2 * self.selfa2 * self.q[:, None]
        return self._gather(e) + out["E"] + 2 * self.selfa2 * mu, G * COUL


def _mat(t6):
    return torch.stack([t6[[0, 3, 4]], t6[[3, 1, 5]], t6[[4, 5, 2]]])


def _lj_forces(x, box, ij, p):
    r = _image(x, box, ij)
    d2 = (r * r).sum(1)
    ins = d2 < p.cutshortrange ** 2
    r, d2, i = r[ins], d2[ins], ij[0][ins]
    s6, c6 = d2 ** -3, p.cutshortrange ** -6
    u = 2.0 * ((s6 * s6 - s6) - (c6 * c6 - c6))           # half of 4 (r^-12 - r^-6), shifted at the cutoff
    w = 24.0 * (2 * s6 * s6 - s6) / d2
    f = torch.zeros_like(x).index_add(0, i, r * w[:, None])
    return f, u.sum(), 0.5 * (w * d2).sum()


def _exact_lj(case, s):
    x, v, box, p = _t(s["pos"]), _t(s["vel"]), _t(np.diag(s["cell"])), s["params"]
    n, dt = len(x), p.dt
    x = x - box * torch.round(x / box)
    ij = _pair_list(x, box, p.cutshortrange + 0.9)
    f, u, vir = _lj_forces(x, box, ij, p)
    th = {k: [] for k in ("e_kin", "temp_r", "u_tot", "e_tot", "h_tot", "u_lj", "pressure_tot")}
    for _ in range(case["steps"]):
        x = x + v * dt + f * (0.5 * dt * dt)
        fo = f
        f, u, vir = _lj_forces(x, box, ij, p)
        v = v + (fo + f) * (0.5 * dt)
        ke = float(0.5 * (v * v).sum())
        th["e_kin"].append(ke / n)
        th["temp_r"].append(2 * ke / (3 * n))
        th["u_tot"].append(float(u) / n)
        th["u_lj"].append(float(u) / n)
        th["e_tot"].append((float(u) + ke) / n)
        th["h_tot"].append((float(u) + ke) / n)
        vol = float(box.prod())
        th["pressure_tot"].append(float(vir) / 3.0 / vol / n + 2 * ke / (3 * n) / vol)
    return dict(pos=x, vel=v, f=f, **{k: np.array(a) for k, a in th.items()})


class _Chain:
    """The Nose-Hoover chain's half step (Suzuki-Yoshida order 3, chain forces kept current)."""

    def __init__(self, p, n):
        self.m, self.kT, self.L, self.dt = p.nhc_n, p.temp * systems.BOLTZ_EV, 3.0 * n, p.dt * TIME
        self.Q = [(p.timesca_thermo * TIME) ** 2 * self.kT * (self.L if k == 0 else 1.0) for k in range(self.m)]
        self.v, self.x, self.mults = [0.0] * self.m, [0.0] * self.m, p.nhc_mults
        w = 1.0 / (2.0 - 2.0 ** (1.0 / 3.0))
        self.w = [w, 1.0 - 2.0 * w, w]

    def _link(self, k, g, dt):
        damp = math.exp(-self.v[k + 1] * dt / 8 / self.Q[k + 1]) if k + 1 < self.m else 1.0
        self.v[k] = (self.v[k] * damp + g * dt / 4) * damp

    def half(self, ke):
        s, v, Q = 1.0, self.v, self.Q
        for _ in range(self.mults):
            for w in self.w:
                dt = w * self.dt / self.mults
                g = [2 * ke * s * s - self.L * self.kT] + [v[k - 1] ** 2 / Q[k - 1] - self.kT for k in range(1, self.m)]
                for k in reversed(range(self.m)):
                    self._link(k, g[k], dt)
                s *= math.exp(-v[0] * dt / 2 / Q[0])
                for k in range(self.m):
                    self.x[k] += v[k] * dt / 2 / Q[k]
                g0 = 2 * ke * s * s - self.L * self.kT
                for k in range(self.m):
                    self._link(k, g0 if k == 0 else v[k - 1] ** 2 / Q[k - 1] - self.kT, dt)
        return s

    def energy(self):
        return (self.L * self.kT * self.x[0] + sum(self.kT * x for x in self.x[1:])
                + sum(v * v / 2 / q for v, q in zip(self.v, self.Q)))


def _ionic(s):
    p = s["params"]
    box = _t(np.diag(s["cell"]))
    x = _t(s["pos"])
    x = x - box * torch.round(x / box)
    return _Ionic(p, s["itype"], x, np.diag(s["cell"]), p.cutlongrange, p.alphaES, p.kES)


def _exact_pim(case, s):
    p, m = s["params"], _ionic(s)
    n, dt = len(m.x), p.dt * TIME
    mass = _t(np.where(s["itype"] == 1, systems.MASS_O, systems.MASS_MG))[:, None]
    v, x = _t(s["vel"]), m.x
    out = m.forces(m.solve())
    chain = _Chain(p, n) if case["ens"] == "nvt" else None
    th = {k: [] for k in THERMO}

    def kin():
        return float(0.5 * (mass * v * v).sum())

    for _ in range(case["steps"]):
        f = out["f"]
        if chain:
            v = v * chain.half(kin())
        v = v + f * (0.5 * dt) / mass
        x = x + v * dt
        mu = m.mu
        m.move(x)
        m.mu = mu
        out = m.forces(m.solve())
        v = v + out["f"] * (0.5 * dt) / mass
        if chain:
            v = v * chain.half(kin())
        ke, up, uc = kin(), float(out["u_pair"]), float(out["u_coul"])
        vol = float(m.box.prod())
        pv = float((out["tn"][:3].sum() + out["tc"][:3].sum()) / 3.0)
        row = dict(e_kin=ke, temp_r=2 * ke / systems.BOLTZ_EV / (3 * n), u_tot=up + uc, e_tot=up + uc + ke,
                   h_tot=up + uc + ke + (chain.energy() if chain else 0.0), u_lj=0.0, u_bmhft=up, u_coul=uc,
                   u_pol=float(out["u_pol"]))
        row["pressure_tot"] = pv + (2 * ke / (3 * n)) / vol / PRESS
        for k in THERMO:
            th[k].append(row[k])
    return dict(pos=x, vel=v, f=out["f"], **{k: np.array(a) for k, a in th.items()})


def _exact_fit(case, seed):
    confs, base, space, theta, noise, tau = _fit_inputs(case, seed)
    start = space.get(base)
    loss, grad = 0.0, torch.zeros(len(theta), dtype=torch.float64, device=_dev())
    for c, ef, et in zip(confs, noise, tau):
        box, B = _t(np.diag(c["cell"])), len(confs)
        x = _t(c["pos"])
        x = x - box * torch.round(x / box)
        m = _Ionic(base, c["itype"], x, np.diag(c["cell"]), c["rc"], c["alpha"], c["kmax"])
        m.r = m.r.contiguous()
        targets = None
        for values in (start, theta):
            th = _t(values).requires_grad_(True)
            named = dict(zip(space.names, th))
            for tab, n in (("Abmhftd", "A"), ("Bbmhftd", "rho"), ("Cbmhftd", "C6"), ("Dbmhftd", "C8")):
                oo, om = named[n + "_OO"], named[n + "_MgO"]
                oo, om = (1.0 / oo, 1.0 / om) if n == "rho" else (oo, om)
                z = torch.zeros_like(oo)
                m.tab[tab] = torch.stack([torch.stack([oo, om]), torch.stack([om, z])])
            m.tab["BDbmhftd"] = torch.where(m.tab["Abmhftd"].detach() != 0, named["b_disp"], m.tab["Abmhftd"].detach() * 0)
            on = torch.as_tensor(np.ctypeslib.as_array(base.ldip_damping)[:2, :2, :2].copy() != 0, device=_dev())
            on = on | on.transpose(1, 2)
            m.db, m.dc = (torch.where(on, named[k], torch.zeros_like(named[k])) for k in ("b_dip", "c_dip"))
            m.alpha_t = torch.stack([named["alpha_O"], torch.zeros_like(named["alpha_O"])])
            mu = m.solve().detach().requires_grad_(True)
            o = m.forces(mu, graph=True)
            tt = _mat(o["tn"] + o["tc"])
            if targets is None:
                targets = o["f"].detach() + _t(ef), tt.detach() + _t(et)
                continue
            L = (((o["f"] - targets[0]) ** 2).sum() / (3.0 * len(x) * B) + 0.01 / (9.0 * B) * ((tt - targets[1]) ** 2).sum())
            gt, gm = torch.autograd.grad(L, (th, mu), retain_graph=True)
            with torch.no_grad():
                lam = m.cg(gm, torch.zeros_like(gm))
            al = m.alpha_t[m.t][:, None]
            inv = torch.where(al > 0, mu.detach() / torch.where(al > 0, al, torch.ones_like(al)), torch.zeros_like(mu))
            grad += gt + torch.autograd.grad((lam * (m.charge_field() - inv)).sum(), th)[0]
            loss += float(L)
    return dict(loss=torch.tensor(loss, dtype=torch.float64), grad=grad)


def _exact_stat(case, seed):
    efg, _, itype = _stat_inputs(case, seed)
    e = efg.transpose(1, 2)
    m = torch.stack([e[..., [0, 3, 4]], e[..., [3, 1, 5]], e[..., [4, 5, 2]]], -2)
    w = torch.as_tensor(np.linalg.eigvalsh(m.cpu().numpy()), device=e.device)
    o = torch.argsort(w.abs(), dim=-1, descending=True)
    vzz, vyy, vxx = (w.gather(-1, o[..., k:k + 1])[..., 0] for k in range(3))
    eta = (vxx - vyy) / vzz
    s3 = 1.0 / math.sqrt(3.0)
    U = torch.stack([e[..., 2] / 2, e[..., 4] * s3, e[..., 5] * s3, e[..., 3] * s3, (e[..., 0] - e[..., 1]) * s3 / 2], -1)
    it = torch.as_tensor(itype, device=e.device)
    rows = [torch.ones_like(it, dtype=torch.bool), it == 1, it == 2]
    nc = case["nconf"]
    stats, mU, m2U = np.zeros((nc, 3, 8)), np.zeros((3, 5)), np.zeros((3, 5, 5))
    for r, sel in enumerate(rows):
        cnt, acc, lo, hi = int(sel.sum()), np.zeros(5), 0.0, 0.0
        u = U[:, sel].reshape(-1, 5)
        mU[r] = u.mean(0).cpu().numpy()
        m2U[r] = np.triu((u.T @ u).cpu().numpy()) / (1.0 if r == 0 else nc * cnt)
        for c in range(nc):   # the reference's loop adds each configuration's sums to the last one's averages
            z, t = vzz[c, sel], eta[c, sel]
            acc = (acc + np.array([float(q) for q in (z.sum(), z.abs().sum(), t.sum(), (z >= 0).sum(), (z * z).sum())])) / cnt
            lo, hi = min(lo, float(z.min())), max(hi, float(z.max()))
            sig = math.sqrt(acc[4] - acc[1] ** 2)
            stats[c, r] = (lo, hi, acc[0], acc[1], acc[2], acc[3], sig / acc[1], sig)
    return dict(stats=stats, mU=mU, m2U=m2U)


def exact(case, seed):
    kind = case["kind"]
    if kind == "rmc" or case.get("ens") == "npt":   # a chain of decisions; a barostat's trajectory
        return None
    if kind == "fit":
        return _exact_fit(case, seed)
    if kind == "stat":
        return _exact_stat(case, seed)
    s = _system(case, seed)
    if kind == "lj":
        return _exact_lj(case, s)
    if kind == "pim":
        return _exact_pim(case, s)
    m = _ionic(s)
    if kind == "silica":
        out = m.forces(m.solve())
        ef, efg = m.efg(m.mu, out)
        return dict(f=out["f"], ef=ef, efg=efg, tau_nonb=_mat(out["tn"]), tau_coul=_mat(out["tc"]),
                    u_coul=float(out["u_coul"]), u_bmhft=float(out["u_pair"]))
    frames = []
    for fr in _frames(case, s, seed):
        x = _t(fr["r"])
        m.move(x - m.box * torch.round(x / m.box))
        out = m.forces(m.solve())
        frames.append(m.efg(m.mu, out)[1])
    return dict(efg=torch.stack(frames))
