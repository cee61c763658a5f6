"""The workloads this framework is measured on, and their exact values.

Every case is a call sequence of a user's program through the public Python entry points
(``Engine``, ``ForceMatchBatch``, ``RDF``), over the systems of ``mdff20_b200.synth`` and
``mdff20_b200.fit``:

* ``lj``     MD of Lennard-Jones argon in reduced units, FP64 NVE (from 256 atoms, where a
             step is launches and latency, to liquids of tens of thousands of atoms);
* ``point``  single points of random silica frames, as a trajectory analysis runs them: new
             positions, new lists, forces, energies and stress (rigid or polarisable ions;
             the induced dipoles start from zero for every frame);
* ``md``     Nose-Hoover-chain MD of polarisable silica between two outputs: a block of
             steps, then the state;
* ``host``   the same MD driven by a host that keeps the state in its own page-locked
             arrays (one call per step, state in and state out);
* ``fit``    one evaluation of the batched force-matching loss and its adjoint gradient at
             a new parameter vector;
* ``rdf``    pair histogram of a few frames handed over as host arrays;
* ``lists``  Verlet lists of a new frame in the reference's CSR form (what the drop-in
             refreshes on every rebuild).

The mixed-precision path carries FP32 accuracy in its double arrays; its results are
returned as float32, the precision a program stores them with.  ``exact`` evaluates the
same model in 64 bits with plain torch operations (direct sums over pairs and k-vectors,
tightly converged dipoles, autograd for the fit's gradient).
"""
from __future__ import annotations

import functools
import math
import os

import numpy as np
import torch

# the fit keeps one stream per configuration in flight (as bench.py and the fit's users set it)
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")

from mdff20_b200 import fit, synth  # noqa: E402
from mdff20_b200.engine import FP64, MIXED, PIM_CG, PIM_CG_FUSED, Engine  # noqa: E402
from mdff20_b200.rdf import RDF, reference_grid  # noqa: E402
from mdff20_b200.system import BOLTZ_UNIT, COUL_UNIT, PRESS_UNIT, TIME_UNIT  # noqa: E402

EQUIL = 6          # MD steps behind the program when a pass begins (the dipole predictor is at its order)
O, SI = synth.O, synth.SI


# ---------------------------------------------------------------------------- cases
def listed():
    return [
        # the LJ argon benchmark itself: 256 atoms, the smallest step there is
        dict(name="lj_md_256_fp64", kind="lj", ncell=4, steps=20),
        # a liquid of ordinary size (15^3 fcc cells), lists rebuilt as atoms move
        dict(name="lj_md_13500_fp64", kind="lj", ncell=15, steps=20),
        # rigid-ion silica, 3000 ions, mixed precision: a frame of a rigid trajectory
        dict(name="rigid_point_3000_mixed", kind="point", n_si=1000, pim=False, mixed=True, kmax=12),
        # polarisable silica, 6000 ions, FP64, dipoles to 1e-8: the reference-quality single point
        dict(name="pim_point_6000_fp64", kind="point", n_si=2000, pim=True, mixed=False, kmax=14),
        # a small cell, as force fields are tried out on: 192 ions, FP64
        dict(name="pim_md_192_fp64", kind="md", cells=2, removed=0, mixed=False, steps=20),
        # FP64 production MD of moderate size
        dict(name="pim_md_3000_fp64", kind="md", cells=5, removed=0, mixed=False, steps=5),
        # the large polarisable NVT run in mixed precision (the headline system)
        dict(name="pim_md_24000_mixed", kind="md", cells=10, removed=0, mixed=True, steps=10),
        # a host program that owns the state: one step per call, a ragged ion count (vacancies)
        dict(name="pim_host_5175_mixed", kind="host", cells=6, removed=3, mixed=True, steps=1),
        # batched force matching in mixed precision, uneven configurations of 96..1536 ions
        dict(name="fit_48_mixed", kind="fit", nconf=48, mixed=True),
        # the FP64 fit it is checked against, fewer configurations
        dict(name="fit_12_fp64", kind="fit", nconf=12, mixed=False),
        # g(r) of two frames of the large system
        dict(name="rdf_24000", kind="rdf", cells=10, removed=0, resg=0.1, frames=2),
        # CSR lists of a 6000-ion frame (short range and Coulomb)
        dict(name="lists_6000", kind="lists", n_si=2000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lj", "point", "md", "host", "fit", "rdf", "lists"])
    if kind == "lj":
        return dict(kind="lj", ncell=rng.randint(4, 15), steps=rng.randint(5, 20))
    if kind == "point":
        pim = rng.random() < 0.6
        mixed = rng.random() < 0.5
        return dict(kind="point", n_si=_log(rng, 64, 2000), pim=pim, mixed=mixed, kmax=rng.randint(9, 14))
    if kind == "md":
        mixed = rng.random() < 0.5
        cells = rng.randint(2, 9) if mixed else rng.randint(2, 5)
        return dict(kind="md", cells=cells, removed=rng.randint(0, cells), mixed=mixed, steps=rng.randint(3, 9))
    if kind == "host":
        return dict(kind="host", cells=rng.randint(4, 8), removed=rng.randint(0, 40), mixed=rng.random() < 0.7, steps=1)
    if kind == "fit":
        mixed = rng.random() < 0.6
        return dict(kind="fit", nconf=_log(rng, 4, 40) if mixed else _log(rng, 3, 11), mixed=mixed)
    if kind == "rdf":
        cells = rng.randint(2, 9)
        return dict(kind="rdf", cells=cells, removed=rng.randint(0, 2 * cells), resg=rng.choice([0.02, 0.05, 0.1]),
                    frames=rng.randint(1, 3))
    return dict(kind="lists", n_si=_log(rng, 64, 2000))


# ---------------------------------------------------------------------------- systems
@functools.lru_cache(maxsize=None)
def _packing(n_si, lo):
    """A random packing (no contact below `lo`: all pairs, or the polarisable table)."""
    return synth.silica(n_si, seed=7, dmin=synth.PIM_DMIN if lo == "pim" else lo, velocities=False)


@functools.lru_cache(maxsize=None)
def _fit_base(c, n):
    return fit.config4_one(c, n)


def _moved(s, rng, rms):
    s = s.copy()
    s.pos = s.pos + rms * rng.standard_normal(s.pos.shape)
    s.pos -= s.cell[0, 0] * np.round(s.pos / s.cell[0, 0])
    return s


def _ewald(s, kmax, skin):
    """rc 10 A, alpha 0.32 where the cell holds them (the benchmark systems), tuned values in smaller cells."""
    L = float(s.cell[0, 0])
    s.skindiff = skin
    if L >= 2.0 * (10.0 + skin):
        s.cutlongrange, s.cutshortrange, s.alphaES, s.kES = 10.0, 7.0, 0.32, (kmax,) * 3
    else:
        ch = fit.ewald_tune(L, s.nion, skin=skin)
        s.cutlongrange, s.cutshortrange, s.alphaES, s.kES = ch.rc, min(7.0, ch.rc), ch.alpha, (ch.kmax,) * 3
    return s


def _point_system(case, seed):
    rng = np.random.default_rng(seed)
    s = _moved(_packing(case["n_si"], "pim" if case["pim"] else 1.4), rng, 0.01)
    if case["pim"]:
        s.polit = np.zeros((2, 3, 3))
        s.polit[O] = np.eye(3)
        s.poldamp = [(O, O, O, 2.0, 1.0, 4), (O, O, SI, 2.0, 1.0, 4)]
        s.conv_tol_ind = 1e-6 if case["mixed"] else 1e-8
    s.integrator = "nve-vv"
    return _ewald(s, case["kmax"], 1.0)


def _md_system(case, seed):
    cells, removed = case["cells"], case["removed"]
    temp = 300.0 if removed else 2500.0 if cells >= 5 else 1000.0
    s = synth.silica(8 * cells ** 3, seed=seed, polarizable=True, kmax=14, temp=temp, conv_tol=1e-6,
                     extrapolate_order=4, dmin=synth.PIM_DMIN, structure="cristobalite")
    if removed:   # whole SiO2 units taken out (a Si and two O next to it): ragged ion counts
        rng = np.random.default_rng(seed)
        n_o, n_si = s.nionit
        L = float(s.cell[0, 0])
        keep = np.ones(s.nion, bool)
        for si in n_o + rng.choice(n_si, removed, replace=False):
            d = s.pos[:n_o] - s.pos[si]
            d2 = ((d - L * np.round(d / L)) ** 2).sum(1)
            d2[~keep[:n_o]] = np.inf
            keep[np.argsort(d2, kind="stable")[:2]] = False
            keep[si] = False
        s.pos, s.vel, s.nionit = s.pos[keep], s.vel[keep], [n_o - 2 * removed, n_si - removed]
    return _ewald(s, 14, 1.0)


def _lj_system(case, seed):
    return synth.lj_fcc(ncell=case["ncell"], seed=seed)


def _fit_sizes(nconf):
    return fit.config4_sizes(nconf)


def _fit_systems(case, seed):
    rng = np.random.default_rng(seed)
    sizes = _fit_sizes(case["nconf"])
    return [_moved(_fit_base(c, n), rng, 0.01) for c, n in enumerate(sizes)]


def _fit_thetas(th0, seed):
    """Parameters along a fit: seeded 1% steps, the first used for the recording in prepare."""
    rng = np.random.default_rng(seed + 1)
    return [th0 * (1.0 + 0.01 * rng.standard_normal(len(th0))) for _ in range(5)]


# ---------------------------------------------------------------------------- the passes
def _as(case, x):
    return np.asarray(x, np.float32) if case.get("mixed") else np.asarray(x, np.float64)


def _engine(case, s):
    e = Engine(s, precision=MIXED if case.get("mixed") else FP64,
               pim_solver=PIM_CG_FUSED if case.get("mixed") else PIM_CG)
    e.gen_verletlist()
    return e


def _pinned(n):
    t = torch.zeros(n, dtype=torch.float64)
    return (t.pin_memory() if torch.cuda.is_available() else t).numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("lj", "md", "host"):
        s = _lj_system(case, seed) if kind == "lj" else _md_system(case, seed)
        e = _engine(case, s)
        e.engforce()
        e.md_steps(1, EQUIL, record=False)
        st = dict(case=case, e=e, step=EQUIL + 1)
        if kind == "host":
            st["host"] = [_pinned(s.nion) for _ in range(9)]
            e.state_soa(*st["host"])
        return st
    if kind == "point":
        s = _point_system(case, seed)
        e = _engine(case, s)
        return dict(case=case, e=e, pos=s.pos, zero=np.zeros((s.nion, 6, 3)))
    if kind == "fit":
        systems = _fit_systems(case, seed)
        th0 = fit.theta_of(systems[0])
        b = fit.ForceMatchBatch(systems, None, precision=FP64)
        b.set_targets(b.forces(fit.perturbed_theta(th0)))
        b.set_precision(MIXED if case["mixed"] else FP64)
        thetas = _fit_thetas(th0, seed)
        b.loss_grad(thetas[0])
        return dict(case=case, batch=b, thetas=thetas, k=1)
    if kind == "rdf":
        frames = [_md_system(dict(case, mixed=False), seed * 16 + f) for f in range(case["frames"])]
        cut, _ = reference_grid(frames[0].cell)
        return dict(case=case, cell=frames[0].cell, frames=[f.pos for f in frames],
                    rdf=RDF(frames[0].nionit, cut, case["resg"]))
    # the caller's CSR arrays have a fixed capacity (the mean count within rc + skin and a quarter more)
    s = _point_system(dict(case, pim=False, mixed=False, kmax=12), seed)
    caps = [int(0.625 * s.nion * (s.nion / s.volume() * 4.0 / 3.0 * math.pi * (rc + s.skindiff) ** 3)) + 1024
            for rc in (s.cutshortrange, s.cutlongrange)]
    return dict(case=case, e=_engine(case, s), pos=s.pos, lists=[np.zeros(c, np.int32) for c in caps])


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind in ("lj", "md"):
        th = st["e"].md_steps(st["step"], case["steps"])
        st["step"] += case["steps"]
        pos, vel, f = st["e"].state()
        return dict(pos=_as(case, pos), vel=_as(case, vel), force=_as(case, f), energies=_as(case, th[:, :9]))
    if kind == "host":
        h = st["host"]
        th = st["e"].md_steps_host(st["step"], 1, h[:6], h)
        st["step"] += 1
        x = _as(case, h)
        return dict(pos=x[0:3], vel=x[3:6], force=x[6:9], energies=_as(case, th[:, :9]))
    if kind == "point":
        e = st["e"]
        e.set_positions(st["pos"])
        e.gen_verletlist()
        if case["pim"]:
            e.set_dipole_history(st["zero"])
        e.engforce()
        t = e.thermo()
        out = dict(force=_as(case, e.forces()), energy=_as(case, [t["u_bhmftd"], t["u_coul"], t["u_pol"]]),
                   stress=_as(case, [t["tau_bhmftd"], t["tau_coul"]]))
        if case["pim"]:
            out["dipoles"] = _as(case, e.dipole_history()[:, 0])
        return out
    if kind == "fit":
        loss, grad = st["batch"].loss_grad(st["thetas"][st["k"]])
        st["k"] = 1 + st["k"] % (len(st["thetas"]) - 1)
        return dict(loss=_as(case, loss), grad=_as(case, grad))
    if kind == "rdf":
        st["rdf"].reset()
        for pos in st["frames"]:
            st["rdf"].add(st["cell"], pos)
        counts, _ = st["rdf"].counts()
        return counts
    e = st["e"]
    e.set_positions(st["pos"])
    e.gen_verletlist()
    out = {}
    for which, name in enumerate(("sr", "co")):
        point, lst = e.verletlist(which)
        st["lists"][which][:len(lst)] = lst
        out["point_" + name], out["list_" + name] = point, st["lists"][which]
    return out


# ---------------------------------------------------------------------------- work
def _silica_flops(n, L, rc_sr, rc_lr, nk, pim, iters):
    """One force evaluation: half-list pairs within the cutoffs and the k sums, plus the
    dipole iterations (a pass over polarisable pairs and both k sums at the O ions)."""
    rho = n / L ** 3
    pairs = lambda rc: 0.5 * n * rho * 4.0 / 3.0 * math.pi * rc ** 3  # noqa: E731
    f = 60.0 * pairs(rc_sr) + (200.0 if pim else 60.0) * pairs(rc_lr) + n * nk * (8.0 + 12.0 if pim else 4.0 + 6.0)
    return f + iters * (4.0 / 9.0 * pairs(rc_lr) * 18.0 + 2.0 / 3.0 * n * nk * 16.0)


def work(case):
    kind = case["kind"]
    if kind == "lj":
        n = 4 * case["ncell"] ** 3
        pairs = 0.5 * n * 0.8442 * 4.0 / 3.0 * math.pi * 2.5 ** 3
        return dict(bytes=8.0 * n * (9 + 9), flops=case["steps"] * (30.0 * pairs + 40.0 * n))
    if kind in ("md", "host"):
        s = _md_system(case, 1)
        nk, it = s.nk(), 2.6 if case["mixed"] else 3.0
        f = _silica_flops(s.nion, s.cell[0, 0], s.cutshortrange, s.cutlongrange, nk, True, it)
        return dict(bytes=8.0 * s.nion * (9 + 9), flops=case["steps"] * f)
    if kind == "point":
        s = _point_system(case, 1)
        it = 0.0 if not case["pim"] else 6.0 if case["mixed"] else 9.0
        return dict(bytes=8.0 * s.nion * 9,
                    flops=_silica_flops(s.nion, s.cell[0, 0], s.cutshortrange, s.cutlongrange, s.nk(), case["pim"], it))
    if kind == "fit":
        f = b = 0.0
        for n in _fit_sizes(case["nconf"]):
            L = (n / fit.NUMBER_DENSITY) ** (1.0 / 3.0)
            ch = fit.ewald_tune(L, n)
            nk = ch.kmax + ch.kmax * (2 * ch.kmax + 1) + ch.kmax * (2 * ch.kmax + 1) ** 2
            # forces, the sensitivities (about twice a force evaluation), forward and adjoint iterations
            f += 3.0 * _silica_flops(n, L, min(7.0, ch.rc), ch.rc, nk, True, 0.0)
            f += _silica_flops(n, L, 0.0, ch.rc, nk, True, 12.0) - _silica_flops(n, L, 0.0, ch.rc, nk, True, 0.0)
            b += 8.0 * 6 * n
        return dict(bytes=b, flops=f)
    if kind == "rdf":
        n = 24 * case["cells"] ** 3 - 3 * case["removed"]
        return dict(bytes=24.0 * n * case["frames"], flops=case["frames"] * 0.5 * n * n * 20.0)
    n = 3 * case["n_si"]
    s = _point_system(dict(case, pim=False, mixed=False, kmax=12), 1)
    rho = n / s.cell[0, 0] ** 3
    m = sum(0.5 * n * rho * 4.0 / 3.0 * math.pi * (rc + 1.0) ** 3 for rc in (s.cutshortrange, s.cutlongrange))
    return dict(bytes=24.0 * n + 4.0 * (m + 2 * n), flops=20.0 * m)


# ---------------------------------------------------------------------------- exact values
class _Silica:
    """(Polarisable) silica in 64 bits: Buckingham pairs plus the Ewald sum of charges and
    Tang-Toennies damped dipoles, by direct sums.  theta: the fit's parameter tensor."""

    def __init__(self, s, theta=None):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda x: torch.as_tensor(np.asarray(x, float), device=self.dev)  # noqa: E731
        self.s, self.L, self.alpha = s, float(s.cell[0, 0]), s.alphaES
        self.th = t(fit.theta_of(s) if s.polit is not None else self._rigid_theta(s)) if theta is None else theta
        self.isO = torch.as_tensor(s.typia() == O, device=self.dev)
        self.pim = s.polit is not None
        K = s.kES[0]
        g = torch.arange(-K, K + 1, dtype=torch.float64, device=self.dev)
        k = torch.cartesian_prod(g, g, g)
        half = (k[:, 0] > 0) | ((k[:, 0] == 0) & ((k[:, 1] > 0) | ((k[:, 1] == 0) & (k[:, 2] > 0))))
        # the half box of the reference: all (ny, nz) for nx > 0, ny > 0 (all nz) and nz > 0 for nx = 0,
        # with nz < 0 kept for ny > 0 (and ny < 0 for nx > 0): exactly one of each +-k pair
        self.k = k[half] * (2.0 * math.pi / self.L)
        kk = (self.k ** 2).sum(1)
        self.Ak = torch.exp(-kk / (4.0 * self.alpha ** 2)) / kk
        self.kk = kk
        self.pref = 4.0 * math.pi / self.L ** 3

    @staticmethod
    def _rigid_theta(s):
        A, B, C = s.Abhmftd, s.Bbhmftd, s.Cbhmftd
        return [A[SI, O], B[SI, O], C[SI, O], A[O, O], B[O, O], C[O, O], s.qit[SI], 1.0, 0.0, 0.0, 0.0, 0.0]

    def charges(self):
        return torch.where(self.isO, -0.5 * self.th[6], self.th[6])

    def place(self, r):
        """Pairs (i < j) within the larger cutoff at positions r, and the phases."""
        n, rc = r.shape[0], max(self.s.cutlongrange, self.s.cutshortrange)
        ii, jj = [], []
        step = max(1, 20_000_000 // n)
        for a in range(0, n, step):
            d = r[a:a + step, None, :] - r[None, :, :]
            d -= self.L * torch.round(d / self.L)
            i, j = torch.nonzero((d ** 2).sum(2) <= rc * rc, as_tuple=True)
            i = i + a
            m = i < j
            ii.append(i[m])
            jj.append(j[m])
        self.i, self.j = torch.cat(ii), torch.cat(jj)
        self.r = r
        ph = r @ self.k.T
        self.C, self.S = torch.cos(ph), torch.sin(ph)

    def vectors(self, r):
        d = r[self.i] - r[self.j]
        return d - self.L * torch.round(d.detach() / self.L)

    def short(self, x):
        """Buckingham energy of the pair vectors."""
        d2 = (x ** 2).sum(1)
        oi, oj = self.isO[self.i], self.isO[self.j]
        oo, so = oi & oj, oi ^ oj
        u = x.new_zeros(())
        for m, p, dd in ((so, 0, 10), (oo, 3, 11)):
            m = m & (d2.detach() < self.s.cutshortrange ** 2)
            d = d2[m].sqrt()
            A, B, C = self.th[p], self.th[p + 1], self.th[p + 2]
            u = u + (A * torch.exp(-B * d) - C / d ** 6 - self.th[dd] / d ** 8).sum()
        return u

    def real(self, x, mu):
        """Real-space electrostatic energy of the pair vectors and dipoles."""
        m = (x.detach() ** 2).sum(1) <= self.s.cutlongrange ** 2
        x, i, j = x[m], self.i[m], self.j[m]
        q, a = self.charges(), self.alpha
        d2 = (x ** 2).sum(1)
        d = d2.sqrt()
        e = torch.exp(-a * a * d2) / math.sqrt(math.pi)
        F0 = torch.erfc(a * d)
        u = (q[i] * q[j] * F0 / d).sum()
        if not self.pim:
            return u
        F1 = F0 + 2.0 * a * d * e
        F2 = F1 + 4.0 * a ** 3 * d ** 3 * e / 3.0
        b, c = self.th[8], self.th[9]
        br = b * d
        tt = 1.0 - c * torch.exp(-br) * (1.0 + br * (1.0 + br / 2.0 * (1.0 + br / 3.0 * (1.0 + br / 4.0))))
        mi, mj = (x * mu[i]).sum(1), (x * mu[j]).sum(1)
        d3 = d2 * d
        u = u + (-(F1 - 1.0 + tt) / d3 * (q[j] * mi - q[i] * mj)).sum()
        return u - (3.0 * F2 / (d3 * d2) * mi * mj - F1 / d3 * (mu[i] * mu[j]).sum(1)).sum()

    def rho(self, mu, C, S):
        q = self.charges()
        re, im = C.T @ q, S.T @ q
        if self.pim:
            re = re - ((S.T @ mu) * self.k).sum(1)
            im = im + ((C.T @ mu) * self.k).sum(1)
        return re, im

    def recip(self, mu, C, S):
        re, im = self.rho(mu, C, S)
        q, a = self.charges(), self.alpha
        return self.pref * (self.Ak * (re ** 2 + im ** 2)).sum() - a / math.sqrt(math.pi) * (
            (q ** 2).sum() + 2.0 * a * a / 3.0 * (mu ** 2).sum())

    def elastic(self, mu):
        return 0.5 * (mu ** 2).sum() / self.th[7]

    def residual(self, mu, x):
        """dU/dmu at the O ions (alpha^-1 mu - E), zero elsewhere."""
        mu = mu.detach().requires_grad_(True)
        u = self.real(x, mu) + self.recip(mu, self.C, self.S) + self.elastic(mu)
        return torch.autograd.grad(u, mu)[0] * self.isO[:, None]

    def solve(self, b, x, start=None, tol=1e-13):
        """A y = b over the O ions; A = alpha^-1 - T (conjugate gradient)."""
        with torch.no_grad():
            zero = torch.zeros_like(b)
        base = self.residual(zero, x)
        apply = lambda y: self.residual(y, x) - base  # noqa: E731
        y = torch.zeros_like(b) if start is None else start.clone()
        r = b - apply(y)
        p, rr, stop = r.clone(), (r * r).sum(), tol ** 2 * (b * b).sum()
        for _ in range(200):
            if rr <= stop:
                break
            Ap = apply(p)
            al = rr / (p * Ap).sum()
            y, r = y + al * p, r - al * Ap
            new = (r * r).sum()
            p, rr = r + new / rr * p, new
        return y

    def dipoles(self, start=None):
        with torch.no_grad():
            x = self.vectors(self.r)
        if not self.pim:
            return torch.zeros_like(self.r)
        b = -self.residual(torch.zeros_like(self.r), x)
        return self.solve(b, x, start)

    def evaluate(self, r, start=None):
        """Forces, dipoles, energies (u_bh, u_coul, u_pol) and stress tensors (bh, coul)."""
        self.place(r)
        mu = self.dipoles(start)
        x = self.vectors(r).requires_grad_(True)
        V = 1.0 / (self.L ** 3 * PRESS_UNIT)
        ub, ur = self.short(x), self.real(x, mu)
        gb = torch.autograd.grad(ub, x, retain_graph=True)[0]
        gr = torch.autograd.grad(ur, x)[0] * COUL_UNIT
        with torch.no_grad():
            f = torch.zeros_like(r)
            f.index_add_(0, self.i, -(gb + gr))
            f.index_add_(0, self.j, gb + gr)
            re, im = self.rho(mu, self.C, self.S)
            q, k = self.charges(), self.k
            w1 = self.C @ (self.Ak * im)[:, None].mul(k) - self.S @ (self.Ak * re)[:, None].mul(k)
            fr = -q[:, None] * w1
            if self.pim:
                kk = (k[:, :, None] * k[:, None, :]).reshape(-1, 9)
                w2 = self.C @ (self.Ak * re)[:, None].mul(kk) + self.S @ (self.Ak * im)[:, None].mul(kk)
                fr = fr + torch.einsum("nab,nb->na", w2.reshape(-1, 3, 3), mu)
            f += 2.0 * self.pref * COUL_UNIT * fr
            amp = self.Ak * (re ** 2 + im ** 2)
            kco = 2.0 / self.kk + 0.5 / self.alpha ** 2
            tr = torch.eye(3, dtype=f.dtype, device=f.device) * amp.sum() - torch.einsum(
                "k,ka,kb->ab", kco * amp, k, k)
            sym = lambda t: 0.5 * (t + t.T)  # noqa: E731
            tb = sym(-(x.T @ gb)) * V
            tc = (sym(-(x.T @ gr)) + self.pref * COUL_UNIT * tr) * V
            u = torch.stack([ub, (ur + self.recip(mu, self.C, self.S)) * COUL_UNIT,
                             self.elastic(mu) * COUL_UNIT])
        return f, mu, u.detach(), torch.stack([tb, tc]).detach()

    def fit_terms(self, r, target):
        """sum |F - F_t|^2 and its gradient in theta (dipoles at their solution)."""
        th = self.th.detach().clone().requires_grad_(True)
        self.place(r)
        with torch.no_grad():
            xs = self.vectors(r)
        mu = self.dipoles()
        self.th = th
        mg, rg = mu.clone().requires_grad_(True), r.clone().requires_grad_(True)
        x = self.vectors(rg)
        ph = rg @ self.k.T
        U = self.short(x) + COUL_UNIT * (self.real(x, mg) + self.recip(mg, torch.cos(ph), torch.sin(ph)))
        F = -torch.autograd.grad(U, rg, create_graph=True)[0]
        sq = ((F - target) ** 2).sum()
        gth, smu = torch.autograd.grad(sq, (th, mg))
        lam = self.solve(smu * self.isO[:, None], xs)
        R = torch.autograd.grad(self.real(xs, mg) + self.recip(mg, self.C, self.S) + self.elastic(mg), mg,
                                create_graph=True)[0]
        gth = gth - torch.autograd.grad((lam.detach() * R).sum(), th)[0]
        self.th = th.detach()
        return sq.detach(), gth

    def forces_of(self, r):
        return self.evaluate(r)[0]


class _Argon:
    def __init__(self, s):
        self.s, self.L = s, float(s.cell[0, 0])
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"

    def evaluate(self, r, start=None):
        n, rc2 = r.shape[0], self.s.cutshortrange ** 2
        f, u, w = torch.zeros_like(r), r.new_zeros(()), r.new_zeros(())
        uc = 4.0 * (1.0 / rc2 ** 6 - 1.0 / rc2 ** 3)
        step = max(1, 20_000_000 // n)
        for a in range(0, n, step):
            d = r[a:a + step, None, :] - r[None, :, :]
            d -= self.L * torch.round(d / self.L)
            d2 = (d ** 2).sum(2)
            i, j = torch.nonzero((d2 < rc2) & (d2 > 0.0), as_tuple=True)
            x, i6 = d[i, j], 1.0 / d2[i, j] ** 3
            g = (24.0 * (2.0 * i6 * i6 - i6) / d2[i, j])[:, None] * x
            f.index_add_(0, i + a, g)
            u = u + 0.5 * (4.0 * (i6 * i6 - i6) - uc).sum()
            w = w + 0.5 * (x * g).sum()
        return f, None, u, w


def _chain(v, mass, xi, vxi, Q, dt, temp, L, mults):
    """One Nose-Hoover-chain half step (Yoshida order 3), with the reference's sweeps."""
    kin = 0.5 * float((mass[:, None] * v * v).sum())
    nn = len(xi)
    w0 = 1.0 / (2.0 - 2.0 ** (1.0 / 3.0))
    s, G = 1.0, [0.0] * nn
    G[0] = 2.0 * kin - L * temp
    for _ in range(mults):
        for w in (w0, 1.0 - 2.0 * w0, w0):
            dts = w * dt / mults
            d2, d4, d8 = dts / 2, dts / 4, dts / 8
            G[nn - 1] = vxi[nn - 2] ** 2 / Q[nn - 2] - temp
            vxi[nn - 1] += G[nn - 1] * d4

            def kick(h):
                vxi[h] *= math.exp(-vxi[h + 1] * d8 / Q[h + 1])
                vxi[h] += G[h] * d4
                vxi[h] *= math.exp(-vxi[h + 1] * d8 / Q[h + 1])

            for h in range(nn - 2, -1, -1):
                kick(h)
            s *= math.exp(-vxi[0] * d2 / Q[0])
            for h in range(nn):
                xi[h] += vxi[h] * d2 / Q[h]
            G[0] = 2.0 * kin * s * s - L * temp
            for h in range(nn - 2):
                kick(h)
                G[h + 1] = vxi[h] ** 2 / Q[h] - temp
            vxi[nn - 1] += G[nn - 1] * d4
    return v * s


def _exact_md(case, seed):
    lj = case["kind"] == "lj"
    s = _lj_system(case, seed) if lj else _md_system(case, seed)
    model = _Argon(s) if lj else _Silica(s)
    t = lambda x: torch.as_tensor(np.asarray(x, float), device=model.dev)  # noqa: E731
    r, v = t(s.pos), t(s.vel)
    mass = t(np.repeat(s.mass, s.nionit))
    im = 1.0 / mass[:, None]
    f, mu, _, _ = model.evaluate(r)
    rows = []
    if lj:
        dt = s.dt
    else:
        dt, temp, ts = s.dt * TIME_UNIT, s.temp * BOLTZ_UNIT, s.timesca_thermo * TIME_UNIT
        L3 = 3.0 * s.nion
        Q = [ts * ts * temp] * s.nhc_n
        Q[0] *= L3
        xi, vxi = [0.0] * s.nhc_n, [0.0] * s.nhc_n
    for step in range(EQUIL + case["steps"]):
        if lj:
            r = r + v * dt + f * (0.5 * dt * dt) * im
            fn, _, u, w = model.evaluate(r)
            v = v + (f + fn) * (0.5 * dt) * im
            f = fn
            kin = 0.5 * float((mass[:, None] * v * v).sum())
            row = [kin, float(u), 0, 0, 0, 0, float(w) / (3.0 * s.volume()), 0, 0]
        else:
            v = _chain(v, mass, xi, vxi, Q, dt, temp, L3, s.nhc_mults)
            v = v + f * (0.5 * dt) * im
            r = r + v * dt
            f, mu, u, tau = model.evaluate(r, mu)
            v = v + f * (0.5 * dt) * im
            v = _chain(v, mass, xi, vxi, Q, dt, temp, L3, s.nhc_mults)
            kin = 0.5 * float((mass[:, None] * v * v).sum())
            nvt = L3 * temp * xi[0] + sum(0.5 * vxi[h] ** 2 / Q[h] for h in range(s.nhc_n)) + temp * sum(xi[1:])
            pv = [float(torch.trace(tau[c])) / 3.0 for c in (0, 1)]
            row = [kin, 0, float(u[0]), float(u[1]), float(u[2]), nvt, 0, pv[0], pv[1]]
        rows.append(row)
    h = lambda x: (x.T.contiguous() if case["kind"] == "host" else x).cpu()  # noqa: E731
    return dict(pos=h(r), vel=h(v), force=h(f), energies=np.array(rows[EQUIL:], float))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("lj", "md", "host"):
        # about 0.5 s per step at 24000 ions
        return _exact_md(case, seed)
    if kind == "point":
        s = _point_system(case, seed)
        m = _Silica(s)
        f, mu, u, tau = m.evaluate(torch.as_tensor(s.pos, device=m.dev))
        if not case["pim"]:
            u[2] = 0.0
        out = dict(force=f.cpu(), energy=u.cpu(), stress=tau.cpu())
        if case["pim"]:
            out["dipoles"] = mu.cpu()
        return out
    if kind == "fit":
        systems = _fit_systems(case, seed)
        th0 = fit.theta_of(systems[0])
        theta, goal = _fit_thetas(th0, seed)[1], fit.perturbed_theta(th0)
        sq, grad = 0.0, 0.0
        for s in systems:
            m = _Silica(s)
            r = torch.as_tensor(s.pos, device=m.dev)
            m.th = torch.as_tensor(goal, device=m.dev)
            target = m.forces_of(r)
            m.th = torch.as_tensor(theta, device=m.dev)
            a, g = m.fit_terms(r, target)
            sq, grad = sq + a, grad + g
        scale = 1.0 / (3.0 * sum(s.nion for s in systems))
        return dict(loss=(sq * scale).cpu(), grad=(grad * scale).cpu())
    return None   # histograms and lists are whole numbers
