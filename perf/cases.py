"""Performance cases of the GFN1-xTB engine: the evaluations its users run, from one water
molecule to a 300-water cluster and a batch of 4096 molecules, through the public Python API.

A case is a dict of plain values:

* ``kind``     "single" (Gfn1NativeCalculator.calculate, one molecule per call),
               "batch" (BatchCalculator.calculate_flat, host buffers in and out),
               "resident" (ResidentBatch: new coordinates, launch, download),
               "hessian" (hessian.hessian_batch) or "optimize" (ResidentBatch.optimize);
* ``set``      monomers: "water", "mixed" (H2O/NH3/CH4) or "hydrides" (SiH4/PH3/H2S/HCl, d shells);
* ``nmol``     molecules of a call;
* ``lo, hi``   monomers per molecule (uniform), equal for one size;
* ``same``     1: all molecules are geometries of one molecule (frames), 0: independent molecules;
* ``grad``     analytic gradient as well as the energy;
* ``guess``    "zero" or "learned" starting charges;
* ``tol``      "default" (1e-6 Eh, 2e-5 e), "bench" (1e-6 Eh, 2e-6 e) or "tight" (1e-8 Eh, 1e-7 e);
* ``steps``    L-BFGS steps ("optimize").

Clusters above 112 waters are the innermost molecules of the packaged 300-water cluster, jittered; the other
molecules are cut from a cubic lattice at the density of the packaged workloads (30 A^3 per
monomer, 64 A^3 for the hydrides) with neighbour-ordered orientations and a 0.05 A (frames: 0.03 A) Gaussian jitter, so that
any size is made quickly and its SCC converges as it does for the packaged clusters.

The Fermi level is left out of the outputs: at 300 K with an open gap every level inside the gap
gives the same occupations, so the electron count fixes it only to rounding.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "gfn1-rs_b200", "python"))

from gfn1_rs import BatchCalculator, Gfn1NativeCalculator, hessian, workloads  # noqa: E402

A2B = 1.8897261246257702
TOL = {"default": (1e-6, 2e-5), "bench": (1e-6, 2e-6), "tight": (1e-8, 1e-7)}
AO = {1: 2, 6: 4, 7: 4, 8: 4, 14: 9, 15: 9, 16: 9, 17: 9}


def _case(name, kind, set_, nmol, lo, hi, same=0, grad=1, guess="zero", tol="default", steps=0):
    c = dict(kind=kind, set=set_, nmol=nmol, lo=lo, hi=hi, same=same, grad=grad, guess=guess, tol=tol, steps=steps)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: one molecule, 8 AOs, energy and forces for an interactive user or an MD driver
        _case("water-1", "single", "water", 1, 1, 1),
        # one mid-size molecule at the convergence used before derivatives: 48 atoms, 128 AOs
        _case("water-16", "single", "water", 1, 16, 16, tol="tight"),
        # one molecule just above the one-SM limit: 120 atoms, 320 AOs
        _case("water-40", "single", "water", 1, 40, 40),
        # the largest system of the packaged workloads: 900 atoms, 2400 AOs
        _case("water-300", "single", "water", 1, 300, 300, tol="tight"),
        # a handful of molecules of odd sizes, as a service collects them from its callers
        _case("mixed-31", "batch", "mixed", 31, 1, 15, guess="learned"),
        # energies only (conformer ranking)
        _case("mixed-250-energy", "batch", "mixed", 250, 2, 9, grad=0),
        # the headline batch: 4096 mixed clusters, learned starting charges, forces
        _case("mixed-4096", "batch", "mixed", 4096, 1, 15, guess="learned", tol="bench"),
        # d shells (Si, P, S, Cl): 512 hydride clusters
        _case("hydrides-512", "batch", "hydrides", 512, 1, 5),
        # 64 frames of a 24-water cluster (192 AOs) kept on the device, new coordinates each pass
        _case("frames-64x24", "resident", "water", 64, 24, 24, same=1, guess="learned"),
        # a short batch of 96-water trajectory frames (768 AOs)
        _case("frames-8x96", "batch", "water", 8, 96, 96, same=1),
        # semi-numerical Hessian of a three-monomer cluster: 6N displaced gradients
        _case("hessian-3", "hessian", "water", 1, 3, 3, tol="tight"),
        # device-resident L-BFGS of 128 small molecules, the first steps
        _case("optimize-128", "optimize", "mixed", 128, 1, 6, steps=4),
    ]


def _cost(c):
    """Matrix work of a pass in units of N^3 (N of the molecules, evaluations of a pass)."""
    per = {"water": 8.0, "mixed": 9.0, "hydrides": 15.0}[c["set"]]
    lo, hi = c["lo"], c["hi"]
    n3 = per ** 3 * sum(k ** 3 for k in range(lo, hi + 1)) / (hi - lo + 1)
    atoms = {"water": 3, "mixed": 4, "hydrides": 4}[c["set"]] * 0.5 * (lo + hi)
    evals = {"hessian": 6 * atoms + 1, "optimize": c["steps"] + 2.0}.get(c["kind"], 1.0)
    return evals * c["nmol"] * n3


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    most = 1.0e10  # below the 300-water cluster
    while True:
        kind = rng.choice(["single", "single", "batch", "batch", "batch", "frames", "resident", "hessian", "optimize"])
        tol = rng.choice(["default", "bench", "tight"])
        grad = rng.choice([0, 1, 1])
        guess = rng.choice(["zero", "learned"])
        if kind == "single":
            k = _log_int(rng, 1, 256)
            c = _case(None, "single", "water" if k > 112 else rng.choice(["water", "mixed"]), 1, k, k, grad=grad, tol=tol)
        elif kind == "batch":
            s = rng.choice(["mixed", "mixed", "water", "hydrides"])
            hi = rng.randint(1, 15 if s != "hydrides" else 6)
            c = _case(None, "batch", s, _log_int(rng, 2, 4096), rng.randint(1, hi), hi, grad=grad,
                      guess=guess if s != "hydrides" else "zero", tol=tol)
        elif kind in ("frames", "resident"):
            k = _log_int(rng, 2, 112)
            c = _case(None, "batch" if kind == "frames" else "resident", "water", _log_int(rng, 2, 256), k, k, same=1,
                      grad=grad, guess=guess, tol=tol)
        elif kind == "hessian":
            k = rng.randint(1, 5)
            c = _case(None, "hessian", "mixed", rng.randint(1, 6), k, k, tol="tight")
        else:
            hi = rng.randint(1, 9)
            c = _case(None, "optimize", "mixed", _log_int(rng, 2, 300), rng.randint(1, hi), hi,
                      steps=rng.randint(2, 5))
        if _cost(c) <= most:
            return c


# ------------------------------------------------------------------ molecules

def _hydride(z, n, r, angle):
    """XH_n with bond length r (A); bent / pyramidal with the H-X-H angle, tetrahedral for n = 4."""
    if n == 1:
        return [z, 1], np.array([[0.0, 0, 0], [r, 0, 0]])
    if n == 2:
        a = math.radians(angle) / 2
        return [z, 1, 1], r * np.array([[0, 0, 0], [math.sin(a), math.cos(a), 0], [-math.sin(a), math.cos(a), 0]])
    if n == 3:
        s = math.sqrt((1.0 - math.cos(math.radians(angle))) / 1.5)
        c = math.sqrt(1.0 - s * s)
        h = [[s * math.cos(2 * math.pi * k / 3), s * math.sin(2 * math.pi * k / 3), -c] for k in range(3)]
        return [z, 1, 1, 1], r * np.array([[0.0, 0, 0]] + h)
    t = 1 / math.sqrt(3.0)
    return [z, 1, 1, 1, 1], r * np.array([[0, 0, 0], [t, t, t], [-t, -t, t], [-t, t, -t], [t, -t, -t]])


MONOMERS = {
    "water": [workloads.MONOMERS["H2O"]],
    "mixed": [workloads.MONOMERS[k] for k in workloads.MONOMER_ORDER],
    "hydrides": [_hydride(14, 4, 1.48, 0), _hydride(15, 3, 1.42, 93.5), _hydride(16, 2, 1.34, 92.1), _hydride(17, 1, 1.28, 0)],
}


def _cluster(set_, kinds, rng):
    """The monomers `kinds` on the lattice sites nearest the origin, each in the one of twelve random
    orientations with the lowest energy of point charges (H positive) and contact repulsion with the
    monomers already placed, as neighbours in a liquid turn to one another."""
    n = len(kinds)
    side = (64.0 if set_ == "hydrides" else 30.0) ** (1.0 / 3.0)
    m = int(math.ceil((n * 2.0) ** (1.0 / 3.0))) + 1
    g = np.arange(-m, m + 1) * side
    sites = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3) + rng.uniform(-0.2, 0.2, 3) * side
    sites = sites[np.argsort((sites ** 2).sum(1), kind="stable")[:n]]
    xs, qs = np.zeros((0, 3)), np.zeros(0)
    for p, k in zip(sites, kinds):
        z, geo = MONOMERS[set_][k]
        q = np.array([-0.3 * (len(z) - 1)] + [0.3] * (len(z) - 1))
        cand = np.stack([geo @ workloads.random_rotation(rng).T for _ in range(12)]) + p
        if len(xs):
            d = np.sqrt(((cand[:, :, None, :] - xs[None, None]) ** 2).sum(-1))
            e = (q[None, :, None] * qs[None, None] / d + np.where(d < 2.5, (1.4 / d) ** 9, 0.0)).sum(axis=(1, 2))
            cand = cand[np.argsort(e, kind="stable")]
        xs, qs = np.concatenate([xs, cand[0]]), np.concatenate([qs, q])
    return xs


_BOX = []  # the packaged 300-water cluster: random orientations at this size often close the gap


def _big_water(n):
    if not _BOX:
        _BOX.append(workloads.water_cluster(300, 1)[1].reshape(300, 3, 3))
    w = _BOX[0]
    d = ((w[:, 0] - w[:, 0].mean(0)) ** 2).sum(1)
    return w[np.argsort(d, kind="stable")[:n]].reshape(-1, 3)


def _molecules(case, seed):
    """Flat arrays (atom_offsets, numbers, xyz in bohr).  Composition and order follow from the case alone, the
    geometries from the seed: at most 96 different clusters, each used for several molecules with a jitter of its own."""
    fixed = np.random.default_rng([17, case["nmol"], case["lo"], case["hi"]])
    rng = np.random.default_rng([int(seed), 19, case["nmol"]])
    base = []
    for _ in range(1 if case["same"] else min(case["nmol"], 96)):
        kinds = fixed.integers(0, len(MONOMERS[case["set"]]), size=int(fixed.integers(case["lo"], case["hi"] + 1)))
        base.append((np.concatenate([MONOMERS[case["set"]][k][0] for k in kinds]).astype(np.uint8),
                     _big_water(len(kinds)) if case["set"] == "water" and len(kinds) > 112 else
                     _cluster(case["set"], kinds, rng)))
    pick = np.arange(case["nmol"]) % len(base)
    fixed.shuffle(pick)
    off = np.concatenate([[0], np.cumsum([len(base[b][0]) for b in pick])]).astype(np.int32)
    z = np.concatenate([base[b][0] for b in pick])
    x = np.concatenate([base[b][1] for b in pick])
    x = x + rng.normal(0.0, 0.03 if case["same"] else 0.05, size=x.shape)
    return off, z, np.ascontiguousarray(x * A2B)


# ------------------------------------------------------------------ state and pass

def prepare(case, seed):
    off, z, x = _molecules(case, seed)
    e, q = TOL[case["tol"]]
    opts = dict(energy_tolerance=e, charge_tolerance=q)
    s = {"case": dict(case), "off": off, "z": z, "x": x}
    if case["kind"] == "single":
        s["calc"] = Gfn1NativeCalculator(**opts)
        s["numbers"], s["positions"] = z.tolist(), x.tolist()
    else:
        s["calc"] = BatchCalculator(learned_guess=case["guess"] == "learned" or None, **opts)
    if case["kind"] in ("resident", "optimize"):
        s["batch"] = s["calc"].resident(off, z, compute_gradient=bool(case["grad"]))
    return s


def _outputs(r, grad):
    out = {"energy": r.energy, "terms": r.terms, "shell_charges": r.shell_charges, "atomic_charges": r.atomic_charges,
           "dipole": r.dipole, "iterations": r.iterations, "status": r.status, "rung": r.rung}
    if grad:
        out["gradient"] = r.gradient
    return out


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "single":
        r = state["calc"].calculate(state["numbers"], state["positions"], unit="bohr", compute_gradient=bool(case["grad"]))
        out = {"energy": np.array([r.energy_hartree]), "terms": np.array([list(r.energy_terms_hartree().values())]),
               "shell_charges": np.array(r.shell_charges), "atomic_charges": np.array(r.charges),
               "dipole": np.array([r.dipole]), "iterations": np.array([r.iterations])}
        if case["grad"]:
            out["gradient"] = np.array(r.gradient_hartree_per_bohr)
        return out
    if kind == "batch":
        return _outputs(state["calc"].calculate_flat(state["off"], state["z"], state["x"],
                                                     compute_gradient=bool(case["grad"])), case["grad"])
    if kind == "resident":
        state["batch"].set_positions(state["x"])
        state["batch"].launch()
        return _outputs(state["batch"].download(), case["grad"])
    if kind == "hessian":
        r = hessian.hessian_batch(state["calc"], state["off"], state["z"], state["x"])
        return {"hessians": list(r["hessians"]), "energy": r["energy"], "gradient": r["gradient"], "status": r["status"]}
    state["batch"].set_positions(state["x"])
    r = state["batch"].optimize(max_iterations=case["steps"])
    return {k: r[k] for k in ("xyz", "energy", "max_gradient", "iterations", "converged", "status")}


def work(case):
    """Bytes: coordinates and elements in, results out.  Operations: per SCC iteration 12 N^3 + 2 N^2 + 2 nsh^2
    (eigensolution, density and the potential), 14 N^3 once, nine iterations."""
    off, z, _ = _molecules(case, 1)
    ao = np.array([AO.get(i, 0) for i in range(128)], dtype=np.float64)
    cum = np.concatenate([[0.0], np.cumsum(ao[z])])
    n = cum[off[1:]] - cum[off[:-1]]
    nat = float(off[-1])
    evals = 1.0
    if case["kind"] == "hessian":
        evals = 6.0 * nat / case["nmol"] + 1.0
    elif case["kind"] == "optimize":
        evals = case["steps"] + 1.0
    flops = evals * float(np.sum(9 * (12 * n ** 3 + 4 * n ** 2) + 14 * n ** 3))
    nbytes = evals * (nat * (3 * 8 + 1) + nat * 8 * (3 * case["grad"] + 1 + 2) + 8.0 * case["nmol"] * 22)
    if case["kind"] == "hessian":
        nbytes = nat * (3 * 8 + 1) + 8.0 * float(np.sum((3.0 * np.diff(off)) ** 2)) + nat * 24
    elif case["kind"] == "optimize":
        nbytes = nat * (6 * 8 + 1) + 8.0 * case["nmol"] * 4
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------ the converged answer in 64 bits
# GFN1-xTB in plain torch from the parameter tables: STO-nG overlap, H0, Klopman-Ohno, D3(BJ) and repulsion as
# functions of the coordinates, a Fermi-smeared SCC with Anderson mixing, and the gradient by automatic differentiation
# of the energy at fixed density, energy-weighted density and shell potential.

EV = 1.0 / 27.21138505
KT = 3.1668115634556e-6 * 300.0


class _Model:
    def __init__(self):
        self.t = {}
        with open(os.path.join(ROOT, "gfn1-rs_b200", "data", "gfn1_tables.txt")) as fh:
            for line in fh:
                p = line.split()
                if p and not line.startswith("#"):
                    self.t[p[0]] = [float(v) for v in p[2:]]
        self.elem = {}

    def g(self, key, default=0.0):
        v = self.t.get(key)
        return v[0] if v else default

    def sto(self, ng, n, l, zeta):
        row = {0: n, 1: 4 + n, 2: 7 + n}[l] - 1
        al = np.array(self.t[f"sto.alpha.{ng}"][row * ng:(row + 1) * ng]) * zeta * zeta
        co = np.array(self.t[f"sto.coeff.{ng}"][row * ng:(row + 1) * ng])
        df = (1.0, 1.0, 3.0)[l]
        return al, co * (2.0 / math.pi * al) ** 0.75 * np.sqrt(4.0 * al) ** l / math.sqrt(df)

    def element(self, z):
        if z in self.elem:
            return self.elem[z]
        e, p = {}, f"elem.{z}."
        ao, lev, ex = self.t[p + "ao"], self.t[p + "lev"], self.t[p + "exp"]
        gam = self.g(p + "gam")
        lpar = [self.g(p + k) for k in ("lpars", "lparp", "lpard")]
        poly = [self.g(p + k) for k in ("polys", "polyp", "polyd")]
        d_kind = self.g("glob.cnd1", -0.5)
        cnf = [self.g("glob.cns", 0.6), self.g("glob.cnp", -0.3), d_kind]
        shells, ref = [], {}
        for k in range(len(lev)):
            n, l = int(ao[2 * k]), int(ao[2 * k + 1])
            ng = (4 if n == 1 else 3) if z <= 2 else (6 if l < 2 else 4)
            a, c = self.sto(ng, n, l, ex[k])
            val = l not in ref
            if not val:  # orthogonalised to the first shell of the same l
                ra, rc = ref[l]
                ov = float(np.sum(rc[:, None] * c[None] * (math.pi / (ra[:, None] + a[None])) ** 1.5))
                a, c = np.concatenate([a, ra]), np.concatenate([c, -ov * rc])
                c = c / math.sqrt(np.sum(c[:, None] * c[None] * (math.pi / (a[:, None] + a[None])) ** 1.5))
            else:
                ref[l] = (a, c)
            shells.append(dict(l=l, a=a, c=c, val=val, h=lev[k] * EV, kcn=-lev[k] * EV * cnf[l] * 0.01,
                               poly=poly[l] * 0.01, occ=self.t["refocc"][3 * z + l] if val else 0.0,
                               hard=gam * (1.0 + 0.1 * lpar[l])))
        e["shells"], e["gam3"] = shells, 0.1 * self.g(p + "gam3")
        e["repa"], e["repb"], e["en"] = self.g(p + "repa"), self.g(p + "repb"), self.t["pauling_en"][z]
        e["rad"] = self.t["atomic_radius_ang"][z] * A2B
        e["rcov"] = 4.0 / 3.0 * self.t["covrad_ang"][z] * A2B
        e["r4r2"] = math.sqrt(0.5 * self.t["d3.r4r2"][z - 1] * math.sqrt(z))
        e["cnref"] = self.t[f"d3.cnref.{z}"][:int(self.t["d3.nref"][z - 1])]
        self.elem[z] = e
        return e

    def kpair(self, li, lj):
        k = [self.g("glob.ks"), self.g("glob.kp"), self.g("glob.kd")]
        return self.g("glob.ksp") if {li, lj} == {0, 1} else 0.5 * (k[li] + k[lj])

    def hscale(self, zi, si, zj, sj):
        kd = self.g("glob.kdiff")
        if si["val"] and sj["val"]:
            de = self.element(zi)["en"] - self.element(zj)["en"]
            pair = self.g(f"pair.{min(zi, zj)}.{max(zi, zj)}", 1.0)
            return pair * self.kpair(si["l"], sj["l"]) * (1.0 + self.g("glob.enscale") * 0.01 * de * de)
        if si["val"]:
            return 0.5 * (self.kpair(si["l"], si["l"]) + kd)
        if sj["val"]:
            return 0.5 * (self.kpair(sj["l"], sj["l"]) + kd)
        return kd


CART = {0: [(0, 0, 0)], 1: [(1, 0, 0), (0, 1, 0), (0, 0, 1)],
        2: [(2, 0, 0), (0, 2, 0), (0, 0, 2), (1, 1, 0), (1, 0, 1), (0, 1, 1)]}
R3 = math.sqrt(3.0)
REAL = {0: [[1.0]], 1: np.eye(3).tolist(),
        2: [[R3 / 2, -R3 / 2, 0, 0, 0, 0], [0.5, 0.5, -1.0, 0, 0, 0], [0, 0, 0, R3, 0, 0], [0, 0, 0, 0, R3, 0], [0, 0, 0, 0, 0, R3]]}


def _overlap(M, shells, R):
    """S over AOs in shell order; `shells`: (atom, shell dict, first AO)."""
    N = shells[-1][2] + 2 * shells[-1][1]["l"] + 1
    S = torch.zeros(N, N, dtype=torch.float64)
    idx = {l: [s for s in shells if s[1]["l"] == l] for l in (0, 1, 2)}
    f64 = lambda v: torch.tensor(v, dtype=torch.float64)  # noqa: E731
    for la in idx:
        for lb in idx:
            if not idx[la] or not idx[lb]:
                continue

            def prims(group):
                n = max(len(s[1]["a"]) for s in group)
                return (f64(np.array([np.pad(s[1]["a"], (0, n - len(s[1]["a"])), constant_values=1.0) for s in group])),
                        f64(np.array([np.pad(s[1]["c"], (0, n - len(s[1]["c"]))) for s in group])))

            aa, ca = prims(idx[la])
            ab, cb = prims(idx[lb])
            A = R[torch.tensor([s[0] for s in idx[la]])]
            B = R[torch.tensor([s[0] for s in idx[lb]])]
            p = aa[:, None, :, None] + ab[None, :, None, :]
            d = A[:, None] - B[None]
            pre = ca[:, None, :, None] * cb[None, :, None, :] * (math.pi / p) ** 1.5
            pre = pre * torch.exp(-(aa[:, None, :, None] * ab[None, :, None, :] / p) * (d ** 2).sum(-1)[..., None, None])
            E = []
            for x in range(3):
                pa = -(ab[None, :, None, :] / p) * d[..., x][..., None, None]
                pb = (aa[:, None, :, None] / p) * d[..., x][..., None, None]
                h = 0.5 / p
                t = {(0, 0): torch.ones_like(p)}
                for i in range(la + 1):
                    for j in range(lb + 1):
                        if i:
                            v = pa * t[i - 1, j]
                            v = v + h * (i - 1) * t[i - 2, j] if i > 1 else v
                            t[i, j] = v + h * j * t[i - 1, j - 1] if j else v
                        elif j:
                            v = pb * t[0, j - 1]
                            t[0, j] = v + h * (j - 1) * t[0, j - 2] if j > 1 else v
                E.append(t)
            blk = torch.stack([torch.stack([(pre * E[0][a[0], b[0]] * E[1][a[1], b[1]] * E[2][a[2], b[2]]).sum((-1, -2))
                                            for b in CART[lb]], -1) for a in CART[la]], -2)
            blk = torch.einsum("ka,ijab,lb->ijkl", f64(REAL[la]), blk, f64(REAL[lb]))
            ra = torch.tensor([[s[2] + k for k in range(2 * la + 1)] for s in idx[la]]).reshape(-1)
            rb = torch.tensor([[s[2] + k for k in range(2 * lb + 1)] for s in idx[lb]]).reshape(-1)
            S = S.index_put((ra[:, None], rb[None]), blk.permute(0, 2, 1, 3).reshape(len(ra), len(rb)))
    return S


def _converged(M, z, x):
    """Energy terms (15), gradient, shell and atomic charges, dipole of one neutral molecule."""
    z = [int(v) for v in z]
    R = torch.tensor(np.asarray(x), dtype=torch.float64, requires_grad=True)
    el = [M.element(v) for v in z]
    nat = len(z)
    shells, o = [], 0
    for a in range(nat):
        for s in el[a]["shells"]:
            shells.append((a, s, o))
            o += 2 * s["l"] + 1
    nsh, N = len(shells), o
    f64 = lambda v: torch.tensor(v, dtype=torch.float64)  # noqa: E731
    at = torch.tensor([s[0] for s in shells])
    of_sh = torch.tensor([i for i, s in enumerate(shells) for _ in range(2 * s[1]["l"] + 1)])
    off = ~torch.eye(nat, dtype=torch.bool)
    d2 = ((R[:, None] - R[None]) ** 2).sum(-1)
    r2 = torch.where(off, d2, torch.ones_like(d2))
    r = torch.sqrt(r2)
    rc = f64([e["rcov"] for e in el])
    count = 1.0 / (1.0 + torch.exp(torch.clamp(-16.0 * ((rc[:, None] + rc[None]) / r - 1.0), -80.0, 80.0)))
    zero = torch.zeros_like(r)
    cn = torch.where(off & (r2 <= 900.0), count, zero).sum(1)
    cnd = torch.where(off & (r2 <= 625.0), count, zero).sum(1)
    # overlap and H0
    inside = (off & (r2 <= 900.0)) | ~off
    S = _overlap(M, shells, R)
    ao_at = at[of_sh]
    S = torch.where(inside[ao_at][:, ao_at], S, torch.zeros_like(S))
    se = f64([s[1]["h"] for s in shells]) - f64([s[1]["kcn"] for s in shells]) * cn[at]
    rad = f64([e["rad"] for e in el])
    rr = torch.sqrt(r / (rad[:, None] + rad[None]))[at][:, at]
    pol = f64([s[1]["poly"] for s in shells])
    key = [(z[s[0]], id(s[1])) for s in shells]
    kinds = sorted(set(key))
    rep = {k: shells[key.index(k)] for k in kinds}
    hk = np.array([[M.hscale(z[rep[a][0]], rep[a][1], z[rep[b][0]], rep[b][1]) for b in kinds] for a in kinds])
    ki = np.array([kinds.index(k) for k in key])
    fac = f64(hk[ki][:, ki]) * (1.0 + pol[:, None] * rr) * (1.0 + pol[None] * rr)
    fac = torch.where(at[:, None] == at[None], torch.ones_like(fac), fac)
    H0 = S * (0.5 * (se[:, None] + se[None]) * fac)[of_sh][:, of_sh]
    # Klopman-Ohno, third order
    hard = f64([s[1]["hard"] for s in shells])
    g = 2.0 / (1.0 / hard[:, None] + 1.0 / hard[None])
    same = at[:, None] == at[None]
    G = torch.where(same, g, 1.0 / torch.sqrt(torch.where(same, torch.ones_like(g), d2[at][:, at]) + 1.0 / (g * g)))
    g3 = f64([e["gam3"] for e in el])
    # repulsion
    ra, rb = f64([e["repa"] for e in el]), f64([e["repb"] for e in el])
    kexp = torch.full_like(r, M.g("glob.kexp"))
    light = f64([1.0 if v <= 2 else 0.0 for v in z])
    kexp = torch.where((light[:, None] * light[None]) > 0, torch.full_like(r, M.g("glob.kexplight", M.g("glob.kexp"))), kexp)
    er = rb[:, None] * rb[None] * torch.exp(-torch.sqrt(ra[:, None] * ra[None]) * r ** kexp) / r
    erep = 0.5 * torch.where(off & (r2 <= 625.0), er, zero).sum()
    # D3(BJ)
    nref = 5
    cref = f64([e["cnref"] + [1e3] * (nref - len(e["cnref"])) for e in el])
    lg = -4.0 * (cnd[:, None] - cref) ** 2
    gw = torch.softmax(lg, dim=1)
    zs = sorted(set(z))
    c6t = np.zeros((len(zs), len(zs), nref, nref))
    for i, a in enumerate(zs):
        for j, b in enumerate(zs):
            hi, lo = max(a, b), min(a, b)
            n1, n2 = len(M.element(hi)["cnref"]), len(M.element(lo)["cnref"])
            blk = np.array(M.t[f"d3.c6.{hi}.{lo}"])[:n1 * n2].reshape(n1, n2)
            blk = blk if a > b else blk.T
            c6t[i, j, :blk.shape[0], :blk.shape[1]] = blk
    zi = np.array([zs.index(v) for v in z])
    c6 = torch.einsum("ia,ijab,jb->ij", gw, f64(c6t[zi][:, zi]), gw)
    r4 = f64([e["r4r2"] for e in el])
    qq = 3.0 * r4[:, None] * r4[None]
    r0 = M.g("glob.a1") * torch.sqrt(qq) + M.g("glob.a2")
    ed = M.g("glob.s6", 1.0) / (r2 ** 3 + r0 ** 6) + M.g("glob.s8") * qq / (r2 ** 4 + r0 ** 8)
    edisp = -0.5 * torch.where(off & (r2 <= 2500.0), c6 * ed, zero).sum()
    # SCC
    Sd, Hd, Gd = S.detach(), H0.detach(), G.detach()
    Li = torch.linalg.inv(torch.linalg.cholesky(Sd))
    occ0 = f64([s[1]["occ"] for s in shells])
    nel = float(occ0.sum())
    one = torch.zeros(nsh, dtype=torch.float64)
    onea = torch.zeros(nat, dtype=torch.float64)

    def potential(q):
        qa = onea.index_add(0, at, q)
        return Gd @ q + (g3 * qa * qa)[at], qa

    def density(q):
        v, _ = potential(q)
        va = v[of_sh]
        F = Hd - 0.5 * Sd * (va[:, None] + va[None])
        eps, Z = torch.linalg.eigh(Li @ F @ Li.T)
        lo, hi = float(eps[0]) - 1.0, float(eps[-1]) + 1.0
        for _ in range(200):
            mu = 0.5 * (lo + hi)
            if float((2.0 / (1.0 + torch.exp(torch.clamp((eps - mu) / KT, -500, 500)))).sum()) < nel:
                lo = mu
            else:
                hi = mu
        f = 2.0 / (1.0 + torch.exp(torch.clamp((eps - 0.5 * (lo + hi)) / KT, -500, 500)))
        C = Li.T @ Z
        P = (C * f) @ C.T
        return occ0 - one.index_add(0, of_sh, (P * Sd).sum(1)), P, C, f, eps

    q, dq, dr = torch.zeros(nsh, dtype=torch.float64), [], []
    last = None
    for _ in range(200):
        qo = density(q)[0]
        res = qo - q
        if float(res.abs().max()) < 1e-11:
            break
        if last is not None:
            dq.append(q - last[0])
            dr.append(res - last[1])
            dq, dr = dq[-12:], dr[-12:]
        last = (q, res)
        q = q + 0.4 * res
        if dr:
            B = torch.stack(dr, 1)
            c = torch.linalg.lstsq(B, res[:, None], driver="gelsd").solution[:, 0]
            q = q - (torch.stack(dq, 1) + 0.4 * B) @ c
    q, P, C, f, eps = density(q)
    W = (C * (f * eps)) @ C.T
    v, qa = potential(q)
    nn = torch.clamp(0.5 * f, 1e-16, 1.0 - 1e-16)
    ts = 2.0 * KT * float((nn * torch.log(nn) + (1.0 - nn) * torch.log(1.0 - nn)).sum())
    e_el, e2, e3 = float((P * Hd).sum()), 0.5 * float(q @ (Gd @ q)), float((qa ** 3 * g3 / 3.0).sum())
    va = v[of_sh]
    L = (P * H0).sum() - 0.5 * (P * S * (va[:, None] + va[None])).sum() - (W * S).sum() + 0.5 * q @ (G @ q) + erep + edisp
    grad, = torch.autograd.grad(L, R)
    erep_v, edisp_v = float(erep.detach()), float(edisp.detach())
    ei = e_el + e2 + e3 + erep_v + edisp_v
    terms = [ei + ts, ei, erep_v, e_el, e2, e3, 0, edisp_v, 0, 0, 0, 0, 0, 0, ts]
    return (np.array(terms), grad.numpy(), q.numpy(), qa.numpy(), (qa[:, None] * R.detach()).sum(0).numpy())


def exact(case, seed):
    """The converged results (to 1e-11 e) where they take some seconds: the tolerance of a case, not rounding, is the
    distance of a pass from them."""
    per = {"water": 8, "mixed": 9, "hydrides": 15}[case["set"]] * 0.5 * (case["lo"] + case["hi"])
    evals = case["nmol"] * (0.25 + (per / 130.0) ** 3)
    if case["kind"] == "optimize" or (case["kind"] == "hessian" and (case["nmol"] > 1 or case["hi"] > 3)) or evals > 16.0:
        return None
    off, z, x = _molecules(case, seed)
    M = _Model()
    if case["kind"] == "hessian":
        h, cols = hessian.DEFAULT_STEP, []
        for c in range(3 * len(z)):
            gp = []
            for s in (h, -h):
                y = x.copy()
                y[c // 3, c % 3] += s
                gp.append(_converged(M, z, y)[1].reshape(-1))
            cols.append((gp[0] - gp[1]) / (2.0 * h))
        hm = np.stack(cols)
        t, g = _converged(M, z, x)[:2]
        return {"hessians": [0.5 * (hm + hm.T)], "energy": t[:1], "gradient": g, "status": None}
    rs = [_converged(M, z[off[m]:off[m + 1]], x[off[m]:off[m + 1]]) for m in range(case["nmol"])]
    out = {"energy": np.array([r[0][0] for r in rs]), "terms": np.stack([r[0] for r in rs]),
           "shell_charges": np.concatenate([r[2] for r in rs]), "atomic_charges": np.concatenate([r[3] for r in rs]),
           "dipole": np.stack([r[4] for r in rs]), "iterations": None}
    if case["grad"]:
        out["gradient"] = np.concatenate([r[1] for r in rs])
    return out
