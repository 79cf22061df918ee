"""What the engine's users have it do, as measurable calls.

Each case is one pass through a public entry point: MD steps of one system or of a batch
(`Batch.run` and the reads a campaign makes after it), single points (`Batch.evaluate`), the
free-energy analysis (`fep.analyze`), the training of the lambda-placement network
(`mlp.train`) and the allocation-free water-water call (`qb_ww_energy_static`).  The systems are
the synthetic ones of `q_b200.synth`: TIP3P spheres, the 56-atom FEP solute in a sphere or a
periodic box, and the polymer sphere.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs, batch or buffers a program holds before the call
    run(state)          one pass
    work(case)          bytes and operations a pass cannot do without
    exact(case, seed)   the outputs in 64 bits, where they have such a value
"""
from __future__ import annotations

import ctypes
import math
import os
import tempfile

import numpy as np
import torch

from q_b200 import FP64, MIXED, Batch, System, fep, mlp, synth
from q_b200._lib import QB_NE, QB_NEQ, check, lib
from q_b200.campaign import open_systems

DENSITY = 0.0334            # waters per cubic Angstrom (the generator's)
MD_STEPS = 50               # two list cycles of the inputs' non_bond 25
PRECISION = {"fp64": FP64, "mixed": MIXED}


def listed():
    return [
        # one call of a host that owns its device memory and wants the water-water terms of a
        # small sphere: the smallest call of the library
        {"name": "static_ww_15A", "kind": "static", "radius": 15.0},
        # a sphere's energies and forces at given coordinates (a frame rescored)
        {"name": "point_sphere_25A_fp64", "kind": "point", "spheres": 1, "radius": 25.0, "precision": "fp64"},
        # frames of many spheres rescored together by the mixed engine
        {"name": "point_spheres16_20A_mixed", "kind": "point", "spheres": 16, "radius": 20.0, "precision": "mixed"},
        # plain MD of one 15 A water sphere: the smallest system, where launches count
        {"name": "md_sphere_15A_fp64", "kind": "md", "system": "sphere", "radius": 15.0, "precision": "fp64"},
        # plain MD of one FEP window: what qdyn runs as one process
        {"name": "md_fep_20A_fp64", "kind": "md", "system": "fep", "radius": 20.0, "windows": 1, "replicas": 1,
         "precision": "fp64"},
        # the protein-ligand sphere (3000-atom polymer, any-atom cut-offs), mixed engine
        {"name": "md_complex_25A_mixed", "kind": "md", "system": "complex", "radius": 25.0, "precision": "mixed"},
        # the FEP solute in a periodic box at constant pressure
        {"name": "md_box_30A_npt_fp64", "kind": "md", "system": "box", "edge": 30.0, "precision": "fp64"},
        # the windows of one perturbation, one replica, mixed engine: an ordinary batch
        {"name": "md_fep_21w_mixed", "kind": "md", "system": "fep", "radius": 20.0, "windows": 21, "replicas": 1,
         "precision": "mixed"},
        # a dense set of reference windows on the parity engine
        {"name": "md_fep_41w_fp64", "kind": "md", "system": "fep", "radius": 20.0, "windows": 41, "replicas": 1,
         "precision": "fp64"},
        # the batched campaign: 21 windows x 4 replicas and 16 water spheres of 15 to 25 A
        {"name": "md_campaign_100_mixed", "kind": "md", "system": "campaign", "windows": 21, "replicas": 4,
         "spheres": 16, "precision": "mixed"},
        # the analysis of a perturbation's energy files
        {"name": "qfep_21w_1000", "kind": "qfep", "windows": 21, "records": 1000, "states": 2, "skip": 100},
        # one training of the placement network (200 perturbations)
        {"name": "placement_train_200", "kind": "train", "samples": 200, "iters": 100},
    ]


def draw(rng):
    kind = rng.choice(["static", "point", "md", "md", "md", "qfep", "train"])
    if kind == "static":
        return {"kind": "static", "radius": round(rng.uniform(9.0, 28.0), 1)}
    if kind == "point":
        return {"kind": "point", "spheres": int(round(math.exp(rng.uniform(0.0, math.log(20.0))))),
                "radius": round(rng.uniform(10.0, 25.0), 1), "precision": rng.choice(["fp64", "mixed"])}
    if kind == "qfep":
        return {"kind": "qfep", "windows": rng.randint(5, 31),
                "records": int(round(math.exp(rng.uniform(math.log(150), math.log(2000))))),
                "states": rng.choice([2, 2, 3, 4]), "skip": rng.randint(0, 100)}
    if kind == "train":
        return {"kind": "train", "samples": rng.randint(40, 250), "iters": rng.randint(50, 100)}
    system = rng.choice(["sphere", "fep", "fep", "fep", "complex", "box"])
    precision = rng.choice(["fp64", "mixed"])
    if system == "sphere":
        return {"kind": "md", "system": system, "radius": round(rng.uniform(11.0, 26.0), 1), "precision": precision}
    if system == "complex":
        return {"kind": "md", "system": system, "radius": 25.0, "precision": precision,
                "lambda": round(rng.uniform(0.05, 0.95), 3)}
    if system == "box":
        return {"kind": "md", "system": system, "edge": round(rng.uniform(29.0, 34.0), 1), "precision": precision}
    return {"kind": "md", "system": "fep", "radius": round(rng.uniform(16.0, 21.0), 1),
            "windows": int(round(math.exp(rng.uniform(0.0, math.log(41.0))))), "replicas": 1, "precision": precision}


# ------------------------------------------------------------------ systems

_root = None
_files = {}


def _generated(kind, size=0.0, variant=0):
    """Input files of one synthetic system, written once per process."""
    global _root
    key = (kind, size, variant)
    if key not in _files:
        if _root is None:
            _root = tempfile.mkdtemp(prefix="q_cases_")
        d = os.path.join(_root, "%s_%g_%d" % key)
        if kind == "sphere":
            g = synth.water_sphere(d, radius=size, seed=1334 + variant, name="sph")
        elif kind == "fep":
            g = synth.fep_solute(d, radius=size, seed=1234)
        elif kind == "complex":
            g = synth.polymer_sphere(d, radius=size, seed=1234)
        else:
            g = synth.fep_box(d, edge=size, seed=1234, constant_pressure=True, volume_change=25)
        _files[key] = g.inp
    return _files[key]


def _systems(case, seed):
    """The prepared systems of an MD or single-point case; the seed gives every system its Maxwell velocities."""
    s0 = 1 + seed % 900000
    if case["kind"] == "point":
        return [System.open(_generated("sphere", case["radius"], k % 4), seed=s0 + k) for k in range(case["spheres"])]
    if case["system"] == "sphere":
        return [System.open(_generated("sphere", case["radius"]), seed=s0)]
    if case["system"] == "complex":
        lam = case.get("lambda", 0.5)
        return [System.open(_generated("complex", case["radius"]), lambdas=(lam, 1.0 - lam), seed=s0)]
    if case["system"] == "box":
        return [System.open(_generated("box", case["edge"]), lambdas=(0.5, 0.5), seed=s0)]
    lams = synth.window_lambdas(case["windows"]) if case["windows"] > 1 else [(0.5, 0.5)]
    systems = open_systems(_generated("fep", case.get("radius", 20.0)), lams, range(s0, s0 + case["replicas"]))
    for k in range(case.get("spheres", 0)):
        systems.append(System.open(_generated("sphere", (15.0, 20.0, 25.0)[k % 3], k % 4), seed=s0 + k))
    return systems


def _jittered(system, rng):
    """The sphere's coordinates with every water moved (0.05 A) and turned (0.2 rad) a little."""
    x = system.array("x0").reshape(-1, 3, 3)
    n = len(x)
    axis = rng.normal(size=(n, 3))
    axis /= np.linalg.norm(axis, axis=1, keepdims=True)
    angle = rng.normal(0.0, 0.2, size=n)
    v = x - x[:, :1]
    c, s = np.cos(angle)[:, None, None], np.sin(angle)[:, None, None]
    k = axis[:, None, :]
    v = v * c + np.cross(np.broadcast_to(k, v.shape), v) * s + k * (k * v).sum(-1, keepdims=True) * (1.0 - c)
    return (x[:, :1] + rng.normal(0.0, 0.05, size=(n, 1, 3)) + v).reshape(-1)


def _series(case, seed):
    """Energy series of every window: q_energies records whose state gap follows a linear-response
    perturbation (mean falling along lambda, 4 kcal/mol wide), as a solvation window's does."""
    rng = np.random.default_rng(seed)
    nw, n, ns = case["windows"], case["records"], case["states"]
    out = []
    for w in range(nw):
        lam = np.zeros(ns)
        lam[0], lam[1] = 1.0 - w / (nw - 1), w / (nw - 1)
        e = np.zeros((n, ns, QB_NEQ))
        base = rng.normal(0.0, 3.0, size=n)
        for st in range(ns):
            parts = rng.normal(0.0, 1.0, size=(n, 4)) + np.array([4.0, 9.0, 6.0, 1.0])
            gap = st * (20.0 - 30.0 * lam[1] + rng.normal(0.0, 4.0, size=n))
            e[:, st, 0] = lam[st]
            e[:, st, 2:6] = parts
            e[:, st, 8] = rng.normal(-12.0, 1.0, size=n)             # qq
            e[:, st, 9] = rng.normal(3.0, 0.5, size=n)
            e[:, st, 12] = base - 60.0 + gap                          # q-water
            e[:, st, 13] = rng.normal(-8.0, 0.5, size=n)
            e[:, st, 6] = e[:, st, 8] + e[:, st, 10] + e[:, st, 12]
            e[:, st, 7] = e[:, st, 9] + e[:, st, 11] + e[:, st, 13]
            # the bonded parts are the same molecule in every state
            if st > 0:
                e[:, st, 2:6], e[:, st, 8:10], e[:, st, 13] = e[:, 0, 2:6], e[:, 0, 8:10], e[:, 0, 13]
                e[:, st, 6] = e[:, st, 8] + e[:, st, 12]
                e[:, st, 7] = e[:, st, 9] + e[:, st, 13]
            e[:, st, 1] = e[:, st, 2:8].sum(1) + e[:, st, 14]
        out.append(e)
    return out


def _training_set(case, seed):
    """Normalised pilot features and the logit corrections they predict (smooth, with sampling noise)."""
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(case["samples"], mlp.IN)).astype(np.float32)
    mix = np.random.default_rng(7).normal(0.0, 0.3, size=(mlp.IN, mlp.OUT))
    t = (np.tanh(x @ mix) * 0.4 + rng.normal(0.0, 0.1, size=(case["samples"], mlp.OUT))).astype(np.float32)
    return x, t


# ------------------------------------------------------------------ the cases

def _static_inputs(case, seed):
    s = System.open(_generated("sphere", case["radius"]), seed=1)
    x = _jittered(s, np.random.default_rng(seed))
    return s, x


def prepare(case, seed):
    kind = case["kind"]
    if kind == "static":
        s, x = _static_inputs(case, seed)
        v = s.view
        n = v.nwat
        return {"kind": kind, "n": n, "par": (v.crg_ow, v.crg_hw, v.A_OO, v.B_OO, 10.0),
                "x": torch.from_numpy(x).cuda(), "grad": torch.empty(9 * n, dtype=torch.float64, device="cuda"),
                "energy": torch.empty(2, dtype=torch.float64, device="cuda"),
                "status": torch.empty(1, dtype=torch.int32, device="cuda")}
    if kind == "qfep":
        p = fep.params(0.592, case["skip"], nbins=20, nmin=5, coeff=(1.0, -1.0) + (0.0,) * (case["states"] - 2))
        return {"kind": kind, "series": _series(case, seed), "params": p}
    if kind == "train":
        x, t = _training_set(case, seed)
        return {"kind": kind, "w": mlp.init(seed % 1000, True), "x": x, "t": t, "iters": case["iters"]}
    systems = _systems(case, seed)
    batch = Batch(systems, precision=PRECISION[case["precision"]])
    # frames and energies of the mixed engine, whose forces are FP32, are kept in single precision
    state = {"kind": kind, "batch": batch, "keep": np.float64 if case["precision"] == "fp64" else np.float32}
    if kind == "point":
        rng = np.random.default_rng(seed)
        state["x"] = np.concatenate([_jittered(s, rng) for s in systems])
    return state


def run(state):
    kind = state["kind"]
    if kind == "static":
        qo, qh, a, b, rc = state["par"]
        check(lib.qb_ww_energy_static(state["x"].data_ptr(), state["n"], qo, qh, a, b, rc, None,
                                      state["grad"].data_ptr(), state["energy"].data_ptr(),
                                      state["status"].data_ptr(),
                                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return {"grad": state["grad"], "energy": state["energy"], "status": state["status"]}
    if kind == "qfep":
        return vars(fep.analyze(state["series"], state["params"]))
    if kind == "train":
        w, loss = mlp.train(state["w"], state["x"], state["t"], state["iters"], lr=2e-3, weight_decay=0.01)
        return {"w": w, "loss": loss}
    batch, keep = state["batch"], state["keep"]
    if kind == "point":
        batch.set_coords_all(state["x"])
        batch.evaluate(True)
        n = len(batch.systems)
        return {"E": np.stack([batch.energy_vectors(s)[0] for s in range(n)]).astype(keep),
                "grad": np.concatenate([batch.gradient(s) for s in range(n)]).astype(keep)}
    # MD: the next MD_STEPS steps of every system; a campaign of the mixed engine keeps the frame and
    # the energy-file records, a plain run the velocities of its restart too
    batch.clear_history()
    batch.run(MD_STEPS)
    counts, records = batch.history_all(1)
    out = {"x": batch.coords_all().astype(keep), "counts": counts, "records": records.astype(keep)}
    if keep is np.float64:
        out["v"] = batch.velocities_all()
    return out


def _waters(radius):
    return DENSITY * 4.0 / 3.0 * math.pi * radius ** 3


def _sphere_pairs(radius, rc=10.0):
    """Expected water pairs within rc in a uniform sphere: n^2/2 times the sphere's pair-distance distribution."""
    n, u = _waters(radius), min(rc / (2.0 * radius), 1.0)
    return 0.5 * n * n * min(1.0, 8.0 * u ** 3 - 9.0 * u ** 4 + 2.0 * u ** 6)


def work(case):
    kind = case["kind"]
    if kind == "static":
        n = _waters(case["radius"])
        return {"bytes": n * 9 * 8 * 2 + 20, "flops": 229.0 * _sphere_pairs(case["radius"])}
    if kind == "point":
        n = _waters(case["radius"])
        lrf = max(0.0, 0.5 * n * n - _sphere_pairs(case["radius"])) * 2 * 3 * 80.0
        return {"bytes": case["spheres"] * n * 9 * 8 * 2,
                "flops": case["spheres"] * (229.0 * _sphere_pairs(case["radius"]) + lrf)}
    if kind == "qfep":
        n = case["windows"] * case["records"]
        return {"bytes": n * case["states"] * QB_NEQ * 8, "flops": n * case["states"] * QB_NEQ + 12 * 30.0 * n}
    if kind == "train":
        w = mlp.IN * mlp.HID + mlp.HID * mlp.HID + mlp.HID * mlp.OUT
        return {"bytes": 8.0 * mlp.NPARAM + 4.0 * case["samples"] * (mlp.IN + mlp.OUT),
                "flops": 6.0 * w * case["samples"] * case["iters"]}
    # per step: 229 operations a water pair; the other terms are a small part
    if case["system"] == "complex":
        atoms, pairs = 3632, 3.0e6 / 7.0          # ~3e5 solute pairs of 37 operations, Q atoms with everything
    elif case["system"] == "box":
        n = DENSITY * case["edge"] ** 3
        atoms, pairs = 3 * n, 0.5 * n * DENSITY * 4.0 / 3.0 * math.pi * 1000.0
    elif case["system"] == "sphere":
        atoms, pairs = 3 * _waters(case["radius"]), _sphere_pairs(case["radius"])
    else:
        m, r = case["windows"] * case["replicas"], case.get("radius", 20.0)
        atoms, pairs = m * 3 * _waters(r), m * _sphere_pairs(r)
        for k in range(case.get("spheres", 0)):
            r = (15.0, 20.0, 25.0)[k % 3]
            atoms, pairs = atoms + 3 * _waters(r), pairs + _sphere_pairs(r)
    return {"bytes": atoms * 24.0 * 4, "flops": MD_STEPS * 229.0 * pairs}


# ------------------------------------------------------------------ 64 bits

class _Sphere:
    """A TIP3P sphere of the engine's model in 64-bit torch: water-water terms within the cut-off, the
    local reaction field beyond it, the radial and polarisation restraints, SHAKE and leap-frog."""

    def __init__(self, system):
        v = self.v = system.view
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=self.dev)
        self.n = v.nwat
        self.q = t([v.crg_ow, v.crg_hw, v.crg_hw])
        self.centre = t([v.xwcent[k] for k in range(3)])
        self.x = t(system.array("x0")).reshape(-1, 3, 3)
        self.vel = t(system.array("v0")).reshape(-1, 3, 3)
        self.mass = t(system.array("mass", 3)).reshape(1, 3)
        self.winv = t(system.array("winv", 3)).reshape(1, 3)
        ns = self.shells = v.nwpolr_shell if v.wpol_restr else 0
        self.rout, self.dr, self.cstb, self.tcorr = (
            [float(p[k]) for k in range(ns)] for p in (v.wshell_rout, v.wshell_dr, v.wshell_cstb,
                                                       v.wshell_theta_corr0))
        self._temperature()

    def _temperature(self):
        v, kb = self.v, float(np.float32(0.001986))
        self.kin = float((0.5 * self.mass[..., None] * self.vel ** 2).sum())
        self.tfree = 2.0 * self.kin / kb / v.Ndegfree
        self.tscale = math.sqrt(1.0 + v.dt / v.tau_T * (v.Temp0 / self.tfree - 1.0)) if self.tfree else 1.0

    def lists(self):
        """Pairs within the cut-off, and the multipole field of all other waters at each water's centre."""
        v, x, n = self.v, self.x, self.n
        o = x[:, 0]
        r2 = ((o[:, None] - o[None]) ** 2).sum(-1)
        self.i, self.j = torch.nonzero(torch.triu(r2 <= v.Rcww ** 2, 1), as_tuple=True)
        self.lc = x.mean(1)
        self.phi = [torch.zeros((n,) + (3,) * k, dtype=torch.float64, device=self.dev) for k in range(4)]
        if not v.use_LRF:
            return
        far = (r2 > v.Rcww ** 2) & (r2 <= v.RcLRF ** 2)
        eye = torch.eye(3, dtype=torch.float64, device=self.dev)
        for a in range(0, n, 128):
            w = far[a:a + 128, :, None].double() * self.q
            d = x[None] - self.lc[a:a + 128, None, None]
            r = (d ** 2).sum(-1).clamp_min(1e-30).sqrt()
            f0, f1 = w / r ** 3, 3.0 * w / r ** 5
            f2 = -3.0 * w / r ** 7
            r2d = (r * r)[..., None] * d
            self.phi[0][a:a + 128] = (w / r).sum((1, 2))
            self.phi[1][a:a + 128] = -torch.einsum("gja,gjab->gb", f0, d)
            self.phi[2][a:a + 128] = torch.einsum("gja,gjab,gjac->gbc", f1, d, d) - eye * f0.sum((1, 2))[:, None, None]
            m = 5.0 * torch.einsum("gja,gjab,gjac,gjad->gbcd", f2, d, d, d)
            s = torch.einsum("gja,gjab->gb", f2, r2d)
            for p, q in (("gb,cd->gbcd", 0), ("gc,bd->gbcd", 0), ("gd,bc->gbcd", 0)):
                m -= torch.einsum(p, s, eye)
            self.phi[3][a:a + 128] = m

    def forces(self):
        v, x = self.v, self.x
        g = torch.zeros_like(x)
        d = x[self.j][:, None] - x[self.i][:, :, None]                  # pair, atom of i, atom of j, xyz
        r = (d ** 2).sum(-1).sqrt()
        qq = self.q[:, None] * self.q[None]
        vel = qq / r
        dv = -vel / r ** 2
        r6 = r[:, 0, 0] ** -6
        va, vb = v.A_OO * r6 * r6, v.B_OO * r6
        dv[:, 0, 0] += (-12.0 * va + 6.0 * vb) / r[:, 0, 0] ** 2
        f = dv[..., None] * d
        g.index_add_(0, self.i, -f.sum(2))
        g.index_add_(0, self.j, f.sum(1))
        E = np.zeros(QB_NE)
        E[19], E[20] = float(vel.sum()), float((va - vb).sum())
        # the Taylor expansion of the field at each atom
        p0, p1, p2, p3 = self.phi
        dr = self.lc[:, None] - x
        h2, h3 = torch.einsum("gbc,gab->gac", p2, dr), torch.einsum("gbcd,gac,gad->gab", p3, dr, dr)
        pot = p0[:, None] + torch.einsum("gb,gab->ga", p1, dr) + 0.5 * (h2 * dr).sum(-1)
        E[2] = float((0.5 * self.q * pot).sum())
        g -= self.q[:, None] * (p1[:, None] + h2 + 0.5 * h3)
        # radial restraint of the oxygens
        u = x[:, 0] - self.centre
        b = u.norm(dim=1)
        shift = math.sqrt(float(np.float32(0.001986)) * self.tfree / v.fk_wsphere) if v.fk_wsphere else 0.0
        db = b - (v.rwat - shift)
        fx = torch.exp(v.awmz * db.clamp_max(0.0))
        out = db > 0
        E[27] = float(torch.where(out, 0.5 * v.fk_wsphere * db ** 2 - v.Dwmz, v.Dwmz * (fx * fx - 2.0 * fx)).sum())
        dv = torch.where(out, v.fk_wsphere * db, -2.0 * v.Dwmz * v.awmz * (fx - fx * fx)) / b
        g[:, 0] += dv[:, None] * u
        # polarisation restraint, shell by shell
        if self.shells:
            mu = x[:, 1] + x[:, 2] - 2.0 * x[:, 0]
            rm = mu.norm(dim=1, keepdim=True)
            mu, uc = mu / rm, u / b[:, None]
            cs = (mu * uc).sum(1).clamp(-1.0, 1.0)
            th = torch.acos(cs)
            shell = torch.full_like(b, -1, dtype=torch.long)
            inner = np.float32(self.rout[-1]) - np.float32(self.dr[-1])
            for k in range(self.shells):                                 # the outermost shell is index 0
                shell[(b > float(inner)) & ((b <= self.rout[k]) | (k == 0))] = k
            for k in range(self.shells):
                w = torch.nonzero(shell == k)[:, 0]
                if not len(w):
                    continue
                w = w[torch.sort(th[w], stable=True).indices]
                rank = torch.arange(1, len(w) + 1, device=self.dev, dtype=torch.float64)
                t0 = torch.acos((1.0 + (1.0 - 2.0 * rank) / len(w)).clamp(-1.0, 1.0))
                t0 = (t0 - 1.5 * torch.sin(t0) * self.cstb[k]).clamp(0.0, math.pi)
                dth = th[w] - t0 + self.tcorr[k]
                E[28] += float((0.5 * v.fkwpol * dth ** 2).sum())
                f0 = -v.fkwpol * dth / torch.sin(th[w]).clamp_min(1e-12)
                f1 = (uc[w] - mu[w] * cs[w, None]) / rm[w]
                f2 = (mu[w] - uc[w] * cs[w, None]) / b[w, None]
                g[w, 0] += f0[:, None] * (f2 - 2.0 * f1)
                g[w, 1] += f0[:, None] * f1
                g[w, 2] += f0[:, None] * f1
        E[23] = E[27] + E[28]
        E[0], E[1] = E[2] + E[19] + E[20] + E[23], self.kin
        return E, g

    def step(self):
        v = self.v
        E, g = self.forces()
        old = self.x
        self.vel = (self.vel - g * self.winv[..., None] * v.dt) * self.tscale
        x = list((old + self.vel * v.dt).unbind(1))
        w = self.winv[0]
        done = [torch.zeros(self.n, dtype=torch.bool, device=self.dev) for _ in range(3)]
        pairs = [(v.shake_i[k], v.shake_j[k], v.shake_dist2[k]) for k in range(3)]
        first = min(p[0] for p in pairs)
        for _ in range(1000):
            for k, (i, j, d2) in enumerate(pairs):
                i, j = i - first, j - first
                d, e = x[i] - x[j], old[:, i] - old[:, j]
                diff = d2 - (d * d).sum(1)
                corr = torch.where(done[k], 0.0, diff / (2.0 * (d * e).sum(1) * (w[i] + w[j])))[:, None] * e
                done[k] = done[k] | (diff.abs() < 0.0001 * d2)
                x[i], x[j] = x[i] + corr * w[i], x[j] - corr * w[j]
            if all(bool(c.all()) for c in done):
                break
        self.x = torch.stack(x, 1)
        self.vel = (self.x - old) / v.dt
        self._temperature()
        E[1] = self.kin
        return E


def _exact_fep(case, seed):
    """qfep's estimators over the series, vectorised (the single-precision quotients it forms are kept)."""
    series = _series(case, seed)
    rt, skip, nbins, nmin = 0.592, case["skip"], 20, 5
    nw, ns = case["windows"], case["states"]
    lam = np.stack([s[0, :, 0] for s in series])
    V = [s[skip:, :, 1] for s in series]
    veff = lambda a, b: sum(lam[a, k] * V[b][:, k] for k in range(ns))
    vg = [0.5 * (u[:, 0] + u[:, 1]) - 0.5 * np.abs(u[:, 0] - u[:, 1]) if ns == 2 else u.min(1) for u in V]
    gap = [u[:, 0] - u[:, 1] for u in V]
    scale = lambda n: float(np.float32(1.0) / np.float32(n))
    av = np.stack([s[skip:].sum(0) * scale(len(s) - skip) for s in series])
    av[:, :, 0] = lam
    z = {k: np.zeros(nw + 2) for k in ("dgf", "dgr", "dgti", "dglu", "dgbar", "dgfsum", "dgrsum", "dG", "dgtisum",
                                       "dglusum", "dgbarsum")}
    for f in range(nw):
        z["dgti"][f + 1] = (V[f][:, 1] - V[f][:, 0]).mean()
        if f:
            z["dgr"][f + 1] = -rt * math.log(np.exp(-(veff(f - 1, f) - veff(f, f)) / rt).mean())
        if f + 1 < nw:
            a, b = veff(f + 1, f) - veff(f, f), veff(f + 1, f + 1) - veff(f, f + 1)
            z["dgf"][f + 1] = -rt * math.log(np.exp(-a / rt).mean())
            c = z["dglu"][f + 1] = -rt * math.log(np.exp(-a / 2 / rt).mean() / np.exp(b / 2 / rt).mean())
            up, down = float(np.float32(len(a)) / np.float32(len(b))), float(np.float32(len(b)) / np.float32(len(a)))
            for _ in range(fep.BAR_MAX_ITER):
                fa, fb = (1 / (1 + up * np.exp((a - c) / rt))).mean(), (1 / (1 + down * np.exp((c - b) / rt))).mean()
                old, c = c, -rt * math.log(fa / fb * math.exp(-c / rt) * up)
                if abs(old - c) <= 0.001:
                    break
            z["dgbar"][f + 1] = c
    for i in range(1, nw):
        for k in ("dgf", "dglu", "dgbar"):
            z[k + "sum"][i + 1] = z[k + "sum"][i] + z[k][i]
        z["dgtisum"][i + 1] = z["dgtisum"][i] + 0.5 * (z["dgti"][i] + z["dgti"][i + 1]) * (lam[i - 1, 0] - lam[i, 0])
        z["dG"][i + 1] = z["dG"][i] + 0.5 * (z["dgf"][i] - z["dgr"][i + 1])
    for i in range(nw, 1, -1):
        z["dgrsum"][i - 1] = z["dgrsum"][i] + z["dgr"][i]
    lo, hi = min(999.0, min(g.min() for g in gap)), max(-999.0, max(g.max() for g in gap))
    xint = (hi - lo) / nbins
    p2, p3 = np.zeros((nw, nbins + 2, fep.PART2_W)), np.zeros((nbins + 2, fep.PART3_W))
    p2[:, 1:nbins + 1, 0] = p3[1:nbins + 1, 0] = lo + np.arange(1, nbins + 1) * xint - xint / 2.0
    for f in range(nw):
        ib = np.clip(((gap[f] - lo) / xint).astype(int) + 1, 0, nbins + 1)
        for b in range(1, nbins + 1):
            m = ib == b
            if m.sum() < nmin:
                continue
            fe = []
            for e in (V[f][m, 0], V[f][m, 1], vg[f][m]):
                e = e - veff(f, f)[m]
                fe.append(z["dG"][f + 1] - rt * math.log(np.exp(-(e - e.mean()) / rt).mean()) + e.mean())
            p2[f, b, 1:] = fe + [m.sum(), 0.0, 0.0, 1.0, 0.0]
    n = p2[:, :, 4].sum(0)
    use = n >= nmin
    mean = np.where(use, (p2[:, :, 3] * p2[:, :, 4]).sum(0) / np.maximum(n, 1), 0.0)
    p3[use, 1], p3[use, 2], p3[use, 3], p3[use, 7] = mean[use], (mean - min(0.0, mean.min()))[use], n[use], 1.0
    return dict(z, lam=lam, npts=None, avEQ=av, bar_iterations=None, gap_range=np.array([lo, hi]), part2=p2, part3=p3)


def _exact_train(case, seed):
    x, t = (torch.from_numpy(a).double() for a in _training_set(case, seed))
    w = torch.from_numpy(mlp.init(seed % 1000, True)).double()
    shapes = [(mlp.HID, mlp.IN), (mlp.HID,), (mlp.HID, mlp.HID), (mlp.HID,), (mlp.OUT, mlp.HID), (mlp.OUT,)]
    sizes = [math.prod(s) for s in shapes]
    decay = torch.cat([torch.full((k,), 0.01 if len(s) == 2 else 0.0, dtype=torch.float64)
                       for k, s in zip(sizes, shapes)])
    m, u, loss = torch.zeros_like(w), torch.zeros_like(w), []
    for it in range(1, case["iters"] + 1):
        p = w.clone().requires_grad_()
        w1, b1, w2, b2, w3, b3 = (a.reshape(s) for a, s in zip(p.split(sizes), shapes))
        h = torch.nn.functional.silu(x @ w1.T + b1)
        h = torch.nn.functional.silu(h @ w2.T + b2)
        e = ((h @ w3.T + b3 - t) ** 2).mean()
        loss.append(float(e.detach()))
        (g,) = torch.autograd.grad(e, p)
        m, u = 0.9 * m + 0.1 * g, 0.999 * u + 0.001 * g * g
        w = w - 2e-3 * (m / (1 - 0.9 ** it) / ((u / (1 - 0.999 ** it)).sqrt() + 1e-8) + decay * w)
    return {"w": w, "loss": np.array(loss)}


def exact(case, seed):
    """None for the MD of systems with a solute (their bonded, exclusion, soft-core and Q-atom terms in
    plain torch would take far longer than the 20 seconds a value may) and of the mixed engine (SHAKE's
    readiness tests turn any rounding of a force into another number of sweeps, so its trajectory has no
    such value; its forces and energies have, in the single points)."""
    kind = case["kind"]
    if kind == "qfep":
        return _exact_fep(case, seed)
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "static":
        s, x = _static_inputs(case, seed)
        e = _Sphere(s)
        e.x = torch.as_tensor(x, device=e.dev).reshape(-1, 3, 3)
        o = e.x[:, 0]
        e.i, e.j = torch.nonzero(torch.triu(((o[:, None] - o[None]) ** 2).sum(-1) <= 100.0, 1), as_tuple=True)
        e.lc, e.shells, e.v.fk_wsphere, e.v.Dwmz = o, 0, 0.0, 0.0
        e.phi = [torch.zeros((e.n,) + (3,) * k, dtype=torch.float64, device=e.dev) for k in range(4)]
        E, g = e.forces()
        return {"grad": g.reshape(-1), "energy": E[19:21], "status": None}
    if kind == "point":
        systems, rng = _systems(case, seed), np.random.default_rng(seed)
        E, G = [], []
        for s in systems:
            e = _Sphere(s)
            e.x = torch.as_tensor(_jittered(s, rng), device=e.dev).reshape(-1, 3, 3)
            e.lists()
            ev, g = e.forces()
            E.append(ev)
            G.append(g.reshape(-1).cpu().numpy())
        return {"E": np.stack(E), "grad": np.concatenate(G)}
    if case["system"] != "sphere" or case["precision"] != "fp64":
        return None
    s = _systems(case, seed)[0]
    e = _Sphere(s)
    rec = []
    for k in range(MD_STEPS):
        if k % s.view.NBcycle == 0:
            e.lists()
        E = e.step()
        if k and k % s.view.iene_cycle == 0:
            rec.append(np.concatenate([[float(k)], E]))
    return {"x": e.x.reshape(-1), "v": e.vel.reshape(-1), "counts": None,
            "records": np.pad(np.stack(rec)[None], ((0, 0), (0, 0), (0, 10 * QB_NEQ + 10)))}
