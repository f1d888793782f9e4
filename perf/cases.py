"""The work that users have this framework do, as measurable cases.

Every case goes through the public entry points a program uses: a Stepper
(or the C ABI behind it) that steps boxes and hands the state back in host
arrays, adjoint.rollout, and the packing and analysis calls.  Sizes and
parameters are those of the repository's own workloads (bench.py,
scenes.py) and of its tests, from a few hundred spheres to a million.

The step cases advance a simulation from one output to the next, as run()
does: some tens to hundreds of steps, then the whole particle state into
pinned host arrays and the walls' state.  A pass continues where the last
one stopped.
"""
import copy
import ctypes
import math

import numpy
import torch

from sphere_b200 import adjoint, scenes
from sphere_b200.runner import HostBonds, HostParticles, Stepper

FIELDS = ("x", "xyzsum", "vel", "force", "angpos", "angvel", "torque",
          "es_dot", "es", "ev_dot", "ev", "p")


def listed():
    return [
        # the smallest call: a test-sized shear box, latency and launches only
        {"name": "shear_fp64_500", "kind": "step", "scene": "shear", "n": 500, "precision": "fp64",
         "launch": "default", "order": "lattice", "steps": 100},
        # the gravity-settling workload (10,000 spheres, walls on all sides)
        {"name": "settle_fp64_10k", "kind": "step", "scene": "settle", "n": 10000,
         "precision": "fp64", "launch": "default", "order": "lattice", "steps": 100},
        # an ordinary sim.run(): FP64, no tuning, spheres in the order of a
        # random deposition
        {"name": "shear_fp64_60k", "kind": "step", "scene": "shear", "n": 60013, "precision": "fp64",
         "launch": "default", "order": "random", "steps": 50},
        # the headline pack in the bit-exact form
        {"name": "shear_fp64_1e6", "kind": "step", "scene": "shear", "n": 1000000,
         "precision": "fp64", "launch": "tuned", "order": "lattice", "steps": 50},
        # a mid-sized pack in the mixed form with lengths in 64 bits, spheres
        # in random order
        {"name": "shear_mixed_20k", "kind": "step", "scene": "shear", "n": 20011,
         "precision": "mixed", "length": "fp64", "launch": "tuned", "order": "random",
         "steps": 100},
        # the headline pack: 1e6 spheres, mixed form
        {"name": "shear_mixed_1e6", "kind": "step", "scene": "shear", "n": 1000000,
         "precision": "mixed", "length": "reference", "launch": "tuned", "order": "lattice",
         "steps": 100},
        # the batched ensemble: 256 boxes of 500 to 20,000 spheres
        {"name": "ensemble_mixed_256", "kind": "ensemble", "boxes": 256, "n_min": 500,
         "n_max": 20000, "steps": 50},
        # the bonded pack: Young's-modulus contacts and linear bonds, in the
        # launch variant the tuner picks for it
        {"name": "bonded_mixed_200k", "kind": "step", "scene": "bonded", "n": 200000,
         "precision": "mixed", "length": "reference", "launch": "split", "order": "lattice",
         "steps": 50},
        # a pack in a Darcy fluid that is solved at every step
        {"name": "darcy_fp64_100k", "kind": "darcy", "n": 100000, "steps": 10},
        # one gradient of a settling/impact run: forward and backward
        {"name": "adjoint_50k", "kind": "adjoint", "n": 50000, "steps": 200, "ckpt": 50},
        # scene packing: overlap-removal sweeps of the headline pack
        {"name": "relax_1e6", "kind": "relax", "n": 1000000, "sweeps": 50},
        # what is read off one output file: image, porosity profile, overlaps
        {"name": "analysis_200k", "kind": "analysis", "n": 200000, "width": 800, "slices": 10},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("step", "step", "step", "step", "ensemble", "darcy", "adjoint", "relax",
                       "analysis"))
    if kind == "step":
        scene = rng.choice(("shear", "shear", "shear", "settle", "bonded"))
        n = {"shear": _log_int(rng, 500, 1000000), "settle": _log_int(rng, 1000, 10000),
             "bonded": _log_int(rng, 5000, 200000)}[scene]
        precision = rng.choice(("fp64", "mixed"))
        launch = "tuned" if rng.random() < (0.8 if n > 100000 else 0.4) else "default"
        if scene == "bonded":
            launch = rng.choice(("split", "default"))
        case = {"kind": "step", "scene": scene, "n": n, "precision": precision, "launch": launch,
                "order": rng.choice(("lattice", "random")) if scene == "shear" else "lattice",
                "steps": 100 if n < 100000 else 50}
        if precision == "mixed":
            case["length"] = rng.choice(("reference", "fp64"))
        return case
    if kind == "ensemble":
        return {"kind": "ensemble", "boxes": rng.randint(8, 256), "n_min": 500,
                "n_max": _log_int(rng, 1000, 20000), "steps": 50}
    if kind == "darcy":
        return {"kind": "darcy", "n": _log_int(rng, 5000, 100000), "steps": 10}
    if kind == "adjoint":
        return {"kind": "adjoint", "n": _log_int(rng, 2000, 50000),
                "steps": rng.choice((60, 100, 150, 200)), "ckpt": rng.choice((20, 50, 100))}
    if kind == "relax":
        return {"kind": "relax", "n": _log_int(rng, 10000, 1000000), "sweeps": 50}
    # slabs thicker than the largest sphere, as the porosity profile asks
    n = _log_int(rng, 5000, 200000)
    slabs = int(0.5 * (2.0 * n * 8.3e-6) ** (1.0 / 3.0) / 0.045)
    return {"kind": "analysis", "n": n, "width": rng.choice((400, 800, 1024)),
            "slices": rng.randint(2, min(slabs, 12))}


# ------------------------------------------------------------------ scenes

_PACKS = {}


def _pack(key, make):
    """The pack behind a case (geometry only: made once, as a program loads
    it once); the seed's variation is applied to a copy."""
    if key not in _PACKS:
        while len(_PACKS) >= 3:
            _PACKS.pop(next(iter(_PACKS)))
        _PACKS[key] = make()
    return copy.deepcopy(_PACKS[key])


def _vary(s, rng, shift=True, vel_sigma=0.002, order="lattice"):
    """The seed's state of a pack: moved by a random vector along its
    periodic axes, free spheres with small random velocities and spins, and
    for order "random" the spheres renumbered."""
    n = int(s.np[0])
    if shift:
        for d in range(2):
            s.x[:, d] = numpy.mod(s.x[:, d] + rng.uniform(0.0, 1.0) * s.L[d], s.L[d])
    free = numpy.asarray(s.fixvel).reshape(-1) == 0.0
    s.vel[free] += rng.normal(0.0, vel_sigma, (n, 3))[free]
    s.angvel[free] = rng.normal(0.0, 0.2, (n, 3))[free]
    if order == "random":
        p = rng.permutation(n)
        for name in ("x", "radius", "vel", "angvel", "fixvel"):
            setattr(s, name, numpy.ascontiguousarray(getattr(s, name)[p]))
    return s


def _sims(case, seed):
    rng = numpy.random.default_rng([int(seed), 7])
    kind, n = case["kind"], case.get("n")
    if kind == "ensemble":
        sims = _pack(("ensemble", case["boxes"], case["n_min"], case["n_max"]),
                     lambda: scenes.shear_ensemble(nboxes=case["boxes"], seed=0, device=0,
                                                   counts=(case["n_min"], case["n_max"])))
        return [_vary(s, rng) for s in sims]
    if kind == "darcy":
        # a shear box of nearly equal spheres filled with water at
        # hydrostatic pressure, the fluid on the box's cell grid
        s = _pack(("darcy", n), lambda: scenes.shear_ensemble(
            nboxes=1, seed=0, device=0, counts=(n, n))[0])
        s.fluid = True
        s.initFluid(cfd_solver=1, mu=8.9e-4, rho=1.0e3, p=0.0, hydrostatic=True)
        s.setFluidCompressibility(1.0e-7)
        s.setPermeabilityGrainSize()
        s.time_file_dt[0] = 1.0
        return [_vary(s, rng)]
    if kind == "adjoint":
        s = _pack(("loose", n), lambda: scenes.loose_pack(n, seed=0, device=0, nsteps=2000))
        s.vel[:] = rng.normal(0.0, 0.1, (n, 3))
        return [s]
    if kind == "relax":
        return [scenes.dense_pack(n, seed=int(seed), relax=lambda *a: 0.0)[0]]
    if kind == "analysis" or case["scene"] == "shear":
        s = _pack(("shear", n), lambda: scenes.sheared_dense_pack(n, seed=0, device=0))
        return [_vary(s, rng, shift=kind != "analysis", order=case.get("order", "lattice"))]
    if case["scene"] == "settle":
        return [_vary(scenes.gravity_settling(n, seed=int(seed)), rng, shift=False)]
    s = _pack(("bonded", n), lambda: scenes.bonded_pack(n, nbonds=3 * n // 2, seed=0, device=0))
    return [_vary(s, rng, shift=False)]


def _pinned(n):
    hp = HostParticles(0)
    for name in FIELDS:
        w = {"x": 4, "vel": 4}.get(name, 3 if name in FIELDS[:7] else 0)
        shape = (n, w) if w else (n,)
        setattr(hp, name, torch.zeros(shape, dtype=torch.float64, pin_memory=True).numpy())
    return hp


class _State(object):
    def __del__(self):
        st = getattr(self, "st", None)
        if st is not None:
            st.close()


def prepare(case, seed):
    q = _State()
    q.case = case
    q.sims = _sims(case, seed)
    kind = case["kind"]
    if kind == "adjoint":
        q.x_target = torch.from_numpy(_target(q.sims[0], seed)).cuda()
        q.v0 = torch.tensor(q.sims[0].vel, dtype=torch.float64, device="cuda")
        return q
    mixed = kind == "ensemble" or case.get("precision") == "mixed"
    q.st = Stepper(q.sims, precision="mixed" if mixed else "fp64",
                   length=case.get("length", "reference"), device=0)
    q.st.upload()
    if kind == "ensemble" or case.get("launch") == "tuned":
        q.st.autotune(steps=10)
    elif case.get("launch") == "split":
        q.st.set_variant(3)
    q.out = _pinned(q.st.ntot)
    q.bonds = HostBonds(q.st.nbonds)
    return q


def _target(s, seed):
    """Final positions to aim at in the adjoint's loss: the spheres' own
    flight and a scatter of the size of a contact's displacement."""
    rng = numpy.random.default_rng([int(seed), 11])
    return s.x + s.vel * float(s.time_dt[0]) * 200 + rng.normal(0.0, 1.0e-5, s.x.shape)


def _download(q):
    ps, bs = q.out.struct(), q.bonds.struct()
    q.st._check(q.st.lib.sph_download(q.st.h, ctypes.byref(ps),
                                      ctypes.byref(bs) if q.st.nbonds else None), "sph_download")
    out = {name: getattr(q.out, name) for name in FIELDS}
    if q.st.nbonds:
        out["bond_delta_n"], out["bond_delta_t"] = q.bonds.delta_n, q.bonds.delta_t
    return out


def run(q):
    kind = q.case["kind"]
    if kind == "adjoint":
        s = q.sims[0]
        one = lambda v: torch.tensor(float(v), dtype=torch.float64, requires_grad=True)  # noqa: E731
        p = [one(s.k_n[0]), one(s.gamma_n[0]), one(s.mu_s[0])]
        v0 = q.v0.clone().requires_grad_(True)
        x = adjoint.rollout(s, p[0], p[1], p[2], v0, nsteps=q.case["steps"], ckpt=q.case["ckpt"])
        loss = ((x - q.x_target) ** 2).sum(1).mean()
        loss.backward()
        return {"x": x.detach(), "k_n": p[0].grad, "gamma_n": p[1].grad, "mu": p[2].grad,
                "v0": v0.grad}
    if kind == "relax":
        worst = q.st.relax(q.case["sweeps"], alpha=0.6, z_top=float(q.sims[0].x[:, 2].max()))
        return {"x": _download(q)["x"], "max_overlap": worst}
    if kind == "analysis":
        img = q.st.render(method=2, maxval=0.01, width=q.case["width"], height=q.case["width"])
        z, por = q.st.porosity(q.case["slices"])
        pairs, delta = q.st.overlaps()
        return {"image": img, "z": z, "porosity": por, "pairs": pairs.astype(numpy.int64),
                "delta_n": delta}
    q.st.step(q.case["steps"])
    out = _download(q)
    if kind == "darcy":
        f = q.st.darcy_get()
        out.update({k: f[k] for k in ("p_f", "v_f", "phi", "k", "f_p")})
    if kind == "ensemble" or q.case.get("scene") == "shear":
        boxes = q.st.boxes()
        out["wall_x"] = numpy.array([b.walls.nx[0][3] for b in boxes])
        out["wall_force"] = numpy.array([b.walls.mvfd[0][2] for b in boxes])
    return out


# ------------------------------------------------------------------ work


def work(case):
    """Per step and sphere the state read and written once (FP64: 352 B,
    mixed: 220 B) and 52 B per directed contact (its id and its history read
    and written); the download's 240 B per sphere; about 200 operations per
    contact and 150 per sphere."""
    kind = case["kind"]
    n = case.get("n") or case["boxes"] * (case["n_min"] + case["n_max"]) / 2.0
    contacts = {"settle": 0.0, "bonded": 6.0}.get(case.get("scene"), 4.0)
    mixed = kind == "ensemble" or case.get("precision") == "mixed"
    state = 220.0 if mixed else 352.0
    if kind == "adjoint":
        # forward, recompute and reverse of every step; few contacts each
        return {"bytes": case["steps"] * n * 3 * 352.0, "flops": case["steps"] * n * 3 * 250.0}
    if kind == "relax":
        return {"bytes": (case["sweeps"] * 64.0 + 240.0) * n, "flops": case["sweeps"] * n * 200.0}
    if kind == "analysis":
        return {"bytes": 3 * 64.0 * n + 12.0 * 3 * n + 3.0 * case["width"] ** 2,
                "flops": 60.0 * n + 100.0 * case["width"] ** 2}
    b = case["steps"] * n * (state + 52.0 * contacts) + 240.0 * n
    f = case["steps"] * n * (150.0 + 200.0 * contacts)
    if kind == "darcy":
        # two thirds as many fluid cells as spheres; the pressure read and
        # written and ten operations per cell and Jacobi iteration, about 100
        # iterations a step on fields that stay in L2
        b += case["steps"] * 0.66 * n * 120.0
        f += case["steps"] * 0.66 * n * 1000.0
    return {"bytes": b, "flops": f}


def tolerance(case):
    """The FP64 form repeats the reference's arithmetic operation for
    operation and the packing, analysis and fluid work is in FP64 with a
    fixed order: the same bits.  The adjoint's sums are atomic: its outputs
    differ by 8e-15 between two runs on the same inputs.  The mixed form
    against exact(), measured: with FP64 lengths forces differ by 1e-6 and
    the frictional heat, which a contact at the edge of slipping switches on
    and off, by up to 3e-5; with the reference's lengths, rounded to 32 bits
    (1e-9 m, where an overlap is 7e-9 m), one last bit of a position moves a
    force by a tenth now and then, and forces differ by 4e-3 to 6e-3 after
    100 steps."""
    kind = case["kind"]
    if kind == "adjoint":
        return {"rel": 1e-12}
    if kind == "ensemble" or case.get("precision") == "mixed":
        if case.get("length", "reference") == "fp64":
            return {"rel": 1.5e-4, "max": 0.1}
        return {"rel": 0.02, "max": 0.99}
    return "exact"


# ------------------------------------------------------------------ exact
#
# The same work in plain torch in 64 bits: the reference's algorithm (linear
# contacts with history, plane walls, linear bonds, third-order Taylor
# integration, wall under normal stress), with lengths rounded to 32 bits
# where the framework's default length mode, the reference's sqrtf, rounds
# them.

PI = 3.14159265358979
PI_E = 3.141592654


def _len(v, f32):
    # the three squares added in order, as the reference adds them
    d = (v[..., 0] * v[..., 0] + v[..., 1] * v[..., 1]) + v[..., 2] * v[..., 2]
    return d.float().sqrt().double() if f32 else d.sqrt()


def _candidates(x, r, base, L, periodic, skin):
    """Directed pairs (i, j) of one box with |x_i - x_j| < r_i + r_j + skin
    under the nearest image, from cells of the largest reach."""
    n, dev = x.shape[0], x.device
    reach = 2.0 * float(r.max()) + skin
    lo = torch.zeros(3, dtype=torch.float64, device=dev)
    top = torch.maximum(torch.tensor(L, dtype=torch.float64, device=dev), x.max(0).values + 1e-9)
    num = [max(1, int(float(top[d]) / reach)) for d in range(3)]
    if periodic and min(num[:2]) < 3 or n < 600:
        ii = torch.arange(n, device=dev).repeat_interleave(n)
        jj = torch.arange(n, device=dev).repeat(n)
        parts = [(ii, jj)]
    else:
        numt = torch.tensor(num, device=dev)
        c = torch.minimum(((x - lo) / (top / numt)).floor().long().clamp(min=0), numt - 1)
        cid = (c[:, 2] * num[1] + c[:, 1]) * num[0] + c[:, 0]
        order = torch.argsort(cid, stable=True)
        start = torch.searchsorted(cid[order], torch.arange(num[0] * num[1] * num[2] + 1, device=dev))
        parts = []
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    q = c + torch.tensor([dx, dy, dz], device=dev)
                    ok = (q[:, 2] >= 0) & (q[:, 2] < num[2])
                    for d in range(2):
                        if periodic:
                            q[:, d] %= num[d]
                        else:
                            ok &= (q[:, d] >= 0) & (q[:, d] < num[d])
                    i = torch.nonzero(ok).flatten()
                    t = (q[i, 2] * num[1] + q[i, 1]) * num[0] + q[i, 0]
                    s, cnt = start[t], start[t + 1] - start[t]
                    for k in range(int(cnt.max()) if len(i) else 0):
                        m = cnt > k
                        parts.append(_near(x, r, i[m], order[s[m] + k], L, periodic, skin))
    if len(parts) == 1:
        parts = [_near(x, r, *parts[0], L, periodic, skin)]
    ii = torch.cat([p[0] for p in parts])
    jj = torch.cat([p[1] for p in parts])
    key = torch.argsort(ii * n + jj)
    return ii[key] + base, jj[key] + base


def _near(x, r, i, j, L, periodic, skin):
    d = x[i] - x[j]
    if periodic:
        for k in range(2):
            d[:, k] -= L[k] * torch.round(d[:, k] / L[k])
    m = ((d * d).sum(1).sqrt() < r[i] + r[j] + skin) & (i != j)
    return i[m], j[m]


class _Exact(object):
    """State of one or more boxes, stepped in 64 bits."""

    def __init__(self, sims, f32):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.tensor(numpy.asarray(a, dtype=numpy.float64), device=dev)  # noqa: E731
        cat = lambda name, w: t(numpy.concatenate(  # noqa: E731
            [numpy.asarray(getattr(s, name), dtype=numpy.float64).reshape((-1, w) if w else -1)
             for s in sims]))
        self.sims, self.f32, self.dev = sims, f32, dev
        self.nb = [int(s.np[0]) for s in sims]
        self.x, self.r, self.v, self.w = cat("x", 3), cat("radius", 0), cat("vel", 3), cat("angvel", 3)
        self.fix = cat("fixvel", 0)
        n = self.n = int(self.x.shape[0])
        self.box = torch.tensor(numpy.repeat(numpy.arange(len(sims)), self.nb), device=dev)
        per = lambda f: t([f(s) for s in sims])[self.box]  # noqa: E731
        self.k_n, self.k_t, self.E = (per(lambda s, a=a: float(getattr(s, a)[0])) for a in ("k_n", "k_t", "E"))
        self.gn, self.gt, self.mu, self.gwn = (per(lambda s, a=a: float(getattr(s, a)[0]))
                                               for a in ("gamma_n", "gamma_t", "mu_s", "gamma_wn"))
        self.dt = per(lambda s: float(s.time_dt[0]))
        self.g = t([numpy.asarray(s.g, dtype=float) for s in sims])[self.box]
        self.L = t([numpy.asarray(s.L, dtype=float) for s in sims])[self.box]
        self.periodic = int(sims[0].periodic[0]) == 1
        self.m = 4.0 / 3.0 * PI * self.r ** 3 * per(lambda s: float(s.rho[0]))
        self.nw = int(sims[0].nw[0])
        first = lambda a: t([float(getattr(s, a)[0]) for s in sims])  # noqa: E731
        if self.nw:
            self.wmode = int(sims[0].wmode[0])
            self.wx, self.wv, self.wm, self.ws = first("w_x"), first("w_vel"), first("w_m"), first("w_sigma0")
            self.wa = torch.zeros_like(self.wx)
        self.wL = t([numpy.asarray(s.L, dtype=float) for s in sims])
        self.wdt = first("time_dt")
        z3 = lambda: torch.zeros(n, 3, dtype=torch.float64, device=dev)  # noqa: E731
        self.xyzsum, self.angpos, self.A, self.O = z3(), z3(), z3(), z3()
        self.es, self.ev = (torch.zeros(n, dtype=torch.float64, device=dev) for _ in range(2))
        self.it = 0
        self.ref = None
        self.H = None
        s = sims[0]
        self.bonds = None
        if int(s.nb0[0]):
            self.bonds = torch.tensor(numpy.asarray(s.bonds).astype(numpy.int64), device=dev)
            self.bdn = torch.zeros(len(self.bonds), dtype=torch.float64, device=dev)
            self.bdt = torch.zeros(len(self.bonds), 3, dtype=torch.float64, device=dev)
            self.bon, self.bot = self.bdn.clone(), self.bdt.clone()
            self.alive = torch.ones(len(self.bonds), dtype=torch.bool, device=dev)

    def pairs(self):
        skin = 0.1 * float(self.r.min())
        with torch.no_grad():
            x = self.x.detach()
            if self.ref is not None:
                d = x - self.ref
                if self.periodic:
                    L = self.L[:, :2]
                    d = torch.cat([d[:, :2] - L * torch.round(d[:, :2] / L), d[:, 2:]], 1)
                if float((d * d).sum(1).max()) < (0.49 * skin) ** 2:
                    return
            ii, jj, o = [], [], 0
            for s, k in zip(self.sims, self.nb):
                a, b = _candidates(x[o:o + k], self.r[o:o + k], o, [float(v) for v in s.L],
                                   self.periodic, skin)
                ii.append(a)
                jj.append(b)
                o += k
            i, j = torch.cat(ii), torch.cat(jj)
        H = torch.zeros(len(i), 3, dtype=torch.float64, device=self.dev)
        if self.H is not None and len(self.i):
            old = self.i * self.n + self.j
            pos = torch.searchsorted(old, i * self.n + j).clamp(max=len(old) - 1)
            same = old[pos] == i * self.n + j
            H = torch.where(same[:, None], self.H[pos], H)
        self.i, self.j, self.H, self.ref = i, j, H, x.clone()

    def image(self, d, i):
        if not self.periodic:
            return d
        L = self.L[i, :2]
        q = d[:, :2]
        q = torch.where(q > 0.5 * L, q - L, torch.where(q < -0.5 * L, q + L, q))
        return torch.cat([q, d[:, 2:]], 1)

    def bond_forces(self, F, T):
        s = self.sims[0]
        bi, bj = self.bonds[:, 0], self.bonds[:, 1]
        dt = float(s.time_dt[0])
        gn, gt, kn, kt = (float(getattr(s, a)[0]) for a in ("gamma_n", "gamma_t", "k_n", "k_t"))
        dot = lambda a, b: (a * b).sum(1, keepdim=True)  # noqa: E731
        cr = lambda a, b: torch.linalg.cross(a, b)  # noqa: E731
        R = float(s.lambda_bar[0]) * torch.minimum(self.r[bi], self.r[bj])
        Ar, I = PI * R * R, 0.25 * PI * R ** 4
        x = self.x[bi] - self.x[bj]
        ln = _len(x, self.f32)
        ov = torch.clamp(ln - (self.r[bi] + self.r[bj]), max=0.0)
        n = x / ln[:, None]
        d0 = self.bdt - n * dot(n, self.bdt)
        dd = (self.v[bi] - self.v[bj] + (self.r[bi] + ov / 2)[:, None] * cr(n, self.w[bi])
              + (self.r[bj] + ov / 2)[:, None] * cr(n, self.w[bj])) * dt
        ddn = -dot(dd, n)[:, 0]
        dn = self.bdn + ddn
        ddt = dd - n * dot(n, dd)
        d1 = d0 + ddt
        fn = (kn * Ar * dn + gn * ddn / dt)[:, None] * n
        ft = -(kt * Ar)[:, None] * d1 - gt * ddt / dt
        o0 = self.bot - n * dot(n, self.bot)
        do = (self.w[bj] - self.w[bi]) * dt
        don = dot(do, -n)[:, 0]
        on = self.bon + don
        o1 = o0 + do + don[:, None] * n
        tn = (kt * 2 * I * on)[:, None] * n
        tt = -(kn * I)[:, None] * o1
        sig = _len(fn, self.f32) / Ar + _len(tt, self.f32) * R / I
        tau = _len(ft, self.f32) / Ar + _len(tn, self.f32) * R / (2 * I)
        self.alive &= ~((sig >= float(s.sigma_b[0])) | (tau >= float(s.tau_b[0])))
        a = self.alive[:, None]
        self.bdt, self.bot = torch.where(a, d1, self.bdt), torch.where(a, o1, self.bot)
        self.bdn = torch.where(self.alive, dn, self.bdn)
        self.bon = torch.where(self.alive, on, self.bon)
        f = torch.where(a, fn + ft, torch.zeros_like(fn))
        t = torch.where(a, tn + tt, torch.zeros_like(fn))
        return F.index_add(0, bi, f).index_add(0, bj, -f), T.index_add(0, bi, -t).index_add(0, bj, t)

    def step(self):
        n, f32 = self.n, self.f32
        self.pairs()
        with torch.no_grad():
            d = self.image(self.x[self.i] - self.x[self.j], self.i)
            hit = torch.nonzero(_len(d, f32) - (self.r[self.i] + self.r[self.j]) < 0.0).flatten()
        i, j = self.i[hit], self.j[hit]
        X = self.image(self.x[i] - self.x[j], i)
        ln = _len(X, f32)
        ra, rb = self.r[i], self.r[j]
        delta = ln - (ra + rb)
        nrm = X / ln[:, None]
        dot = lambda a, b: (a * b).sum(1, keepdim=True)  # noqa: E731
        cr = lambda a, b: torch.linalg.cross(a, b)  # noqa: E731
        sa, sb = (ra + delta / 2)[:, None], (rb + delta / 2)[:, None]
        vl = self.v[i] - self.v[j]
        vel = vl + sa * cr(nrm, self.w[i]) + sb * cr(nrm, self.w[j])
        vn = -dot(vl, nrm)[:, 0]
        vt = vel - nrm * dot(nrm, vel)
        vtl = _len(vt.detach(), f32)
        kn, kt = self.k_n[i], self.k_t[i]
        ke = PI_E / 2.0 * self.E[i] * (ra + rb) / 2.0
        kn, kt = torch.where(self.E[i] > .001, ke, kn), torch.where(self.E[i] > .001, ke, kt)
        gn, gt, mu, dt = self.gn[i], self.gt[i], self.mu[i], self.dt[i]
        h0 = self.H[hit]
        d0 = h0 - nrm * dot(nrm, h0)
        fn = torch.clamp(-kn * delta + gn * vn, min=0.0)[:, None] * nrm
        safe = lambda v: (v * v).sum(1).clamp(min=1e-300).sqrt()  # noqa: E731
        ln_of = (lambda v: _len(v, True)) if f32 else safe
        fnl = ln_of(fn)
        tang = (_len(d0.detach(), f32) > 0.0) | (vtl > 0.0)
        dtv = d0 + vt * dt[:, None]
        ft0 = -kt[:, None] * dtv - gt[:, None] * vt
        ftl = ln_of(ft0)
        lim = mu * fnl
        slip = tang & (ftl.detach() > lim.detach())
        one = torch.ones_like(ftl)
        tdir = ft0 / torch.where(slip, ftl, one)[:, None]
        fts = lim[:, None] * tdir
        dns = (-1.0 / kt)[:, None] * (lim[:, None] * tdir + gt[:, None] * vt)
        ft = torch.where(slip[:, None], fts, ft0)
        dnew = torch.where(slip[:, None], dns, dtv)
        ft = torch.where(tang[:, None], ft, torch.zeros_like(ft))
        dnew = torch.where(tang[:, None], dnew, torch.zeros_like(dnew))
        z1 = lambda: torch.zeros(n, dtype=torch.float64, device=self.dev)  # noqa: E731
        z3 = lambda: torch.zeros(n, 3, dtype=torch.float64, device=self.dev)  # noqa: E731
        F = z3().index_add(0, i, fn + ft)
        T = z3().index_add(0, i, -sa * cr(nrm, ft))
        p = z1().index_add(0, i, fnl / (4.0 * PI * ra * ra))
        ev = z1().index_add(0, i, 0.5 * gn * vn * vn + torch.where(tang, 0.5 * gt * vtl * vtl, 0.0 * vtl))
        es = z1().index_add(0, i, torch.where(slip, 0.5 * ln_of(ft) * vtl, 0.0 * vtl))
        self.H = torch.zeros_like(self.H).index_copy(0, hit, dnew)
        # plane walls: the top (a dynamic wall when there is one), the bottom,
        # and the sides of a box that is not periodic
        kw = torch.where(self.E > .001, PI_E / 2.0 * self.E * self.r, self.k_n)
        top = self.wx[self.box] if self.nw else self.L[:, 2]
        walls = [(2, top, -1.0), (2, 0.0 * self.r, 1.0)]
        if not self.periodic:
            walls += [(0, self.L[:, 0], -1.0), (0, 0.0 * self.r, 1.0),
                      (1, self.L[:, 1], -1.0), (1, 0.0 * self.r, 1.0)]
        cols = [0.0, 0.0, 0.0]
        for q, (axis, pos, sgn) in enumerate(walls):
            dw = pos - (self.x[:, axis] + self.r) if sgn < 0 else self.x[:, axis] - self.r - pos
            vw = sgn * self.v[:, axis]
            on = dw.detach() < 0.0
            fw = torch.where(on, torch.clamp(-kw * dw - self.gwn * vw, min=0.0), 0.0 * dw)
            if q == 0:
                w0 = fw
            cols[axis] = cols[axis] + sgn * fw
            p = p + fw.detach() / (4.0 * PI * self.r * self.r)
            ev = ev + torch.where(on, self.gwn * vw * vw, 0.0 * dw)
        F = F + torch.stack([c if torch.is_tensor(c) else z1() for c in cols], 1)
        if self.bonds is not None:
            F, T = self.bond_forces(F, T)
        acc = F / self.m[:, None] + self.g
        ang = T / (2.0 / 5.0 * self.m * self.r * self.r)[:, None]
        held = ((self.fix > 1e-4) & (self.fix < 10.0))[:, None]
        keep = torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64, device=self.dev)
        acc = torch.where(held, (F / self.m[:, None]) * keep, acc)
        ang = torch.where(held, torch.zeros_like(ang), ang)
        h = self.dt[:, None]
        ja = (acc - (self.A if self.it else 0.0 * acc)) / h
        jo = (ang - (self.O if self.it else 0.0 * ang)) / h
        dx = self.v * h + 0.5 * acc * h * h + (1.0 / 6.0) * ja * h * h * h
        self.x = self.x + dx
        self.xyzsum = self.xyzsum + dx.detach()
        self.v = self.v + acc * h + 0.5 * ja * h * h
        self.angpos = self.angpos + (self.w * h + 0.5 * ang * h * h + (1.0 / 6.0) * jo * h * h * h).detach()
        self.w = self.w + ang * h + 0.5 * jo * h * h
        self.A, self.O = acc, ang
        if self.periodic:
            xy, L = self.x[:, :2], self.L[:, :2]
            xy = torch.where(xy < 0.0, xy + L, xy)
            self.x = torch.cat([torch.where(xy > L, xy - L, xy), self.x[:, 2:]], 1)
        self.F, self.T, self.p, self.es_dot, self.ev_dot = F, T, p, es.detach(), ev.detach()
        self.es = self.es + self.es_dot * self.dt
        self.ev = self.ev + self.ev_dot * self.dt
        if self.nw:
            fsum = torch.zeros_like(self.wx).index_add(0, self.box, w0)
            self.wf = fsum
            acc = (fsum - self.ws * self.wL[:, 0] * self.wL[:, 1]) / self.wm
            if self.wmode == 2:
                acc = 0.0 * acc
            j = (acc - (self.wa if self.it else 0.0 * acc)) / self.wdt
            self.wx = self.wx + self.wv * self.wdt + 0.5 * acc * self.wdt ** 2 + (1.0 / 6.0) * j * self.wdt ** 3
            self.wv = self.wv + acc * self.wdt + 0.5 * j * self.wdt ** 2
            self.wa = acc
        self.it += 1


def _exact_steps(case, seed):
    sims = _sims(case, seed)
    e = _Exact(sims, case.get("length", "reference") == "reference")
    with torch.no_grad():
        for _ in range(case["steps"]):
            e.step()
    out = {"x": torch.cat([e.x, e.r[:, None]], 1), "vel": torch.cat([e.v, e.fix[:, None]], 1),
           "xyzsum": e.xyzsum, "force": e.F, "angpos": e.angpos, "angvel": e.w, "torque": e.T,
           "es_dot": e.es_dot, "es": e.es, "ev_dot": e.ev_dot, "ev": e.ev, "p": e.p}
    if e.bonds is not None:
        out["bond_delta_n"], out["bond_delta_t"] = e.bdn, e.bdt
    if case["kind"] == "ensemble" or case.get("scene") == "shear":
        out["wall_x"], out["wall_force"] = e.wx, e.wf
    return {k: v.cpu().numpy() for k, v in out.items()}


def _exact_adjoint(case, seed):
    s = _sims(case, seed)[0]
    e = _Exact([s], False)
    p = [torch.tensor(float(v[0]), dtype=torch.float64, device=e.dev, requires_grad=True)
         for v in (s.k_n, s.gamma_n, s.mu_s)]
    # rollout() differentiates k_n with k_t held, and the walls' normal
    # stiffness is k_n
    e.k_n, e.gn, e.mu = (q.expand(e.n) for q in p)
    v0 = e.v.clone().requires_grad_(True)
    e.v = v0
    for _ in range(case["steps"]):
        e.step()
    loss = ((e.x - torch.from_numpy(_target(s, seed)).to(e.dev)) ** 2).sum(1).mean()
    loss.backward()
    return {"x": e.x.detach(), "k_n": p[0].grad, "gamma_n": p[1].grad, "mu": p[2].grad, "v0": v0.grad}


def _exact_relax(case, seed):
    s = _sims(case, seed)[0]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.tensor(s.x, dtype=torch.float64, device=dev)
    r = torch.tensor(s.radius, dtype=torch.float64, device=dev)
    L = [float(v) for v in s.L]
    z_top = float(s.x[:, 2].max())
    skin = 0.2 * float(r.min())
    ref, worst = None, 0.0
    for _ in range(case["sweeps"]):
        if ref is None or float(((x - ref) ** 2).sum(1).max()) > (0.49 * skin) ** 2:
            i, j = _candidates(x, r, 0, L, True, skin)
            ref = x.clone()
        d = x[i] - x[j]
        for k in range(2):
            d[:, k] -= L[k] * torch.round(d[:, k] / L[k])
        ln = (d * d).sum(1).sqrt()
        ov = torch.clamp(r[i] + r[j] - ln, min=0.0)
        step = torch.zeros_like(x).index_add(0, i, (0.5 * 0.6 * ov / ln)[:, None] * d)
        below, above = r - x[:, 2], x[:, 2] + r - z_top
        step[:, 2] += torch.clamp(below, min=0.0) - torch.clamp(above, min=0.0)
        worst = max(float(ov.max()), float(below.max()), float(above.max()))
        x = x + step
        for k in range(2):
            x[:, k] = torch.where(x[:, k] < 0.0, x[:, k] + L[k], x[:, k])
            x[:, k] = torch.where(x[:, k] >= L[k], x[:, k] - L[k], x[:, k])
        x[:, 2] = x[:, 2].clamp(min=0.0)
    return {"x": torch.cat([x, r[:, None]], 1).cpu().numpy(), "max_overlap": worst}


def _exact_analysis(case, seed):
    s = _sims(case, seed)[0]
    k = case["slices"]
    h = float(s.w_x[0]) / k
    z, r = s.x[:, 2], s.radius

    def cap(c):
        return math.pi * c * c / 3.0 * (3.0 * r - c)

    # the reference's terms: a sphere cut by a slab's face counts with its cap
    # on the slab's side, or, centre inside, with its volume plus the other cap
    vol, por = 4.0 / 3.0 * math.pi * r ** 3, []
    for q in range(k):
        lo, hi = q * h, (q + 1) * h
        t = numpy.where((lo <= z - r) & (z + r <= hi), vol, 0.0)
        part = t == 0.0
        t += numpy.where(part & (lo >= z) & (lo <= z + r), cap(z + r - lo), 0.0)
        t += numpy.where(part & (lo < z) & (lo > z - r), vol + cap(lo - z + r), 0.0)
        t += numpy.where(part & (hi <= z) & (hi >= z - r), cap(hi - z + r), 0.0)
        t += numpy.where(part & (hi > z) & (hi < z + r), vol + cap(z + r - hi), 0.0)
        por.append(1.0 - t.sum() / (h * float(s.L[0]) * float(s.L[1])))
    i, j = _candidates(torch.tensor(s.x), torch.tensor(r), 0, [float(v) for v in s.L], False, 0.0)
    pairs = torch.stack([i, j], 1)[i < j].numpy()
    d = numpy.sqrt(((s.x[pairs[:, 1]] - s.x[pairs[:, 0]]) ** 2).sum(1)) - r[pairs[:, 0]] - r[pairs[:, 1]]
    free = numpy.asarray(s.fixvel).reshape(-1) == 0.0
    m = (d < 0.0) & free[pairs[:, 0]] & free[pairs[:, 1]]
    pairs, d = pairs[m], d[m]
    return {"image": None, "z": (numpy.arange(k) + 0.5) * h, "porosity": numpy.array(por),
            "pairs": pairs, "delta_n": d}


def exact(case, seed):
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed)
    if case["kind"] == "relax":
        return _exact_relax(case, seed)
    if case["kind"] == "analysis":
        return _exact_analysis(case, seed)
    if case["kind"] == "darcy":
        return None
    return _exact_steps(case, seed)
