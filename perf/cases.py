"""The work that this framework's users have it do, as cases that can be timed and compared.

A case is one call pattern of a user's program on an open engine: advance a simulation by an output interval and read
its state back, with or without uploading a state first; a fluid-coupled interval; an ensemble of boxes; an image.
Workloads are those of `sphere_b200.configs`, at their published sizes and at sizes between them.

`exact` restates the physics in plain torch FP64 (all pairs of a neighbour list at once) for the dry, bonded and
Darcy-coupled runs; it uses this package only for the workload generators, as `prepare` does.
"""
import math

import numpy
import torch

from sphere_b200 import configs
from sphere_b200.engine import Batch, Engine

PACKED = 100000          # spheres of the packing that ships with the package


def listed():
    return [
        # a few hundred spheres under a wall, the size of the reference's own tests: launch latency is all there is
        {"name": "box_400_faithful", "kind": "dry", "scene": "box", "n": 400, "precision": "faithful", "steps": 100,
         "exchange": False},
        # dry settling of the 10,000-sphere lattice, the configuration sphere itself runs
        {"name": "settle_10k_faithful", "kind": "dry", "scene": "lattice", "n": 10000, "precision": "faithful",
         "steps": 200, "exchange": False},
        # a host program that uploads positions and velocities every few steps, odd size, the other contact model
        {"name": "coupled_20k_viscous", "kind": "dry", "scene": "box", "model": 1, "n": 20011, "precision": "fp64",
         "steps": 20, "exchange": True},
        # the headline workload: dense shear of 100,000 spheres, one output interval
        {"name": "shear_100k_mixed", "kind": "dry", "scene": "packing", "n": PACKED, "precision": "mixed", "steps": 100,
         "exchange": False},
        # the same as the drop-in default runs it
        {"name": "shear_100k_faithful", "kind": "dry", "scene": "packing", "n": PACKED, "precision": "faithful",
         "steps": 100, "exchange": False},
        # bonded polydisperse packing, larger than every cache
        {"name": "cohesive_1m_faithful", "kind": "dry", "scene": "cohesive", "n": 1000000, "precision": "faithful",
         "steps": 10, "exchange": False},
        # an ensemble of independent shear boxes of 2,000 to 20,000 spheres in one launch
        {"name": "ensemble_128_mixed", "kind": "ensemble", "nbox": 128, "n_min": 2000, "n_max": 20000,
         "precision": "mixed", "steps": 50},
        # Darcy-coupled consolidation on the 40 x 40 x 80 grid, started from the previous solution
        {"name": "darcy_100k", "kind": "darcy", "n": PACKED, "precision": "faithful", "warm_start": 0, "steps": 4},
        # the same with the learned start: extrapolation, network prediction and one training step per solve
        {"name": "darcy_100k_learned", "kind": "darcy", "n": PACKED, "precision": "mixed", "warm_start": 1, "steps": 4},
        # Navier-Stokes flow through the packing, held in place, on the same grid
        {"name": "navier_stokes_100k", "kind": "ns", "n": PACKED, "precision": "faithful", "steps": 10},
        # the ray-traced image at the reference's default size
        {"name": "render_100k_800", "kind": "render", "n": PACKED, "width": 800, "height": 800, "method": 1},
        # the diagnostics read between output files: energies, porosity profile, coordination number
        {"name": "diagnostics_100k", "kind": "diagnostics", "n": PACKED, "slices": 20},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["dry", "dry", "dry", "dry", "ensemble", "darcy", "ns", "render", "diagnostics"])
    if kind == "dry":
        scene = rng.choice(["lattice", "box", "box", "box", "cohesive"])
        n = {"lattice": size(1000, 100000), "box": size(300, 200000), "cohesive": size(20000, 1000000)}[scene]
        case = {"kind": kind, "scene": scene, "n": n, "precision": rng.choice(["faithful", "fp64", "mixed"]),
                "steps": 10 if scene == "cohesive" else rng.randint(5, 100), "exchange": rng.random() < 0.3}
        if scene == "box":
            case["model"] = rng.choice([1, 2])
        return case
    if kind == "ensemble":
        return {"kind": kind, "nbox": rng.randint(3, 64), "n_min": size(300, 2000), "n_max": size(4000, 20000),
                "precision": rng.choice(["faithful", "mixed"]), "steps": rng.randint(10, 50)}
    if kind == "darcy":
        return {"kind": kind, "n": size(2000, 100000), "precision": rng.choice(["faithful", "mixed"]),
                "warm_start": rng.choice([0, 0, 1, 2]), "steps": rng.randint(2, 4)}
    if kind == "ns":
        return {"kind": kind, "n": size(2000, 100000), "precision": "faithful", "steps": rng.randint(2, 10)}
    if kind == "render":
        return {"kind": kind, "n": size(1000, 100000), "width": rng.randint(200, 800), "height": rng.randint(200, 800),
                "method": rng.randint(0, 5)}
    return {"kind": kind, "n": size(1000, 100000), "slices": rng.randint(5, 40)}


# ---------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------
_packings = {}


def _packed():
    """The settled packing under shear (read from the package once)."""
    if "shear" not in _packings:
        _packings["shear"] = configs.shear_benchmark(n=PACKED, seed=1)
    return _packings["shear"].copy()


def _consolidation(n, seed):
    """A dense box under a 10 kPa wall, ready for a fluid: the settled packing on the 40 x 40 x 80 grid at its own
    size, a face-centred cubic start on the sorting grid otherwise."""
    if n == PACKED:
        if "fluid" not in _packings:
            _packings["fluid"] = configs.darcy_benchmark(n=PACKED, seed=1)
        return _packings["fluid"].copy()
    d = _dense_box(n, seed, sigma0=10e3)
    d.fixvel[:] = 0
    d.E = 7e8
    d.gamma_wn = 1.0e4
    configs.init_temporal(d, total=1.0, file_dt=1.0)
    configs.init_fluid_darcy(d, mu=1.797e-6, rho_f=1000.0, k_c=3.5e-13, beta_f=4.5e-10, tolerance=1e-8, maxiter=200000,
                             bottom_no_flow=True)
    return d


def _dense_box(n, seed, sigma0=20e3, shear_velocity=1e-4, mu=0.5, model=2):
    """A shear box as `configs.fcc_shear_box` makes it, at rest under its load: radii equal but for a few parts in 1e5,
    so that about two thirds of the lattice's neighbours touch with the overlaps that sigma0 gives them."""
    d = configs.fcc_shear_box(n, seed, r_min=0.01, r_max=0.01, sigma0=sigma0, shear_velocity=shear_velocity, mu=mu,
                              contactmodel=model)
    rng = numpy.random.default_rng(seed)
    d.x[:, :2] += 0.0035     # off the periodic faces
    d.radius = 0.01001 + rng.normal(2e-7, 4e-7, size=n)
    d.w_x[0] = float(numpy.max(d.x[:, 2] + d.radius))
    d.w_m[0] = float(numpy.sum(d.rho * 4.0 / 3.0 * math.pi * d.radius ** 3))
    d.vel += rng.normal(0.0, 1e-3, size=(n, 3)) * (d.fixvel == 0)[:, None]
    d.angvel = rng.normal(0.0, 1e-2, size=(n, 3)) * (d.fixvel == 0)[:, None]
    if model == 1:
        d.gamma_n = d.gamma_t = 50.0
    return d


def _ensemble(case, seed):
    """Boxes with the counts, loads, velocities and friction of `configs.batch_shear_boxes`."""
    rng = numpy.random.default_rng(seed)
    boxes = []
    for b in range(case["nbox"]):
        # counts spread evenly over the logarithm, in no order of size
        n = int(round(case["n_min"] * (case["n_max"] / case["n_min"]) ** ((0.618033988749895 * (b + 1)) % 1.0)))
        boxes.append(_dense_box(n, seed * 1009 + b, sigma0=float(rng.choice([10e3, 20e3, 40e3, 80e3, 160e3])),
                                shear_velocity=float(rng.uniform(1e-5, 1e-3)), mu=float(rng.uniform(0.3, 0.6))))
    return boxes


def _scene(case, seed):
    """The workload of a case as a BinData; every input that a run may vary is drawn from the seed."""
    rng = numpy.random.default_rng(seed)
    kind, n = case["kind"], case.get("n")
    if kind in ("darcy", "ns"):
        d = _consolidation(n, seed)
        if kind == "ns":
            # flow through a bed of held spheres
            configs.init_fluid_ns(d, mu=8.9e-4, rho_f=1000.0, hydrostatic=True)
            d.v_f = rng.normal(0.0, 1e-4, size=d.v_f.shape)
            d.vel[:] = 0.0
            d.angvel[:] = 0.0
            d.fixvel[:] = -1.0
            return d
        d.vel = rng.normal(0.0, 1e-3, size=(n, 3))
        d.angvel[:] = 0.0
        return d
    scene = case.get("scene", "packing" if n == PACKED else "box")
    if scene == "packing":
        d = _packed()
        d.vel += rng.normal(0.0, 1e-3, size=(n, 3)) * (d.fixvel == 0)[:, None]
        d.angvel = rng.normal(0.0, 1e-2, size=(n, 3)) * (d.fixvel == 0)[:, None]
    elif scene == "cohesive":
        d = configs.large_cohesive_packing(n=n, seed=seed)
    elif scene == "box":
        d = _dense_box(n, seed, model=case.get("model", 2))
    else:
        side = max(3, int(math.ceil(n ** (1.0 / 3.0))))
        d = configs.settling_lattice(n=n, seed=seed, nx=side, ny=side, nz=side)
    return d


class _Run:
    """An open engine and the host buffers its user reads into and uploads from."""

    def __init__(self, eng, fields, uploads=()):
        self.eng, self.fields, self.uploads = eng, fields, uploads
        self.out = {}
        for f in fields:
            a = eng.get(f)
            self.out[f] = torch.from_numpy(a).pin_memory().numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        b = Batch(_ensemble(case, seed), precision=case["precision"])
        b.step(WARM_STEPS)   # a running ensemble, its launch shape chosen on its first steps
        return {"case": case, "batch": b}
    d = _scene(case, seed)
    if kind == "dry":
        eng = Engine(d, precision=case["precision"])
        return {"case": case, "run": _Run(eng, ("x", "vel", "angvel", "force", "torque"),
                                          ("x", "vel", "angvel") if case["exchange"] else ())}
    if kind == "darcy":
        eng = Engine(d, fluid=True, precision=case["precision"], warm_start=case["warm_start"])
        return {"case": case, "run": _Run(eng, ("x", "vel", "darcy_p", "darcy_phi", "darcy_v"))}
    if kind == "ns":
        eng = Engine(d, fluid=True, precision=case["precision"])
        return {"case": case, "run": _Run(eng, ("x", "vel", "darcy_p", "darcy_phi", "darcy_v", "ns_f_sum"))}
    eng = Engine(d, precision="fp64")
    eng.step(10)             # an image or a diagnostic is of a state that has contacts
    return {"case": case, "eng": eng, "slices": _slices(case, d)}


def run(state):
    case = state["case"]
    if case["kind"] == "ensemble":
        b = state["batch"]
        b.step(case["steps"])
        return {"x": numpy.concatenate([b.get(i, "x") for i in range(case["nbox"])]),
                "vel": numpy.concatenate([b.get(i, "vel") for i in range(case["nbox"])])}
    if case["kind"] == "render":
        return {"image": state["eng"].render(method=case["method"], max_val=_max_val(case["method"]),
                                             width=case["width"], height=case["height"])}
    if case["kind"] == "diagnostics":
        e = state["eng"]
        phi, depth = e.porosity(state["slices"])
        return {"energy": {m: e.energy(m) for m in ENERGIES}, "porosity": phi, "depth": depth,
                "coordination": e.coordination_number()}
    r = state["run"]
    for f in r.uploads:
        r.eng.set(f, r.out[f])
    r.eng.step(case["steps"])
    for f in r.fields:
        r.eng.get(f, r.out[f])
    return r.out


ENERGIES = ("pot", "kin", "rot", "shear", "visc_n")


def _slices(case, d):
    """Slabs of the porosity profile; a slab is higher than a sphere."""
    top = float(d.w_x[0]) if d.nw else float(d.L[2])
    return max(1, min(case.get("slices", 1), int(top / (2.2 * float(numpy.max(d.radius))))))


WARM_STEPS = 256         # enough for the ensemble to choose its launch shape


def _max_val(method):
    """The colour scale a user gives: the range that the values of these packings have."""
    return {0: 1.0, 1: 1e5, 2: 2e-3, 3: 5e-2, 4: 1e-7, 5: 1e-6}[method]


# ---------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------
_CONTACTS = {"packing": 2.8, "lattice": 0.0, "box": 7.0, "cohesive": 0.0}


def _dry_work(n, steps, z, bonds=0.0):
    """Per particle and step: position, velocities, angle, accelerations and displacement sums in, the same and the
    forces out (440 bytes), 56 for the partner and the history of each contact; per bond its history in and out and
    its particles (136 bytes).  About 150 operations to integrate, 180 per contact, 200 per bond."""
    return {"bytes": n * steps * (440.0 + 56.0 * z + 136.0 * bonds),
            "flops": n * steps * (150.0 + 180.0 * z + 200.0 * bonds)}


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
        mean = (case["n_max"] - case["n_min"]) / (hi - lo)
        return _dry_work(case["nbox"] * mean, case["steps"], _CONTACTS["box"])
    if kind == "dry":
        w = _dry_work(case["n"], case["steps"], _CONTACTS[case["scene"]], 2.35 if case["scene"] == "cohesive" else 0.0)
        if case["exchange"]:
            w["bytes"] += 256.0 * case["n"]
        return w
    n = case["n"]
    if kind in ("darcy", "ns"):
        # the fluid fields in and out once per step; about 30 operations per cell and pressure iteration, some 400
        # iterations from the previous solution, half as many from the extrapolation, 60 for Navier-Stokes
        cells = 128000 if n == PACKED else 0.9 * n
        w = _dry_work(n, case["steps"], 2.8)
        iters = 60 if kind == "ns" else 200 if case["warm_start"] else 400
        w["bytes"] += case["steps"] * cells * (120.0 if kind == "darcy" else 350.0)
        w["flops"] += case["steps"] * cells * iters * 30.0
        return w
    if kind == "render":
        # the spheres and the image once; some ten spheres tested per ray at 25 operations
        px = case["width"] * case["height"]
        return {"bytes": 60.0 * n + 4.0 * px, "flops": 250.0 * px}
    return {"bytes": n * (5 * 80.0 + 40.0 + 64.0 + 24.0), "flops": n * 400.0}


def tolerance(case):
    kind = case["kind"]
    if kind == "render":
        return "exact"
    if kind == "dry" and case["precision"] in ("faithful", "fp64"):
        return "exact"       # every path keeps the reference's operation order
    if kind == "diagnostics":
        return {"rel": 1e-12, "max": 1e-9, "differ": 0.0}   # FP64 sums in another order
    if kind in ("darcy", "ns"):
        if case.get("warm_start"):
            # the start of a solve decides where within its tolerance it stops
            return {"rel": 1e-6, "max": 1e-3}
        if case["precision"] == "faithful":
            return {"rel": 1e-9, "max": 1e-6}
    # FP32 contact laws: rounding of single contacts, carried through the steps
    return {"rel": 1e-5, "max": 1e-2}


# ---------------------------------------------------------------------
# the same physics in plain FP64
# ---------------------------------------------------------------------
def _t(a, dev):
    return torch.as_tensor(numpy.ascontiguousarray(a), dtype=torch.float64, device=dev)


def _cross(a, b):
    return torch.linalg.cross(a, b)


def _dot(a, b):
    return (a * b).sum(dim=1, keepdim=True)


def _neighbours(x, r, L, skin):
    """Directed pairs (i, j) with |x_i - x_j| < r_i + r_j + skin, x and y periodic."""
    dev, n = x.device, x.shape[0]
    width = float(2.0 * r.max() + skin)
    num = [max(3, int(L[0] / width)), max(3, int(L[1] / width)), max(1, int(math.ceil(float(L[2]) / width)))]
    cell = torch.stack([(x[:, 0] / L[0] * num[0]).long() % num[0], (x[:, 1] / L[1] * num[1]).long() % num[1],
                        (x[:, 2] / width).long().clamp(0, num[2] - 1)], dim=1)
    key = cell[:, 0] + num[0] * (cell[:, 1] + num[1] * cell[:, 2])
    key_s, order = torch.sort(key)
    first = torch.searchsorted(key_s, torch.arange(num[0] * num[1] * num[2] + 1, device=dev))
    found = []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                cz = cell[:, 2] + dz
                ok = (cz >= 0) & (cz < num[2])
                other = (cell[:, 0] + dx) % num[0] + num[0] * ((cell[:, 1] + dy) % num[1] + num[1] * cz.clamp(0, num[2] - 1))
                lo = first[other]
                count = (first[other + 1] - lo) * ok
                i = torch.repeat_interleave(torch.arange(n, device=dev), count)
                start = torch.cumsum(count, 0) - count
                j = order[lo[i] + torch.arange(i.shape[0], device=dev) - start[i]]
                d = _image(x[i] - x[j], L)
                keep = (i != j) & ((d * d).sum(dim=1) < (r[i] + r[j] + skin) ** 2)
                found.append(torch.stack([i[keep], j[keep]]))
    i, j = torch.cat(found, dim=1)
    return i, j


def _image(d, L):
    d = d.clone()
    d[:, 0] -= L[0] * torch.round(d[:, 0] / L[0])
    d[:, 1] -= L[1] * torch.round(d[:, 1] / L[1])
    return d


class _Dem:
    """Spheres with periodic sides, a fixed bottom and at most one moving top wall, advanced pair-wise in FP64."""

    def __init__(self, d, dev):
        self.d, self.n, self.dev = d, d.np, dev
        self.x, self.v, self.w = _t(d.x, dev), _t(d.vel, dev), _t(d.angvel, dev)
        self.r, self.fix = _t(d.radius, dev), _t(d.fixvel, dev)
        self.L = [float(v) for v in d.L]
        self.g = _t(d.g, dev)
        self.a0, self.b0 = torch.zeros_like(self.x), torch.zeros_like(self.x)
        self.m = 4.0 / 3.0 * math.pi * self.r ** 3 * d.rho
        self.skin = 0.1 * float(self.r.min())
        self.i = self.j = torch.zeros(0, dtype=torch.long, device=dev)
        self.hist = torch.zeros((0, 3), dtype=torch.float64, device=dev)
        self.rebuild()
        self.wall = None
        if d.nw:
            self.wall = [float(d.w_x[0]), float(d.w_vel[0]), 0.0]
        self.bonds = None
        if d.nb0:
            self.bonds = torch.as_tensor(numpy.asarray(d.bonds).astype(numpy.int64), device=dev)
            self.bond_d, self.bond_w = (torch.zeros((d.nb0, 4), dtype=torch.float64, device=dev) for _ in range(2))
            self.bond_ok = torch.ones(d.nb0, dtype=torch.bool, device=dev)

    def rebuild(self):
        """The neighbour list at the present positions; pairs that stay keep their tangential displacement."""
        key, hist = self.i * self.n + self.j, self.hist
        self.i, self.j = _neighbours(self.x, self.r, self.L, self.skin)
        self.x_built = self.x.clone()
        self.hist = torch.zeros((self.i.shape[0], 3), dtype=torch.float64, device=self.dev)
        if len(key):
            key, order = torch.sort(key)
            new = self.i * self.n + self.j
            at = torch.searchsorted(key, new).clamp(max=len(key) - 1)
            kept = key[at] == new
            self.hist[kept] = hist[order[at[kept]]]

    def pairs(self, F, T):
        d, i, j = self.d, self.i, self.j
        xab = _image(self.x[i] - self.x[j], self.L)
        ln = xab.norm(dim=1, keepdim=True)
        ra, rb = self.r[i][:, None], self.r[j][:, None]
        delta = ln - (ra + rb)
        c = torch.nonzero(delta[:, 0] < 0.0)[:, 0]
        i, j, xab, ln, ra, rb, delta = i[c], j[c], xab[c], ln[c], ra[c], rb[c], delta[c]
        n = xab / ln
        vl = self.v[i] - self.v[j]
        vel = vl + (ra + delta / 2) * _cross(n, self.w[i]) + (rb + delta / 2) * _cross(n, self.w[j])
        vn = _dot(vl, n)
        vt = vel - n * _dot(n, vel)
        vt_len = vt.norm(dim=1, keepdim=True)
        kn = math.pi / 2 * d.E * (ra + rb) / 2 if d.E > 1e-3 else torch.full_like(ra, d.k_n)
        kt = kn if d.E > 1e-3 else torch.full_like(ra, d.k_t)
        fn = (-kn * delta - d.gamma_n * vn).clamp(min=0.0) * n
        fn_len = fn.norm(dim=1, keepdim=True)
        if d.contactmodel == 1:
            limit = torch.where(vt_len > 1e-3, d.mu_d, d.mu_s) * fn_len
            ft = -torch.minimum(d.gamma_t * vt_len, limit) * vt / vt_len.clamp(min=1e-300)
        else:
            h = self.hist[c]
            h = h - n * _dot(n, h) + vt * d.time_dt
            ft = -kt * h - d.gamma_t * vt
            ft_len = ft.norm(dim=1, keepdim=True)
            limit = d.mu_s * fn_len
            t = ft / ft_len.clamp(min=1e-300)
            slip = ft_len > limit
            h = torch.where(slip, -(d.mu_d * fn_len * t + d.gamma_t * vt) / kt, h)
            ft = torch.where(slip, limit * t, ft)
            self.hist.zero_()
            self.hist[c] = h
        F.index_add_(0, i, fn + ft)
        T.index_add_(0, i, _cross(-(ra + delta / 2) * n, ft))

    def walls(self, F, T):
        d = self.d
        pos, wv = (self.wall[0], self.wall[1]) if self.wall else (self.L[2], 0.0)
        total = torch.zeros(1, dtype=torch.float64, device=self.dev)
        for sign, vel_w in ((-1.0, wv), (1.0, 0.0)):
            delta = pos - (self.x[:, 2] + self.r) if sign < 0 else self.x[:, 2] - self.r - float(d.origo[2])
            c = torch.nonzero(delta < 0.0)[:, 0]
            if not len(c):
                continue
            n = torch.zeros((len(c), 3), dtype=torch.float64, device=self.dev)
            n[:, 2] = sign
            ra, dl = self.r[c][:, None], delta[c][:, None]
            vel = self.v[c] + (ra + dl / 2) * _cross(n, self.w[c]) + vel_w
            vt = vel - n * _dot(n, vel)
            vt_len = vt.norm(dim=1, keepdim=True)
            kn = math.pi / 2 * d.E * ra if d.E > 1e-3 else d.k_n
            fn = (-kn * dl - d.gamma_wn * _dot(self.v[c], n)).clamp(min=0.0) * n
            ft = -torch.minimum(d.gamma_wt * vt_len, d.mu_wd * fn.norm(dim=1, keepdim=True)) * vt / vt_len.clamp(min=1e-300)
            F.index_add_(0, c, fn + ft)
            T.index_add_(0, c, _cross(-(ra + dl / 2) * n, ft))
            if sign < 0:
                total = total + _dot(fn, n).sum()
        return float(total)

    def bond_forces(self, F, T):
        d, dt = self.d, self.d.time_dt
        i, j = self.bonds[:, 0], self.bonds[:, 1]
        ri, rj = self.r[i][:, None], self.r[j][:, None]
        R = d.lambda_bar * torch.minimum(ri, rj)
        A, I = math.pi * R ** 2, 0.25 * math.pi * R ** 4
        J = 2 * I
        x = self.x[i] - self.x[j]
        ln = x.norm(dim=1, keepdim=True)
        over = (ln - (ri + rj)).clamp(max=0.0)
        n = x / ln
        d0, w0 = self.bond_d, self.bond_w
        dt0 = d0[:, :3] - n * _dot(n, d0[:, :3])
        dd = (self.v[i] - self.v[j] + (ri + over / 2) * _cross(n, self.w[i]) + (rj + over / 2) * _cross(n, self.w[j])) * dt
        ddn = -_dot(dd, n)
        dn = d0[:, 3:] + ddn
        ddt = dd - n * _dot(n, dd)
        dtt = dt0 + ddt
        fn = (d.k_n * A * dn + d.gamma_n * ddn / dt) * n
        ft = -d.k_t * A * dtt - d.gamma_t * ddt / dt
        nn = -n
        wt0 = w0[:, :3] - nn * _dot(w0[:, :3], nn)
        dw = (self.w[j] - self.w[i]) * dt
        dwn = _dot(dw, nn)
        wn = w0[:, 3:] + dwn
        wt = wt0 + dw - dwn * nn
        tn, tt = -d.k_t * J * wn * nn, -d.k_n * I * wt
        sigma = fn.norm(dim=1, keepdim=True) / A + tt.norm(dim=1, keepdim=True) * R / I
        tau = ft.norm(dim=1, keepdim=True) / A + tn.norm(dim=1, keepdim=True) * R / J
        self.bond_ok &= ((sigma < d.sigma_b) & (tau < d.tau_b))[:, 0]
        ok = self.bond_ok[:, None]
        self.bond_d = torch.where(ok, torch.cat([dtt, dn], dim=1), d0)
        self.bond_w = torch.where(ok, torch.cat([wt, wn], dim=1), w0)
        f, t = (fn + ft) * ok, (tn + tt) * ok
        F.index_add_(0, i, f)
        F.index_add_(0, j, -f)
        T.index_add_(0, i, -t)
        T.index_add_(0, j, t)

    def step(self, fluid=None):
        d, dt = self.d, float(self.d.time_dt)
        F, T = torch.zeros_like(self.x), torch.zeros_like(self.x)
        self.pairs(F, T)
        top = self.walls(F, T)
        if self.bonds is not None:
            self.bond_forces(F, T)
        if fluid is not None:
            fluid.step(self, F)
        self.F, self.T = F, T
        m = self.m[:, None]
        a = F / m + self.g
        b = T / (0.4 * m * self.r[:, None] ** 2)
        held = (self.fix > 1e-4) & (self.fix < 10.0)
        a = torch.where(held[:, None], torch.stack([torch.zeros_like(a[:, 0]), torch.zeros_like(a[:, 0]),
                                                    a[:, 2] - self.g[2]], dim=1), a)
        b = torch.where(held[:, None], torch.zeros_like(b), b)
        da, db = a - self.a0, b - self.b0
        self.x = self.x + self.v * dt + 0.5 * a * dt ** 2 + da * dt ** 2 / 6.0
        self.v = self.v + a * dt + 0.5 * da * dt
        self.w = self.w + b * dt + 0.5 * db * dt
        self.a0, self.b0 = a, b
        for k in (0, 1):
            self.x[:, k] -= self.L[k] * torch.floor(self.x[:, k] / self.L[k])
        if self.wall:
            acc = (top - float(d.w_sigma0[0]) * self.L[0] * self.L[1]) / float(d.w_m[0])
            da = acc - self.wall[2]
            self.wall[0] += self.wall[1] * dt + 0.5 * acc * dt ** 2 + da * dt ** 2 / 6.0
            self.wall[1] += acc * dt + 0.5 * da * dt
            self.wall[2] = acc
        moved = _image(self.x - self.x_built, self.L).norm(dim=1).max()
        if float(moved) > 0.45 * self.skin:
            self.rebuild()


def _wide(f, d):
    """A cell field (x, y, z) with one layer around it: periodic sides, the bottom mirrored at its first cells, the top
    repeated."""
    f = torch.cat([f[-1:], f, f[:1]], dim=0)
    f = torch.cat([f[:, -1:], f, f[:, :1]], dim=1)
    return torch.cat([f[:, :, 1:2], f, f[:, :, -1:]], dim=2)


class _Darcy:
    """The porosity-coupled pressure of a box with periodic sides, a no-flow bottom and a Dirichlet top."""

    def __init__(self, d, dev):
        self.d = d
        self.num = [int(v) for v in d.num]
        self.h = [float(d.L[k]) / self.num[k] for k in range(3)]
        self.wall_iz = int(float(d.w_x[0]) / self.h[2])
        self.p, self.phi = _t(d.p_f, dev), _t(d.phi, dev)
        self.n_steps = 0

    def weights(self, x, L):
        """For each of the 27 cells around a sphere's own: cell indices, and one minus the distance per axis."""
        num, h = self.num, self.h
        c = [torch.floor(x[:, k] / h[k]).long().clamp(0, num[k] - 1) for k in range(3)]
        for a in (-1, 0, 1):
            for b in (-1, 0, 1):
                for e in (-1, 0, 1):
                    w = 1.0
                    for k, o in ((0, a), (1, b), (2, e)):
                        w = w * (1.0 - (x[:, k] - (c[k].double() + o + 0.5) * h[k]).abs() / h[k]).clamp(min=0.0)
                    yield c[0] + a, c[1] + b, c[2] + e, w

    def step(self, dem, F):
        d, num, h = self.d, self.num, self.h
        dt, L = float(d.time_dt), dem.L
        nx, ny, nz = num
        vol = 4.0 / 3.0 * math.pi * dem.r ** 3
        # force of the present pressure gradient on the spheres
        P = _wide(self.p, d)
        grad = [(P[2:, 1:-1, 1:-1] - P[:-2, 1:-1, 1:-1]) / (2 * h[0]), (P[1:-1, 2:, 1:-1] - P[1:-1, :-2, 1:-1]) / (2 * h[1]),
                (P[1:-1, 1:-1, 2:] - P[1:-1, 1:-1, :-2]) / (2 * h[2])]
        grad = [_wide(q, d) for q in grad]
        at = torch.zeros_like(dem.x)
        for ix, iy, iz, w in self.weights(dem.x, L):
            out = ((ix < 0) | (ix >= nx)).int() + ((iy < 0) | (iy >= ny)).int() + ((iz < 0) | (iz >= nz)).int()
            w = w * (out < 2)
            for k in range(3):
                q = grad[k][ix + 1, iy + 1, iz + 1]
                if k == 2:
                    q = q * ((iz >= 0) & (iz < self.wall_iz - 1))
                at[:, k] += w * q
        fp = -(at + float(d.rho_f) * dem.g) * vol[:, None]
        above = torch.floor(dem.x[:, 2] / h[2]) >= self.wall_iz
        fp[:, 2] = torch.where(above, torch.zeros_like(fp[:, 2]), fp[:, 2])
        F += fp
        # porosity now and after the step, and the solid's velocity
        cells = nx * ny * nz

        def spread(x, val):
            f = torch.zeros(cells, dtype=torch.float64, device=x.device)
            own = torch.floor(dem.x[:, 2] / h[2]).long()       # a sphere is found from the cells around its present one
            c = [torch.floor(dem.x[:, k] / h[k]).long() for k in range(3)]
            for a in (-1, 0, 1):
                for b in (-1, 0, 1):
                    for e in (-1, 0, 1):
                        w = 1.0
                        for k, o in ((0, a), (1, b), (2, e)):
                            w = w * (1.0 - (x[:, k] - (c[k].double() + o + 0.5) * h[k]).abs() / h[k]).clamp(min=0.0)
                        z = c[2] + e
                        # cells of the bottom layer count the layer above them twice
                        w = w * torch.where((z == 0) & (own == 1), 2.0, 1.0) * ((z >= 0) & (z < nz))
                        q = ((c[0] + a) % nx * ny + (c[1] + b) % ny) * nz + z.clamp(0, nz - 1)
                        f.index_add_(0, q, w * val)
            return f.view(nx, ny, nz)

        volume = torch.full((nx, ny, nz), h[0] * h[1] * h[2], dtype=torch.float64, device=dem.dev)
        volume[:, :, -1] *= 0.875
        solid = spread(dem.x, vol)
        phi = (1.0 - solid / volume).clamp(0.1, 0.9)
        if self.n_steps == 0:
            dphi = torch.zeros_like(phi)
            vp = [torch.zeros_like(phi)] * 3
        else:
            moved = (1.0 - spread(dem.x + dem.v * dt, vol) / volume).clamp(0.1, 0.9)
            dphi = 0.5 * (moved - self.phi)
            vp = [spread(dem.x, vol * dem.v[:, k]) / solid.clamp(min=1e-16) for k in range(3)]
        self.phi = phi
        k = (float(d.k_c) * phi ** 3 / (1.0 - phi) ** 2).clamp(max=2.7e-10)
        W, K = _wide(phi, d), _wide(k, d)
        mid = (slice(1, -1),) * 3
        sides = []
        for ax in range(3):
            for s in (slice(2, None), slice(None, -2)):
                at_ = list(mid)
                at_[ax] = s
                sides.append(tuple(at_))
        face = [2.0 * K[s] * k / (K[s] + k) for s in sides]
        grad_phi = [(W[sides[2 * q]] - W[sides[2 * q + 1]]) / (2 * h[q]) for q in range(3)]
        ndt = float(d.ndem) * dt
        a = ndt / (float(d.beta_f) * phi * float(d.mu))
        src = ndt / (float(d.beta_f) * phi * (1.0 - phi)) * (dphi / ndt + sum(vp[q] * grad_phi[q] for q in range(3)))
        free = torch.ones_like(phi)
        free[:, :, min(self.wall_iz, nz - 1):] = 0.0

        def change(p):
            Q = _wide(p, d)
            div = 0.0
            for q in range(3):
                up, dn = Q[sides[2 * q]] - p, p - Q[sides[2 * q + 1]]
                if q == 2:
                    dn = dn.clone()
                    dn[:, :, 0] = 0.0
                div = div + (face[2 * q] * up - face[2 * q + 1] * dn) / h[q] ** 2
            return (a * div - src) * free

        old = self.p
        base = old + 0.5 * change(old)
        p = old
        for it in range(int(d.maxiter)):
            new = 0.95 * p + 0.05 * (base + 0.5 * change(p))
            worst = ((new - p) / (p + 1e-16)).abs().max() if it % 10 == 0 else None
            p = new
            if worst is not None and float(worst) <= float(d.tolerance):
                break
        self.p = p
        P = _wide(p, d)
        self.v = torch.stack([-k / float(d.mu) * (P[sides[2 * q]] - P[sides[2 * q + 1]]) / (2 * h[q]) / phi
                              for q in range(3)], dim=3)
        self.n_steps += 1


def _four(a, w=None):
    out = torch.zeros((a.shape[0], 4), dtype=torch.float64, device=a.device)
    out[:, :3] = a
    if w is not None:
        out[:, 3] = w
    return out.cpu().numpy()


def _cells(f):
    """A cell field (x, y, z, ...) in the engine's order: x fastest."""
    return f.transpose(0, 2).contiguous().reshape((-1,) + tuple(f.shape[3:])).cpu().numpy()


def _cap(h, r):
    return math.pi * h * h / 3.0 * (3.0 * r - h)


def _exact_diagnostics(s, slices):
    """The sums and lists of a state: energies, porosity of slabs with sphere's case analysis, overlaps of free pairs."""
    g = float(s.g.norm())
    energy = {"pot": float((s.m * g * s.x[:, 2]).sum()), "kin": float((0.5 * s.m * (s.v ** 2).sum(dim=1)).sum()),
              "rot": float((0.2 * s.m * s.r ** 2 * (s.w ** 2).sum(dim=1)).sum()), "shear": None, "visc_n": None}
    top = s.wall[0] if s.wall else s.L[2]
    high = top / slices
    c, r = s.x[:, 2], s.r
    lo, hi = c - r, c + r
    whole = 4.0 / 3.0 * math.pi * r ** 3
    none = torch.zeros_like(r)
    porosity, depth = [], []
    for q in range(slices):
        a, b = q * high, (q + 1) * high
        inside = (a <= lo) & (hi <= b)
        below = torch.where((a >= c) & (a <= hi), _cap(hi - a, r), torch.where((a < c) & (a > lo), whole + _cap(a - lo, r), none))
        above = torch.where((b <= c) & (b >= lo), _cap(b - lo, r), torch.where((b > c) & (b < hi), whole + _cap(hi - b, r), none))
        solid = float(torch.where(inside, whole, below + above).sum())
        porosity.append(1.0 - solid / (high * s.L[0] * s.L[1]))
        depth.append(a + 0.5 * high)
    i, j = s.i, s.j
    keep = (i < j) & (s.fix[i] == 0) & (s.fix[j] == 0)
    i, j = i[keep], j[keep]
    over = (s.x[j] - s.x[i]).norm(dim=1) - (s.r[i] + s.r[j])
    hit = over < 0
    return {"energy": energy, "porosity": numpy.array(porosity), "depth": numpy.array(depth),
            "coordination": torch.bincount(torch.cat([i[hit], j[hit]]), minlength=s.n).cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if kind == "ensemble":
        if case["nbox"] * (WARM_STEPS + case["steps"]) > 12000:
            return None      # box after box, over 20 seconds
        xs, vs = [], []
        for d in _ensemble(case, seed):
            s = _Dem(d, dev)
            for _ in range(WARM_STEPS + case["steps"]):
                s.step()
            xs.append(_four(s.x, s.r))
            vs.append(_four(s.v, s.fix))
        return {"x": numpy.concatenate(xs), "vel": numpy.concatenate(vs)}
    if kind == "render":
        return None          # bytes
    d = _scene(case, seed)
    if kind == "diagnostics":
        s = _Dem(d, dev)
        for _ in range(10):
            s.step()
        return _exact_diagnostics(s, _slices(case, d))
    if kind == "ns":
        # the porosity of the bed, which does not move; the flow through it is not restated here
        x, r = _t(d.x, dev), _t(d.radius, dev)
        num = [int(q) for q in d.num]
        h = [float(d.L[q]) / num[q] for q in range(3)]
        R = min(h)
        void = torch.full((num[0] * num[1] * num[2],), 4.0 / 3.0 * math.pi * R ** 3, dtype=torch.float64, device=dev)
        whole = float(void[0])
        c = [torch.floor(x[:, q] / h[q]).long() for q in range(3)]
        for a in range(-2, 3):
            for b in range(-2, 3):
                for e in range(-2, 3):
                    z = c[2] + e
                    dist = torch.stack([x[:, 0] - (c[0].double() + a + 0.5) * h[0],
                                        x[:, 1] - (c[1].double() + b + 0.5) * h[1],
                                        x[:, 2] - (z.double() + 0.5) * h[2]]).norm(dim=0)
                    cap = math.pi * (R + r - dist) ** 2 * (dist ** 2 + 2 * dist * r - 3 * r ** 2 + 2 * dist * R
                                                           + 6 * r * R - 3 * R ** 2) / (12.0 * dist)
                    part = ((R - r) < dist) & (dist < R + r)
                    inside = dist <= R - r
                    val = torch.where(part, cap, torch.where(inside, 4.0 / 3.0 * math.pi * r ** 3, 0.0))
                    val = val * ((z >= 0) & (z < num[2]))
                    q = ((c[0] + a) % num[0] * num[1] + (c[1] + b) % num[1]) * num[2] + z.clamp(0, num[2] - 1)
                    void.index_add_(0, q, -val)
        phi = (void / whole).clamp(0.0, 1.0).view(*num)
        return {"x": None, "vel": None, "darcy_p": None, "darcy_phi": _cells(phi), "darcy_v": None, "ns_f_sum": None}
    s = _Dem(d, dev)
    if kind == "darcy":
        f = _Darcy(d, dev)
        for _ in range(case["steps"]):
            s.step(f)
        return {"x": _four(s.x, s.r), "vel": _four(s.v, s.fix), "darcy_p": _cells(f.p), "darcy_phi": _cells(f.phi),
                "darcy_v": _cells(f.v)}
    for _ in range(case["steps"]):
        s.step()
    return {"x": _four(s.x, s.r), "vel": _four(s.v, s.fix), "angvel": _four(s.w), "force": _four(s.F),
            "torque": _four(s.T)}
