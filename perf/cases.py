"""The work this framework is used for, as cases that can be timed and checked.

Every case goes through the public Python entry points (DemEngine, Surrogate)
with inputs made from a seed; what a program holds before the call (the engine
with its particles uploaded, page-locked host buffers for the results, the
network) is made in `prepare`.

A step case is a stretch of time steps between two outputs of one simulation:
`step(k)`, the balances and the state read back. Its handle is kept, so the
next pass continues the simulation. A drum run starts over in every pass: a
bed without a lid loosens while its first overlaps relax, and every pass is to
find it in contact.
"""
import math

import numpy as np
import torch

from mercurydpm_fork_b200 import DemEngine, _abi, calibration, scenarios
from mercurydpm_fork_b200.surrogate import Surrogate

SMALL_D = 1e-3


def listed():
    return [
        # one time step per call with its .ene line, as the drop-in MercuryDPM
        # binding and drivers with a hook after every step do it
        dict(name="box_single_step", kind="box", n=1000, steps=1, law="sliding"),
        # the settling box (5,000 spheres, six walls) between two outputs
        dict(name="box_5k", kind="box", n=5000, steps=100, law="sliding"),
        # a short run of a drum of the size most reference drivers have, from
        # host arrays to host arrays
        dict(name="drum_30k_run", kind="drum", n=30_011, steps=100, law="mindlin_rolling_torsion"),
        # the periodic inclined chute, two HGrid levels, fixed base
        dict(name="chute_200k", kind="chute", n=200_000, steps=50),
        # the benchmark's drum from host arrays to host arrays: upload, the
        # initial evaluation, a window of time steps, the state read back
        dict(name="drum_1m_run", kind="drum", n=1_000_000, steps=60, law="mindlin_rolling_torsion"),
        # spheres landing on a triangulated floor
        dict(name="floor_50k", kind="floor", n=50_000, steps=50),
        # one trace interval of the calibration's batch: many small heaps in one handle
        dict(name="heaps_1024x600", kind="heaps", instances=1024, spheres=600, steps=50),
        # the chute's coarse-grained fields, depth profiles along the flow
        dict(name="cg_xz_chute", kind="cg", n=200_000, coordinates="XZ", nx=100, ny=1, nz=50, width=1.0),
        # fields resolved in three dimensions over a box
        dict(name="cg_xyz_box", kind="cg", n=20_000, coordinates="XYZ", nx=20, ny=20, nz=24, width=1.0),
        # what the .fstat and .restart writers read: contacts, their geometry, forces
        dict(name="records_50k", kind="records", n=50_000),
        # the surrogate's candidates of one calibration round
        dict(name="predict_65536", kind="predict", rows=65_536),
        # an epoch of the surrogate's training
        dict(name="train_2x1024", kind="train", rows=2048, batch=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box", "drum", "drum", "chute", "floor", "heaps", "cg", "records", "predict", "train"])
    if kind == "box":
        return dict(kind=kind, n=_log(rng, 300, 60_000), steps=rng.choice([1, 10, 37, 100]),
                    law=rng.choice(["sliding", "mindlin", "mindlin_rolling_torsion"]))
    if kind == "drum":
        return dict(kind=kind, n=_log(rng, 3000, 500_000), steps=rng.choice([1, 20, 57, 100]),
                    law=rng.choice(["mindlin_rolling_torsion", "mindlin"]))
    if kind == "chute":
        return dict(kind=kind, n=_log(rng, 5000, 200_000), steps=rng.choice([10, 21, 50]))
    if kind == "floor":
        return dict(kind=kind, n=_log(rng, 12_000, 150_000), steps=rng.choice([5, 21, 50]))
    if kind == "heaps":
        return dict(kind=kind, instances=_log(rng, 16, 1024), spheres=_log(rng, 150, 700), steps=rng.choice([10, 25, 50]))
    if kind == "cg":
        if rng.random() < 0.5:
            return dict(kind=kind, n=_log(rng, 5000, 150_000), coordinates="XZ", nx=rng.randint(20, 100), ny=1,
                        nz=rng.randint(11, 50), width=rng.choice([0.75, 1.0, 1.5]))
        return dict(kind=kind, n=_log(rng, 2000, 20_000), coordinates="XYZ", nx=rng.randint(7, 20),
                    ny=rng.randint(7, 20), nz=rng.randint(7, 24), width=rng.choice([0.75, 1.0]))
    if kind == "records":
        return dict(kind=kind, n=_log(rng, 2000, 50_000))
    if kind == "predict":
        return dict(kind=kind, rows=_log(rng, 100, 65_536))
    return dict(kind=kind, rows=_log(rng, 300, 4096), batch=rng.choice([256, 1000, 1024]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _mindlin(rolling_torsion):
    """The drum's Hertz-Mindlin species."""
    E, nu = 1e7, 0.3
    return scenarios.hertz_mindlin_species(E, E / 2 * (1 + nu), 0.7, 0.4, 0.05 if rolling_torsion else 0.0,
                                           rolling_torsion=rolling_torsion)


def _box(n, seed, law):
    """A jittered lattice whose neighbours overlap by 0.1 % of a diameter,
    filling a closed box of six walls."""
    s = 0.999
    nx = max(2, round(n ** (1 / 3)))
    nz = -(-n // (nx * nx))
    edge = lambda k: k * s * (1 + 1e-9)
    sc = scenarios.settling_box(n=n, seed=seed, box=(edge(nx), edge(nx), edge(nz)), spacing=s, jitter=0.005)
    if law != "sliding":
        sc.species = [_mindlin(law == "mindlin_rolling_torsion")]
    return sc


def _chute(n, seed):
    """The periodic chute started as close-packed layers, its area scaled with
    the number of spheres (100 x 50 small diameters for 200,000)."""
    f = math.sqrt(n / 200_000)
    return scenarios.periodic_chute(n_flow=n, seed=seed, packing="layers", lx=max(14.0, 100.0 * f),
                                    ly=max(14.0, 50.0 * f), base_fraction=0.4)


def _drum(n, seed, law):
    """The rotating drum (10 % of the spheres three times larger, 60 small
    diameters long) with a bed whose neighbours touch, its radius scaled with
    the number of spheres (175 small diameters for 1,000,000)."""
    R = scenarios.DRUM_RADIUS_D * math.sqrt(n / 1e6) + 6.0 * (n < 50_000)
    sc = scenarios.rotating_drum(n=n, seed=seed, radius_d=R, length_d=59.941, site_spacing=0.999, touch_wall=0.05,
                                 vstd=0.005)
    sc.species = [_mindlin(law == "mindlin_rolling_torsion")] * len(sc.species)
    return sc


def _scenario(case, seed):
    kind = case["kind"]
    if kind == "cg":
        kind = "chute" if case["coordinates"] == "XZ" else "box"
    if kind == "records":  # one packing, so that the number of contacts does not hang on the seed
        sc = _drum(case["n"], 1, "mindlin_rolling_torsion")
        sc.velocity = np.random.default_rng([seed, 9]).normal(0.0, 0.05, (sc.n, 3))
        return sc
    if kind == "drum":
        return _drum(case["n"], seed, case["law"])
    if kind == "box":
        return _box(case["n"], seed, case.get("law", "sliding"))
    if kind == "chute":
        return _chute(case["n"], seed)
    return scenarios.triangle_floor(n=case["n"], seed=seed, drop_d=0.02, v0=0.5,
                                    l_d=max(20.0, 100.0 * math.sqrt(case["n"] / 200_000)))


def _pinned(shape, dtype=torch.float64):
    return torch.zeros(shape, dtype=dtype, pin_memory=True).numpy()


def _pin(a):
    out = _pinned(a.shape, torch.from_numpy(a[:0].copy()).dtype)
    out[...] = a
    return out


def _state_buffers(n):
    return dict(position=_pinned((n, 3)), velocity=_pinned((n, 3)), angular_velocity=_pinned((n, 3)),
                orientation=_pinned((n, 4)))


# Time steps before the fields are read; the records are those of the initial
# evaluation.
STEPS_BEFORE_READING = dict(cg=10, records=0)


def _grid(case, sc):
    """Points, bounds and width of a coarse-graining case."""
    coord = _abi.DEM_CG_XZ if case["coordinates"] == "XZ" else _abi.DEM_CG_XYZ
    lo, hi = sc.instance.domain_min, sc.instance.domain_max
    top = float(sc.position[:, 2].max()) + SMALL_D
    return coord, (case["nx"], case["ny"], case["nz"]), lo, (hi[0], hi[1], top), case["width"] * SMALL_D


def _network(seed):
    """Parameters of the 4-256-256-256-3 network, uniform by fan-in."""
    g = np.random.default_rng([seed, 7])
    parts = []
    for rows, cols in ((256, 4), (256, 256), (256, 256), (3, 256)):
        a = math.sqrt(6.0 / cols)
        parts += [g.uniform(-a, a, rows * cols), g.uniform(-0.05, 0.05, rows)]
    return np.concatenate(parts).astype(np.float32)


def _samples(rows, seed):
    """Contact parameters in the calibration's box and smooth responses to them."""
    g = np.random.default_rng([seed, 8])
    lo, hi = calibration.PARAM_BOX[:, 0], calibration.PARAM_BOX[:, 1]
    u = g.uniform(size=(rows, 4))
    y = np.stack([15 + 20 * u[:, 0] + 9 * u[:, 0] * u[:, 1], 0.6 - 0.1 * u[:, 1] + 0.05 * u[:, 3],
                  0.1 + 0.2 * u[:, 2] * u[:, 2]], 1) * (1 + 0.01 * g.normal(size=(rows, 3)))
    return (lo + (hi - lo) * u).astype(np.float32), y.astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("predict", "train"):
        x, y = _samples(case["rows"], seed)
        s = Surrogate(capacity=65_536 if kind == "predict" else 4096, seed=0)
        s.fit_normalisation(x, y)
        s.set_params(_network(seed))
        return dict(case=case, net=s, x=x, y=y)
    if kind == "heaps":
        b, _, _ = calibration.heap_batch(case["instances"], seed=seed, n_range=(case["spheres"], case["spheres"]),
                                         spacing=1.0, v0=0.5)
        e = b.engine()
        e.step(0)
        return dict(case=case, engine=e, out=dict(position=_pinned((b.n, 3)), velocity=_pinned((b.n, 3))))
    sc = _scenario(case, seed)
    if kind == "drum":
        e = DemEngine(sc.time_step, [sc.instance], sc.species, sc.walls, rotation=sc.rotation)
        args = [_pin(a) for a in (sc.position, sc.velocity, sc.radius, sc.inv_mass, sc.inv_inertia)]
        return dict(case=case, engine=e, args=args + [_pin(sc.species_index), _pin(sc.ids)], out=_state_buffers(sc.n))
    e = sc.engine()
    if kind in ("cg", "records"):
        e.step(STEPS_BEFORE_READING[kind])
        return dict(case=case, engine=e, grid=_grid(case, sc) if kind == "cg" else None)
    e.step(0)
    return dict(case=case, engine=e, out=_state_buffers(sc.n))


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "predict":
        return state["net"].predict(state["x"])
    if kind == "train":
        net = state["net"]
        losses = net.fit(state["x"], state["y"], epochs=1, batch=case["batch"])
        return dict(losses=np.array(losses), params=net.params())
    e = state["engine"]
    if kind == "heaps":
        rows = e.batch_run(case["steps"])
        return dict(rows=rows, state=e.download(state["out"]))
    if kind == "cg":
        coord, n, lo, hi, width = state["grid"]
        return e.cg(coord, n, lo, hi, width)
    if kind == "records":
        force, torque = e.forces()
        return dict(contacts=e.contacts(), geometry=e.contact_geometry(), force=force, torque=torque)
    if kind == "drum":
        e.upload(*state["args"])
        e.step(case["steps"])
        return e.download(state["out"])
    e.step(case["steps"])
    return dict(balances=e.reduce(), state=e.download(state["out"]))


# Contacts per sphere of each kind of bed (pairs and walls), for the bytes of
# a step: 248 B per sphere, 64 B per contact of a law with one spring, 160 B
# with three.
CONTACTS = dict(box=2.5, drum=1.7, chute=2.0, floor=0.3, heaps=0.7, cg=2.0, records=1.7)


def work(case):
    kind = case["kind"]
    if kind in ("predict", "train"):
        flops = 2 * (4 * 256 + 2 * 256 * 256 + 3 * 256)
        n = case["rows"]
        if kind == "predict":
            return dict(bytes=n * (4 + 3) * 4 + 133_635 * 2, flops=float(n) * flops)
        steps = -(-n // case["batch"])
        return dict(bytes=n * (4 + 3) * 4 + steps * 133_635 * 4 * 7, flops=3.0 * n * flops)
    n = case["instances"] * case["spheres"] if kind == "heaps" else case["n"]
    c = n * CONTACTS[kind]
    if kind == "cg":
        pts = case["nx"] * case["ny"] * case["nz"]
        # a sphere or contact reaches about pi (3 w)^2 points of an XZ grid of
        # spacing w, 4/3 pi (3 w)^3 of an XYZ one
        reach = 28 * case["width"] ** 2 if case["coordinates"] == "XZ" else 113 * case["width"] ** 3
        return dict(bytes=n * 100 + c * 250 + pts * 29 * 8, flops=reach * (n * 60 + c * 200))
    if kind == "records":
        return dict(bytes=n * 2 * 48 + c * 2 * (16 + 8 * 22), flops=0)
    per_contact = 160 if kind == "heaps" or case.get("law") == "mindlin_rolling_torsion" else 64
    state = n * (48 if kind == "heaps" else 104)
    upload = n * 80 if kind == "drum" else 0
    return dict(bytes=case["steps"] * (n * 248 + c * per_contact) + state + upload,
                flops=case["steps"] * (n * 150 + c * 350))


# ---------------------------------------------------------------------------
# the same results in plain torch, 64 bits
# ---------------------------------------------------------------------------
class _Plain:
    """The DEM time step restated over arrays of pairs: linear viscoelastic
    with sliding friction, or Hertz with Mindlin (rolling, torsion) friction;
    flat walls and a cylinder about x; periodic boxes."""

    def __init__(self, sc):
        dev = self.dev = torch.device("cuda")
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
        self.sc, self.dt, self.sp = sc, sc.time_step, sc.species[0]
        self.x, self.v, self.r = t(sc.position), t(sc.velocity), t(sc.radius)
        self.im, self.ii = t(sc.inv_mass), t(sc.inv_inertia)
        self.n = len(sc.radius)
        self.w = torch.zeros_like(self.x)
        self.q = torch.zeros((self.n, 4), dtype=torch.float64, device=dev)
        self.q[:, 0] = 1.0
        self.g = t(sc.instance.gravity)
        self.fixed = self.im == 0
        self.L = torch.zeros(3, dtype=torch.float64, device=dev)
        for k in range(3):
            if sc.instance.periodic_mask >> k & 1:
                self.L[k] = sc.instance.periodic_max[k] - sc.instance.periodic_min[k]
        self.margin = 0.4 * float(self.r.min())
        self.moved = 1e30
        self.keys = torch.zeros(0, dtype=torch.int64, device=dev)
        self.springs = torch.zeros((0, 3, 3), dtype=torch.float64, device=dev)
        self.evaluation = 0

    def _near(self):
        """Pairs (i < j) closer than their radii plus the margin, by cells of a
        size per pair of radius classes."""
        x, r, n, dev = self.x, self.r, self.n, self.dev
        classes = [torch.arange(n, device=dev)]
        rmax = float(r.max())
        if rmax > 1.5 * float(r.min()):
            cut = 0.5 * rmax * 1.15
            classes = [torch.nonzero(r <= cut).flatten(), torch.nonzero(r > cut).flatten()]
        found = []
        lo = x.min(0).values
        span = x.max(0).values - lo + 1e-9
        for a in range(len(classes)):
            for b in range(a, len(classes)):
                A, B = classes[a], classes[b]
                if not len(A) or not len(B):
                    continue
                size = float(r[A].max() + r[B].max()) + self.margin
                dims = torch.floor(torch.where(self.L > 0, self.L, span) / size).clamp(min=1).long()
                width = torch.where(self.L > 0, self.L / dims, torch.full_like(self.L, size))
                org = torch.where(self.L > 0, torch.zeros_like(lo), lo)
                dims = torch.where(self.L > 0, dims, torch.floor(span / size).long() + 1)
                cell = lambda p: torch.minimum(torch.floor((p - org) / width).long().clamp(min=0), dims - 1)
                cb = cell(x[B])
                kb = (cb[:, 2] * dims[1] + cb[:, 1]) * dims[0] + cb[:, 0]
                kb, order = torch.sort(kb)
                Bs = B[order]
                ca = cell(x[A])
                for o in range(27):
                    off = torch.tensor([o % 3 - 1, o // 3 % 3 - 1, o // 9 - 1], device=dev)
                    c = ca + off
                    ok = torch.ones(len(A), dtype=torch.bool, device=dev)
                    for k in range(3):
                        if self.L[k] > 0:
                            if dims[k] < 3:
                                raise ValueError("a period of fewer than three cells")
                            c[:, k] %= dims[k]
                        else:
                            ok &= (c[:, k] >= 0) & (c[:, k] < dims[k])
                    key = (c[:, 2] * dims[1] + c[:, 1]) * dims[0] + c[:, 0]
                    first = torch.searchsorted(kb, key)
                    count = torch.where(ok, torch.searchsorted(kb, key, right=True) - first, torch.zeros_like(first))
                    for s in range(0, len(A), 200_000):
                        m = count[s:s + 200_000]
                        i = torch.repeat_interleave(A[s:s + 200_000], m)
                        at = torch.arange(len(i), device=dev) - torch.repeat_interleave(torch.cumsum(m, 0) - m, m)
                        j = Bs[torch.repeat_interleave(first[s:s + 200_000], m) + at]
                        keep = i < j if a == b else torch.ones_like(i, dtype=torch.bool)
                        i, j = i[keep], j[keep]
                        d = self._image(x[i] - x[j])
                        near = ((d * d).sum(1) < (r[i] + r[j] + self.margin) ** 2) & ~(self.fixed[i] & self.fixed[j])
                        found.append(torch.minimum(i[near], j[near]) * n + torch.maximum(i[near], j[near]))
        keys = torch.unique(torch.cat(found))
        self.pi, self.pj = keys // n, keys % n
        self.moved = 0.0

    def _image(self, d):
        for k in range(3):
            if self.L[k] > 0:
                d[:, k] -= self.L[k] * torch.round(d[:, k] / self.L[k])
        return d

    def _law(self, n, overlap, dist, vrel, vpi, wpi, im, curv, s, wall):
        """Force and torque of the first body, springs after, elastic energy, friction force."""
        sp, dt = self.sp, self.dt
        dot = lambda a, b: (a * b).sum(1, keepdim=True)
        cross = lambda a, b: torch.linalg.cross(a, b, dim=1)
        vn = dot(vrel, n)
        vt = vrel - n * vn
        touching = overlap > 0
        if sp.normal_law == _abi.DEM_NORMAL_LINEAR_VISCOELASTIC:
            fn = torch.where(touching, sp.stiffness * overlap - sp.dissipation * vn, torch.zeros_like(vn))
            energy = torch.where(touching, 0.5 * sp.stiffness * overlap ** 2, torch.zeros_like(vn))
            slide = s[:, 0]
            step = vt if wall else vt - dot(slide, vpi) * n / dist
            slide = torch.where(touching, slide + step * dt, slide)
            ft = -sp.sliding_stiffness * slide - sp.sliding_dissipation * vt
            size = ft.norm(dim=1, keepdim=True)
            slips = size > sp.sliding_mu * fn.abs()
            ft = torch.where(slips, ft * (sp.sliding_mu * fn.abs() / size.clamp(min=1e-300)), ft)
            slide = torch.where(slips & touching, -(ft + sp.sliding_dissipation * vt) / sp.sliding_stiffness, slide)
            ft = torch.where(touching, ft, torch.zeros_like(ft))
            energy = energy + 0.5 * sp.sliding_stiffness * dot(slide, slide)
            return fn * n + ft, torch.zeros_like(ft), torch.stack([slide, s[:, 1], s[:, 2]], 1), energy, ft
        reff, meff = 1 / curv, 1 / im
        over = overlap.clamp(min=1e-300)
        k = 4 / 3 * sp.elastic_modulus * torch.sqrt(reff * over)
        fn = torch.where(touching, k * overlap - sp.dissipation * torch.sqrt(meff * k) * vn, torch.zeros_like(vn))
        energy = torch.where(touching, 0.4 * k * overlap ** 2, torch.zeros_like(vn))
        size = fn.abs()
        kt = 8 * sp.shear_modulus * torch.sqrt(reff * over)

        def turned(a):
            L = a.norm(dim=1, keepdim=True)
            b = a - dot(a, n) * n
            return torch.where(L > 1e-10, b * (L / b.norm(dim=1, keepdim=True).clamp(min=1e-300)), a)

        slide = turned(s[:, 0]) + vt * dt
        ft = -2 / 3 * kt * slide
        fl = ft.norm(dim=1, keepdim=True)
        sticks = fl < sp.sliding_mu * size
        slipped = ft * (sp.sliding_mu * size / fl.clamp(min=1e-300))
        slide = torch.where(sticks, slide, -(slipped / (2 / 3 * kt)))
        ft = torch.where(sticks, ft - sp.sliding_dissipation * torch.sqrt(meff * kt) * vt, slipped)
        torque = torch.zeros_like(ft)
        roll, tors = s[:, 1], s[:, 2]
        if sp.friction_law == _abi.DEM_FRICTION_MINDLIN_ROLLING_TORSION:
            if sp.torsion_mu != 0:
                raise ValueError("torsion is not restated")
            if sp.rolling_mu != 0:
                vr = -reff * cross(n, wpi)
                roll = turned(roll) + vr * dt
                fr = -kt * roll - sp.rolling_dissipation * vr
                fl = fr.norm(dim=1, keepdim=True)
                slips = fl > sp.rolling_mu * size
                fr = torch.where(slips, fr * (sp.rolling_mu * size / fl.clamp(min=1e-300)), fr)
                roll = torch.where(slips, -(fr + sp.rolling_dissipation * vr) / kt, roll)
                torque = reff * cross(n, fr)
        live = size != 0
        pick = lambda a, b: torch.where(live, a, b)
        springs = torch.stack([pick(slide, s[:, 0]), pick(roll, s[:, 1]), tors], 1)
        ft, torque = pick(ft, torch.zeros_like(ft)), pick(torque, torch.zeros_like(ft))
        return fn * n + ft, torque, springs, energy, ft

    def _walls(self):
        """Distance to and outward normal of each wall: (index, distance, normal, angular velocity, position)."""
        for k, w in enumerate(self.sc.walls):
            q0, q1, q2, q3 = w.orientation
            a = torch.tensor([q0 * q0 - q3 * q3 + q1 * q1 - q2 * q2, 2 * (q1 * q2 + q3 * q0), 2 * (q1 * q3 - q2 * q0)],
                             dtype=torch.float64, device=self.dev)
            pos = torch.tensor(list(w.position), dtype=torch.float64, device=self.dev)
            om = torch.tensor(list(w.angular_velocity), dtype=torch.float64, device=self.dev)
            if w.type == _abi.DEM_WALL_INFINITE:
                yield k, ((pos - self.x) * a).sum(1), a.expand(self.n, 3), om, pos
            else:
                d = self.x - pos
                d = d - (d * a).sum(1, keepdim=True) * a
                rho = d.norm(dim=1, keepdim=True)
                yield k, w.faces[0][3] - rho[:, 0], d / rho.clamp(min=1e-300), om, pos

    def forces(self):
        if self.moved > 0.45 * self.margin:
            self._near()
        x, v, w, r = self.x, self.v, self.w, self.r
        self.F = torch.zeros_like(x)
        self.T = torch.zeros_like(x)
        i, j = self.pi, self.pj
        raw = x[i] - x[j]
        br = self._image(raw.clone())
        d2 = (br * br).sum(1)
        hit = d2 < (r[i] + r[j]) ** 2
        i, j, br, per = i[hit], j[hit], br[hit], ((raw - br)[hit] != 0).any(1)
        dist = br.norm(dim=1, keepdim=True)
        n = br / dist
        overlap = (r[i] + r[j])[:, None] - dist
        c = -(r[i][:, None] - 0.5 * overlap) * n  # contact point from P
        cross = lambda a, b: torch.linalg.cross(a, b, dim=1)
        vrel = (v[i] - cross(c, w[i])) - (v[j] - cross(c + br, w[j]))
        key = [i * self.n + j]
        old = [self._old(key[0])]
        F, T, s, e, ft = self._law(n, overlap, dist, vrel, v[i] - v[j], w[i] - w[j], (self.im[i] + self.im[j])[:, None],
                                   (1 / r[i] + 1 / r[j])[:, None], old[0], False)
        if self.evaluation == 1 and bool(per.any()):
            # the first step shares its time stamp with the initial evaluation:
            # a pair across the boundary keeps its spring of that evaluation
            was = per & self._had(key[0])
            s = torch.where(was[:, None, None], old[0], s)
        self.F.index_add_(0, i, F)
        self.F.index_add_(0, j, -F)
        self.T.index_add_(0, i, T - cross(-c, F))
        self.T.index_add_(0, j, -T + cross(-(c + br), F))
        out = [dict(p=i, i=j, wall=torch.zeros_like(i), per=per.long(), s=s, F=F, o=overlap[:, 0], c=c + x[i], n=n, ft=ft,
                    e=e, br=br)]
        self.F += torch.where(self.fixed[:, None], torch.zeros_like(x), self.g * (1 / self.im.clamp(min=1e-300))[:, None])
        for k, dist, nrm, om, pos in self._walls():
            at = torch.nonzero((dist < r) & ~self.fixed).flatten()
            n = -nrm[at]
            dist = dist[at][:, None]
            overlap = r[at][:, None] - dist
            c = -(r[at][:, None] - 0.5 * overlap) * n
            key.append(-(at * 64 + k) - 1)
            vrel = (v[at] - cross(c, w[at])) + cross(c + x[at] - pos, om.expand(len(at), 3))
            F, T, s, e, ft = self._law(n, overlap, dist, vrel, v[at], w[at] - om, self.im[at][:, None],
                                       (1 / r[at])[:, None], self._old(key[-1]), True)
            self.F.index_add_(0, at, F)
            self.T.index_add_(0, at, T - cross(-c, F))
            one = torch.ones_like(at)
            out.append(dict(p=at, i=one * k, wall=one, per=0 * one, s=s, F=F, o=overlap[:, 0], c=c + x[at], n=n, ft=ft,
                            e=e, br=torch.zeros_like(F)))
        self.contacts = {f: torch.cat([o[f] for o in out]) for f in out[0]}
        keys, springs = torch.cat(key), self.contacts["s"]
        if self.evaluation == 1:  # what the first step does not touch outlives it
            gone = ~torch.isin(self.keys, keys)
            keys, springs = torch.cat([keys, self.keys[gone]]), torch.cat([springs, self.springs[gone]])
        self.keys, order = torch.sort(keys)
        self.springs = springs[order]
        self.evaluation += 1

    def _had(self, key):
        if not len(self.keys):
            return torch.zeros(len(key), dtype=torch.bool, device=self.dev)
        at = torch.searchsorted(self.keys, key).clamp(max=len(self.keys) - 1)
        return self.keys[at] == key

    def _old(self, key):
        s = torch.zeros((len(key), 3, 3), dtype=torch.float64, device=self.dev)
        if len(self.keys):
            at = torch.searchsorted(self.keys, key).clamp(max=len(self.keys) - 1)
            s = torch.where((self.keys[at] == key)[:, None, None], self.springs[at], s)
        return s

    def steps(self, count):
        if self.evaluation == 0:
            self.forces()
        dt = self.dt
        for _ in range(count):
            self.v += self.F * (0.5 * dt * self.im)[:, None]
            self.x += self.v * dt
            self.moved += float((self.v * dt).norm(dim=1).max())
            for k in range(3):
                if self.L[k] > 0:
                    lo = self.sc.instance.periodic_min[k]
                    self.x[:, k] += self.L[k] * ((self.x[:, k] < lo).double() - (self.x[:, k] > lo + self.L[k]).double())
            self.w += self.T * (0.5 * dt * self.ii)[:, None]
            q, a = self.q, self.w * dt
            d = 0.5 * torch.stack([-q[:, 1] * a[:, 0] - q[:, 2] * a[:, 1] - q[:, 3] * a[:, 2],
                                   q[:, 0] * a[:, 0] + q[:, 3] * a[:, 1] - q[:, 2] * a[:, 2],
                                   -q[:, 3] * a[:, 0] + q[:, 0] * a[:, 1] + q[:, 1] * a[:, 2],
                                   q[:, 2] * a[:, 0] - q[:, 1] * a[:, 1] + q[:, 0] * a[:, 2]], 1)
            self.q = (q + d) / (q + d).norm(dim=1, keepdim=True)
            self.forces()
            self.v += self.F * (0.5 * dt * self.im)[:, None]
            self.w += self.T * (0.5 * dt * self.ii)[:, None]

    def state(self):
        return dict(position=self.x.cpu().numpy(), velocity=self.v.cpu().numpy(), angular_velocity=self.w.cpu().numpy(),
                    orientation=self.q.cpu().numpy())

    def balances(self, steps):
        move = ~self.fixed
        m, x, v, w = 1 / self.im[move], self.x[move], self.v[move], self.w[move]
        inertia = 1 / self.ii[move]
        c = self.contacts
        num = lambda a: a.cpu().numpy()
        com = (m[:, None] * x).sum(0) / m.sum()
        return dict(kinetic_energy=float(0.5 * (m * (v * v).sum(1)).sum()),
                    rotational_energy=float(0.5 * (inertia * (w * w).sum(1)).sum()),
                    gravitational_energy=float(-(m[:, None] * x * self.g).sum()), elastic_energy=float(c["e"].sum()),
                    momentum=num((m[:, None] * v).sum(0)), angular_momentum=num((inertia[:, None] * w).sum(0)),
                    mass=float(m.sum()), centre_of_mass=num(com), n_contacts=int((c["wall"] == 0).sum()),
                    n_wall_contacts=int(c["wall"].sum()), time=steps * self.dt, n_steps=steps)

    def sorted_contacts(self):
        c = self.contacts
        order = torch.argsort((c["wall"] * self.n + c["p"]) * (self.n + 64) + c["i"])
        return {k: a[order] for k, a in c.items()}


def _plain_fields(p, case, grid):
    """The 29 fields of every point by direct sums over spheres and contacts."""
    _, n, lo, hi, width = grid
    dev = p.dev
    xyz = case["coordinates"] == "XYZ"
    dims = [0, 1, 2] if xyz else [0, 2]
    cut = 3.0 * width
    f64 = dict(dtype=torch.float64, device=dev)
    idx = torch.stack(torch.meshgrid(*[torch.arange(k, device=dev) for k in n], indexing="ij"), -1).reshape(-1, 3)
    lo_t, hi_t = torch.tensor(lo, **f64), torch.tensor(hi, **f64)
    n_t = torch.tensor(n, **f64)
    delta = (hi_t - lo_t) / n_t
    pts = lo_t + 0.5 * delta + delta * idx
    root2, rootpi = math.sqrt(2.0), math.sqrt(math.pi)
    one = 1 / (root2 * rootpi * width)
    ratio = cut / width
    if xyz:
        pre = one ** 3 / (math.erf(ratio / root2) - root2 / rootpi * ratio * math.exp(-0.5 * ratio ** 2))
        line = one ** 2 / (1 - math.exp(-0.5 * ratio ** 2))
    else:
        pre = one ** 2 / (1 - math.exp(-0.5 * ratio ** 2))
        line = one / math.erf(cut / (width * root2))
    move = ~p.fixed
    x, v, r, m = p.x[move], p.v[move], p.r[move], 1 / p.im[move]
    val = [4 / 3 * math.pi * r ** 3, m] + [v[:, a] * m for a in range(3)]
    val += [v[:, a] * v[:, b] * m for a, b in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))]
    val = torch.stack(val + [r ** k for k in range(6)], 1)
    c = p.contacts
    pf, wall = p.fixed[c["p"]], c["wall"] == 1
    jf = torch.where(wall, torch.ones_like(wall), p.fixed[torch.where(wall, torch.zeros_like(c["i"]), c["i"])])
    both = ~(pf & jf)
    c = {k: a[both] for k, a in c.items()}
    pf, jf, wall = pf[both], jf[both], wall[both]
    P, C, nn = p.x[c["p"]], c["c"], c["n"]
    wpos = torch.tensor([list(w.position) for w in p.sc.walls] or [[0.0] * 3], **f64)
    I = torch.where(wall[:, None], wpos[torch.where(wall, c["i"], torch.zeros_like(c["i"]))],
                    p.x[torch.where(wall, torch.zeros_like(c["i"]), c["i"])])
    dist = c["br"].norm(dim=1, keepdim=True)
    branch = torch.where(pf[:, None], nn * dist + C - P, torch.where(jf[:, None], P - C, nn * dist))
    ifd = torch.where(pf[:, None], -c["F"], torch.where(jf[:, None], c["F"], torch.zeros_like(c["F"])))
    stress = (c["F"][:, :, None] * branch[:, None, :]).reshape(-1, 9)
    ie, pe = torch.where(jf[:, None] & ~pf[:, None], C, I), torch.where(pf[:, None], C, P)
    sel = torch.zeros(3, **f64)
    sel[dims] = 1.0
    nl = (nn * sel).norm(dim=1, keepdim=True)
    nh = nn * sel / nl if not xyz else nn
    length = ((pe - ie) * nh).sum(1)
    ws = width * root2
    b = cut + length
    a = -cut
    prefactor = line * 0.5 / (torch.erf(b / ws) * b + ws / rootpi * torch.exp(-(b / ws) ** 2)
                              - math.erf(a / ws) * a - ws / rootpi * math.exp(-(a / ws) ** 2))
    end = torch.where(jf[:, None], C, I)
    inv = n_t / (hi_t - lo_t)
    ends = torch.stack([(P - lo_t) * inv - 0.5, (end - lo_t) * inv - 0.5])
    first = torch.floor(ends.min(0).values - cut * inv + 1).clamp(min=0)
    last = torch.floor(ends.max(0).values + cut * inv + 1).clamp(min=0)
    out = torch.zeros((len(pts), 29), **f64)
    for s in range(0, len(pts), 64):
        q, qi = pts[s:s + 64, None, :], idx[s:s + 64, None, :]
        d2 = (((x[None] - q) * sel) ** 2).sum(2)
        f = torch.where(d2 > cut * cut, torch.zeros_like(d2), pre * torch.exp(-d2 / (2 * width * width))) @ val
        out[s:s + 64, :11], out[s:s + 64, 23:] = f[:, :11], f[:, 11:]
        for t in range(0, len(P), 100_000):
            at = slice(t, t + 100_000)
            iN = ((ie[at] - q) * nh[at]).sum(2)
            pN = ((pe[at] - q) * nh[at]).sum(2)
            t2 = (((P[at] - q) * sel) ** 2).sum(2) - pN * pN
            inside = torch.ones_like(iN, dtype=torch.bool)
            for k in dims:
                if n[k] > 1:
                    inside &= (qi[:, :, k] >= first[at, k]) & (qi[:, :, k] < last[at, k])
            psi = prefactor[at] * (torch.erf(pN / ws) - torch.erf(iN / ws)) * torch.exp(-0.5 * t2 / width ** 2)
            psi = torch.where(inside & (iN <= cut) & (pN >= -cut) & (t2 <= cut * cut), psi, torch.zeros_like(psi))
            out[s:s + 64, 11:20] += psi @ stress[at]
            d2 = (((C[at] - q) * sel) ** 2).sum(2)
            phi = torch.where(inside & (d2 <= cut * cut), pre * torch.exp(-d2 / (2 * width * width)), torch.zeros_like(d2))
            out[s:s + 64, 20:23] += phi @ ifd[at]
    return (out / (1.0 if xyz else hi[1] - lo[1])).cpu().numpy()


def _plain_network(flat, x, norm):
    at = 0
    h = (x - norm[0]) / norm[1]
    for k, (rows, cols) in enumerate(((256, 4), (256, 256), (256, 256), (3, 256))):
        W = flat[at:at + rows * cols].reshape(rows, cols)
        h = h @ W.T + flat[at + rows * cols:at + rows * cols + rows]
        at += rows * cols + rows
        if k < 3:
            h = torch.nn.functional.gelu(h)
    return h


def exact(case, seed):
    kind = case["kind"]
    if kind in ("heaps", "floor"):
        return None  # heaps on their disk with deletion, grouped triangles: no plain restatement here
    if kind in ("predict", "train"):
        x, y = _samples(case["rows"], seed)
        t = lambda a: torch.as_tensor(np.asarray(a, np.float64))
        std = lambda a: np.maximum(np.asarray(a, np.float64).std(0), 1e-6)
        norm = [t(np.float32(a)) for a in (np.float64(x).mean(0), std(x), np.float64(y).mean(0), std(y))]
        flat = t(_network(seed))
        if kind == "predict":
            return (_plain_network(flat, t(x), norm) * norm[3] + norm[2]).numpy()
        m, v, losses = torch.zeros_like(flat), torch.zeros_like(flat), []
        order = np.random.default_rng(0).permutation(len(x))
        for step, a in enumerate(range(0, len(x), case["batch"]), 1):
            at = order[a:a + case["batch"]]
            flat = flat.detach().requires_grad_(True)
            loss = ((_plain_network(flat, t(x[at]), norm) - (t(y[at]) - norm[2]) / norm[3]) ** 2).mean()
            g, = torch.autograd.grad(loss, flat)
            losses.append(float(loss.detach()))
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            flat = flat.detach() - 1e-3 * (m / (1 - 0.9 ** step)) / (torch.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
        return dict(losses=np.array([np.mean(losses)]), params=flat.numpy())
    sc = _scenario(case, seed)
    p = _Plain(sc)
    if kind in ("cg", "records"):
        p.steps(STEPS_BEFORE_READING[kind])
        if kind == "cg":
            return _plain_fields(p, case, _grid(case, sc))
        c = p.sorted_contacts()
        num = lambda a: a.cpu().numpy()
        whole = lambda k: num(c[k]).astype(np.int32)
        return dict(contacts=dict(id_p=whole("p"), id_i=whole("i"), is_wall=whole("wall"), periodic=whole("per"),
                                  springs=num(c["s"].reshape(-1, 9)), force=num(c["F"]), overlap=num(c["o"])),
                    geometry=dict(contact_point=num(c["c"]), normal=num(c["n"]), tangential_force=num(c["ft"])),
                    force=num(p.F), torque=num(p.T))
    p.steps(case["steps"])
    if kind == "drum":
        return p.state()
    return dict(balances=p.balances(case["steps"]), state=p.state())
