"""Workloads the engine's speed is measured on, through its public entry points.

A case is one way a program uses the engine: stepping a scene between two reads of its state
(``GpuEngine.run`` + ``state``), coupling it to another solver (``set_state`` + ``run`` +
``state``, ``run_with_impulses``), advancing a batch of scenes, serving jobs, or reading its
observables; in the FP64 form (the drop-in, whose candidate list is rebuilt every `up` steps) and
the mixed form, from a few dozen spheres to two million, with the linear and the Hertz laws,
equal and polydisperse radii, fixed and turning walls.

Every scene comes from vedo_gb300.scenes with its sizes chosen so that spheres touch from the first
step.  ``exact`` restates the time step in plain 64-bit torch (every contact of the step at once,
summed by index).
"""
import math

import numpy as np
import torch

from vedo_gb300 import scenes
from vedo_gb300.engine import STATE_FIELDS, BatchEngine, GpuEngine
from vedo_gb300.serve import Server

MOTION = ("position", "velocity", "angular_velocity")
IMPULSES = ("impact", "angular_impact")
FOREVER = 10 ** 8          # steps until t_stop: no pass reaches it


def listed():
    return [
        # one step of a small linear-law scene with the list rebuilt every step (anne's default
        # UpIact of 1): the shortest call, and the one a debugging or teaching run makes
        {"name": "fp64_small_step", "kind": "run", "scene": "cluster", "n": 64, "form": "fp64", "up": 1, "steps": 1},
        # the 8,000-sphere linear box between two reads, list every 20 steps: the plain drop-in run
        {"name": "fp64_box", "kind": "run", "scene": "box", "n": 8000, "form": "fp64", "up": 20, "steps": 20},
        # the polydisperse drum (32 radii, turning shell and end plates) in the drop-in form
        {"name": "fp64_drum", "kind": "run", "scene": "drum", "n": 150001, "form": "fp64", "up": 20, "steps": 20},
        # a dense Hertz packing coupled to a fluid solver: forces in, one step, motion out
        {"name": "fp64_coupled_step", "kind": "impulses", "scene": "pack", "n": 300000, "form": "fp64", "up": 20,
         "steps": 1},
        # the same box in the mixed form as it comes out of the constructor (no tuning)
        {"name": "mixed_box", "kind": "run", "scene": "box", "n": 8000, "form": "mixed", "steps": 30},
        # the bulk run of the mixed form: a dense packing, every pair in contact, tuned settings
        {"name": "mixed_pack", "kind": "run", "scene": "pack", "n": 1000000, "form": "mixed", "tick": "pair",
         "steps": 20},
        # the polydisperse drum in the mixed form with the settings the tuner picks for it
        {"name": "mixed_drum", "kind": "run", "scene": "drum", "n": 400000, "form": "mixed", "tick": "pair",
         "steps": 40},
        # a large loose bed (nothing touches yet) with rods and a moving top plate, light tick
        {"name": "mixed_loose_bed", "kind": "run", "scene": "bed", "n": 2000000, "form": "mixed", "tick": "split",
         "steps": 20},
        # a coupling loop that owns the state: upload, 10 steps, download
        {"name": "mixed_coupled", "kind": "assigned", "scene": "hopper", "n": 60000, "form": "mixed", "steps": 10},
        # many hoppers of uneven sizes with different materials in one engine: a parameter study
        {"name": "hopper_batch", "kind": "batch", "scenes": 48, "n": 700000, "tick": "pair", "steps": 20},
        # a few short jobs submitted to the job server and their results collected
        {"name": "serve_jobs", "kind": "serve", "scenes": 6, "n": 60000, "steps": 100},
        # energies, contacts and coordination numbers of a running simulation (post-processing hook)
        {"name": "monitor", "kind": "monitor", "scene": "pack", "n": 500000, "form": "mixed"},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["run", "run", "run", "run", "impulses", "assigned", "batch", "serve", "monitor"])
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(2, 48), "n": size(5000, 500000),
                "tick": rng.choice(["full", "pair", "split"]), "steps": rng.randint(5, 20)}
    if kind == "serve":
        return {"kind": kind, "scenes": rng.randint(1, 8), "n": size(5000, 60000), "steps": rng.randint(20, 150)}
    form = rng.choice(["fp64", "mixed"])
    scene = rng.choice(["cluster", "box", "pack", "drum", "hopper", "bed", "job"])
    if kind == "monitor":
        return {"kind": kind, "scene": rng.choice(["box", "pack", "hopper"]), "n": size(500, 500000), "form": form}
    if kind in ("impulses", "assigned"):
        scene = rng.choice(["box", "pack", "hopper"])
    limits = {"cluster": (20, 3000), "box": (500, 60000), "pack": (2000, 300000), "drum": (5000, 150000),
              "hopper": (500, 100000), "bed": (20000, 400000), "job": (2000, 60000)}
    case = {"kind": kind, "scene": scene, "n": size(*limits[scene]), "form": form,
            "steps": 1 if kind == "impulses" else rng.randint(1, 40)}
    if form == "fp64":
        case["up"] = rng.choice([1, 5, 20, 50])
    else:
        case["tick"] = rng.choice(["full", "pair", "split"])
    return case


# ---- inputs -----------------------------------------------------------------------------------
def _scene(kind, n, seed):
    if kind == "cluster":                      # colliding linear-law spheres in a small box
        return scenes.cluster(n=n, seed=seed, steps=FOREVER, spacing=2.002e-3, vel_sigma=0.2)
    if kind == "box":                          # linear law, nearly touching cubic lattice, open box
        side = max(4, round(n ** (1.0 / 3.0)))
        return scenes.lsd_box(n_side=side, seed=seed, steps=FOREVER, spacing=2.001e-3, jitter=2e-6,
                              box_width=side * 2.001e-3 + 1e-4, box_height=side * 2.001e-3 + 1e-2)
    if kind == "pack":                         # Hertz law, face-centred packing, 12 contacts a sphere
        return scenes.dense_pack(n=n, seed=seed, steps=FOREVER)
    if kind == "drum":                         # 32 radii in touching layers, turning shell
        return scenes.hertz_drum(n=n, seed=seed, steps=FOREVER, fill="lattice", gap=0.0, vel_sigma=1e-3)
    if kind == "hopper":                       # Hertz law, draining column
        return _hopper(n, seed, seed)
    if kind == "bed":                          # loose bed, rods, moving top plate
        return scenes.compressed_bed(n=n, seed=seed, steps=FOREVER, box=max(0.03, 0.4 * math.sqrt(n / 16e6)),
                                     cylinders=max(1, 32 * n // 16000000), packing="fcc")
    # the serving stream's polydisperse job
    return scenes.serving_job("settle" if seed % 2 else "projectile", n, "lsd" if seed % 4 < 2 else "hertz", seed,
                              steps=FOREVER)


def _hopper(n, seed, material):
    rng = np.random.default_rng(material)
    sc = scenes.hopper(n=n, seed=seed, friction=rng.uniform(0.2, 0.6), restitution=rng.uniform(0.5, 0.9),
                       orifice=rng.uniform(6e-3, 12e-3), steps=FOREVER, touching=True)
    sc.velocity[:n] = np.random.default_rng(seed).normal(0.0, 1e-2, size=(n, 3))
    return sc


def _share(n, parts):
    """n spheres over `parts` scenes of uneven sizes (the largest about 20 times the smallest)."""
    w = np.exp(np.linspace(0.0, math.log(20.0), parts))
    return [max(200, int(n * x / w.sum())) for x in w]


def _scenes(case, seed):
    sizes = _share(case["n"], case["scenes"])
    if case["kind"] == "batch":
        return [_hopper(k, seed + 17 * q, seed + q) for q, k in enumerate(sizes)]
    return [scenes.serving_job("settle" if q % 2 else "projectile", k, "lsd" if q % 4 < 2 else "hertz", seed + q,
                               steps=FOREVER) for q, k in enumerate(sizes)]


def _fields(case):
    if case.get("form") == "fp64":
        return STATE_FIELDS
    return MOTION if case["n"] >= 300000 else MOTION + IMPULSES


def _options(case):
    if case.get("form") == "fp64":
        return {"up_iact": case["up"]}
    tick = case.get("tick", "full")
    opts = {"precision": 1}
    if tick == "pair":                       # what the tuner settles on for packed scenes
        opts.update(pair_pass=True, stored_splits=True, tick_block=64)
    elif tick == "split":                      # ... and for loose ones
        opts.update(split_tick=True, stored_splits=True)
    return opts


def _pinned(n, fields):
    return {f: torch.zeros((n, 3), dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy() for f in fields}


def _impulses(n, seed):
    """Forces of a coupled solver on every object over one step, about a sphere's weight."""
    rng = np.random.default_rng(seed + 5)
    j = 2e-10 * rng.standard_normal((n, 3))
    return j, 1e-14 * rng.standard_normal((n, 3))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        jobs = _scenes(case, seed)
        return {"kind": kind, "server": Server(), "jobs": jobs, "steps": case["steps"]}
    if kind == "batch":
        opts = _options(dict(case, form="mixed"))
        opts.pop("precision")
        eng = BatchEngine(_scenes(case, seed), **opts)
        return {"kind": "run", "engine": eng, "steps": case["steps"], "out": _pinned(eng.n, _fields(case))}
    scene = _scene(case["scene"], case["n"], seed)
    eng = GpuEngine(scene, **_options(case))
    state = {"kind": kind, "engine": eng, "steps": case.get("steps", 0), "out": _pinned(eng.n, _fields(case))}
    if kind == "assigned":
        state["given"] = _pinned(eng.n, MOTION)
        for f in MOTION:
            state["given"][f][:] = getattr(scene, f)
    elif kind == "impulses":
        state["impulses"] = _pinned(eng.n, IMPULSES)
        j, ja = _impulses(eng.n, seed)
        state["impulses"]["impact"][:], state["impulses"]["angular_impact"][:] = j, ja
    elif kind == "monitor":
        lo, hi = scene.position.min(0), scene.position.max(0)
        state["box"] = [float(x) for k in range(3) for x in (lo[k] + 0.2 * (hi[k] - lo[k]), lo[k] + 0.8 * (hi[k] - lo[k]))]
    return state


def run(state):
    kind = state["kind"]
    if kind == "serve":
        ids = [state["server"].submit(sc, state["steps"]) for sc in state["jobs"]]
        out = []
        for j in ids:
            info = state["server"].wait(j)
            if info["status"] != "done":
                raise RuntimeError("job %d: %s" % (j, info["status"]))
            out.append(state["server"].result(j, MOTION + IMPULSES))
        return out
    eng = state["engine"]
    if kind == "monitor":
        below, touching, average = eng.coordination(state["box"])
        return {"observables": eng.observables(), "below": below.view(np.int32), "touching": touching.view(np.int32),
                "average": average}
    if kind == "impulses":
        eng.run_with_impulses(state["impulses"]["impact"], state["impulses"]["angular_impact"])
    else:
        if kind == "assigned":
            eng.set_state(**state["given"])
        eng.run(state["steps"])
    return eng.state(tuple(state["out"]), out=state["out"])


# ---- what a pass cannot do without ----------------------------------------------------------------
#: contacts per sphere and prefilter candidates per sphere at the start of each scene
CONTACTS = {"cluster": 1.0, "box": 0.8, "pack": 5.9, "drum": 1.5, "hopper": 1.5, "bed": 0.0, "job": 0.0}


def work(case):
    n = case["n"]
    if case["kind"] == "monitor":              # positions, velocities, radii in; two counts out
        return {"bytes": n * (72.0 + 8.0 + 8.0), "flops": n * 120.0}
    fp64 = case.get("form") == "fp64"
    z = CONTACTS[case.get("scene", "hopper" if case["kind"] == "batch" else "job")]
    # per step: position, velocity, spin (and, FP64, orientation) read and written, each contact's
    # history read and written with its two indices, the radius; per pass: the state to the host
    state, hist = (120.0, 32.0) if fp64 else (72.0, 16.0)
    per_step = 2.0 * state + z * (2.0 * hist + 8.0) + 8.0
    sync = 24.0 * len(_fields(case)) * (2.0 if case["kind"] == "assigned" else 1.0)
    flops = 60.0 + z * 250.0 + (150.0 if fp64 else 0.0)
    return {"bytes": n * (case["steps"] * per_step + sync), "flops": n * case["steps"] * flops}


# ---- the same step in plain 64-bit torch -----------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        # every scene alone; the batch's objects are numbered scene after scene
        fields = _fields(case) if kind == "batch" else MOTION + IMPULSES
        each = [_Step(sc).run(case["steps"], fields) for sc in _scenes(case, seed)]
        return each if kind == "serve" else {f: np.concatenate([e[f] for e in each]) for f in fields}
    scene = _scene(case["scene"], case["n"], seed)
    step = _Step(scene)
    if kind == "monitor":
        lo, hi = scene.position.min(0), scene.position.max(0)
        return step.monitor([float(x) for k in range(3) for x in (lo[k] + 0.2 * (hi[k] - lo[k]),
                                                                  lo[k] + 0.8 * (hi[k] - lo[k]))])
    ext = _impulses(scene.num_objects, seed) if kind == "impulses" else None
    return step.run(case["steps"], _fields(case), ext)


SPHERE, CYLINDER, PLATE, SHELL = 1, 6, 7, 32
MOBILE, ORBITAL = 3, 4


class _Step:
    """Spheres against spheres and walls by the linear (ISwBSDBF) or Hertz (ISwH) law."""

    def __init__(self, sc):
        dev = self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
        self.sc, self.dt = sc, sc.sp.time_interval
        self.P, self.V, self.W = t(sc.position), t(sc.velocity), t(sc.angular_velocity)
        self.X, self.Z = t(sc.orientation_x), t(sc.orientation_z)
        self.model = torch.as_tensor(sc.model_index.astype(np.int64), device=dev)
        an = [m.analysis() for m in sc.models]
        shape = np.array([m.shape for m in sc.models])
        beh = np.array([m.behavior for m in sc.models])
        moves = (shape == SPHERE) & (beh == MOBILE)
        self.sudo = t(np.where(shape == SPHERE, [a[3] for a in an], 0.0))[self.model]
        self.mass = t([a[2] for a in an])[self.model]
        self.inertia = t([a[4][0] for a in an])[self.model]
        self.r = t([m.attrs[0] if m.shape == SPHERE else 0.0 for m in sc.models])[self.model]
        self.moves = torch.as_tensor(moves, device=dev)[self.model]
        wall = shape[sc.model_index] != SPHERE
        self.walls = [int(i) for i in np.flatnonzero(wall)]
        self.balls = torch.as_tensor(np.flatnonzero(~wall), device=dev)
        self.g = t(sc.sp.field_acceleration)
        self._tables(an)
        self._pairs()

    def _tables(self, an):
        sc, nm = self.sc, len(self.sc.models)
        by = {}
        for im in sc.iact_models:
            by.setdefault(frozenset((im.master_group, im.slave_group)), im)
        tab, hertz = np.zeros((nm, nm, 6)), False
        for a, A in enumerate(sc.models):
            if A.shape != SPHERE:
                continue
            for b, B in enumerate(sc.models):
                im = by.get(frozenset((A.group, B.group)))
                if im is None:
                    continue
                get = dict(im.mechanisms).get
                if im.equation_type == "ISwH":
                    hertz = True
                    tab[a, b] = [get(k) for k in ("HertzNormalStiffness", "EquivalentMass", "ShearStiffnessCoefficient1",
                                                  "ShearStiffnessCoefficient2", "DampingRatio",
                                                  "KineticFrictionCoefficient")]
                else:
                    ma, mb = an[a][3], (an[b][3] if B.shape == SPHERE else 0.0)
                    me = ma if mb == 0.0 else 0.5 * (ma + mb)
                    kn, ks = get("NormalStiffness"), get("ShearStiffness")
                    tab[a, b] = [kn, ks, get("NormalDampingRatio") * 2.0 * math.sqrt(me * kn),
                                 get("ShearDampingRatio") * 2.0 * math.sqrt(me * ks), get("FrictionCoefficient"), 0.0]
        self.tab, self.hertz = torch.as_tensor(tab, device=self.dev), hertz

    def _pairs(self):
        """Sphere pairs within the largest radius sum and a margin: each cell of a grid against half of its neighbours."""
        b, p = self.balls, self.P[self.balls]
        reach = 2.0 * float(self.r.max())
        self.margin = 0.15 * float(self.r[b].min())
        h = reach + self.margin
        c = torch.floor((p - p.min(0).values) / h).long() + 1
        dim = c.max(0).values + 2
        key = (c[:, 0] * dim[1] + c[:, 1]) * dim[2] + c[:, 2]
        key, order = torch.sort(key, stable=True)
        got = []
        for q in range(14):                    # itself, then the 13 neighbours after it
            d = [(q // 9) % 3, (q // 3) % 3, q % 3] if q == 0 else [(13 + q) // 9 - 1, ((13 + q) // 3) % 3 - 1, (13 + q) % 3 - 1]
            other = key + (d[0] * dim[1] + d[1]) * dim[2] + d[2]
            lo = torch.searchsorted(key, other, right=False)
            hi = torch.searchsorted(key, other, right=True)
            if q == 0:
                lo = torch.arange(1, len(key) + 1, device=self.dev)
            cnt = (hi - lo).clamp(min=0)
            i = torch.repeat_interleave(torch.arange(len(key), device=self.dev), cnt)
            j = torch.arange(len(i), device=self.dev) - torch.repeat_interleave(torch.cumsum(cnt, 0) - cnt, cnt) + lo[i]
            i, j = b[order[i]], b[order[j]]
            near = (self.P[i] - self.P[j]).norm(dim=1) <= self.r[i] + self.r[j] + self.margin
            got.append(torch.stack([torch.minimum(i, j)[near], torch.maximum(i, j)[near]]))
        s, m = torch.cat(got, 1)
        self.s, self.m = [s], [m]              # then each wall's spheres: the sphere is the slave
        for w in self.walls:
            depth, _ = self._wall(w, b)
            k = b[depth > -self.margin]
            self.s.append(k)
            self.m.append(torch.full_like(k, w))
        self.start = self.P.clone()
        par = [self.tab[self.model[s], self.model[m]] for s, m in zip(self.s, self.m)]
        self.par = torch.cat(par)
        n = len(self.par)
        self.shear = torch.zeros((n, 3), dtype=torch.float64, device=self.dev)
        self.kn = torch.zeros(n, dtype=torch.float64, device=self.dev)
        self.held = torch.zeros(n, dtype=torch.bool, device=self.dev)

    def _wall(self, w, s):
        """Overlap of spheres s with wall w and the direction to its nearest point."""
        md = self.sc.models[int(self.sc.model_index[w])]
        P, c, z, x = self.P[s], self.P[w], self.Z[w], self.X[w]
        d = P - c
        if md.shape == PLATE:
            cap = P - ((d @ z) / z.norm() / z.norm())[:, None] * z - c
            y = torch.linalg.cross(z, x)
            u = (cap @ x).clamp(-0.5 * md.attrs[0], 0.5 * md.attrs[0])
            v = (cap @ y).clamp(-0.5 * md.attrs[2], 0.5 * md.attrs[2])
            to = u[:, None] * x + v[:, None] * y + c - P
            return self.r[s] + 0.5 * md.attrs[1] - _len(to), _dir(to)
        if md.shape == CYLINDER:
            a = (d @ z).clamp(-0.5 * md.attrs[1], 0.5 * md.attrs[1])
            to = c + a[:, None] * z - P
            return self.r[s] + md.attrs[0] - _len(to), _dir(to)
        a = d @ z                              # the inside of a hollow cylinder
        rad = d - a[:, None] * z
        rim = c + a.clamp(-0.5 * md.attrs[1], 0.5 * md.attrs[1])[:, None] * z + md.attrs[0] * _dir(rad) - P
        inside = (a.abs() <= 0.5 * md.attrs[1])
        depth = torch.where(inside, self.r[s] + _len(rad) - md.attrs[0], self.r[s] - _len(rim))
        return depth, torch.where(inside[:, None], _dir(rad), _dir(rim))

    def _contacts(self):
        to = self.P[self.m[0]] - self.P[self.s[0]]
        depth, n = [self.r[self.s[0]] + self.r[self.m[0]] - _len(to)], [_dir(to)]
        for w, s in zip(self.walls, self.s[1:]):
            dw, nw = self._wall(w, s)
            depth.append(dw)
            n.append(nw)
        return torch.cat(depth), torch.cat(n)

    def run(self, steps, fields, ext=None):
        dt, S, M = self.dt, torch.cat(self.s), torch.cat(self.m)
        for _ in range(steps):
            depth, n = self._contacts()
            on = depth > 0.0
            self.shear[~on], self.kn[~on], self.held[~on] = 0.0, 0.0, False
            k = torch.nonzero(on)[:, 0]
            s, m, d, nk, c = S[k], M[k], depth[k], n[k], self.par[k]
            point = self.P[s] + (self.r[s] - 0.5 * d)[:, None] * nk
            ra, rb = point - self.P[s], point - self.P[m]
            v = self.V[s] - self.V[m] + _cross(self.W[s], ra) - _cross(self.W[m], rb)
            vn = (v * nk).sum(1)[:, None] * nk
            vs = v - vn
            old = self.shear[k]
            turned = torch.where((old * vs).sum(1) <= 0.0, -_len(old), _len(old))[:, None] * _dir(vs)
            if self.hertz:
                beta = c[:, 4]
                coef = torch.where(beta < 0.99, 0.957832746294131 / (1.0 - beta * beta), torch.full_like(beta, 479.155951122633))
                vl = _len(vn)
                first = torch.where(vl == 0.0, c[:, 0], coef * c[:, 1] ** 0.2 * c[:, 0] ** 0.8 * vl ** 0.4)
                kn = torch.where(self.held[k], self.kn[k], first)
                fn = -(kn * d)[:, None] * nk - (2.0 * torch.sqrt(c[:, 1] * kn) * beta)[:, None] * vn
                ks = c[:, 2] * (c[:, 3] * (kn * d).abs()) ** (1.0 / 3.0)
                fs = turned - (ks * dt)[:, None] * vs
                top = c[:, 5] * kn * d
                fs = torch.where((_len(fs) >= top)[:, None], top[:, None] * _dir(fs), fs)
                self.kn[k] = kn
            else:
                fn = -(c[:, 0] * d)[:, None] * nk - c[:, 2:3] * vn
                fs = turned - (c[:, 1] * dt)[:, None] * vs
                top = c[:, 4] * c[:, 0] * d
                fs = torch.where((_len(fs) > top)[:, None], top[:, None] * _dir(fs), fs - c[:, 3:4] * vs)
            self.shear[k], self.held[k] = fs, True
            f = fn + fs
            J, A = torch.zeros_like(self.P), torch.zeros_like(self.P)
            J.index_add_(0, s, f * dt)
            J.index_add_(0, m, -f * dt)
            A.index_add_(0, s, dt * _cross(ra, f))
            A.index_add_(0, m, -dt * _cross(rb, f))
            J += self.sudo[:, None] * (self.g * dt)
            if ext is not None:
                J += torch.as_tensor(ext[0], device=self.dev)
                A += torch.as_tensor(ext[1], device=self.dev)
            self._respond(J, A)
        if float((self.P - self.start)[self.balls].norm(dim=1).max()) > 0.5 * self.margin:
            return None                        # the candidate pairs may be incomplete
        all_ = dict(position=self.P, velocity=self.V, angular_velocity=self.W, orientation_x=self.X, orientation_z=self.Z,
                    impact=J, angular_impact=A)
        return {f: all_[f].cpu().numpy() for f in fields}

    def _respond(self, J, A):
        dt, mv = self.dt, self.moves[:, None]
        sudo = torch.where(self.sudo > 0.0, self.sudo, torch.ones_like(self.sudo))
        r = torch.where(self.r > 0.0, self.r, torch.ones_like(self.r))
        dv = torch.where(mv, J / sudo[:, None], torch.zeros_like(J))
        dw = torch.where(mv, 2.5 * A / (sudo * r * r)[:, None], torch.zeros_like(A))
        turns = mv.clone()
        for w in self.walls:
            turns[w] = self.sc.models[int(self.sc.model_index[w])].behavior == ORBITAL
        self.P = torch.where(turns, self.P + dt * (self.V + 0.5 * dv), self.P)
        ang = dt * (self.W + 0.5 * dw)
        a = _len(ang)[:, None]
        u, cos = _dir(ang) * torch.sin(0.5 * a), torch.cos(0.5 * a)
        for name in ("X", "Z"):
            p = getattr(self, name)
            q = cos * cos * p + (p * u).sum(1)[:, None] * u + 2.0 * cos * _cross(u, p) + _cross(u, _cross(u, p))
            setattr(self, name, torch.where(turns, q, p))
        self.V, self.W = self.V + dv, self.W + dw

    def monitor(self, box):
        mv = self.moves.double()
        V, W, m = self.V, self.W, self.mass * mv
        vl, wl = _len(V)[self.moves], _len(W)[self.moves]
        I = (self.inertia * mv)[:, None].expand(-1, 3)
        mom, ang = m[:, None] * V, _cross(I, W)
        cnt = mv.sum()
        depth, _ = self._contacts()
        o = [-(m * (self.P @ self.g)).sum(), (0.5 * m * _len(V) ** 2).sum(), (0.5 * (I * W * W).sum(1)).sum(),
             vl.min(), vl.max(), wl.min(), wl.max(), (_len(mom - mom.sum(0) / cnt) * mv).sum(),
             (_len(ang - ang.sum(0) / cnt) * mv).sum(), (depth > 0.0).sum()]
        o += [(m * self.P[:, k]).sum() / m.sum() for k in range(3)]
        s, t = self.s[0], self.m[0]
        d, rs = _len(self.P[s] - self.P[t]), self.r[s] + self.r[t]
        count = []
        for hit in (d < rs, d <= rs):
            c = torch.zeros(len(self.P), dtype=torch.int32, device=self.dev)
            one = torch.ones(int(hit.sum()), dtype=torch.int32, device=self.dev)
            c.index_add_(0, s[hit], one)
            c.index_add_(0, t[hit], one)
            count.append(c)
        ball = torch.zeros(len(self.P), dtype=torch.bool, device=self.dev)
        ball[self.balls] = True
        for k in range(3):
            ball &= (self.P[:, k] < box[2 * k + 1] + self.r) & (self.P[:, k] > box[2 * k] - self.r)
        return {"observables": np.array([float(x) for x in o]), "below": count[0].cpu().numpy(),
                "touching": count[1].cpu().numpy(), "average": float(count[1][ball].double().mean())}


def _len(v):
    return torch.sqrt(v[:, 0] * v[:, 0] + v[:, 1] * v[:, 1] + v[:, 2] * v[:, 2])


def _dir(v):
    n = _len(v)[:, None]
    return torch.where(n > 0.0, v / torch.where(n > 0.0, n, torch.ones_like(n)), torch.zeros_like(v))


def _cross(a, b):
    return torch.linalg.cross(a, b)
