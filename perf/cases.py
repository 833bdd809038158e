"""The work that a user of the engine has it do, as measurable cases.

Three kinds of pass, each through the package's public entry points:

* ``step``: simulations resident in a context advance by a number of steps and their
  state is read back (a control loop, an interactive viewer, one generation's chunk).
  ``settle`` steps are taken before the first pass, so the pass meets the regime that
  most of a 10^4..10^5 step run is spent in; without them it meets a fresh creature's.
* ``load``: VXA texts in, parsed and built, run for a number of steps, results and
  poses out, simulations freed: what an evolution loop does with each generation.
* ``serve``: requests of uneven sizes and horizons submitted to the serving queue and
  polled until all are done.

Creatures are random fills of a lattice (largest connected part) with random actuation
phases, as in the repository's benchmark and tests: 0.01 m voxels, four materials with E
log-uniform in [1e5, 1e7] Pa (one or two actuated), floor, gravity and friction; the
self-colliding ones use three materials, one of them soft (E = 1e5), and contract only.
"""
import json
import math
import time
import zlib

import numpy as np
import torch

import gpuvoxels_gb300 as g
from gpuvoxels_gb300 import synth

CHUNK = 64        # steps between two polls of the serving queue


def _step(name, n, side, fill, steps, settle=0, collide=False, fma=False):
    return {"name": name, "kind": "step", "n": n, "side_lo": side[0], "side_hi": side[1], "fill_lo": fill[0], "fill_hi": fill[1],
            "flat": False, "steps": steps, "settle": settle, "collide": collide, "fma": fma}


def listed():
    return [
        # a controller that takes one step of one small creature at a time and reads its state
        _step("control_step_6", 1, (6, 6), (0.9, 0.9), 1),
        # the plain single creature (10^3 lattice, fill 0.6), one chunk of its run
        _step("creature_10", 1, (10, 10), (0.6, 0.6), 64),
        # one large creature, odd side, settled
        _step("creature_33_settled", 1, (33, 33), (0.6, 0.6), 32, settle=192),
        # a few dozen uneven creatures: a small population
        _step("population_32", 32, (6, 20), (0.3, 0.9), 20),
        # the same through the contracted-multiply-add build that callers may choose
        _step("population_32_fma", 32, (6, 20), (0.3, 0.9), 20, fma=True),
        # the batched configuration at a quarter of its size, in the settled regime
        _step("population_128_settled", 128, (6, 20), (0.3, 0.9), 20, settle=256),
        # the batched configuration: 512 uneven creatures
        _step("population_512", 512, (6, 20), (0.3, 0.9), 20),
        # a small soft creature folding onto itself (contacts and watch lists)
        _step("collide_12", 1, (12, 12), (0.5, 0.5), 64, settle=512, collide=True),
        # the collision configuration at an eighth of its size
        _step("collide_8x40", 8, (40, 40), (0.5, 0.5), 16, settle=64, collide=True),
        # one large solid body: a slab half as high as it is wide
        dict(_step("slab_120x120x60", 1, (120, 120), (1.0, 1.0), 10), flat=True),
        # a generation of 64 creatures from VXA text to fitness and poses
        {"name": "generation_64", "kind": "load", "n": 64, "side_lo": 6, "side_hi": 20, "fill_lo": 0.3, "fill_hi": 0.9, "steps": 20},
        # a serving stream of uneven requests, a fifth of them with self-collision
        {"name": "serve_12", "kind": "serve", "n": 12, "v_lo": 100, "v_hi": 10000, "h_lo": 100, "h_hi": 400},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "collide", "one", "slab", "load", "serve"])
    if kind == "load":
        n = _log(rng, 4, 64)
        lo = rng.randint(4, 12)
        return {"kind": "load", "n": n, "side_lo": lo, "side_hi": rng.randint(lo, 20), "fill_lo": 0.3, "fill_hi": 0.9, "steps": _log(rng, 10, 40)}
    if kind == "serve":
        return {"kind": "serve", "n": rng.randint(4, 12), "v_lo": 100, "v_hi": _log(rng, 1000, 10000), "h_lo": 100, "h_hi": rng.randint(150, 400)}
    c = _step("", 1, (6, 20), (0.3, 0.9), 20)
    del c["name"]
    c["fma"] = rng.random() < 0.1
    if kind == "step":
        c["n"] = _log(rng, 2, 256)
        c["side_lo"] = rng.randint(3, 12)
        c["side_hi"] = rng.randint(c["side_lo"], 20)
        c["steps"] = _log(rng, 1, 40)
        c["settle"] = rng.choice([0, 0, rng.randint(32, 256)])
    elif kind == "collide":
        c["collide"] = True
        c["side_lo"] = c["side_hi"] = _log(rng, 8, 40)
        c["n"] = max(1, min(8, int(4e5 / c["side_lo"] ** 3)))
        c["fill_lo"] = c["fill_hi"] = rng.uniform(0.4, 0.7)
        c["steps"] = _log(rng, 4, 48)
        c["settle"] = rng.choice([0, rng.randint(16, 256)])
    elif kind == "one":
        c["side_lo"] = c["side_hi"] = _log(rng, 2, 48)
        c["fill_lo"] = c["fill_hi"] = rng.uniform(0.5, 1.0)
        c["steps"] = _log(rng, 1, 96)
        c["settle"] = rng.choice([0, rng.randint(32, 256)])
    else:
        c["side_lo"] = c["side_hi"] = _log(rng, 20, 110)
        c["fill_lo"] = c["fill_hi"] = 1.0
        c["flat"] = True
        c["steps"] = rng.randint(2, 12)
    return c


# ---------------------------------------------------------------- inputs
class _Body:
    """One creature: lattice (0 empty, k = materials[k-1]), phases in cycles, materials, self-collision.
    The body plan comes from `plan`, what it is made of and how it moves from `rng`."""

    def __init__(self, plan, rng, side, fill, mats, collide):
        X, Y, Z = side
        cells = plan.random((Z, Y, X)) < fill
        if not cells.any():
            cells[0, 0, 0] = True
        if fill < 1.0:
            cells = synth.largest_component(cells)
        self.grid = np.where(cells, rng.integers(1, len(mats) + 1, size=cells.shape), 0).astype(np.int32)
        self.phase = rng.random(cells.shape)
        self.mats, self.collide = mats, collide

    def vxa(self, **kw):
        return synth.vxa_document(self.grid, self.phase, self.mats, collision=self.collide, expansion=not self.collide, **kw)

    @property
    def num_voxel(self):
        return int((self.grid > 0).sum())


def _soft_materials():
    return [dict(E=e, rho=1000.0, nu=0.35, cte=c, mus=1.0, muk=0.5) for e, c in ((1e5, 0.01), (1e6, 0.01), (1e6, 0.0))]


def _bodies(case, seed):
    """The case's creatures and horizons: body plans (and so all sizes) are the case's, materials and phases the seed's."""
    plan = np.random.default_rng(zlib.crc32(json.dumps(case, sort_keys=True).encode()))
    rng = np.random.default_rng([int(seed), 77])
    out = []
    for _ in range(case["n"]):
        if case["kind"] == "serve":
            v = math.exp(plan.uniform(math.log(case["v_lo"]), math.log(case["v_hi"])))
            fill, collide, flat = float(plan.uniform(0.5, 0.9)), bool(plan.random() < 0.2), False
            s = max(2, int(round((v / fill) ** (1.0 / 3.0))))
        else:
            s = int(plan.integers(case["side_lo"], case["side_hi"] + 1))
            fill = float(plan.uniform(case["fill_lo"], case["fill_hi"]))
            collide, flat = bool(case.get("collide")), bool(case.get("flat"))
        if flat:
            mats = [dict(E=1e6, rho=1000.0, nu=0.35, cte=0.01, mus=1.0, muk=0.5)]
        else:
            mats = _soft_materials() if collide and case["kind"] == "step" else synth.config1_materials(rng)
        out.append(_Body(plan, rng, (s, s, max(1, s // 2) if flat else s), fill, mats, collide))
    horizons = [int(h) for h in plan.integers(case["h_lo"], case["h_hi"] + 1, size=case["n"])] if case["kind"] == "serve" else []
    return out, horizons


def _budget(bodies):
    return (384 << 20) + 4096 * sum(b.num_voxel for b in bodies)


def prepare(case, seed):
    bodies, horizons = _bodies(case, seed)
    ctx = g.Context(0, _budget(bodies))
    if case.get("fma"):
        ctx.set_precision(g.FMA)
    docs = [b.vxa().encode() for b in bodies]
    s = {"case": case, "ctx": ctx}
    if case["kind"] == "step":
        s["ids"] = ctx.load_many(docs)
        if case["settle"]:
            ctx.step(s["ids"], case["settle"])
    elif case["kind"] == "load":
        s["docs"] = docs
    else:
        s["docs"], s["horizons"] = docs, horizons
        ctx.set_serving(g.SERVE_LEAST_WORK, 150000)
    return s


def _results(rs):
    return {"steps": np.array([r.steps for r in rs], np.int64), "status": np.array([r.status for r in rs], np.int64),
            "time": np.array([r.current_time for r in rs]), "fitness": np.array([r.fitness_score for r in rs]),
            "com": np.array([list(r.current_center_of_mass) for r in rs])}


def run(s):
    case, ctx = s["case"], s["ctx"]
    if case["kind"] == "step":
        ctx.step(s["ids"], case["steps"])
        pos, q, fl, _ = ctx.get_states(s["ids"])
        return {"pos": pos, "orient": q, "flags": fl}
    if case["kind"] == "load":
        ids = ctx.load_many(s["docs"])
        ctx.run(ids, g.BATCHED, case["steps"])
        out = _results([ctx.result(i) for i in ids])
        pos, q, fl, _ = ctx.get_states(ids)
        for i in ids:
            ctx.free(i)
        return {"pos": pos, "orient": q, "flags": fl, **out}
    ids = ctx.load_many(s["docs"])
    for i, h in zip(ids, s["horizons"]):
        ctx.submit(i, h)
    done, t0 = {}, time.monotonic()
    while ctx.pending() > 0 and time.monotonic() - t0 < 60:
        for r in ctx.poll(CHUNK):
            done[r.id] = r
    out = _results([done[i] for i in ids])
    pos, q, fl, _ = ctx.get_states(ids)
    for i in ids:
        ctx.free(i)
    return {"pos": pos, "orient": q, "flags": fl, **out}


def work(case):
    """Per step: a voxel's state (13 doubles) read and written, each link's nine doubles read and
    written and its two end forces and moments (12 doubles) formed; about 230 floating-point
    operations a voxel and 350 a link in 64 bits."""
    if case["kind"] == "serve":
        v = case["n"] * (case["v_hi"] - case["v_lo"]) / math.log(case["v_hi"] / case["v_lo"])
        fill, steps = 0.7, 0.5 * (case["h_lo"] + case["h_hi"])
    else:
        lo, hi = case["side_lo"], case["side_hi"]
        sides = [float(s) ** 3 * (0.5 if case.get("flat") else 1.0) for s in range(lo, hi + 1)]
        fill = 0.5 * (case["fill_lo"] + case["fill_hi"])
        v, steps = case["n"] * fill * sum(sides) / len(sides), case["steps"]
    links = 3.0 * fill * v
    return {"bytes": steps * (208.0 * v + 240.0 * links), "flops": steps * (230.0 * v + 350.0 * links)}


# ---------------------------------------------------------------- the same in 64 bits
# The soft-body step of the reference's CPU path in plain torch: 64-bit state, and 32 bits
# where that path holds 32 bits (materials, temperatures, strains, stresses, contact forces).
F64, F32 = torch.float64, torch.float32


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _f(x):
    return np.float32(x)


def _voxel_material(m, nom):
    """The 32-bit constants of a palette material."""
    E, nu, rho = _f(m["E"]), _f(m["nu"]), _f(m["rho"])
    one, two = _f(1), _f(2)
    d = dict(E=E, nu=nu, cte=_f(m["cte"]), mus=_f(m["mus"]), muk=_f(m["muk"]), eHat=E / ((one - two * nu) * (one + nu)))
    d["mass"] = _f(nom * nom * nom * float(rho))
    inertia = _f(float(d["mass"]) * nom * nom / 6.0)
    d["massInv"], d["sqrtMass"], d["Iinv"] = one / d["mass"], np.sqrt(d["mass"]), one / inertia
    c2m = _f(2.0 * math.sqrt(float(d["mass"] * E) * nom))
    c2i = _f(2.0 * math.sqrt(float(inertia * E) * nom * nom * nom))
    zi, zc, zg = _f(1.0), _f(0.8), _f(0.01)
    d["dampNum"] = two * d["sqrtMass"] * zi
    d["gDampT"], d["gDampR"], d["cDampT"] = zg * c2m, zg * c2i, zc * c2m
    d["grav"] = -d["mass"] * _f(9.80665) * _f(_f(9.81) / 9.80665)
    d["pen"] = _f(2 * float(E) * nom)
    return d


def _link_material(a, b, nom):
    one, two = _f(1), _f(2)
    E = two * a["E"] * b["E"] / (a["E"] + b["E"])
    hat = two * a["eHat"] * b["eHat"] / (a["eHat"] + b["eHat"])
    c2 = _f(float((hat - E) / (two * hat)) + 0.0625)
    nu = _f(float(np.sqrt(c2)) - 0.25)
    L = _f(nom)
    d = dict(nu=nu, eHat=E / ((one - two * nu) * (one + nu)), a2=E * L * L * L / (_f(12) * (one + nu)), b1=E * L, b2=E * L * L / two,
             b3=E * L * L * L / _f(6))
    d["sqA1"], d["sqA2"], d["sqB1"] = np.sqrt(E * L), np.sqrt(d["a2"] * L * L / _f(6)), np.sqrt(d["b1"])
    d["sqB2"], d["sqB3"] = np.sqrt(d["b2"] * L / two), np.sqrt(d["b3"] * L * L / _f(6))
    return d


def _qmul(a, f):
    (aw, ax, ay, az), (fw, fx, fy, fz) = a, f
    return (aw * fw - ax * fx - ay * fy - az * fz, aw * fx + ax * fw + ay * fz - az * fy, aw * fy - ax * fz + ay * fw + az * fx,
            aw * fz + ax * fy - ay * fx + az * fw)


def _qrot(q, f):
    (w, x, y, z), (fx, fy, fz) = q, f
    tw, tx, ty, tz = fx * x + fy * y + fz * z, fx * w - fy * z + fz * y, fx * z + fy * w - fz * x, -fx * y + fy * x + fz * w
    return (w * tx + x * tw + y * tz - z * ty, w * ty - x * tz + y * tw + z * tx, w * tz + x * ty - y * tx + z * tw)


def _qrotinv(q, f):
    (w, x, y, z), (fx, fy, fz) = q, f
    tw, tx, ty, tz = x * fx + y * fy + z * fz, w * fx - y * fz + z * fy, w * fy + x * fz - z * fx, w * fz - x * fy + y * fx
    return (tw * x + tx * w + ty * z - tz * y, tw * y - tx * z + ty * w + tz * x, tw * z + tx * y - ty * x + tz * w)


def _rotvec(q):
    w, x, y, z = q
    unit = (w >= 1) | (w <= -1)
    ws = torch.where(unit, torch.zeros_like(w), w)
    sl = 1 - ws * ws
    s = torch.where(sl < 2.4e-3, torch.sqrt((2 - 2 * ws) / sl), torch.acos(ws) * (1 / torch.sqrt(sl)))
    s = torch.where(unit, torch.zeros_like(s), s)
    return (2 * x * s, 2 * y * s, 2 * z * s)


def _from_rotvec(v):
    x, y, z = (0.5 * c for c in v)
    m2 = x * x + y * y + z * z
    small = m2 * m2 < 5.328e-15
    m = torch.sqrt(torch.where(small, torch.ones_like(m2), m2))
    w = torch.where(small, 1 - 0.5 * m2, torch.cos(m))
    s = torch.where(small, 1 - m2 / 6, torch.sin(m) / m)
    return (w, x * s, y * s, z * s)


def _angle_to_x(r):
    """The rotation of r onto +x (identity for a zero vector)."""
    x, y, z = r
    yox, zox = y / x, z / x
    turn = (yox.abs() < 1.732e-2) & (zox.abs() < 1.732e-2)
    ty, tz = 0.5 * zox, -0.5 * yox
    li = 1 / torch.sqrt(x * x + y * y + z * z)
    nx, ny, nz = x * li, y * li, z * li
    theta = torch.acos(nx.clamp(-1, 1))
    ami = 1 / torch.sqrt(nz * nz + ny * ny)
    s, c = torch.sin(0.5 * theta), torch.cos(0.5 * theta)
    back = theta > 3.14159265358979 - 1e-7
    one, nil = torch.ones_like(x), torch.zeros_like(x)
    pick = lambda a, b, d, e: torch.where((x == 0) & (y == 0) & (z == 0), e, torch.where(turn, a, torch.where(back, b, d)))  # noqa: E731
    return (pick(1 + 0.5 * (-ty * ty - tz * tz), nil, c, one), nil, pick(ty, one, nz * ami * s, nil), pick(tz, nil, -ny * ami * s, nil))


def _to_x(axis, v):
    x, y, z = v
    a1, a2 = axis == 1, axis == 2
    return (torch.where(a1, y, torch.where(a2, z, x)), torch.where(a1, -x, y), torch.where(a2, -x, z))


def _from_x(axis, v):
    x, y, z = v
    a1, a2 = axis == 1, axis == 2
    return (torch.where(a1, -y, torch.where(a2, -z, x)), torch.where(a1, x, y), torch.where(a2, x, z))


class _World:
    """Several bodies side by side: they do not touch one another, and each has its own time step."""

    def __init__(self, bodies):
        dev, nom = _device(), 0.01
        self.dev, self.nom, self.collide = dev, nom, bodies[0].collide
        ijk, vmat, phase, body, neg, pos, ax, lmat, vms, lms = [], [], [], [], [], [], [], [], [], []
        for b, B in enumerate(bodies):
            at = len(vms)
            vms += [_voxel_material(m, nom) for m in B.mats]
            k = len(B.mats)
            lat = len(lms)
            lms += [_link_material(vms[at + i], vms[at + j], nom) for i in range(k) for j in range(k)]
            base = sum(len(p) for p in phase)
            cells = np.argwhere(B.grid > 0)
            num = -np.ones(B.grid.shape, np.int64)
            num[tuple(cells.T)] = base + np.arange(len(cells))
            ijk.append(cells[:, ::-1])
            vm = B.grid[tuple(cells.T)] - 1
            vmat.append(at + vm)
            phase.append(B.phase[tuple(cells.T)])
            body.append(np.full(len(cells), b))
            for a in range(3):
                lo, hi = np.moveaxis(num, 2 - a, 0)[:-1], np.moveaxis(num, 2 - a, 0)[1:]
                both = (lo >= 0) & (hi >= 0)
                neg.append(lo[both])
                pos.append(hi[both])
                ax.append(np.full(int(both.sum()), a))
                lmat.append(lat + vm[lo[both] - base] * k + vm[hi[both] - base])
        cat = lambda v: torch.from_numpy(np.ascontiguousarray(np.concatenate(v))).to(dev)  # noqa: E731
        self.ijk, self.phase, self.body = cat(ijk), cat(phase), cat(body)
        self.neg, self.pos, self.axis = cat(neg), cat(pos), cat(ax)
        vmat, lmat = cat(vmat), cat(lmat)
        table = lambda ms, k: torch.from_numpy(np.array([m[k] for m in ms], np.float32)).to(dev)  # noqa: E731
        self.V = {k: table(vms, k)[vmat] for k in vms[0]}
        self.L = {k: table(lms, k)[lmat] for k in lms[0]}
        n, nl = len(self.ijk), len(self.neg)
        self.n = n
        self.slot = torch.full((6, n), nl, dtype=torch.int64, device=dev)   # link in each direction; nl: none
        ids = torch.arange(nl, device=dev)
        self.slot[2 * self.axis, self.neg] = ids
        self.slot[2 * self.axis + 1, self.pos] = ids
        self.has = self.slot < nl
        self.surface = ~self.has.all(0)
        zero = lambda k: tuple(torch.zeros(k, dtype=F64, device=dev) for _ in range(3))  # noqa: E731
        self.p = tuple(self.ijk[:, k].to(F64) * nom for k in range(3))
        self.q = (torch.ones(n, dtype=F64, device=dev),) + zero(n)
        self.lm, self.am = zero(n), zero(n)
        self.ps = torch.zeros((3, n), dtype=F32, device=dev)
        self.static = torch.ones(n, dtype=torch.bool, device=dev)
        self.floor = torch.zeros(n, dtype=torch.bool, device=dev)
        self.old = (zero(nl), zero(nl), zero(nl))
        self.small = torch.ones(nl, dtype=torch.bool, device=dev)
        self.valid = torch.zeros(nl, dtype=torch.bool, device=dev)
        self.t = torch.zeros(len(bodies), dtype=F64, device=dev)
        self.steps = 0
        self._temperature()
        self._time_step(len(bodies))
        self.pairs = self.seen = None
        if self.collide:
            self._near()

    def _temperature(self):
        T = 39.0 * torch.sin(float(_f(2 * 3.1415926)) * (self.t[self.body] / 0.2 + self.phase))
        if self.collide:
            T = torch.where(T > 0, torch.zeros_like(T), T)
        self.temp = T.to(F32)
        self.size = self.nom * (1 + self.temp * self.V["cte"]).to(F64)
        self.rest = 0.5 * (self.size[self.neg] + self.size[self.pos])

    def _time_step(self, nb):
        s2 = _f(self.nom) * _f(self.nom)
        k = (self.L["eHat"] * float(s2)).to(F64) / self.rest
        f2 = k.to(F32) / torch.minimum(self.V["mass"][self.neg], self.V["mass"][self.pos])
        best = torch.zeros(nb, dtype=F32, device=self.dev)
        best.scatter_reduce_(0, self.body[self.neg], f2, "amax")
        alone = (self.V["E"].to(F64) * self.nom / self.V["mass"].to(F64)).to(F32)
        own = torch.zeros(nb, dtype=F32, device=self.dev).scatter_reduce_(0, self.body, alone, "amax")
        best = torch.where(best > 0, best, own)
        opt = 1.0 / (float(_f(6.283185)) * torch.sqrt(best.cpu()).numpy().astype(np.float32)).astype(np.float32)
        self.dt = torch.from_numpy((0.95 * opt.astype(np.float32).astype(np.float64)).astype(np.float32)).to(self.dev)

    def _near(self):
        """Pairs of voxels at most five links apart, as sorted keys a * n + b."""
        n = self.n
        a, b = torch.cat([self.neg, self.pos]), torch.cat([self.pos, self.neg])
        order = torch.argsort(a)
        nb_of = torch.full((n, 6), -1, dtype=torch.int64, device=self.dev)
        nb_of[self.neg, 2 * self.axis] = self.pos
        nb_of[self.pos, 2 * self.axis + 1] = self.neg
        del order, a, b
        near = torch.arange(n, device=self.dev) * (n + 1)
        front = near
        for _ in range(5):
            i, j = front // n, front % n
            k = nb_of[j]
            front = (i[:, None] * n + k)[k >= 0].unique()
            near = torch.cat([near, front]).unique()
        self.near = near

    def _contacts(self, F):
        """The contact forces of the overlapping surface pairs, taken off F."""
        n, nom = self.n, self.nom
        P = torch.stack(self.p, 1)
        s = torch.nonzero(self.surface).flatten()
        if self.seen is None or bool((((P[s] - self.seen) ** 2).sum(1) > (0.5 * nom) ** 2).any()):
            self.seen = P[s].to(F32).to(F64)
            found = []
            r2 = float(_f(2.5 * nom) ** 2)
            for b in range(len(self.t)):
                sb = s[self.body[s] == b]
                Pb = P[sb]
                for c in range(0, len(sb), 4096):
                    d = sum((Pb[c:c + 4096, k, None] - Pb[None, :, k]) ** 2 for k in range(3))
                    i, j = torch.nonzero(d <= r2, as_tuple=True)
                    i = i + c
                    found.append((sb[i] * n + sb[j])[i < j])
            pairs = torch.cat(found)
            at = torch.searchsorted(self.near, pairs).clamp(max=len(self.near) - 1)
            self.pairs = pairs[self.near[at] != pairs].sort().values
        a, b = self.pairs // n, self.pairs % n
        V = self.V
        off = [(self.p[k][b] - self.p[k][a]).to(F32) for k in range(3)]
        avg = (self.size + self.size + self.size) / 3.0
        reach = ((avg[a] + avg[b]) * 0.625).to(F32)
        ln = torch.sqrt(off[0] * off[0] + off[1] * off[1] + off[2] * off[2])
        rel = reach - ln
        hit = rel > 0
        a, b, rel, ln, off = a[hit], b[hit], rel[hit], ln[hit], [o[hit] for o in off]
        inv = torch.where(ln > 0, 1 / ln, torch.ones_like(ln))
        u = [inv * o for o in off]
        speed = lambda v: sum(self.lm[k][v] * V["massInv"][v].to(F64) * u[k].to(F64) for k in range(3))  # noqa: E731
        rv = (speed(a) - speed(b)).to(F32)
        k = 2.0 / (1.0 / V["pen"][a] + 1.0 / V["pen"][b])
        f = k * rel + 0.5 * (V["cDampT"][a] + V["cDampT"][b]) * rv
        return tuple(F[i].index_add(0, a, -(f * u[i]).to(F64)).index_add(0, b, (f * u[i]).to(F64)) for i in range(3))

    def step(self):
        V, L, neg, pos, axis = self.V, self.L, self.neg, self.pos, self.axis
        D = lambda x: x.to(F64)  # noqa: E731
        if self.steps:
            self._temperature()
        # links
        d = _to_x(axis, tuple(c[pos] - c[neg] for c in self.p))
        q1, q2 = ((c[0],) + _to_x(axis, c[1:]) for c in (tuple(c[neg] for c in self.q), tuple(c[pos] for c in self.q)))
        conj = (q1[0], -q1[1], -q1[2], -q1[3])
        p2, a2 = _qrot(conj, d), _qmul(conj, q2)
        turn, ext = ((p2[2].abs() + p2[1].abs()) / p2[0]).to(F32), (1 - p2[0] / self.rest).abs().to(F32)
        hb, he = float(_f(1.2) * _f(0.05)), float(_f(1.2) * _f(0.5))
        into = ~self.small & (turn < float(_f(0.05))) & (ext < 0.5)
        leave = self.small & ((turn > hb) | (ext > he))
        small, valid = (self.small | into) & ~leave, self.valid & ~into & ~leave
        q_on = _angle_to_x(p2)
        one, nil = torch.ones_like(p2[0]), torch.zeros_like(p2[0])
        ident = (one, nil, nil, nil)
        a1 = tuple(torch.where(small, i, c) for i, c in zip(ident, q_on))
        a2 = tuple(torch.where(small, i, c) for i, c in zip(a2, _qmul(q_on, a2)))
        ln = torch.sqrt(p2[0] * p2[0] + p2[1] * p2[1] + p2[2] * p2[2])
        p2 = (torch.where(small, p2[0], ln) - self.rest, torch.where(small, p2[1], nil), torch.where(small, p2[2], nil))
        r1, r2 = _rotvec(a1), _rotvec(a2)
        dP, d1, d2 = (tuple(0.5 * (x - y) for x, y in zip(new, old)) for new, old in zip((p2, r1, r2), self.old))
        self.old, self.small = (p2, r1, r2), small
        ta, tb = (axis == 0).long(), 2 - (axis == 2).long()
        s2 = float(_f(self.nom) * _f(self.nom))

        def across(v):
            pa, pb = self.ps[ta, v], self.ps[tb, v]
            return (s2 * (1 + D(pa)) * (1 + D(pb))).to(F32), pa + pb

        (aN, sN), (aP, sP) = across(neg), across(pos)
        area, tss = 0.5 * (aN + aP), 0.5 * (sN + sP)
        strain = (p2[0] / self.rest).to(F32)
        stress = L["eHat"] * ((1 - L["nu"]) * strain + L["nu"] * tss)
        b1, b2, b3, k2 = D(L["b1"]), D(L["b2"]), D(L["b3"]), D(L["a2"])
        fN = (D(stress * area), b1 * p2[1] - b2 * (r1[2] + r2[2]), b1 * p2[2] + b2 * (r1[1] + r2[1]))
        fP = tuple(-c for c in fN)
        mN = (k2 * (r2[0] - r1[0]), -b2 * p2[2] - b3 * (2 * r1[1] + r2[1]), b2 * p2[1] - b3 * (2 * r1[2] + r2[2]))
        mP = (k2 * (r1[0] - r2[0]), -b2 * p2[2] - b3 * (r1[1] + 2 * r2[1]), b2 * p2[1] - b3 * (r1[2] + 2 * r2[2]))
        c1, c2, c3, c4, c5 = (D(L[k]) for k in ("sqA1", "sqA2", "sqB1", "sqB2", "sqB3"))
        damp = V["dampNum"] / self.dt[self.body]
        gN, gP = (torch.where(valid, D(damp[v]), nil) for v in (neg, pos))
        pc = (c1 * dP[0], c3 * dP[1] - c4 * (d1[2] + d2[2]), c3 * dP[2] + c4 * (d1[1] + d2[1]))
        tN = (-c2 * (d2[0] - d1[0]), c4 * dP[2] + c5 * (2 * d1[1] + d2[1]), -c4 * dP[1] + c5 * (2 * d1[2] + d2[2]))
        tP = (c2 * (d2[0] - d1[0]), c4 * dP[2] + c5 * (d1[1] + 2 * d2[1]), -c4 * dP[1] + c5 * (d1[2] + 2 * d2[2]))
        fN, fP = tuple(f + gN * c for f, c in zip(fN, pc)), tuple(f - gP * c for f, c in zip(fP, pc))
        mN, mP = tuple(m - 0.5 * gN * c for m, c in zip(mN, tN)), tuple(m - 0.5 * gP * c for m, c in zip(mP, tP))
        self.valid = torch.ones_like(valid)
        fN, mN = (tuple(torch.where(small, x, y) for x, y in zip(f, _qrotinv(a1, f))) for f in (fN, mN))
        fN, mN, fP, mP = (_from_x(axis, f) for f in (fN, mN, _qrotinv(a2, fP), _qrotinv(a2, mP)))
        ratio = V["E"][pos] / V["E"][neg]
        eN, eP = 2.0 * strain / (1.0 + ratio), 2.0 * strain * ratio / (1.0 + ratio)

        # voxels: the six directions' links in order
        def gather(onN, onP):
            total = torch.zeros(self.n, dtype=onN.dtype, device=self.dev)
            z = torch.zeros(1, dtype=onN.dtype, device=self.dev)
            onN, onP = torch.cat([onN, z]), torch.cat([onP, z])
            for k in range(6):
                total = total + (onP if k & 1 else onN)[self.slot[k]]
            return total

        F = _qrot(self.q, tuple(gather(a, b) for a, b in zip(fN, fP)))
        M = _qrot(self.q, tuple(gather(a, b) for a, b in zip(mN, mP)))
        vel, gd = tuple(D(V["massInv"]) * c for c in self.lm), D(V["gDampT"])
        F = tuple(f - gd * v for f, v in zip(F, vel))
        F = (F[0], F[1], F[2] + D(V["grav"]))
        if self.collide:
            F = self._contacts(F)
        # floor and friction
        avg = (self.size + self.size + self.size) / 3.0
        pen = (0.5 * avg - 0.5 * self.nom - self.p[2]).to(F32)
        on = pen >= 0
        normal = V["pen"] * pen
        fz = torch.where(on, F[2] + (D(normal) - D(V["cDampT"]) * vel[2]), F[2])
        side = (F[0] * F[0] + F[1] * F[1]).to(F32)
        slip = side > (V["mus"] * normal) * (V["mus"] * normal)
        hl = torch.sqrt(vel[0] * vel[0] + vel[1] * vel[1])
        inv = torch.where(hl > 0, 1 / hl, torch.ones_like(hl))
        kin = D(V["muk"] * normal)
        slide = on & ~self.static
        fx, fy = (torch.where(slide, F[k] - kin * (inv * vel[k]), F[k]) for k in (0, 1))
        static = self.static & on & ~slip
        dt = self.dt[self.body]
        lm = tuple(c + D(dt) * f for c, f in zip(self.lm, (fx, fy, fz)))
        sdt = D(dt * V["massInv"])
        tr = tuple(sdt * c for c in lm)
        work_ = (fx - F[0]) * tr[0] + (fy - F[1]) * tr[1]
        energy = 0.5 * D(V["massInv"]) * (lm[0] * lm[0] + lm[1] * lm[1])
        static = on & (static | (energy + work_ <= 0))
        zero = torch.zeros_like(tr[0])
        hold = lambda c: torch.where(static, zero, c)  # noqa: E731
        self.lm = (hold(lm[0]), hold(lm[1]), lm[2])
        self.p = (self.p[0] + hold(tr[0]), self.p[1] + hold(tr[1]), self.p[2] + tr[2])
        self.static = static
        w = tuple(D(V["Iinv"]) * c for c in self.am)
        M = tuple(m - D(V["gDampR"]) * c for m, c in zip(M, w))
        self.am = tuple(c + D(dt) * m for c, m in zip(self.am, M))
        sI = D(dt * V["Iinv"])
        self.q = _qmul(_from_rotvec(tuple(sI * c for c in self.am)), self.q)
        # the next step's Poisson strain
        z = torch.zeros(1, dtype=F32, device=self.dev)
        eN, eP = torch.cat([eN, z]), torch.cat([eP, z])
        ten, s = [], []
        for k in range(3):
            both = self.has[2 * k] & self.has[2 * k + 1]
            v = eN[self.slot[2 * k]] + eP[self.slot[2 * k + 1]]
            s.append(torch.where(both, v * 0.5, v))
            ten.append(both)
        add = sum(torch.where(t, c, torch.zeros_like(c)) for t, c in zip(ten, s))
        free = (D(1 + add) ** -D(V["nu"])).to(F32) - 1
        self.ps = torch.stack([torch.where(t, c, free) for t, c in zip(ten, s)])
        self.t = self.t + D(self.dt)
        self.steps += 1

    def out(self):
        flags = self.static.to(torch.uint8) | ((~self.surface).to(torch.uint8) << 1)
        return {"pos": torch.stack(self.p, 1).cpu().numpy(), "orient": torch.stack(self.q, 1).cpu().numpy(), "flags": flags.cpu().numpy()}


def exact(case, seed):
    bodies, _ = _bodies(case, seed)
    if case["kind"] == "serve":
        return None          # every request has a horizon of its own, to hundreds of steps: too long
    w = _World(bodies)
    n = case["steps"] + case.get("settle", 0)
    for _ in range(n):
        w.step()
    out = w.out()
    out["flags"] = None       # flags also say what the engine alone keeps
    if case["kind"] == "load":
        mass = w.V["mass"].to(F64)
        com = [[float((c[w.body == b] * mass[w.body == b]).sum() / mass[w.body == b].sum()) for c in w.p] for b in range(len(bodies))]
        out.update(time=w.t.cpu().numpy(), com=np.array(com), steps=None, status=None, fitness=None)
    return out
