"""The work that programs have this framework do, as cases that can be timed and compared.

Every case goes through the public entry points: ``Scene.run``/``one``/``sync``, ``S.dem.con``,
``Batch.run``, the serving ``SlotPool``, ``wg_run_host`` and ``pack_rsa``. Scenes follow the
repository's own configurations (box settle, periodic shear, rotating drum with facets, parametric
batch, serving slots) at sizes from a few hundred spheres to a million, in both precision modes.
The sphere beds are made here, from the seed alone: a small random packing in a periodic cube,
relaxed until its spheres just touch, repeated over the volume of the scene.

In FP32-force mode the forces are FP32 numbers and the velocities integrate them; those outputs are
returned in that type, positions (accumulated in FP64) as they are.
"""
import math

import numpy as np
import torch

STATE = ("pos", "ori", "vel", "angVel", "force", "torque")
# Law2_L6Geom_HertzPhys_DMT caps the shear force at zero under compression: in the drum, torques and
# angular velocities hold rounding errors alone and are not returned
DRUM = ("pos", "ori", "vel", "force")


def _names(case):
    return DRUM if case["kind"] in ("drum", "host") else STATE


# ------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # a script that looks at a small running scene after every step: launches, waits and copies only
        dict(name="look-300-fp64", kind="box", n=300, precision="fp64", steps=1, warm=60, damping=0.2, young=1e7, dyndt=0, count=False),
        # the default engines (with DynDt) of a small interactive script that reads the contacts
        dict(name="script-2803-fp64", kind="box", n=2803, precision="fp64", steps=100, warm=0, damping=0.2, young=1e7, dyndt=50, count=True),
        # the box settle configuration, in both precision modes
        dict(name="settle-10k-fp64", kind="box", n=10000, precision="fp64", steps=200, warm=0, damping=0.2, young=1e7, dyndt=0, count=False),
        dict(name="settle-10k-fp32", kind="box", n=10000, precision="fp32", steps=200, warm=0, damping=0.2, young=1e7, dyndt=0, count=False),
        # the periodic shear configuration with its stress tensor, in both precision modes
        dict(name="shear-200k-fp64", kind="shear", n=200000, precision="fp64", steps=20, rate=1.0),
        dict(name="shear-200k-fp32", kind="shear", n=200000, precision="fp32", steps=100, rate=1.0),
        # the rotating drum (facets, Hertz): the plain mode at a quarter of the size, the headline at full size
        dict(name="drum-250k-fp64", kind="drum", n=250007, precision="fp64", steps=40),
        dict(name="drum-1m-fp32", kind="drum", n=1000000, precision="fp32", steps=400),
        # a host that keeps the state itself and steps one by one from page-locked arrays
        dict(name="host-100k-fp32", kind="host", n=100003, precision="fp32", steps=1),
        # the parametric study: uneven scenes advanced together
        dict(name="batch-64-fp32", kind="batch", scenes=64, nmin=1000, nmax=50000, precision="fp32", steps=200),
        # the serving loop's tick: a job goes into a slot, all slots run, the slot's result is read
        dict(name="serve-8-fp32", kind="serve", slots=8, n=6000, precision="fp32", steps=100),
        # scene generation on the device
        dict(name="insert-30k", kind="insert", n=30000, fill=0.35),
    ]


def _logint(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["box", "box", "box", "shear", "drum", "drum", "host", "batch", "serve", "insert"])
    prec = rng.choice(["fp64", "fp32"])
    if kind == "box":
        n = _logint(rng, 200, 60000)
        one = rng.random() < 0.2
        return dict(kind=kind, n=n, precision=prec, steps=1 if one else rng.randint(50, 200), warm=rng.randint(40, 80) if one else 0,
                    damping=round(rng.uniform(0.0, 0.4), 3), young=round(math.exp(rng.uniform(math.log(1e6), math.log(1e8))), 1),
                    dyndt=rng.choice([0, 0, 30, 100]), count=rng.random() < 0.3)
    if kind == "shear":
        return dict(kind=kind, n=_logint(rng, 4000, 250000), precision=prec, steps=rng.randint(10, 30), rate=round(rng.uniform(0.2, 2.0), 3))
    if kind == "drum":
        return dict(kind=kind, n=_logint(rng, 20000, 600000 if prec == "fp32" else 200000), precision=prec, steps=rng.randint(20, 60))
    if kind == "host":
        return dict(kind=kind, n=_logint(rng, 5000, 200000), precision=prec, steps=rng.randint(1, 3))
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(3, 40), nmin=500, nmax=_logint(rng, 2000, 30000), precision=prec, steps=rng.randint(20, 80))
    if kind == "serve":
        return dict(kind=kind, slots=rng.randint(2, 12), n=_logint(rng, 800, 12000), precision=prec, steps=rng.randint(20, 100))
    return dict(kind=kind, n=_logint(rng, 2000, 30000), fill=round(rng.uniform(0.2, 0.36), 3))


def work(case):
    """Bytes and operations a pass cannot do without: per step the state of each sphere (position,
    velocity, orientation, constants, force and torque) read and written once, the persistent state
    of each touching contact read and written once, the particle ids of every other potential
    contact; once per pass the state handed to the host."""
    k = case["kind"]
    if k == "insert":
        return dict(bytes=case["n"] * 32.0, flops=case["n"] * 400.0)
    if k == "batch":
        n = sum(_study_sizes(case))
    else:
        n = case["n"] * (case["slots"] if k == "serve" else 1)
    real, other = {"box": (0.8, 1.6), "batch": (0.8, 1.6), "serve": (0.8, 1.6)}.get(k, (2.6, 3.0))
    br = 192.0 if case["precision"] == "fp64" else 124.0
    per_step = n * (260.0 + real * br + other * 16.0)
    out = case["n"] if k == "serve" else n
    host = out * 152.0 * (2 if k in ("host", "serve") else 1)
    return dict(bytes=case["steps"] * per_step + host, flops=case["steps"] * n * (250.0 + real * 400.0))


# ------------------------------------------------------------------------------------ the beds
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _tile(radii, fill, seed, sweeps=220):
    """Centres of spheres in a periodic cube at solid fraction ``fill``, moved apart until they
    overlap no more than the fraction demands (numpy array), and the cube's side."""
    dev = _device()
    r = torch.as_tensor(radii, dtype=torch.float64, device=dev)
    side = float((4 / 3 * math.pi * np.sum(np.asarray(radii) ** 3) / fill) ** (1 / 3))
    x = torch.as_tensor(np.random.default_rng(seed).uniform(0, side, (len(radii), 3)), device=dev)
    rr = r[:, None] + r[None, :]
    rr.fill_diagonal_(0.0)
    for _ in range(sweeps):
        w = torch.zeros_like(rr)
        dd = []
        for a in range(3):
            d = x[:, None, a] - x[None, :, a]
            d = d - side * torch.round(d / side)
            dd.append(d)
            w += d * d
        dist = torch.sqrt(w).clamp_min_(1e-12)
        w = (rr - dist).clamp_min_(0.0) / dist
        x = x + 0.4 * torch.stack([(w * d).sum(1) for d in dd], dim=1)
    x = x - side * torch.floor(x / side)
    return x.cpu().numpy(), side


def _repeat(x, side, k):
    g = np.stack(np.meshgrid(*[np.arange(q) for q in k], indexing="ij"), axis=-1).reshape(-1, 1, 3)
    return (x[None, :, :] + side * g).reshape(-1, 3), len(g)


def _box_bed(n, radius, seed, fill=0.5, tile=None):
    """``n`` spheres of one radius on their way down in a box: positions, velocities, box corners."""
    rng = np.random.default_rng(seed)
    m = max(1, int((n / 1200.0) ** (1 / 3)))
    per = int(math.ceil(n / float(m ** 3)))
    if tile is None:
        x, side = _tile(np.ones(per), fill, seed)
        k = (m, m, m)
    else:
        x, side = tile
        x = x[:, rng.permutation(3)]
        q = max(1, int(round((n / (2.0 * len(x))) ** (1 / 3))))
        k = (q, q, int(math.ceil(n / float(len(x) * q * q))))
    c, _ = _repeat(x, side, k)
    c = c[np.argsort(c[:, 2], kind="stable")[:n]] * radius
    lo = c.min(0) - radius * (1 - 1e-3)
    hi = c.max(0) + radius * (1 - 1e-3)
    hi[2] += 4 * radius
    v = rng.normal(0.0, 0.15, (n, 3))
    v[:, 2] -= 0.4
    return c, v, lo, hi


def _drum_radii(n, rng):
    return np.clip(3e-3 * np.exp(0.25 * rng.standard_normal(n)), 1.5e-3, 6e-3)


def _drum_bed(n, seed):
    """Centres, radii and velocities of a bed in the lower part of an x-axis drum, with a few spheres
    in flight above it, and the drum's diameter, length and mesh divisions."""
    rng = np.random.default_rng(seed)
    s = (n / 1e6) ** (1 / 3)
    R, length = 0.6 * s, 0.6 * s
    div, ax = max(16, int(round(200 * s))) + 1, max(4, int(round(50 * s)))
    m = 1300
    r0 = _drum_radii(m, rng)
    x, side = _tile(r0, 0.605, seed)
    k = (int(length / side) + 1, int(2 * R / side) + 1, int(1.1 * R / side) + 1)
    c, reps = _repeat(x, side, k)
    r = np.tile(r0, reps)
    c = c - np.array([0.0, 0.5 * k[1] * side, R])
    inside = (np.hypot(c[:, 1], c[:, 2]) + r < R * math.cos(math.pi / (div - 1)) - 1e-5) & (c[:, 0] > r) & (c[:, 0] + r < length)
    c, r = c[inside], r[inside]
    nf = n // 200
    low = np.argsort(c[:, 2], kind="stable")[: n - nf]
    if len(low) < n - nf:
        raise RuntimeError("the drum is too small for its bed")
    c, r = c[low], r[low]
    top = float(np.max(c[:, 2] + r))
    p = 0.013
    gx, gy, gz = np.arange(p, length - p, p), np.arange(-R, R, p), np.arange(top + p, R, p)
    f = np.stack(np.meshgrid(gx, gy, gz, indexing="ij"), axis=-1).reshape(-1, 3)
    f = f[np.hypot(f[:, 1], f[:, 2]) < R - p]
    f = f[np.sort(rng.permutation(len(f))[:nf])]
    if len(f) < nf:
        raise RuntimeError("the drum is too small for the spheres in flight")
    c = np.concatenate([c, f])
    r = np.concatenate([r, _drum_radii(nf, rng)])
    # the bed is landing: it closes on its own middle, so that its contacts carry load
    v = rng.normal(0.0, 0.01, (n, 3)) - (c - c[: n - nf].mean(0)) / R
    v[n - nf:] = rng.normal(0.0, 0.4, (nf, 3)) + np.array([0.0, 0.5, -0.5])
    return c, r, v, 2 * R, length, div, ax


def _shear_bed(n, seed):
    rng = np.random.default_rng(seed)
    k = max(1, int((n / 1200.0) ** (1 / 3)))
    per = n // k ** 3
    r0 = rng.uniform(2e-3, 4e-3, per)
    x, side = _tile(r0, 0.605, seed)
    c, reps = _repeat(x, side, (k, k, k))
    r = np.tile(r0 * 1.0005, reps)
    # insertion leaves the spheres in no spatial order
    o = rng.permutation(len(c))
    return c[o], r[o], rng.normal(0.0, 0.02, (len(c), 3)), k * side


def _mono_tile(seed):
    return _tile(np.ones(1100), 0.5, seed)


def _study_sizes(case):
    """Log-uniform sizes in no order; they belong to the case, not to the seed."""
    q = (np.random.default_rng(17).permutation(case["scenes"]) + 0.5) / case["scenes"]
    return [int(case["nmin"] * (case["nmax"] / case["nmin"]) ** v) for v in q]


def _study(case, seed):
    """Parameters and beds of the scenes of a parametric study."""
    rng = np.random.default_rng(seed)
    tile = _mono_tile(seed)
    out = []
    for n in _study_sizes(case):
        k = len(out)
        radius = rng.uniform(3e-3, 6e-3)
        p = dict(radius=radius, young=math.exp(rng.uniform(math.log(1e6), math.log(1e8))),
                 tanPhi=math.exp(rng.uniform(math.log(0.2), math.log(0.8))), damping=rng.uniform(0.0, 0.4))
        out.append((p, _box_bed(n, radius, seed * 1000 + k, tile=tile)))
    return out


def _jobs(case, seed, count=4):
    """Jobs of a serving stream: sizes just below the slots' capacity."""
    rng = np.random.default_rng(seed)
    tile = _mono_tile(seed)
    out = []
    for k in range(count):
        n = case["n"] - k * (case["n"] // 16)
        radius = rng.uniform(3e-3, 6e-3)
        p = dict(radius=radius, young=math.exp(rng.uniform(math.log(1e6), math.log(1e8))),
                 tanPhi=math.exp(rng.uniform(math.log(0.2), math.log(0.8))), damping=rng.uniform(0.0, 0.4))
        out.append((p, _box_bed(n, radius, seed * 1000 + k, tile=tile)))
    return out


def _insert_radii(case, seed):
    r = np.random.default_rng(seed).uniform(2e-3, 4e-3, case["n"])
    return r, float((4 / 3 * math.pi * np.sum(r ** 3) / case["fill"]) ** (1 / 3))


# ------------------------------------------------------------------------------------ prepare, run
def _velocities(S, v):
    soa = S.dem._nodes.soa
    soa.col("vel")[len(soa) - len(v):] = v


def _box_scene(bed, p, precision, dyndt=0):
    from woodem_gb300 import utils
    from woodem_gb300.core import Scene
    from woodem_gb300.dem import DemField, FrictMat
    c, v, lo, hi = bed
    S = Scene(fields=[DemField(gravity=(0, 0, -9.81))])
    S.gpu.precision = precision
    mat = FrictMat(density=3000.0, young=p["young"], ktDivKn=0.2, tanPhi=p["tanPhi"])
    S.dem.par.add(utils.wallBox((lo, hi), mat=mat))
    S.dem.par.addSpheres(c, p["radius"], mat)
    S.engines = utils.defaultEngines(damping=p["damping"], verletDist=-0.1, dynDtPeriod=dyndt)
    S.dt = 0.3 * utils.pWaveDt(S)
    _velocities(S, v)
    return S


def _box_params(case):
    return dict(radius=5e-3, young=case["young"], tanPhi=0.5, damping=case["damping"])


def _shear_scene(case, seed):
    from woodem_gb300 import utils
    from woodem_gb300.core import Cell, Scene
    from woodem_gb300.dem import DemField, FrictMat
    c, r, v, side = _shear_bed(case["n"], seed)
    S = Scene(fields=[DemField(gravity=(0, 0, 0))])
    S.gpu.precision = case["precision"]
    S.periodic = True
    S.cell.setBox(side, side, side)
    S.cell.homoDeform = Cell.HomoGradV2
    S.dem.par.addSpheres(c, r, FrictMat(density=2600.0, young=5e7, tanPhi=0.4, ktDivKn=0.2))
    S.engines = utils.defaultEngines(damping=0.2, verletDist=-0.1, dynDtPeriod=0)
    S.engines[2].evalStress = True
    S.dt = 0.3 * utils.pWaveDt(S)
    _velocities(S, v)
    g = np.zeros((3, 3))
    g[0, 2] = case["rate"]
    S.cell.nextGradV = g
    return S


def _drum_scene(case, seed):
    from woodem_gb300 import scenes
    c, r, v, dia, length, div, ax = _drum_bed(case["n"], seed)
    o = scenes.spatial_order(c, 12e-3)
    return scenes.hertz_drum_from_state(c[o], r[o], vel=v[o], diameter=dia, length=length, div=div, axDiv=ax,
                                        precision=case["precision"])


class _State:
    pass


def prepare(case, seed):
    st = _State()
    st.case, st.turn = case, 0
    k = case["kind"]
    if k == "box":
        st.S = _box_scene(_box_bed(case["n"], 5e-3, seed), _box_params(case), case["precision"], case["dyndt"])
        if case["warm"]:
            st.S.run(case["warm"])
    elif k == "shear":
        st.S = _shear_scene(case, seed)
    elif k == "drum":
        st.S = _drum_scene(case, seed)
    elif k == "host":
        st.S = _drum_scene(case, seed)
        st.sim = st.S._ensure_sim()
        soa = st.S.dem._nodes.soa
        st.host = [torch.from_numpy(np.ascontiguousarray(soa.col(q))).clone() for q in STATE]
        if torch.cuda.is_available():
            st.host = [t.pin_memory() for t in st.host]
        st.n0 = len(soa) - case["n"]
    elif k == "batch":
        from woodem_gb300.batch import Batch
        st.scenes = [_box_scene(bed, p, case["precision"]) for p, bed in _study(case, seed)]
        st.batch = Batch(st.scenes)
    elif k == "serve":
        from woodem_gb300 import _plan
        from woodem_gb300.serve import SlotPool
        st.jobs = [_plan.compile_scene(_box_scene(bed, p, case["precision"])) for p, bed in _jobs(case, seed)]
        st.pool = SlotPool([case["n"] + 6] * case["slots"], precision=case["precision"], template=st.jobs[0])
        for q in range(case["slots"]):
            st.pool.load(q, st.jobs[(q + 1) % len(st.jobs)], 1 << 40)
    else:
        st.radii, st.side = _insert_radii(case, seed)
        st.seed = seed
    return st


def _typed(out, precision):
    out = {q: torch.from_numpy(v) if isinstance(v, np.ndarray) else v for q, v in out.items()}
    if precision == "fp32":
        out = {q: v if q in ("pos", "hSize") else v.to(torch.float32) for q, v in out.items()}
    return out


def run(st):
    case = st.case
    k = case["kind"]
    if k == "insert":
        from woodem_gb300 import scenes
        return scenes.pack_rsa(st.radii, (0, 0, 0), (st.side,) * 3, region=2, seed=st.seed, device=True)
    if k == "host":
        from woodem_gb300 import _native
        H = st.sim.H
        H.check(H.L.wg_run_host(H.h, case["steps"], *[_native.ptr(t.numpy()) for t in st.host]), "run_host")
        return _typed({q: t[st.n0:] for q, t in zip(STATE, st.host) if q in DRUM}, case["precision"])
    if k == "batch":
        st.batch.run(case["steps"])
        st.batch.pull()
        nodes = [S.dem._nodes.soa for S in st.scenes]
        return _typed({q: torch.cat([torch.from_numpy(d.col(q)[6:]) for d in nodes]) for q in STATE}, case["precision"])
    if k == "serve":
        q, A = st.turn % case["slots"], st.jobs[st.turn % len(st.jobs)]
        st.turn += 1
        st.pool.clear(q)
        st.pool.load(q, A, 1 << 40)
        st.pool.run(case["steps"])
        out = st.pool.nodes(q, A.n_nodes)
        return _typed({q: v[6:] for q, v in out.items()}, case["precision"])
    S = st.S
    if case["steps"] == 1:
        S.one()
    else:
        S.run(case["steps"])
    S.sync()
    soa = S.dem._nodes.soa
    out = _typed({q: soa.col(q)[len(soa) - _spheres(case):] for q in _names(case)}, case["precision"])
    if k == "shear":
        out["hSize"], out["stress"] = np.array(S.cell.hSize), np.array(S.engines[2].stress)
    if k == "box" and case["dyndt"]:
        out["dt"] = float(S.dt)
    if k == "box" and case["count"]:
        out["real"] = S.dem.con.countReal()
    return out


def _spheres(case):
    if case["kind"] != "shear":
        return case["n"]
    k = max(1, int((case["n"] / 1200.0) ** (1 / 3)))
    return (case["n"] // k ** 3) * k ** 3


# ------------------------------------------------------------------------------------ exact
# The same scenes in 64 bits, in plain torch: Leapfrog, contact geometry (sphere-sphere, wall-sphere,
# facet-sphere), the two contact laws, the periodic cell and DynDt.
def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _dot(a, b):
    return (a * b).sum(-1, keepdim=True)


def _unit(a):
    return a / torch.sqrt(_dot(a, a)).clamp_min(1e-300)


def _ranges(beg, end):
    """(index of the range, value) of every integer of the ranges [beg, end)."""
    n = end - beg
    i = torch.repeat_interleave(torch.arange(len(n), device=n.device), n)
    off = torch.cumsum(n, 0) - n
    return i, beg[i] + torch.arange(len(i), device=n.device) - off[i]


def _near_spheres(x, reach, H=None):
    """Pairs (i < j) of points whose boxes of half-edge reach/2 may overlap; with a periodic cell H
    the nearest images."""
    dev = x.device
    if H is None:
        q = x - x.min(0).values
        n = torch.floor(q.max(0).values / reach).long() + 1
        c = torch.minimum(torch.floor(q / reach).long(), n - 1)
    else:
        s = x @ torch.linalg.inv(H).T
        s = s - torch.floor(s)
        edge = 1.0 / torch.linalg.norm(torch.linalg.inv(H), dim=1)
        n = torch.clamp(torch.floor(edge / reach).long(), min=1)
        c = torch.minimum((s * n).long(), n - 1)
    key = (c[:, 2] * n[1] + c[:, 1]) * n[0] + c[:, 0]
    sk, o = torch.sort(key)
    ii, jj = [], []
    nn = [int(v) for v in n]
    offs = [[d for d in (-1, 0, 1)] if (H is None or m >= 3) else list(range(m)) for m in nn]
    for dz in offs[2]:
        for dy in offs[1]:
            for dx in offs[0]:
                d = c + torch.tensor([dx, dy, dz], device=dev)
                if H is None:
                    ok = ((d >= 0) & (d < n)).all(1)
                else:
                    d = d % n
                    ok = torch.ones(len(d), dtype=torch.bool, device=dev)
                k = (d[:, 2] * n[1] + d[:, 1]) * n[0] + d[:, 0]
                a = torch.searchsorted(sk, k)
                b = torch.where(ok, torch.searchsorted(sk, k, right=True), a)
                i, p = _ranges(a, b)
                j = o[p]
                keep = i < j
                i, j = i[keep], j[keep]
                dd = x[j] - x[i]
                if H is not None:
                    dd = dd - torch.round(dd @ torch.linalg.inv(H).T) @ H.T
                keep = (dd.abs() <= reach).all(1)
                ii.append(i[keep])
                jj.append(j[keep])
    i, j = torch.cat(ii), torch.cat(jj)
    u = torch.unique(i * len(x) + j)  # few cells per axis meet a pair more than once
    return u // len(x), u % len(x)


def _near_facets(x, r, verts, margin):
    """(facet, sphere) pairs whose boxes, grown by the margin, overlap."""
    lo, hi = verts.min(1).values - margin, verts.max(1).values + margin
    cell = float((hi - lo).max()) + 2 * float(r.max()) + 2 * margin
    q = torch.floor((x - lo.min(0).values) / cell).long() + 2
    mid = torch.floor((0.5 * (lo + hi) - lo.min(0).values) / cell).long() + 2
    n = torch.maximum(q.max(0).values, mid.max(0).values) + 3
    key = (q[:, 2] * n[1] + q[:, 1]) * n[0] + q[:, 0]
    sk, o = torch.sort(key)
    ff, ss = [], []
    for d in np.ndindex(3, 3, 3):
        m = mid + torch.tensor(d, device=x.device) - 1
        k = (m[:, 2] * n[1] + m[:, 1]) * n[0] + m[:, 0]
        f, p = _ranges(torch.searchsorted(sk, k), torch.searchsorted(sk, k, right=True))
        s = o[p]
        keep = ((x[s] - r[s, None] <= hi[f]) & (x[s] + r[s, None] >= lo[f])).all(1)
        ff.append(f[keep])
        ss.append(s[keep])
    return torch.cat(ff), torch.cat(ss)


def _segment(P, A, B):
    BA = B - A
    u = (_dot(P, BA) - _dot(A, BA)) / _dot(BA, BA)
    return A + u.clamp(0.0, 1.0) * BA


class _Kind:
    """The contacts of one kind (sphere, wall, facet with sphere) and their persistent state."""

    def __init__(self, dev):
        self.key = torch.zeros(0, dtype=torch.int64, device=dev)
        self.st = torch.zeros((0, 19), dtype=torch.float64, device=dev)  # real, c0, c1, cp, phys 5, ft 2, uN first

    def renew(self, key):
        key = torch.unique(key)
        st = torch.zeros((len(key), 19), dtype=torch.float64, device=key.device)
        if len(self.key) and len(key):
            p = torch.searchsorted(key, self.key).clamp_max(len(key) - 1)
            hit = key[p] == self.key
            st[p[hit]] = self.st[hit]
        self.key, self.st = key, st


class _Dem:
    def __init__(self, x, v, r, m, p, walls=(), facets=None, cell=None, gravity=(0, 0, 0)):
        self.dev = dev = _device()
        t = lambda a: torch.as_tensor(np.array(a, dtype=float), device=dev)  # noqa: E731
        self.x, self.v, self.r = t(x), t(v), t(r)
        n = len(self.x)
        self.m = t(m)[:, None]
        self.I = 0.4 * self.m * self.r[:, None] ** 2
        self.w, self.F, self.T = (torch.zeros((n, 3), dtype=torch.float64, device=dev) for _ in range(3))
        self.q = torch.zeros((n, 4), dtype=torch.float64, device=dev)
        self.q[:, 0] = 1
        self.p, self.dt, self.g, self.step, self.time = p, p["dt"], t(gravity), 0, 0.0
        self.walls = [(ax, sense, float(c), t(w)) for ax, sense, c, w in walls]
        self.verts = None if facets is None else t(facets[0])
        self.fake = None if facets is None else t(facets[1])
        self.H = None if cell is None else t(cell[0])
        self.L, self.nextL = torch.zeros((3, 3), dtype=torch.float64, device=dev), None if cell is None else t(cell[1])
        self.last, self.margin = None, 0.2 * float(self.r.min())
        self.kinds = [_Kind(dev), _Kind(dev), _Kind(dev)]
        self.stress, self.nextDt, self.real = None, None, 0

    def leapfrog(self):
        dt, d = self.dt, self.p["damping"]
        a, al = self.F / self.m, self.T / self.I
        fv, fw = self.v, self.w
        if self.H is not None:
            fv = self.v - (self.x - dt / 2 * self.v) @ self.L.T
            fw = self.w - self.spin(self.L)
        if d:
            a = a * (1 - d * torch.sign(self.F * (fv + 0.5 * dt * a)))
            al = al * (1 - d * torch.sign(self.T * (fw + 0.5 * dt * al)))
        if self.H is None:
            self.v = self.v + dt * a
            self.w = self.w + dt * al
        else:
            I = torch.eye(3, dtype=torch.float64, device=self.dev)
            q = (self.nextL + self.L) * dt / 4
            self.v = (self.x @ (self.nextL - self.L).T + self.v @ (I + q).T + a * dt) @ torch.linalg.inv(I - q).T
            self.w = self.w + dt * al - (self.spin(self.nextL) - self.spin(self.L))
        self.x = self.x + dt * self.v
        ang = torch.sqrt(_dot(self.w, self.w))
        s, c = torch.sin(0.5 * ang * dt), torch.cos(0.5 * ang * dt)
        av = self.w / ang.clamp_min(1e-300) * s
        w0, v0 = self.q[:, :1], self.q[:, 1:]
        q = torch.cat([c * w0 - _dot(av, v0), c * v0 + w0 * av + _cross(av, v0)], dim=1)
        self.q = q / torch.linalg.norm(q, dim=1, keepdim=True)

    @staticmethod
    def spin(L):
        W = (L - L.T) / 2
        return 0.5 * torch.stack([W[1, 2] - W[2, 1], W[2, 0] - W[0, 2], W[0, 1] - W[1, 0]])

    def candidates(self):
        if self.last is not None and float((self.x - self.last).abs().max()) < 0.25 * self.margin:
            return
        self.last = self.x.clone()
        n = len(self.x)
        reach = 2 * float(self.r.max()) + self.margin
        i, j = _near_spheres(self.x, reach, self.H)
        dx = self.x[j] - self.x[i]
        if self.H is not None:
            dx = dx - torch.round(dx @ torch.linalg.inv(self.H).T) @ self.H.T
        keep = (dx * dx).sum(1) <= (self.r[i] + self.r[j] + self.margin) ** 2
        self.kinds[0].renew(i[keep] * n + j[keep])
        wk = [k * n + torch.nonzero((self.x[:, ax] - c).abs() <= self.r + self.margin).flatten()
              for k, (ax, _, c, _) in enumerate(self.walls)]
        if wk:
            self.kinds[1].renew(torch.cat(wk))
        if self.verts is not None:
            f, s = _near_facets(self.x, self.r, self.verts, self.margin)
            self.kinds[2].renew(f * n + s)

    def geometry(self, kind, st, key):
        """Of the contacts that touch or did: their row, pA's id (or -1) and pB's, normal, overlap,
        contact point, both positions, velocities, angular velocities and radii."""
        n = len(self.x)
        a, b = key // n, key % n
        was = st[:, 0] > 0
        z = torch.zeros_like
        if kind == 0:
            sh = None
            dx = self.x[b] - self.x[a]
            if self.H is not None:
                cd = -torch.round(dx @ torch.linalg.inv(self.H).T)
                sh = cd @ self.H.T
                dx = dx + sh
            rr = self.r[a] + self.r[b]
            row = torch.nonzero(was | ((dx * dx).sum(1) <= rr * rr)).flatten()
            a, b, dx, rr = a[row], b[row], dx[row], rr[row, None]
            dist = torch.sqrt(_dot(dx, dx))
            nrm, u = dx / dist, dist - rr
            r1, r2 = self.r[a, None], self.r[b, None]
            pos1 = self.x[a]
            vel2 = self.v[b]
            if sh is not None:
                vel2 = vel2 + cd[row] @ (self.L @ self.Hmid).T
            return row, a, b, nrm, u, pos1 + (r1 + 0.5 * u) * nrm, pos1, self.v[a], self.w[a], pos1 + dx, vel2, self.w[b], r1, r2
        r = self.r[b, None]
        if kind == 1:
            ax = torch.tensor([w[0] for w in self.walls], device=self.dev)[a]
            sense = torch.tensor([float(w[1]) for w in self.walls], dtype=torch.float64, device=self.dev)[a][:, None]
            c = torch.tensor([w[2] for w in self.walls], dtype=torch.float64, device=self.dev)[a][:, None]
            aw = torch.stack([w[3] for w in self.walls])[a]
            e = torch.nn.functional.one_hot(ax, 3).to(torch.float64)
            x = self.x[b]
            d = _dot(x, e) - c
            row = torch.nonzero(was | (d.abs() <= r).flatten()).flatten()
            b, e, x, d, r, sense, aw = b[row], e[row], x[row], d[row], r[row], sense[row], aw[row]
            nrm, cp = e * sense, x - d * e
            wp = c[row] * e
            return row, b * 0 - 1, b, nrm, sense * d - r, cp, wp, z(x), aw, x, self.v[b], self.w[b], -r, r
        p0, p1, p2 = (self.verts[a, k] for k in range(3))
        x = self.x[b]
        nn = _cross(p1 - p0, p2 - p0)
        fn = _unit(nn)
        pd = _dot(x - p0, fn)
        fc = x - pd * fn
        l0, l1, l2 = (_dot(_cross(q1 - q0, nn), fc - q0) > 0 for q0, q1 in ((p0, p1), (p1, p2), (p2, p0)))
        code = (l0.long() + 2 * l1.long() + 4 * l2.long()).flatten()
        opts = torch.stack([fc, _segment(fc, p0, p1), _segment(fc, p1, p2), p1, _segment(fc, p2, p0), p0, p2, fc], dim=1)
        cp = opts[torch.arange(len(code), device=self.dev), code]
        d = x - cp
        dist = torch.sqrt(_dot(d, d))
        row = torch.nonzero(was | ((pd.abs() <= r) & (dist <= r)).flatten()).flatten()
        a, b, cp, d, dist, r, x = a[row], b[row], cp[row], d[row], dist[row], r[row], x[row]
        return row, b * 0 - 1, b, d / dist, dist - r, cp, cp, self.fake[a], z(x), x, self.v[b], self.w[b], r, r

    def law(self, kind, k):
        st, p, dt = k.st, self.p, self.dt
        row, a, b, nrm, u, cp, pos1, v1, w1, pos2, v2, w2, r1, r2 = self.geometry(kind, st, k.key)
        s = st[row]
        real = s[:, :1] > 0
        # new contacts: frame and material constants
        ref = torch.zeros_like(nrm)
        yz = (nrm[:, 1].abs() < nrm[:, 2].abs())
        ref[:, 1], ref[:, 2] = yz.to(ref.dtype), (~yz).to(ref.dtype)
        y = _cross(nrm, ref)
        y = _unit(y - nrm * _dot(y, nrm))
        l0, l1 = r1.abs() + u / 2, r2.abs() + u / 2
        l0, l1 = torch.where(l0 < 0, l1, l0), torch.where(l1 < 0, l0, l1)
        E, nu = p["young"], p.get("poisson", 0.2)
        if p["law"] == 0:
            rc = torch.where(r1 > 0, torch.minimum(r1, r2), r2)
            kn = 1 / (1 / (E * math.pi * rc * rc / l0) + 1 / (E * math.pi * rc * rc / l1))
            ph = torch.cat([kn, p["ktDivKn"] * kn, torch.full_like(kn, p["tanPhi"]), kn * 0, kn * 0], dim=1)
        else:
            K = 4 / 3 / ((1 - nu * nu) / E * 2)
            R = 1 / (1 / l0 + 1 / l1)
            kn0 = K * torch.sqrt(R)
            G = E / (2 * (1 + nu))
            m2 = self.m[b]
            mbar = torch.where((a >= 0)[:, None], self.m[a.clamp_min(0)] * m2 / (self.m[a.clamp_min(0)] + m2), m2)
            le = math.log(p["en"])
            visc = -math.sqrt(5.0) * le / math.sqrt(le * le + math.pi ** 2) * torch.sqrt(mbar * kn0)
            ph = torch.cat([kn0, 2 * torch.sqrt(4 * R) * G / (2 - nu), torch.full_like(kn0, p["tanPhi"]), visc, R], dim=1)
        # existing contacts: frame update and relative velocity
        pn, pc, pcp = s[:, 1:4], s[:, 4:7], s[:, 7:10]
        mid = _unit(0.5 * (pn + nrm))
        rt = _cross(pn, nrm) + mid * dt * 0.5 * _dot(mid, w1 + w2)
        m1 = pc - _cross(pc, rt) / 2
        m2v = _cross(mid, m1)
        c1 = pc - _cross(m1, rt)
        if self.step % 100 == 0:
            c1 = _unit(c1 - nrm * _dot(c1, nrm))
        mc = 0.5 * (pcp + cp)
        b1, b2 = mc - (pos1 - dt / 2 * v1), mc - (pos2 - dt / 2 * v2)
        rel = (v2 + _cross(w2, b2)) - (v1 + _cross(w1, b1))
        lv = torch.cat([_dot(mid, rel), _dot(m1, rel), _dot(m2v, rel)], dim=1)
        lv = torch.where(real, lv, torch.zeros_like(lv))
        c0, c1 = nrm, torch.where(real, c1, y)
        ph = torch.where(real, s[:, 10:15], ph)
        ft = torch.where(real, s[:, 15:17], torch.zeros_like(s[:, 15:17]))
        u0 = torch.where(real, s[:, 18:19], u)
        keep = u <= 0
        if p["law"] == 0:
            fn = ph[:, :1] * u
            ft = ft + dt * ph[:, 1:2] * lv[:, 1:]
            cap = fn.abs() * ph[:, 2:3]
            f = torch.sqrt(_dot(ft, ft))
            ft = torch.where(f > cap, ft * (cap / f.clamp_min(1e-300)), ft)
            kn, kt = ph[:, :1], ph[:, 1:2]
        else:
            su = torch.sqrt((-u).clamp_min(0))
            fe = -ph[:, :1] * su ** 3
            eta = ph[:, 3:4] * torch.sqrt(su)
            fv = eta * lv[:, :1]
            fv = torch.where(fe + fv > 0, -fe, fv)
            fn = fe + fv
            kn, kt = 1.5 * ph[:, :1] * su, ph[:, 1:2] * su
            ft = dt * kt * lv[:, 1:]
            cap = fn.clamp_min(0) * ph[:, 2:3]
            f = torch.sqrt(_dot(ft, ft))
            ft = torch.where(f > cap, ft * (cap / f.clamp_min(1e-300)), ft + eta * lv[:, 1:])
        Fg = fn * c0 + ft[:, :1] * c1 + ft[:, 1:] * _cross(c0, c1)
        Fg = torch.where(keep, Fg, torch.zeros_like(Fg))
        self.F.index_add_(0, b, -Fg)
        self.T.index_add_(0, b, _cross(cp - pos2, -Fg))
        if kind == 0:
            self.F.index_add_(0, a, Fg)
            self.T.index_add_(0, a, _cross(cp - pos1, Fg))
            if self.H is not None:
                self.stress = Fg.T @ (pos2 - pos1)
        st[row] = torch.cat([keep.to(st.dtype), c0, c1, cp, ph, ft, u, u0], dim=1) * keep
        self.real += int(keep.sum())
        if self.due:
            n2 = c0 * c0
            add = torch.where(keep, n2 * (kn - kt) + kt, torch.zeros_like(n2))
            rv = torch.stack([n2[:, 1] + n2[:, 2], n2[:, 2] + n2[:, 0], n2[:, 0] + n2[:, 1]], dim=1) * kt * keep
            self.kt.index_add_(0, b, add)
            self.kr.index_add_(0, b, rv * (r2.abs() + u0 / 2) ** 2)
            if kind == 0:
                self.kt.index_add_(0, a, add)
                self.kr.index_add_(0, a, rv * (r1.abs() + u0 / 2) ** 2)

    def one(self):
        if self.H is not None:
            I = torch.eye(3, dtype=torch.float64, device=self.dev)
            h = self.H
            self.H = torch.linalg.inv(I - self.L * self.dt / 2) @ (I + self.L * self.dt / 2) @ h
            self.Hmid = 0.5 * (h + self.H)
        self.leapfrog()
        self.candidates()
        self.F = (self.m * self.g).expand(-1, 3).clone()
        self.T = torch.zeros_like(self.F)
        period = self.p.get("dyndt", 0)
        self.due = bool(period) and self.step % period == 0
        if self.due:
            self.kt, self.kr = torch.zeros_like(self.F), torch.zeros_like(self.F)
        self.real = 0
        for kind, k in enumerate(self.kinds):
            if len(k.key):
                self.law(kind, k)
        new = self.dt
        if self.due:
            sq = torch.stack([torch.where(self.kt != 0, self.m / self.kt.abs(), math.inf).min(),
                              torch.where(self.kr != 0, self.I / self.kr.abs(), math.inf).min()]).min()
            crit = math.sqrt(2 * float(sq))
            prev = getattr(self, "prev", self.step)
            if math.isfinite(crit):
                new = min(crit * 0.9, self.dt * (1 + 1e-4) ** (self.step - prev))
            self.prev = self.step
        if self.nextL is not None:
            self.L = self.nextL
        self.step += 1
        self.time += self.dt
        self.dt = new

    def out(self):
        return {"pos": self.x, "ori": self.q, "vel": self.v, "angVel": self.w, "force": self.F, "torque": self.T}


def _exact_box(bed, p, steps, dyndt=0):
    c, v, lo, hi = bed
    r = np.full(len(c), p["radius"])
    m = 4 / 3 * math.pi * r ** 3 * 3000.0
    walls = [(ax, s, side[ax], (0, 0, 0)) for s, side in ((1, lo), (-1, hi)) for ax in range(3)]
    dt = 0.3 * p["radius"] / math.sqrt(p["young"] / 3000.0)
    D = _Dem(c, v, r, m, dict(law=0, young=p["young"], ktDivKn=0.2, tanPhi=p["tanPhi"], damping=p["damping"], dt=dt, dyndt=dyndt),
             walls=walls, gravity=(0, 0, -9.81))
    for _ in range(steps):
        D.one()
    return D


def exact(case, seed):
    k = case["kind"]
    if k == "insert":
        return None
    if k == "box":
        D = _exact_box(_box_bed(case["n"], 5e-3, seed), _box_params(case), case["warm"] + case["steps"], case["dyndt"])
        out = D.out()
        if case["dyndt"]:
            out["dt"] = D.dt
        if case["count"]:
            out["real"] = None
        return out
    if k == "batch":
        parts = [_exact_box(bed, p, case["steps"]).out() for p, bed in _study(case, seed)] if case["scenes"] * case["steps"] <= 1500 else None
        return parts and {q: torch.cat([o[q] for o in parts]) for q in STATE}
    if k == "serve":
        p, bed = _jobs(case, seed, 1)[0]
        return _exact_box(bed, p, case["steps"]).out()
    if k == "shear":
        c, r, v, side = _shear_bed(case["n"], seed)
        g = np.zeros((3, 3))
        g[0, 2] = case["rate"]
        m = 4 / 3 * math.pi * r ** 3 * 2600.0
        D = _Dem(c, v, r, m, dict(law=0, young=5e7, ktDivKn=0.2, tanPhi=0.4, damping=0.2, dt=0.3 * float(r.min()) / math.sqrt(5e7 / 2600.0)),
                 cell=(np.diag([side] * 3), g))
        for _ in range(case["steps"]):
            D.one()
        return dict(D.out(), hSize=D.H, stress=D.stress / torch.linalg.det(D.H))
    # the drum, as triangulated.cylinder meshes it
    c, r, v, dia, length, div, ax = _drum_bed(case["n"], seed)
    o = _morton(c, 12e-3)
    c, r, v = c[o], r[o], v[o]
    R = dia / 2
    th = np.linspace(0, 2 * math.pi, num=div)[:-1]
    xs = np.linspace(0, length, num=ax + 1)
    e1, e2 = np.array([0.0, 0, 1]), np.array([0.0, -1, 0])
    ring = R * (np.cos(th)[:, None] * e1 + np.sin(th)[:, None] * e2)
    P = xs[:, None, None] * np.array([1.0, 0, 0]) + ring[None]
    a, b, cc, d = P[:-1], np.roll(P, -1, 1)[:-1], P[1:], np.roll(P, -1, 1)[1:]
    tri = np.stack([np.stack([a, cc, b], -2), np.stack([b, cc, d], -2)], 2).reshape(-1, 3, 3)
    nrm = np.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0])
    flip = (nrm * (tri.mean(1) * np.array([0, 1.0, 1]))).sum(1) < 0
    tri[flip] = tri[flip][:, [0, 2, 1]]
    nrm[flip] = -nrm[flip]
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    fake = -R * 1.0 * np.cross(nrm, np.array([1.0, 0, 0]))
    walls = [(0, 1, 0.0, (1.0, 0, 0)), (0, -1, length, (1.0, 0, 0))]
    m = 4 / 3 * math.pi * r ** 3 * 2500.0
    D = _Dem(c, v, r, m, dict(law=1, young=1e8, poisson=0.25, en=0.6, tanPhi=0.5, damping=0.0, dt=0.3 * float(r.min()) / math.sqrt(1e8 / 2500.0)),
             walls=walls, facets=(tri, fake), gravity=(0, 0, -9.81))
    for _ in range(case["steps"]):
        D.one()
    return {q: v for q, v in D.out().items() if q in DRUM}


def _morton(points, cell):
    """The order of points along a Z-curve over cubes of side ``cell`` (stable)."""
    q = np.floor((points - points.min(axis=0)) / cell).astype(np.uint64)
    code = np.zeros(len(points), np.uint64)
    for bit in range(21):
        for ax in range(3):
            code |= ((q[:, ax] >> np.uint64(bit)) & np.uint64(1)) << np.uint64(3 * bit + ax)
    return np.argsort(code, kind="stable")
