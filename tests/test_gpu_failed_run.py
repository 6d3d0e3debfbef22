"""A collider run that fails (a box that is not finite, no memory left) leaves the contacts, their state and their
forces as they were: they list as before, and with the cause mended the scene goes on as one restored from them.
The run is one that parts touching pairs (real contacts without an overlap) and brings many new ones (every array grows)."""
import ctypes as C

import numpy as np
import pytest

from woodem_gb300 import _native, checkpoint, utils
from woodem_gb300.core import Cell, Scene
from woodem_gb300.dem import DemField, FrictMat

pytestmark = pytest.mark.gpu

R, PAIRS, LOOSE = 5e-3, 24, 480
KEYS = ("pos", "ori", "vel", "angVel", "force", "torque")


def build(precision, periodic):
    """PAIRS pairs that touch and roll, and LOOSE spheres that touch nothing (the last ones)."""
    rng = np.random.default_rng(7)
    g = lambda n, pitch, at: np.stack(np.meshgrid(*[np.arange(8)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * pitch + at
    a = g(PAIRS, 8 * R, [.1, .1, .1])
    b = a + 1.97 * R * np.array([0.6, 0.64, 0.48])
    c = np.concatenate([np.stack([a, b], 1).reshape(-1, 3), g(LOOSE, 6 * R, [.1, .1, .6])])
    S = Scene(fields=[DemField(gravity=(0, 0, 0))])
    S.gpu.precision = precision
    if periodic:
        S.periodic = True
        S.cell.setBox(1.0, 1.0, 1.0)
        S.cell.homoDeform = Cell.HomoNone
    S.dem.par.addSpheres(c, R, FrictMat(density=3000., young=1e7, ktDivKn=.2, tanPhi=.5))
    nd = S.dem._nodes.soa
    nd.col("vel")[:2 * PAIRS] = rng.uniform(-.02, .02, (2 * PAIRS, 3))
    nd.col("angVel")[:2 * PAIRS] = rng.uniform(-5, 5, (2 * PAIRS, 3))
    S.engines = utils.defaultEngines(damping=.1, verletDist=-.4, dynDtPeriod=0)
    S.dt = .2 * utils.pWaveDt(S)
    return S


class Raw:
    """The C calls of one scene."""

    def __init__(self, S):
        self.S, self.sim = S, S._ensure_sim()
        self.L, self.h = self.sim.H.L, self.sim.H.h
        self.n = len(S.dem._nodes.soa)
        self.due = 0

    def run(self, n):
        return self.L.wg_run(self.h, n)

    def nodes(self):
        out = [np.empty((self.n, w)) for w in (3, 4, 3, 3, 3, 3)]
        self.sim.H.check(self.L.wg_get_nodes(self.h, *[_native.ptr(a) for a in out]), "get_nodes")
        return out

    def energy(self):
        v, c = np.zeros(32), np.zeros(32, np.int32)
        self.sim.H.check(self.L.wg_get_energy(self.h, _native.ptr(v), _native.ptr(c, _native.P_I32)), "get_energy")
        return np.concatenate([v, c])

    def put(self, nodes):
        self.sim.H.check(self.L.wg_put_state(self.h, *[_native.ptr(a) for a in nodes]), "put_state")

    def apart(self):
        """Whether the boxes of each pair of the last full run are apart."""
        mn, mx = np.empty((self.n, 3)), np.empty((self.n, 3))
        self.sim.H.check(self.L.wg_get_aabbs(self.h, _native.ptr(mn), _native.ptr(mx)), "get_aabbs")
        a, b = np.arange(0, 2 * PAIRS, 2), np.arange(1, 2 * PAIRS, 2)
        return np.any((mn[a] > mx[b]) | (mx[a] < mn[b]), axis=1)

    def contacts(self):
        from woodem_gb300 import _plan
        c = _plan.read_contacts(self.L, self.h, "wg")
        r = c["real"] != 0
        return c, {k: c[k][r] for k in ("id_lo", "id_hi", "id_a", "cell_dist", "fglob", "local", "trsf")}

    def state(self):
        c = checkpoint.contact_snapshot(self.S)
        r = (c["con_flags"] & 1) != 0  # C_REAL
        # the FP32-force mode keeps no contact points (the first three columns) of two spheres
        kept = c["con_state"][r][:, 3 if self.S.gpu.precision == "fp32" else 0:]
        return c, [c["con_key"][r], c["con_flags"][r], c["con_step0"][r], c["con_cell_dist"][r], kept]


def crowd(nodes):
    """The loose spheres brought together (their boxes overlap many others), and every third pair parted."""
    out = [a.copy() for a in nodes]
    rng = np.random.default_rng(3)
    at = np.stack(np.meshgrid(*[np.arange(8)] * 3, indexing="ij"), -1).reshape(-1, 3)[:LOOSE] * 2.05 * R + [.1, .1, .6]
    out[0][2 * PAIRS:] = at + rng.uniform(-.02 * R, .02 * R, at.shape)
    out[0][1:2 * PAIRS:6] += 3 * R
    return out


def same(a, b):
    for k in a:
        assert np.array_equal(a[k], b[k]), k


def fails_and_goes_on(precision, periodic, cause, read):
    """cause(raw, nodes): makes the next run fail, returns the nodes it may then go on from. False: it did not fail."""
    S = build(precision, periodic)
    raw = Raw(S)
    assert raw.run(4) == 0
    if read:
        raw.contacts()
    nodes = crowd(raw.nodes())
    twin = build(precision, periodic)  # the same steps, never failing
    t = Raw(twin)
    assert t.run(4) == 0
    before, (snap, state) = t.contacts()[1], t.state()
    assert len(before["id_lo"]) == PAIRS and np.any(before["fglob"])
    step = t.sim.clock()[0]
    twin.close()

    mend = cause(raw, nodes)
    r = raw.run(3)
    mend()
    if r == 0:
        S.close()
        return False
    assert raw.sim.clock()[0] == step
    c, real = raw.contacts()
    same(real, before)
    for a, b in zip(raw.state()[1], state):
        assert np.array_equal(a, b)
    assert raw.sim.stats().n_real == PAIRS
    # on from the nodes as they are meant to be, beside a scene restored from the snapshot
    raw.put(nodes)
    T = build(precision, periodic)
    T.step = step
    t = Raw(T)
    t.put(nodes)
    checkpoint.restore_contacts(T, snap)
    for steps in (1, 2, 40):
        assert raw.run(steps) == 0 and t.run(steps) == 0
        if steps == 1:  # the run met real contacts without an overlap, which the merge finds by being repeated
            assert np.all(raw.apart()[::3]) and not np.any(raw.apart()[1::3])
        for a, b, k in zip(raw.nodes(), t.nodes(), KEYS):
            assert np.array_equal(a, b), k
        same(raw.contacts()[1], t.contacts()[1])
    assert raw.sim.clock()[0] == step + 43
    T.close()
    S.close()
    return True


MODES = [("fp32", False), ("fp64", False), ("fp32", True), ("fp64", True)]


@pytest.mark.parametrize("precision,periodic", MODES)
@pytest.mark.parametrize("read", [False, True])
def test_position_that_is_not_finite(precision, periodic, read, gpu_lib):
    def cause(raw, nodes):
        bad = [a.copy() for a in nodes]
        bad[0][-1] = np.inf
        raw.put(bad)
        return lambda: None
    assert fails_and_goes_on(precision, periodic, cause, read)


@pytest.mark.parametrize("precision,periodic", MODES)
def test_no_memory(precision, periodic, gpu_lib):
    """Every allocation of the run fails in turn (the entry that says so hands out no memory; nothing is used up)."""
    k = 0
    while True:
        def cause(raw, nodes):
            raw.put(nodes)
            raw.L.wg_fail_alloc(raw.h, k)
            return lambda: raw.L.wg_fail_alloc(raw.h, -1)
        if not fails_and_goes_on(precision, periodic, cause, False):
            break
        k += 1
    assert k > 20


@pytest.mark.parametrize("precision,periodic", MODES)
def test_no_memory_at_the_first_run(precision, periodic, gpu_lib):
    want = None
    for k in range(-1, 200):
        S = build(precision, periodic)
        raw = Raw(S)
        assert raw.run(0) == 0  # the upload
        start = [np.ascontiguousarray(S.dem._nodes.soa.col(q)) for q in KEYS]
        raw.put(start)
        raw.L.wg_fail_alloc(raw.h, k)
        r = raw.run(5)
        raw.L.wg_fail_alloc(raw.h, -1)
        done = r == 0
        if not done:
            assert raw.contacts()[0]["real"].sum() == 0
            raw.put(start)
            assert raw.run(5) == 0
        got = (raw.nodes(), raw.contacts()[0])
        S.close()
        if k < 0:
            want = got
            continue
        for a, b in zip(got[0], want[0]):
            assert np.array_equal(a, b)
        same(got[1], want[1])
        if done:
            break
    assert k > 25


@pytest.mark.parametrize("precision,periodic", MODES)
def test_goes_on_as_if_it_had_not_failed(precision, periodic, gpu_lib):
    """Failed runs, the first ones of a scene and later ones, and the steps after them beside a scene that never failed."""
    def go(fails):
        S = build(precision, periodic)
        S.trackEnergy = not periodic
        raw = Raw(S)
        assert raw.run(0) == 0
        failed = 0
        for steps, crowded in ((4, False), (3, True), (1, False), (30, False)):
            if crowded:
                raw.put(crowd(raw.nodes()))
            for k in fails:
                raw.L.wg_fail_alloc(raw.h, k)
                failed += raw.run(steps) != 0
                raw.L.wg_fail_alloc(raw.h, -1)
                if raw.sim.clock()[0] == raw.due + steps:
                    break
            rest = raw.due + steps - raw.sim.clock()[0]
            assert raw.run(rest) == 0
            raw.due += steps
        out = (raw.nodes(), raw.contacts()[0], raw.sim.clock()[:2], raw.energy())
        S.close()
        return out, failed
    want, none = go([])
    got, failed = go([0, 7, 3])
    assert none == 0 and failed >= 6
    for a, b in zip(got[0], want[0]):
        assert np.array_equal(a, b)
    same(got[1], want[1])
    assert got[2] == want[2] and np.array_equal(got[3], want[3])


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("scenes_", [1, 3])
def test_failure_among_queued_steps(scenes_, precision, gpu_lib):
    """Spheres fall into a heap; whenever a run needs larger arrays, it first fails: every step, time and DynDt count as if
    it had not, in a scene and in a batch."""
    from woodem_gb300 import scenes
    from woodem_gb300.batch import Batch

    def go(fail):
        mix = []
        for q in range(scenes_):
            S = scenes.box_settle_scaled(500 + 150 * q, 5e-3, seed=q, precision=precision)
            S.engines = utils.defaultEngines(damping=.2, verletDist=-.1, dynDtPeriod=70)
            nd = S.dem._nodes.soa
            nd.col("vel")[6:] = np.random.default_rng(q).uniform(-.3, .3, (len(nd) - 6, 3)) + [0, 0, -1.]
            mix.append(S)
        B = Batch(mix) if scenes_ > 1 else mix[0]._ensure_sim()
        H, step, time = B.H, C.c_int64(), C.c_double()
        done = failed = inside = 0
        while done < 2500:
            if fail:
                H.L.wg_fail_alloc(H.h, 0)
            r = H.L.wg_run(H.h, 2500 - done)
            H.L.wg_fail_alloc(H.h, -1)
            H.check(H.L.wg_get_clock(H.h, 0, C.byref(step), C.byref(time), None, None), "get_clock")
            failed += r != 0
            inside += r != 0 and step.value > done
            done = step.value
            if r:  # once more with memory, up to the next need
                H.check(H.L.wg_run(H.h, min(10, 2500 - done)), "run")
                done += min(10, 2500 - done)
        times = []
        for k in range(scenes_):
            H.check(H.L.wg_get_clock(H.h, k, C.byref(step), C.byref(time), None, None), "get_clock")
            times += [step.value, time.value]
        n = sum(len(S.dem._nodes.soa) for S in mix)
        out = [np.empty((n, w)) for w in (3, 4, 3, 3, 3, 3)]
        H.check(H.L.wg_get_nodes(H.h, *[_native.ptr(a) for a in out]), "get_nodes")
        (B if scenes_ > 1 else mix[0]).close()
        return out, times, failed, inside
    want, got = go(False), go(True)
    assert want[2] == 0 and got[2] >= 3 and got[3] >= 1
    assert got[1] == want[1]
    for a, b in zip(got[0], want[0]):
        assert np.array_equal(a, b)
