"""Small scenes run many steps in one launch; a contact block size set by the caller runs them as a launch
per kernel. Both end bitwise the same: part warps of nodes and contacts, walls, facets that stand or turn,
a periodic cell, several scenes, and runs that end a launch at every step (no verlet distance)."""
import numpy as np
import pytest

from woodem_gb300 import scenes, tune
from woodem_gb300.batch import Batch

pytestmark = pytest.mark.gpu

KEYS = ("pos", "ori", "vel", "angVel", "force", "torque")


def _box(n, verletRel=0.1):
    return lambda p: scenes.box_settle_scaled(n, 5e-3, seed=n, verletRel=verletRel, precision=p)


def _peri(p):
    S = scenes.periodic_shear(n=333, seed=21, fill_fraction=0.4, shear_rate=0.0, precision=p)
    g = -40.0 * np.eye(3)
    g[0, 2] = 20.0
    S.cell.nextGradV = g
    return S


BUILD = {
    "one": (_box(1), 300),
    "warp": (_box(26), 3000),  # 26 spheres and 6 walls: 32 nodes
    "warp+1": (_box(27), 3000),
    "part": (_box(700), 3000),
    "many": (_box(100003), 40),
    "no verlet": (_box(100, 0.0), 3000),
    "periodic": (_peri, 300),
    "drum": (lambda p: scenes.hertz_drum(n=1500, seed=2, diameter=0.3, length=0.12, div=31, axDiv=6, fill_fraction=0.3, precision=p), 300),
}


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("kind", sorted(BUILD))
def test_one_launch_is_many(kind, precision, gpu_lib):
    build, steps = BUILD[kind]
    out = []
    for block in (0, 128):
        S = build(precision)
        S.run(1)
        tune.set_launch(S._sim, block, 32)
        S.run(steps)
        st = S._sim.stats()
        S.sync()
        nd = S.dem._nodes.soa
        out.append(({k: nd.col(k).copy() for k in KEYS}, S.step, st.n_full_runs, st.n_contacts, st.n_real))
        S.close()
    for k in KEYS:
        assert np.array_equal(out[0][0][k], out[1][0][k]), k
    assert out[0][1:] == out[1][1:]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_one_launch_is_many_in_a_batch(precision, gpu_lib):
    out = []
    for block in (0, 128):
        mix, _ = scenes.batch_study(n_scenes=4, seed=9, nmin=1, nmax=600, precision=precision)
        B = Batch(mix)
        B.run(1)
        tune.set_launch(B, block, 32)
        B.run(3000)
        B.pull()
        out.append([[S.dem._nodes.soa.col(k).copy() for k in KEYS] for S in mix])
        B.close()
    for a, b in zip(*out):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)


def test_simulations_side_by_side(gpu_lib):
    """Scenes of both precisions in threads of their own, each launch with a grid barrier beside the others'."""
    from concurrent.futures import ThreadPoolExecutor
    jobs = [(n, p) for n in (700, 4000, 26) for p in ("fp64", "fp32")]

    def go(job):
        S = scenes.box_settle_scaled(job[0], 5e-3, seed=job[0], precision=job[1])
        for _ in range(20):
            S.run(100)
        S.sync()
        out = [S.dem._nodes.soa.col(k).copy() for k in KEYS]
        S.close()
        return out
    alone = [go(j) for j in jobs]
    with ThreadPoolExecutor(len(jobs)) as ex:
        beside = list(ex.map(go, jobs))
    for a, b in zip(alone, beside):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
