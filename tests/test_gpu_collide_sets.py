"""Collider runs whose result is not the ordinary one: real contacts whose boxes no longer overlap (spheres
that part by more than the verlet distance in one step, a law that keeps contacts, no verlet distance), sets
that come and go empty, and the sphere-sphere records that go from one packed set to the next."""
import numpy as np
import pytest

from woodem_gb300 import _plan, scenes, utils
from woodem_gb300.batch import Batch

from test_gpu_parity import _run_pair

pytestmark = pytest.mark.gpu


def fast_box(n=300, verletRel=1e-3, noBreak=False, precision="fp64", speed=1.5, seed=4):
    S = scenes.box_settle_small(n=n, seed=seed, precision=precision)
    S.engines = utils.defaultEngines(damping=.1, verletDist=-verletRel, dynDtPeriod=0, noBreak=noBreak)
    nd = S.dem._nodes.soa
    v = np.random.default_rng(seed).uniform(-speed, speed, (n, 3))
    nd.col("vel")[-n:] = v
    return S


@pytest.mark.parametrize("verletRel,noBreak", [(1e-3, False), (0.0, False), (0.005, True), (0.0, True)])
def test_parting_contacts_are_the_oracles(verletRel, noBreak, gpu_lib):
    S = fast_box(verletRel=verletRel, noBreak=noBreak)
    _run_pair(S, 12, 25)
    S.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n", [1, 2, 300])
def test_lists_between_runs(n, precision, gpu_lib):
    """Contacts read back between the steps (from the packed records, then from their columns) change nothing."""
    out = []
    for read in (False, True):
        S = fast_box(n, 1e-2, precision=precision)
        S.run(1)
        for _ in range(60):
            if read:
                c = S._sim.contacts()
                assert len(c["real"]) == S._sim.stats().n_contacts
            S.run(5)
        S.sync()
        nd = S.dem._nodes.soa
        c = S._sim.contacts()
        out.append([nd.col(k).copy() for k in ("pos", "vel", "angVel", "force", "torque")] + [c[k] for k in sorted(c)])
        S.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_scenes_of_very_different_sizes(precision, gpu_lib):
    """A grid of its own for each scene: 1, 2, 40 and 400 spheres of different radii in one batch."""
    def build():
        out = [scenes.box_settle_scaled(n, r, seed=n, precision=precision) for n, r in ((1, 5e-3), (400, 2e-3), (2, 9e-3), (40, 6e-3))]
        for S in out:
            nd = S.dem._nodes.soa
            nd.col("vel")[6:] = np.random.default_rng(3).uniform(-1, 1, (len(nd) - 6, 3))
        return out
    mix = build()
    B = Batch(mix)
    B.run(600)
    B.pull()
    lists = [B.contacts(k) for k in range(len(mix))]
    B.close()
    for S, T, c in zip(build(), mix, lists):
        S.run(600)
        S.sync()
        real = S._sim.contacts()
        r = real["real"] != 0
        q = c["real"] != 0
        assert np.array_equal(real["id_lo"][r], c["id_lo"][q]) and np.array_equal(real["id_hi"][r], c["id_hi"][q])
        for k in ("pos", "vel", "angVel"):
            assert np.array_equal(S.dem._nodes.soa.col(k), T.dem._nodes.soa.col(k)), k
        S.close()
