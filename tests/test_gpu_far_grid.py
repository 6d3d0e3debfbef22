"""The broad phase far from the origin: the cells are as long as the largest box wherever the scene stands (a number
of cells makes them longer only), and the pairs are those of the boxes."""
import ctypes as C

import numpy as np
import pytest

from woodem_gb300 import _native, _plan, scenes, utils
from woodem_gb300.core import Scene
from woodem_gb300.dem import DemField, FrictMat

from helpers import brute_force_pairs

pytestmark = pytest.mark.gpu


def spheres(n):
    rng = np.random.default_rng(n)
    S = Scene(fields=[DemField(gravity=(0, 0, 0))])
    S.dem.par.addSpheres(rng.uniform(0, 9 * n ** (1 / 3), (n, 3)) * 1e-3, rng.uniform(3e-3, 5e-3, n),
                         FrictMat(density=3000., young=1e7, ktDivKn=.2, tanPhi=.5))
    S.engines = utils.defaultEngines(verletDist=-.1, dynDtPeriod=0)
    S.dt = 1e-9
    return S


def collide(S):
    """The boxes, the pairs found and the grid (edge, cells per axis)."""
    A = _plan.compile_scene(S)
    sim = S._ensure_sim()
    L, h = sim.H.L, sim.H.h
    sim.H.check(L.wg_collide_only(h), "collide_only")
    n = A.n_particles
    mn, mx = np.empty((n, 3)), np.empty((n, 3))
    sim.H.check(L.wg_get_aabbs(h, _native.ptr(mn), _native.ptr(mx)), "get_aabbs")
    c = _plan.read_contacts(L, h, "wg")
    org, edge, dims = np.empty(3), C.c_double(), np.empty(3, np.int32)
    sim.H.check(L.wg_get_grid(h, 0, _native.ptr(org), C.byref(edge), _native.ptr(dims, _native.P_I32)), "get_grid")
    got = set(zip(c["id_lo"].tolist(), c["id_hi"].tolist()))
    assert got == brute_force_pairs(A, mn, mx) and len(got) > 0
    ball = A.particles["shape"] == 0
    assert np.array_equal(org, mn[ball].min(0))
    out = mn[ball], mx[ball], edge.value, dims
    S.close()
    return out


@pytest.mark.parametrize("kind", ["spheres", "drum"])
@pytest.mark.parametrize("offset", [0., 1e2, 1e4, 1e6, -1e6, 1e9])
def test_cells_are_the_largest_box(kind, offset, gpu_lib):
    S = spheres(1500) if kind == "spheres" else scenes.hertz_drum(n=1500, seed=2, diameter=0.3, length=0.12, div=31, axDiv=6,
                                                                  fill_fraction=0.3)
    S.dem._nodes.soa.col("pos")[:] += offset * np.array([1., -.7, .3])
    mn, mx, edge, dims = collide(S)
    assert np.prod(dims.astype(float)) < 2 ** 15  # not so many that the cells were made longer
    assert np.max(mx - mn) <= edge <= 1.00001 * np.max(mx - mn)


@pytest.mark.parametrize("at", [1e7, 1e20, 1e38, 1e39, 1e300])
def test_one_sphere_far_away(at, gpu_lib):
    """Its neighbours are found, and it is no error past the range of FP32 numbers."""
    S = spheres(300)
    S.dem._nodes.soa.col("pos")[7] = (at, -.5 * at, 0.)
    collide(S)


def test_one_scene_of_a_batch_far_away(gpu_lib):
    """Its pairs and those of the others are what each scene has alone."""
    from woodem_gb300.batch import Batch
    from woodem_gb300 import _plan
    at = (0., 1e6, 3.)
    pairs = []
    for q in at:
        S = spheres(400)
        S.dem._nodes.soa.col("pos")[:] += q
        sim = S._ensure_sim()
        sim.H.check(sim.H.L.wg_collide_only(sim.H.h), "collide_only")
        c = _plan.read_contacts(sim.H.L, sim.H.h, "wg")
        pairs.append((c["id_lo"], c["id_hi"]))
        S.close()
    mix = [spheres(400) for _ in at]
    for S, q in zip(mix, at):
        S.dem._nodes.soa.col("pos")[:] += q
    B = Batch(mix)
    B.H.check(B.H.L.wg_collide_only(B.H.h), "collide_only")
    for k, (lo, hi) in enumerate(pairs):
        c = B.contacts(k)
        assert len(lo) > 100 and np.array_equal(c["id_lo"], lo) and np.array_equal(c["id_hi"], hi)
    B.close()
