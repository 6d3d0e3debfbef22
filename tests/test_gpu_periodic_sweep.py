"""The periodic broad phase against the exact overlap test pair by pair: cells of 1 to 7 grid cells per
axis, spheres on and across the boundary and several periods away, and positions on a lattice whose
boxes touch exactly (the FP32 fractions of the sweep cannot decide those: they go to the FP64 test)."""
import numpy as np
import pytest

from woodem_gb300 import _native, _plan, utils
from woodem_gb300.core import Cell, Scene
from woodem_gb300.dem import DemField, FrictMat

from test_oracle_pbc import _overlap_peri

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1.25, 1.25, 1.25), (1.25, 2.0, 3.5), (1.0625, 1.5, 1.75), (0.9, 3.5, 1.3)])
@pytest.mark.parametrize("lattice", [True, False])
@pytest.mark.parametrize("shear", [0.0, 0.21])
def test_pairs_are_the_exact_overlaps(size, lattice, shear, gpu_lib):
    if lattice and (shear or min(size) < 1.0):
        pytest.skip("sheared edges are not exact, and boxes of half the cell raise an error")
    rng = np.random.default_rng(int(100 * sum(size)) + lattice)
    n = 150
    r = np.full(n, 0.25) if lattice else rng.uniform(0.08, 0.2, n)
    c = rng.integers(-24, 40, (n, 3)) / 8.0 if lattice else rng.uniform(-3.0, 5.0, (n, 3))
    S = Scene(fields=[DemField()])
    S.periodic = True
    S.cell.setBox(*size)
    if shear:
        h = np.array(S.cell.hSize)
        h[0, 2] = shear * size[0]
        S.cell.hSize = h
    S.cell.homoDeform = Cell.HomoNone
    S.dem.par.addSpheres(c, r, FrictMat(density=1e3, young=1e7, ktDivKn=.2, tanPhi=.5))
    S.engines = utils.defaultEngines(verletDist=0.0, dynDtPeriod=0)
    S.dt = 1e-9
    sim = S._ensure_sim()
    L, h = sim.H.L, sim.H.h
    mn, mx = np.empty((n, 3)), np.empty((n, 3))
    sim.H.check(L.wg_collide_only(h), "collide_only")
    sim.H.check(L.wg_get_aabbs(h, _native.ptr(mn), _native.ptr(mx)), "get_aabbs")
    got = _plan.read_contacts(L, h, "wg")
    edges = np.linalg.norm(np.asarray(S.cell.hSize, float), axis=0)
    want = {}
    for a in range(n):
        for b in range(a + 1, n):
            ok, per = _overlap_peri(mn, mx, a, b, edges)
            if ok:
                want[(a, b)] = tuple(per)
    assert len(want) > 50
    assert {(int(a), int(b)): tuple(int(v) for v in d) for a, b, d in zip(got["id_lo"], got["id_hi"], got["cell_dist"])} == want
    S.close()
