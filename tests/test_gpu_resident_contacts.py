"""The resident grid that walks facet, wall and packed sphere-sphere contacts together, against one contact
per thread: bitwise the same at the edges of its chunks (32) and of the packed tiles (1024), with real and
other contacts mixed, with no mixed contacts and with as many as spheres."""
import numpy as np
import pytest

from woodem_gb300 import tune, utils
from woodem_gb300.core import Scene
from woodem_gb300.dem import DemField, FrictMat

pytestmark = pytest.mark.gpu

R = 5e-3


def chain(n, wall):
    """n spheres along x, n - 1 potential contacts, two of three of them overlapping; with ``wall`` each
    sphere also presses on one plane."""
    rng = np.random.default_rng(n)
    gap = np.where(np.arange(n - 1) % 3 == 2, 2.15 * R, 1.98 * R)
    x = np.concatenate([[0.], np.cumsum(gap)])
    c = np.stack([x, rng.uniform(-1e-5, 1e-5, n), np.full(n, 0.9999 * R)], 1)
    S = Scene(fields=[DemField(gravity=(0, 0, -9.81) if wall else (0, 0, 0))])
    S.gpu.precision = "fp32"
    mat = FrictMat(density=3000., young=1e7, ktDivKn=.2, tanPhi=.5)
    if wall:
        S.dem.par.add(utils.wall(0., axis=2, sense=1, mat=mat))
    S.dem.par.addSpheres(c, R, mat)
    nd = S.dem._nodes.soa
    nd.col("angVel")[-n:] = rng.uniform(-5, 5, (n, 3))
    nd.col("vel")[-n:] = rng.uniform(-.01, .01, (n, 3))
    S.engines = utils.defaultEngines(damping=.1, verletDist=-.1, dynDtPeriod=0)
    S.dt = .2 * utils.pWaveDt(S)
    return S


@pytest.mark.parametrize("wall", [False, True])
@pytest.mark.parametrize("n", [2, 33, 34, 1024, 1025, 1026, 2050, 30000])
def test_resident_grid_is_one_thread_a_contact(n, wall, gpu_lib):
    out = []
    for block, graph in ((256, False), (-256, True)):  # as a graph: one launch per kernel at every size
        S = chain(n, wall)
        S.run(1)
        tune.set_launch(S._sim, block, 2, graph)
        S.run(12)
        S.sync()
        c = S._sim.contacts()
        out.append([S.dem._nodes.soa.col(k).copy() for k in ("pos", "vel", "angVel", "force", "torque")] + [c[k] for k in sorted(c)])
        assert len(c["real"]) >= n - 1 and (n == 2 or 0 < np.count_nonzero(c["real"]) < len(c["real"]))
        S.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
