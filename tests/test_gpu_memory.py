"""Device memory of a scene whose potential contacts are mostly dormant: what only active contacts use (their packed
state, 80 bytes twice, and their two ends, 24 bytes each) is not held for all of them."""
import numpy as np
import pytest

from woodem_gb300 import utils
from woodem_gb300.core import Scene
from woodem_gb300.dem import DemField, FrictMat

pytestmark = pytest.mark.gpu


def test_packed_state_is_sized_by_active_contacts(gpu_lib):
    torch = pytest.importorskip("torch")
    torch.zeros(1, device="cuda")
    r, k = 5e-3, 46
    c = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3) * 2.05 * r
    S = Scene(fields=[DemField(gravity=(0, 0, 0))])
    S.gpu.precision = "fp32"
    S.dem.par.addSpheres(c, r, FrictMat(density=3000., young=1e7, ktDivKn=.2, tanPhi=.5))
    # boxes of 2.8 r: 26 neighbours overlap, of which the 6 nearest are within 2 verletDist (0.8 r) of touching
    S.engines = utils.defaultEngines(verletDist=-.4, dynDtPeriod=0)
    S.dt = 1e-9
    sim = S._ensure_sim()
    sim.H.check(sim.H.L.wg_run(sim.H.h, 0), "run")  # the upload
    before = torch.cuda.mem_get_info()[0]
    S.run(2)
    used = before - torch.cuda.mem_get_info()[0]
    n = sim.stats().n_contacts
    near = 3 * k * k * (k - 1)
    assert n > 12 * k ** 3 and near < n / 4
    S.close()
    # two sets of contacts (key, flags, step, cell distance, 5 FP64 and 11 FP32 columns: 104 bytes) with half as many
    # again, less the first arrays (6 a particle), pairs twice (8), keys, lists, slots, counts and items (52, half
    # as many again), places (4, half as many again), packed places (8), sort scratch (10, half as many again)
    rest = 2 * 104 * 1.5 * n - 2 * 104 * 6 * k ** 3 + (2 * 8 + 52 * 1.5 + 4 * 1.5 + 8 + 10 * 1.5) * n
    active = near * 1.25 * (2 * 80 + 2 * 24)
    assert used < rest + active + (64 << 20)  # 64 MB for the sphere grid, granularity and the rest
    assert n * 1.25 * (2 * 80 + 2 * 24) > active + (2 * 64 << 20)  # what all contacts would take stands out
