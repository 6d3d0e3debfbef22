"""What the host is told about a device scene, by the shorter ways: the clock of a scene against its
statistics, contacts counted on the device against their list, and the state of many nodes copied in
pieces by several threads against single copies."""
import ctypes as C

import numpy as np
import pytest

from woodem_gb300 import _native, scenes
from woodem_gb300.batch import Batch

pytestmark = pytest.mark.gpu


def _counts(sim):
    st, c = sim.stats(), sim.contacts()
    assert st.n_real == int(np.count_nonzero(c["real"]))
    assert st.n_contacts == len(c["real"])
    return st


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("periodic", [False, True])
def test_clock_and_counts(precision, periodic, gpu_lib):
    if periodic:
        S = scenes.periodic_shear(n=400, seed=21, fill_fraction=0.4, shear_rate=0.0, precision=precision)
        S.cell.nextGradV = -10.0 * np.eye(3)
    else:
        S = scenes.box_settle_small(n=700, seed=5, precision=precision)
    for steps in (1, 400 if periodic else 12000, 1):
        S.run(steps)
        st = _counts(S._sim)
        step, time, full, stress = S._sim.clock()
        assert (step, time, full) == (st.step, st.time, st.n_full_runs) == (S.step, st.time, st.n_full_runs)
        assert np.array_equal(stress, np.array(st.stress))
    assert st.n_contacts > 50
    assert periodic or st.n_real > 50
    S.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_clocks_of_a_batch(precision, gpu_lib):
    mix, _ = scenes.batch_study(n_scenes=3, seed=7, nmin=300, nmax=700, precision=precision)
    B = Batch(mix)
    B.run(6000)
    step, time = C.c_int64(), C.c_double()
    total = 0
    for k, S in enumerate(mix):
        st, c = B.scene_stats(k), B.contacts(k)
        B.H.check(B.H.L.wg_get_clock(B.H.h, k, C.byref(step), C.byref(time), None, None), "get_clock")
        assert (step.value, time.value) == (st.step, st.time) == (S.step, S.time)
        assert st.n_real == int(np.count_nonzero(c["real"]))
        total += st.n_real
    assert total > 20
    for k in (-1, len(mix)):
        assert B.H.L.wg_get_clock(B.H.h, k, C.byref(step), C.byref(time), None, None) != 0
    B.close()


@pytest.mark.parametrize("n", [27000, 90000])  # 4.1 and 13.7 MB in all: one piece an array, then two
def test_state_in_pieces_is_the_state(n, gpu_lib):
    S = scenes.box_settle_scaled(n, 2e-3, seed=3)
    S.run(2)
    S.sync()
    nd = S.dem._nodes.soa
    m = len(nd)
    one = {}
    for q, (k, w) in enumerate((("pos", 3), ("ori", 4), ("vel", 3), ("angVel", 3), ("force", 3), ("torque", 3))):
        a = np.empty((m, w))
        args = [None] * 6
        args[q] = _native.ptr(a)
        S._sim.H.check(S._sim.H.L.wg_get_nodes(S._sim.H.h, *args), "get_nodes")
        one[k] = a
    for k, a in one.items():
        assert np.array_equal(a, nd.col(k)), k
    assert np.any(one["vel"])
    S.close()
