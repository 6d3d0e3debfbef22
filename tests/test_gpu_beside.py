"""Simulations in a run at the same time share the SMs, and large ones go over to a launch per kernel: each ends bitwise
as it does alone, more of them at once than can have their quarter of the SMs, and sizes on both sides of the change."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from woodem_gb300 import scenes

pytestmark = pytest.mark.gpu

KEYS = ("pos", "ori", "vel", "angVel", "force", "torque")


def go(job):
    n, precision, runs, steps = job
    S = scenes.box_settle_scaled(n, 5e-3, seed=n, precision=precision)
    for _ in range(runs):
        S.run(steps)
    S.sync()
    out = [S.dem._nodes.soa.col(k).copy() for k in KEYS]
    S.close()
    return out


@pytest.mark.parametrize("jobs", [
    [(n, p, 10, 60) for n in (65530, 65531, 900, 4000) for p in ("fp64", "fp32")],  # 65 536 nodes with the walls, and one more
    [(400 + 150 * q, ("fp64", "fp32")[q % 2], 20, 100) for q in range(20)],
], ids=["sizes", "many"])
def test_beside_is_alone(jobs, gpu_lib):
    alone = [go(j) for j in jobs]
    with ThreadPoolExecutor(len(jobs)) as ex:
        beside = list(ex.map(go, jobs))
    for a, b in zip(alone, beside):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
