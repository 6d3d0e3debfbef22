"""The FP32 test that decides most overlaps of a contact's boxes in a periodic cell (overlapPeriQuick of
csrc/wg_geom.cuh), restated operation by operation: where it decides, the FP64 test says the same."""
import numpy as np
import pytest

from test_oracle_pbc import _overlap_peri

f4 = np.float32


def quick(mn1, mx1, mn2, mx2, size):
    res = 1
    for q in range(3):
        dim, m1, m2 = f4(size[q]), f4(mn1[q]), f4(mn2[q])
        e1, e2 = f4(mx1[q] - mn1[q]) / dim, f4(mx2[q] - mn2[q]) / dim
        d = f4(mn2[q] - mn1[q]) / dim
        lim = f4(1e6) * dim
        if not (abs(m1) < lim and abs(m2) < lim and 1e-4 < e1 < f4(.4) and 1e-4 < e2 < f4(.4)):
            return 2
        f = d - np.rint(d)
        over = e1 - f if f >= 0 else e2 + f
        if not abs(over) > f4(2e-6) * (f4(1) + abs(d)):
            return 2
        if over < 0:
            res = 0
    return res


@pytest.mark.parametrize("kind", ["random", "touching", "far", "same minimum", "half a period", "small boxes"])
def test_decisions_are_exact(kind):
    rng = np.random.default_rng(len(kind))
    size = np.array([1.25, 2.0, 0.75])
    decided = 0
    for _ in range(3000):
        e1, e2 = rng.uniform(.05, .45, 3) * size, rng.uniform(.05, .45, 3) * size
        a = rng.uniform(-3, 3, 3) * size
        d = rng.uniform(-.5, .5, 3) * size
        k = rng.integers(-4, 5, 3) * size
        if kind == "touching":  # within a few roundings of either edge, FP32 and FP64 ones
            edge = np.where(rng.random(3) < .5, e1, -e2)
            d = np.where(rng.random(3) < .6, edge * (1 + rng.choice([0, 1e-16, -3e-16, 1e-9, -1e-7, 3e-6, -3e-6], 3)), .5 * edge)
        elif kind == "far":
            k = rng.integers(-10 ** 5, 10 ** 5, 3) * size
        elif kind == "same minimum":
            d = rng.choice([0., 1e-17, -1e-17, 1e-9, -1e-9], 3)
        elif kind == "half a period":
            d = .5 * size * (1 + rng.choice([0., 1e-16, -1e-16, 1e-8, -1e-8], 3))
        elif kind == "small boxes":
            e1, e2 = e1 * 10. ** rng.uniform(-6, 0, 3), e2 * 10. ** rng.uniform(-6, 0, 3)
            d = rng.choice([-1, 1], 3) * np.maximum(e1, e2) * rng.uniform(0, 1.2, 3)
        mn = np.array([a, a + d + k])
        mx = mn + np.array([e1, e2])
        q = quick(mn[0], mx[0], mn[1], mx[1], size)
        if q == 2:
            continue
        decided += 1
        assert bool(q) == bool(_overlap_peri(mn, mx, 0, 1, size)[0])
    assert decided > 0
