"""overlapPeriQuick of csrc/wg_geom.cuh as compiled, on the host and on the device: where it decides, it says what the
exact test says, about its margins, at any sizes of box, cell and coordinates."""
import numpy as np
import pytest

from woodem_gb300 import _native

from test_oracle_pbc import _overlap_peri

KINDS = ["random", "touching", "margin", "far", "same minimum", "half a period", "small boxes", "limits", "odd"]
SIZE = np.array([1.25, 2.0, 0.75])


def boxes(kind, n, size):
    rng = np.random.default_rng(len(kind))
    e1, e2 = rng.uniform(.05, .45, (n, 3)) * size, rng.uniform(.05, .45, (n, 3)) * size
    a = rng.uniform(-3, 3, (n, 3)) * size
    d = rng.uniform(-.5, .5, (n, 3)) * size
    k = rng.integers(-4, 5, (n, 3)) * size
    edge = np.where(rng.random((n, 3)) < .5, e1, -e2)
    if kind == "touching":  # within a few roundings of either edge
        d = np.where(rng.random((n, 3)) < .6, edge * (1 + rng.choice([0, 1e-16, -3e-16, 1e-9, -1e-7], (n, 3))), .5 * edge)
    elif kind == "margin":  # about the margin of 2e-6 periods
        d = np.where(rng.random((n, 3)) < .6, edge + size * rng.uniform(-6e-6, 6e-6, (n, 3)), .5 * edge)
    elif kind == "far":
        k = rng.integers(-10 ** 5, 10 ** 5, (n, 3)) * size
    elif kind == "same minimum":
        d = rng.choice([0., 1e-17, -1e-17, 1e-9, -1e-9], (n, 3))
    elif kind == "half a period":
        d = .5 * size * (1 + rng.choice([0., 1e-16, -1e-16, 1e-8, -1e-8], (n, 3)))
    elif kind == "small boxes":
        e1, e2 = e1 * 10. ** rng.uniform(-6, 0, (n, 3)), e2 * 10. ** rng.uniform(-6, 0, (n, 3))
        d = rng.choice([-1, 1], (n, 3)) * np.maximum(e1, e2) * rng.uniform(0, 1.2, (n, 3))
    elif kind == "limits":  # boxes about 1e-4 and 0.4 periods, minima about 1e6 periods away
        e1 = size * np.where(rng.random((n, 3)) < .5, 1e-4, .4) * (1 + rng.uniform(-1e-6, 1e-6, (n, 3)))
        a = rng.choice([-1, 1, 0], (n, 3)) * 1e6 * size * (1 + rng.uniform(-1e-6, 1e-6, (n, 3)))
        k = rng.integers(-2, 3, (n, 3)) * size
    mn = np.stack([a, a + d + k], 1)
    mx = mn + np.stack([e1, e2], 1)
    if kind == "odd":  # what no scene has: not decided
        mx[::3, 0] = np.array([np.inf, np.nan, -1e300])
        mn[1::3, 1] = np.nan
        mn[2::3], mx[2::3] = 1e38 * mn[2::3], 1e38 * mx[2::3]
    return np.ascontiguousarray(mn), np.ascontiguousarray(mx)


def decide(mn, mx, size, device):
    n = len(mn)
    q, e = np.full(n, -7, np.int32), np.full(n, -7, np.int32)
    P, I = _native.ptr, _native.P_I32
    r = _native.lib().wg_selftest_overlap(n, P(mn), P(mx), P(size), P(q, I), P(e if device else None, I))
    assert r == 0
    return q, e


@pytest.mark.parametrize("scale", [1., 1e-3, 1e5])
@pytest.mark.parametrize("kind", KINDS)
def test_on_the_host(kind, scale, gpu_lib):
    size = SIZE * scale
    mn, mx = boxes(kind, 2000, size)
    q, _ = decide(mn, mx, size, False)
    if kind == "odd":
        assert np.all(q == 2)
        return
    for i in np.nonzero(q != 2)[0]:
        assert bool(q[i]) == bool(_overlap_peri(mn[i], mx[i], 0, 1, size)[0])
    assert np.any(q != 2) or kind in ("same minimum", "touching")
    # a cell too small or too large for FP32 numbers: nothing is decided
    for s in (1e-31, 1e31):
        assert np.all(decide(mn, mx, SIZE * s, False)[0] == 2)


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1., 1e-3, 1e5])
@pytest.mark.parametrize("kind", KINDS)
def test_on_the_device(kind, scale, gpu_lib):
    size = SIZE * scale
    mn, mx = boxes(kind, 400001, size)
    q, e = decide(mn, mx, size, True)
    if kind == "odd":
        assert np.all(q == 2)
        return
    d = q != 2
    assert np.array_equal(q[d], e[d])
    assert kind != "random" or (np.mean(d) > .3 and 0 < np.mean(q[d]) < 1)
