"""The quotients of csrc/wg_div.cuh as compiled: bit for bit those of a division, inside the exponent range of the
short way, at its ends and outside, for zeros of either sign, subnormal numbers, infinities and NaN."""
import numpy as np
import pytest

from woodem_gb300 import _native

pytestmark = pytest.mark.gpu


def numbers(rng, shape, kind):
    m = rng.uniform(1, 2, shape) * rng.choice([-1., 1.], shape)
    if kind == "near a power of two":
        m = np.where(rng.random(shape) < .5, 2. - rng.integers(1, 200, shape) * 2. ** -52, 1. + rng.integers(0, 200, shape) * 2. ** -52)
    if kind == "ends":
        return np.ldexp(m, rng.choice([-503, -502, -501, -500, -499, 0, 498, 499, 500, 501, 502, 503], shape))
    if kind == "all":
        x = rng.integers(0, 2 ** 64, shape, dtype=np.uint64).view(np.float64)
        odd = np.array([0., -0., 5e-324, -5e-324, 2. ** -1022, np.inf, -np.inf, np.nan, 1., -1.])
        return np.where(rng.random(shape) < .2, rng.choice(odd, shape), x)
    if kind == "zeros":
        return np.where(rng.random(shape) < .5, rng.choice([0., -0.], shape), m)
    return np.ldexp(m, rng.integers(-60, 60, shape))


def same(got, want):
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got.view(np.int64)[~nan], want.view(np.int64)[~nan])


@pytest.mark.parametrize("kind", ["random", "near a power of two", "quotient near one", "ends", "all", "zeros"])
def test_bitwise(kind, gpu_lib):
    rng = np.random.default_rng(len(kind))
    n = 1000003
    a, b = numbers(rng, (n, 3), kind), numbers(rng, (n, 3), kind)
    if kind == "quotient near one":
        a = b + np.spacing(b) * rng.integers(-8, 9, (n, 3))
    if kind != "all":
        b = np.abs(b)
    a, b, out = np.ascontiguousarray(a), np.ascontiguousarray(b), np.empty((n, 13))
    with np.errstate(all="ignore"):
        z = np.where(b != 0, 1. / b, 0.)  # as the scene's nodes keep it
        P = _native.ptr
        assert _native.lib().wg_selftest_quotients(n, P(a), P(b), P(np.ascontiguousarray(z)), P(out)) == 0
        same(out[:, :3].copy(), a / b[:, :1])
        same(out[:, 3:6].copy(), a / b)
        sq = (a[:, 0] * a[:, 0] + a[:, 1] * a[:, 1]) + a[:, 2] * a[:, 2]
        same(out[:, 6:9].copy(), np.where(sq[:, None] > 0, a / np.sqrt(sq)[:, None], a))
        w = b[:, 0]
        nrm = np.sqrt(((a[:, 0] * a[:, 0] + a[:, 1] * a[:, 1]) + a[:, 2] * a[:, 2]) + w * w)
        same(out[:, 9:].copy(), np.stack([w, a[:, 0], a[:, 1], a[:, 2]], 1) / nrm[:, None])
