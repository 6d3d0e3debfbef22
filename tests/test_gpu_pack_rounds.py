"""The device packer against its own rules restated on the host: rounds over a window of unplaced
spheres, bit for bit (the batches of rounds that the device tests at once change nothing)."""
import numpy as np
import pytest

from woodem_gb300 import _native

pytestmark = pytest.mark.gpu
M = (1 << 64) - 1


def _mix(z):
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _uni(seed, i, a, k):
    i, a = i.astype(np.uint64), a.astype(np.uint64)
    h = _mix(np.uint64(seed) ^ _mix(i * np.uint64(0x9E3779B97F4A7C15) + np.uint64(0x632BE59BD9B4E019)) ^
             _mix(a * np.uint64(0xD1B54A32D192ED03) + np.uint64((k * 0x8CB92BA72F3D8DD7 + 1) & M)))
    return (h >> np.uint64(11)).astype(float) * (1.0 / 9007199254740992.0)


def _clash(c, r, p, q, L, peri):
    """Pairs (rows of c, rows of p) that overlap."""
    d2 = np.zeros((len(c), len(p)))
    for k in range(3):
        d = c[:, None, k] - p[None, :, k]
        if peri:
            d = d - L[k] * np.rint(d / L[k])
        d2 = d2 + d * d
    rr = r[:, None] + q[None, :]
    return d2 < rr * rr


def _host(radii, lo, hi, kind, cyl, seed, most):
    n = len(radii)
    L, peri = hi - lo, kind == 2
    state, att = np.zeros(n, int), np.zeros(n, np.int64)
    pos = np.zeros((n, 3))
    W = min(32768, max(256, n // 64))
    w0 = 0
    while True:
        while w0 < n and state[w0] == 1:
            w0 += 1
        if w0 == n or state[w0] == 2:
            return w0, pos
        w1 = min(n, w0 + W)
        for _ in range(16):
            u = w0 + np.nonzero(state[w0:w1] == 0)[0]
            if not len(u):
                break
            r = radii[u]
            m = 0.0 if peri else r
            c = np.stack([(lo[k] + m) + _uni(seed, u, att[u], k) * (L[k] - 2 * m) for k in range(3)], axis=1)
            ok = np.ones(len(u), bool)
            if kind == 1:
                dy, dz = c[:, 1] - cyl[0], c[:, 2] - cyl[1]
                ok = ~(np.sqrt(dy * dy + dz * dz) > cyl[2] - r) & ~(c[:, 2] + r > cyl[3])
            done = np.nonzero(state == 1)[0]
            ok &= ~_clash(c, r, pos[done], radii[done], L, peri).any(1)
            lower = np.tril(_clash(c, r, c, r, L, peri) & ok[None, :], -1).any(1)
            take = ok & ~lower
            pos[u[take]] = c[take]
            state[u[take]] = 1
            rest = u[~take]
            att[rest] += 1
            state[rest[att[rest] >= most]] = 2


@pytest.mark.parametrize("n,kind,fill,most", [(1, 2, 0.1, 50), (257, 0, 0.2, 400), (700, 2, 0.33, 2000), (500, 1, 0.1, 4000), (600, 2, 0.5, 100)])
def test_device_rounds(n, kind, fill, most, gpu_lib):
    rng = np.random.default_rng(n)
    radii = np.sort(rng.uniform(2e-3, 4e-3, n))[::-1].copy()
    side = (4 / 3 * np.pi * np.sum(radii ** 3) / fill) ** (1 / 3)
    lo, hi = np.zeros(3), np.full(3, max(side, 0.01))
    cyl = np.array([hi[1] / 2, hi[2] / 2, hi[1] / 2, 0.9 * hi[2]])
    out = np.zeros((n, 3))
    p = _native.ptr
    got = _native.lib().wg_pack_rsa_device(n, p(radii), p(lo), p(hi), kind, p(cyl), 12345, most, p(out))
    want, pos = _host(radii, lo, hi, kind, cyl, 12345, most)
    assert got == want and (fill < 0.5) == (want == n)
    assert np.array_equal(out[:want], pos[:want])
