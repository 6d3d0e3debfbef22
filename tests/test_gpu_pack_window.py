"""The device packer's windows of more than 1024 unplaced spheres (over 65 536 in all), which are gone through round by
round, and the change from those to batches of rounds: against the rules restated on the host, bit for bit."""
import numpy as np
import pytest

from woodem_gb300 import _native

from test_gpu_pack_rounds import _clash, _uni

pytestmark = pytest.mark.gpu


def _near(tree, pos, radii, c, r, lo, L, rmax, peri):
    """Rows of c that overlap a sphere of the tree (whose spheres are pos, radii)."""
    hit = np.zeros(len(c), bool)
    for q, js in enumerate(tree.query_ball_point(c - lo, r + rmax * (1 + 1e-9))):
        if js:
            hit[q] = _clash(c[q:q + 1], r[q:q + 1], pos[js], radii[js], L, peri).any()
    return hit


def _host(radii, lo, hi, kind, seed, most):
    from scipy.spatial import cKDTree
    n, L, peri, rmax = len(radii), hi - lo, kind == 2, radii.max()
    state, att, pos = np.zeros(n, int), np.zeros(n, np.int64), np.zeros((n, 3))
    W, w0, rounds = min(32768, max(256, n // 64)), 0, 0
    while True:
        while w0 < n and state[w0] == 1:
            w0 += 1
        if w0 == n or state[w0] == 2:
            return w0, pos, rounds
        w1 = min(n, w0 + W)
        old = np.nonzero(state == 1)[0]
        tree = cKDTree((pos[old] - lo) % L if peri else pos[old] - lo, boxsize=L if peri else None) if len(old) else None
        rounds += np.count_nonzero(state[w0:w1] == 0) > 1024
        for _ in range(16):
            u = w0 + np.nonzero(state[w0:w1] == 0)[0]
            if not len(u):
                break
            r = radii[u]
            m = 0.0 if peri else r
            c = np.stack([(lo[k] + m) + _uni(seed, u, att[u], k) * (L[k] - 2 * m) for k in range(3)], axis=1)
            ok = np.ones(len(u), bool)
            if tree is not None:
                ok &= ~_near(tree, pos[old], radii[old], c, r, lo, L, rmax, peri)
            new = w0 + np.nonzero(state[w0:w1] == 1)[0]
            new = new[~np.isin(new, old)]
            if len(new):
                ok &= ~_clash(c, r, pos[new], radii[new], L, peri).any(1)
            lower = np.tril(_clash(c, r, c, r, L, peri) & ok[None, :], -1).any(1)
            take = ok & ~lower
            pos[u[take]] = c[take]
            state[u[take]] = 1
            rest = u[~take]
            att[rest] += 1
            state[rest[att[rest] >= most]] = 2


@pytest.mark.parametrize("kind", [0, 2])
def test_wide_windows(kind, gpu_lib):
    pytest.importorskip("scipy")
    n, fill = 70000, 0.2
    rng = np.random.default_rng(n + kind)
    radii = np.sort(rng.uniform(2e-3, 4e-3, n))[::-1].copy()
    side = (4 / 3 * np.pi * np.sum(radii ** 3) / fill) ** (1 / 3)
    lo, hi = np.zeros(3), np.full(3, side)
    cyl, out = np.zeros(4), np.zeros((n, 3))
    p = _native.ptr
    got = _native.lib().wg_pack_rsa_device(n, p(radii), p(lo), p(hi), kind, p(cyl), 12345, 2000, p(out))
    want, pos, wide = _host(radii, lo, hi, kind, 12345, 2000)
    assert wide > 10  # windows of the old kind were met, and between them batches for the stragglers
    assert got == want == n
    assert np.array_equal(out, pos)
