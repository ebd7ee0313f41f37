"""Closest and any hits of rays on which a box test goes wrong first: axis-
aligned directions (zero and negative-zero components), components below the
reciprocal's clamp, directions of very different lengths, origins on the
walls and edges, and geometry far from the coordinate origin.  The reference
tests every triangle with the published watertight test (Woop, Benthin, Wald
2013; the kx / ky swap included), each operation rounded to float32, so
primitive ids, barycentrics and t must agree bit for bit."""
import numpy as np
import pytest

import oracle
from helpers import edge_targets, seeded_rays
from vision_b200 import scenes

pytestmark = pytest.mark.gpu


def _rays(pos, idx, lo, hi, n, seed):
    rng = np.random.default_rng(seed)
    rays = seeded_rays(n, lo, hi, seed, targets=edge_targets(pos, idx))
    d, k = rays[:, 4:7], n // 8
    # One or two components zero (of either sign) or below the clamp.
    tiny = np.array([0.0, -0.0, 1e-35, -1e-35, 1e-30, -3e-31], np.float32)
    for a in range(3):
        rows = rng.random(n) < 0.25
        d[rows, a] = rng.choice(tiny, rows.sum())
    dead = np.abs(d).max(1) < 1e-6
    d[dead, 0] = 1.0
    # Lengths from 1e-4 to 1e4.
    d *= (10.0 ** rng.uniform(-4, 4, (n, 1))).astype(np.float32)
    # Origins exactly on vertices and edge midpoints.
    tg = edge_targets(pos, idx)
    rays[:k, 0:3] = tg[rng.integers(0, len(tg), k)]
    return rays


def _brute_force(tris, rays):
    """(prim, u, v, t) of the closest hits: ties in t to the lower primitive."""
    f = np.float32
    n = rays.shape[0]
    prim = np.full(n, 0xffffffff, np.uint32)
    uvt = np.zeros((n, 3), f)
    with np.errstate(all='ignore'):
        for i in range(0, n, 512):
            o, d, tmax = rays[i:i + 512, 0:3], rays[i:i + 512, 4:7], rays[i:i + 512, 7:8]
            a = np.abs(d)
            kz = np.where(a[:, 0] > a[:, 1], np.where(a[:, 0] > a[:, 2], 0, 2), np.where(a[:, 1] > a[:, 2], 1, 2))
            kx, ky = (kz + 1) % 3, (kz + 2) % 3
            r = np.arange(len(o))
            neg = d[r, kz] < 0
            kx, ky = np.where(neg, ky, kx), np.where(neg, kx, ky)
            sx, sy, sz = (d[r, kx] / d[r, kz])[:, None], (d[r, ky] / d[r, kz])[:, None], (f(1) / d[r, kz])[:, None]
            V = [tris[None, :, v, :] - o[:, None, :] for v in range(3)]
            ax = [[np.take_along_axis(v, k[:, None, None].repeat(v.shape[1], 1), 2)[..., 0] for k in (kx, ky, kz)]
                  for v in V]
            (Ax, Ay), (Bx, By), (Cx, Cy) = [(x - sx * z, y - sy * z) for x, y, z in ax]
            U, W, X = Cx * By - Cy * Bx, Ax * Cy - Ay * Cx, Bx * Ay - By * Ax
            z = (U == 0) | (W == 0) | (X == 0)
            g = np.float64
            U = np.where(z, (g(1) * Cx * By - g(1) * Cy * Bx).astype(f), U)
            W = np.where(z, (g(1) * Ax * Cy - g(1) * Ay * Cx).astype(f), W)
            X = np.where(z, (g(1) * Bx * Ay - g(1) * By * Ax).astype(f), X)
            out = ((U < 0) | (W < 0) | (X < 0)) & ((U > 0) | (W > 0) | (X > 0))
            det = (U + W) + X
            T = (U * (sz * ax[0][2]) + W * (sz * ax[1][2])) + X * (sz * ax[2][2])
            t = T / det
            hit = ~out & (det != 0) & (t > 0) & (t < tmax)
            t = np.where(hit, t, f(np.inf))
            best = t.argmin(1)  # the first of equal minima: the lowest primitive
            ok = hit[r, best]
            assert T.dtype == f and t.dtype == f
            prim[i:i + 512][ok] = best[ok]
            uvt[i:i + 512][ok] = np.stack([W / det, X / det, t], 2)[r, best][ok]
    return prim, uvt


@pytest.mark.parametrize('offset', [0.0, 300.0])
@pytest.mark.parametrize('soup', [0, 3000])
def test_degenerate_rays_bit_exact(vb, gpu_ctx, offset, soup):
    sc = scenes.box_room(width=4, height=4)
    for s in sc['shapes']:
        m = s['param']['transform']['param']['matrix4x4']
        m[3][0] += offset
        m[3][2] -= offset
    if soup:
        rng = np.random.default_rng(3)
        c = rng.random((soup, 1, 3)) * 0.8 + [[-0.4 + offset, 0.1, -0.4 - offset]]
        P = (c + 0.05 * rng.normal(size=(soup, 3, 3))).astype(np.float32)
        sc['shapes'].append({'type': 'mesh', 'name': 'soup', 'param': {
            'positions': P.reshape(-1).tolist(), 'indices': list(range(3 * soup)), 'material': 'Floor'}})
    s = vb.Scene(gpu_ctx, sc).build_accel()
    pos, idx = s.export('pos', np.float32), s.export('idx', np.uint32)
    rays = _rays(pos, idx, [-0.6 + offset, -0.1, -0.6 - offset], [0.6 + offset, 1.1, 1.9 - offset],
                 6000 if soup else 1 << 16, 17)
    prim, uvt = _brute_force(pos.reshape(-1, 3)[idx.reshape(-1, 3)], rays)
    hits, t = s.trace_closest(rays)
    miss = prim == 0xffffffff
    assert 0.0 < miss.mean() < 0.95
    assert np.array_equal(hits[:, 1], prim)
    assert np.array_equal(hits[~miss, 2:], uvt[~miss, :2].copy().view(np.uint32))
    assert np.array_equal(t[~miss], uvt[~miss, 2])
    assert np.array_equal(s.trace_any(rays) != 0, ~miss)


@pytest.mark.parametrize('offset, size, spread', [(1e8, 3e2, 3e3), (5e8, 3e3, 2e4), (3e9, 2e4, 1e5)])
def test_axis_parallel_rays_far_from_the_origin(vb, gpu_ctx, offset, size, spread):
    # A direction component of zero times a coordinate above 3.4e8 overflows
    # in a box test that multiplies by the reciprocal.
    rng = np.random.default_rng(1)
    P = (rng.random((300, 1, 3)) * spread + size * rng.normal(size=(300, 3, 3)) + offset).astype(np.float32)
    sc = scenes.box_room(width=4, height=4)
    sc['shapes'].append({'type': 'mesh', 'name': 'soup', 'param': {
        'positions': P.reshape(-1).tolist(), 'indices': list(range(900)), 'material': 'Floor'}})
    s = vb.Scene(gpu_ctx, sc).build_accel()
    pos, idx = s.export('pos', np.float32), s.export('idx', np.uint32)
    tris = pos.reshape(-1, 3)[idx.reshape(-1, 3)]
    n = 4096
    rays = np.zeros((n, 8), np.float32)
    axis, sign = rng.integers(0, 3, n), rng.choice([-1.0, 1.0], n)
    rays[np.arange(n), 4 + axis] = sign
    rays[:, 0:3] = tris[rng.integers(len(tris) - 300, len(tris), n)].mean(1) - 2 * spread * rays[:, 4:7]
    negative = (rays[:, 4:7] == 0.0) & (rng.random((n, 1)) < 0.5)
    rays[:, 4:7][negative] = -0.0
    rays[:, 7] = 1e30
    prim, uvt = _brute_force(tris, rays)
    hits, t = s.trace_closest(rays)
    hit = prim != 0xffffffff
    assert hit.mean() > 0.9
    assert np.array_equal(hits[:, 1], prim)
    assert np.array_equal(hits[hit, 2:], uvt[hit, :2].copy().view(np.uint32))
    assert np.array_equal(t[hit], uvt[hit, 2])
    assert np.array_equal(s.trace_any(rays) != 0, hit)


@pytest.mark.parametrize('n', [1, 31, 33, 127, 129, 5000, 300001])
def test_batch_sizes_bit_exact(vb, gpu_ctx, n):
    s = vb.Scene(gpu_ctx, scenes.box_room()).build_accel()
    o = oracle.OracleScene(s)
    rays = seeded_rays(n, [-0.6, -0.1, -0.6], [0.6, 1.1, 1.9], seed=n)
    h_gpu, t_gpu = s.trace_closest(rays)
    h_cpu, t_cpu = o.trace_closest(rays)
    miss = h_cpu[:, 1] == 0xffffffff
    assert np.array_equal(h_gpu[:, :2], h_cpu[:, :2])
    assert np.array_equal(h_gpu[~miss, 2:], h_cpu[~miss, 2:])
    assert np.array_equal(t_gpu.view(np.uint32), t_cpu.view(np.uint32))
    assert np.array_equal(s.trace_any(rays), o.trace_any(rays))
