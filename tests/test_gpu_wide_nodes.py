"""The 4-wide nodes the renders and closest-hit rays walk (folded on the device from the binary tree,
enlarged centre / half-extent boxes) against every triangle tested without a tree, on the rays on
which a box test goes wrong first.  Closest hits must agree exactly (triangle and distance)."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import same_bits
from vira_gb300 import Mesh, Scene, capi, synthetic
from vira_gb300.spectral import FOUR_BAND

pytestmark = pytest.mark.gpu
F = np.float32


def _dem(n, posting=10.0, offset=0.0):
    z = synthetic.fbm_heights(n, 0.8, seed=n, lo=-100.0, hi=100.0)
    m = Mesh.from_dem(z, posting)
    if offset:
        m.positions = (m.positions + F(offset)).astype(F)
    return m


def _flat(n):
    return Mesh.from_dem(np.zeros((n, n), F), 1.0)     # boxes of no height, every plane shared


def _sliver():
    """Triangles of 1000 x 0.001 x 0 side by side, and one triangle alone far away."""
    x = np.arange(65, dtype=F) * F(1e-3)
    p = np.concatenate([np.stack([x, np.zeros(65, F), np.zeros(65, F)], 1),
                        np.stack([x, np.full(65, 1000, F), np.zeros(65, F)], 1),
                        np.array([[5e4, 0, 0], [5e4, 1, 0], [5e4, 0, 1]], F)]).astype(F)
    i = np.arange(64)
    t = np.concatenate([np.stack([i, i + 1, i + 65], 1), np.stack([i + 1, i + 66, i + 65], 1), [[130, 131, 132]]])
    return Mesh(positions=p, indices=t.astype(np.uint32))


def _nested(k):
    """k triangles, each a quarter of the size of the one before, all around the origin: a deep tree."""
    s = (F(0.25) ** np.arange(k, dtype=F) * F(1e6)).astype(F)
    p = np.stack([np.stack([s, s, s], 1), np.stack([s * F(1.5), s, s], 1), np.stack([s, s * F(1.5), s], 1)], 1)
    return Mesh(positions=p.reshape(-1, 3).astype(F), indices=np.arange(3 * k, dtype=np.uint32).reshape(-1, 3))


MESHES = {"one": lambda: Mesh(positions=np.array([[0, 0, 0], [9, 0, 0], [0, 9, 1]], F),
                              indices=np.array([[0, 1, 2]], np.uint32)),
          "quad": lambda: _dem(2), "dem3": lambda: _dem(3), "dem5": lambda: _dem(5), "dem66": lambda: _dem(66),
          "offset": lambda: _dem(33, offset=3.0e4), "flat": lambda: _flat(33), "sliver": _sliver,
          "nested": lambda: _nested(24)}


def _rays(mesh, rng):
    p = mesh.positions.astype(np.float64)
    lo, hi = p.min(0), p.max(0)
    c, e = (lo + hi) / 2, np.maximum(hi - lo, 1.0)
    tri = mesh.indices[rng.integers(0, mesh.indices.shape[0], 1500)]
    w = rng.dirichlet([1, 1, 1], 1500)
    on = (p[tri] * w[:, :, None]).sum(1)
    v = p[rng.integers(0, p.shape[0], 1500)]
    o, d = [], []
    for axis in range(3):                                    # parallel to an axis, through vertices and faces
        for sign in (1.0, -1.0):
            u = np.zeros(3)
            u[axis] = sign
            for x in (v[:300], on[:300]):
                o.append(x - u * e[axis] * 2)
                d.append(np.broadcast_to(u, x.shape))
    for far in (2.0, 50.0):                                  # through vertices, edges' ends and faces, near and far
        src = c + e.max() * far * _unit(rng, 1500)
        for x in (v, on):
            o.append(src)
            d.append(x - src)                                # not normalised
    o.append(on)                                             # from the surface, any way
    d.append(_unit(rng, 1500) * rng.choice([1e-3, 1.0, 1e3], 1500)[:, None])
    o.append(on[:300] + 0.1 * e * _unit(rng, 300))           # a direction whose reciprocal is subnormal
    d.append(_unit(rng, 300) * 3e38)
    o.append(v)                                              # from a vertex, in a plane of the axes
    f = _unit(rng, 1500)
    f[np.arange(1500), rng.integers(0, 3, 1500)] = 0.0
    d.append(f)
    return np.concatenate(o).astype(F), np.concatenate(d).astype(F)


def _unit(rng, n):
    x = rng.standard_normal((n, 3))
    return x / np.linalg.norm(x, axis=1, keepdims=True)


def _brute(positions, indices, o, d):
    """The watertight test (Woop, Benthin, Wald 2013) of every ray with every triangle in FP32, each
    operation rounded by itself; closest t, ties to the smaller triangle."""
    import torch

    dev = "cuda"
    p = torch.from_numpy(positions).to(dev)[torch.from_numpy(indices.astype(np.int64)).to(dev)]      # [T][3][3]
    o, d = torch.from_numpy(o).to(dev), torch.from_numpy(d).to(dev)
    tri = torch.full((o.shape[0],), -1, dtype=torch.int64, device=dev)
    tt = torch.full((o.shape[0],), float("inf"), device=dev)
    step = max(1, 8000000 // p.shape[0])
    for i in range(0, o.shape[0], step):
        oo, dd = o[i:i + step], d[i:i + step]
        a = dd.abs()
        kz = torch.where(a[:, 0] > a[:, 1], torch.where(a[:, 0] > a[:, 2], 0, 2), torch.where(a[:, 1] > a[:, 2], 1, 2))
        kx, ky = (kz + 1) % 3, (kz + 2) % 3
        g = lambda x, k: torch.gather(x, 1, k[:, None])                      # noqa: E731
        dz = g(dd, kz)
        kx, ky = torch.where(dz[:, 0] < 0, ky, kx), torch.where(dz[:, 0] < 0, kx, ky)
        sx, sy, sz = g(dd, kx) / dz, g(dd, ky) / dz, 1.0 / dz
        X, Y, Z = [], [], []
        for c in range(3):
            q = p[None, :, c, :] - oo[:, None, :]
            at = lambda k: torch.gather(q, 2, k[:, None, None].expand(-1, q.shape[1], 1))[..., 0]    # noqa: E731
            z = at(kz)
            X.append(at(kx) - sx * z)
            Y.append(at(ky) - sy * z)
            Z.append(sz * z)
        cr = lambda j, k: X[j] * Y[k] - Y[j] * X[k]                          # noqa: E731
        cr64 = lambda j, k: (X[j].double() * Y[k].double() - Y[j].double() * X[k].double()).float()   # noqa: E731
        U, V, W = cr(2, 1), cr(0, 2), cr(1, 0)
        z = (U == 0) | (V == 0) | (W == 0)
        U, V, W = torch.where(z, cr64(2, 1), U), torch.where(z, cr64(0, 2), V), torch.where(z, cr64(1, 0), W)
        det = U + V + W
        t = ((U * Z[0] + V * Z[1]) + W * Z[2]) * (1.0 / det)
        out = ((U < 0) | (V < 0) | (W < 0)) & ((U > 0) | (V > 0) | (W > 0))
        t = torch.where(out | (det == 0) | ~(t > 0), torch.full_like(t, float("inf")), t)
        m, k = t.min(dim=1)
        first = torch.where(t == m[:, None], torch.arange(p.shape[0], device=dev)[None], p.shape[0]).min(dim=1).values
        tt[i:i + step] = m
        tri[i:i + step] = torch.where(torch.isfinite(m), first, -1)
    return tri.cpu().numpy(), tt.cpu().numpy()


def _check(scene, rng):
    m = scene.meshes[0]
    o, d = _rays(m, rng)
    tri, t, _ = scene.intersect(o, d)
    rt, rtt = _brute(np.ascontiguousarray(m.positions), m.indices, o, d)
    assert (rt >= 0).any()
    assert np.array_equal(tri.astype(np.int64), np.where(rt < 0, int(capi.NO_HIT), rt))
    assert same_bits(t, rtt)


@pytest.mark.parametrize("builder", [0, 1], ids=["sah", "lbvh"])
@pytest.mark.parametrize("name", list(MESHES))
def test_closest_hits_equal_every_triangle_tested(gpu, name, builder):
    s = Scene(FOUR_BAND, device=0)
    s.new_instance(s.add_mesh(MESHES[name]()))
    s.bvh_options = capi.BvhOptions(0, builder, 0, 0)
    s.build_tlas()
    _check(s, np.random.default_rng(len(name)))
    s.close()


def test_moved_vertices_move_the_wide_boxes(gpu):
    mesh = _dem(40)
    s = Scene(FOUR_BAND, device=0)
    s.new_instance(s.add_mesh(mesh))
    s.build_tlas()
    rng = np.random.default_rng(3)
    s.update_positions(0, (mesh.positions + rng.normal(0, 30.0, mesh.positions.shape)).astype(F))
    _check(s, rng)
    s.close()
