"""Traversal at the sizes and rays where its launch and its float decisions
can go wrong, against the oracle: launches smaller than the grid (the rays
are spread over the resident warps in smaller groups), and double rays whose
float rounding matters (aimed at vertices and edge midpoints, from origins far
outside the scene, with tmin or tmax exactly at the hit)."""
import numpy as np
import pytest

import scene_fixtures as sf
from skwarka_gb300 import scenes
from skwarka_gb300.accel import Primitive, TriangleAccelerator, TriangleMesh, unpack_hits, unpack_hits_d

pytestmark = pytest.mark.gpu


def _scene(oracle):
    meshes = sf.small_query_scene()
    acc = TriangleAccelerator([Primitive(TriangleMesh(v, t)) for v, t in meshes])
    return meshes, acc, oracle.accel(meshes)


# one ray, the edges of a warp, of a block, and of one ray per resident warp
@pytest.mark.parametrize("n", [1, 31, 32, 33, 129, 3647, 3648, 3649, 116735, 116737])
def test_small_launches(gpu, oracle, n):
    import torch
    meshes, acc, oa = _scene(oracle)
    lo, hi = scenes.scene_bounds(meshes)
    rays = scenes.uniform_rays(n, lo, hi, 41, tmax_range=(0.0, 3.0))
    want, occ = oa.intersect(rays), oa.intersect_test(rays)
    got = unpack_hits(acc.intersect(torch.from_numpy(rays).cuda()))
    assert np.array_equal(got["prim"], want["prim"]) and np.array_equal(got["tri"], want["tri"])
    assert np.array_equal(acc.intersect_test(torch.from_numpy(rays).cuda()).cpu().numpy(), occ)
    d = rays.astype(np.float64)
    got = unpack_hits_d(acc.intersect_d(torch.from_numpy(d).cuda()))
    want = oa.intersect_d(d)
    assert np.array_equal(got["prim"], want["prim"]) and np.array_equal(got["tri"], want["tri"])
    assert np.array_equal(got["t"].view(np.uint64), want["t"].view(np.uint64))


def _all_t(meshes, rays):
    """(rays, triangles) exact t of the reference's Moller-Trumbore test in its operation order, inf where the
    barycentric tests reject (TriangleAccelerator.cpp:240-273)."""
    corners = np.concatenate([v.astype(np.float64)[t] for v, t in meshes])
    v0, e1, e2 = corners[:, 0], corners[:, 1] - corners[:, 0], corners[:, 2] - corners[:, 0]

    def cross(a, b):
        return [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]

    def dot(a, b):
        return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]

    out = np.empty((len(rays), len(corners)))
    for i, r in enumerate(rays):
        d, e1c, e2c = r[3:6], e1.T, e2.T
        s1 = cross(d, e2c)
        with np.errstate(all="ignore"):
            inv = 1.0 / dot(s1, e1c)
            dd = [r[k] - v0[:, k] for k in range(3)]
            b1 = dot(dd, s1) * inv
            s2 = cross(dd, e1c)
            b2 = dot(d, s2) * inv
            t = dot(e2c, s2) * inv
            eps = 2.220446049250313e-16
            out[i] = np.where((b1 > -eps) & (b1 < 1.0 + eps) & (b2 > -eps) & (b1 + b2 < 1.0 + eps), t, np.inf)
    return out


@pytest.mark.parametrize("distance", [0.0, 1.0, 50.0, 1e4])
def test_double_rays_at_the_float_bounds(gpu, distance):
    """Against brute force over all triangles in the reference's double arithmetic: rays through vertices and along
    edges graze the boxes of the leaves too, where the reference's own walk drops some by rounding, so its tree walk
    is no oracle for them; the GPU's widened boxes drop none.  The nearest t is unique, the triangle need not be."""
    import torch
    meshes = sf.small_query_scene()
    acc = TriangleAccelerator([Primitive(TriangleMesh(v, t)) for v, t in meshes])
    rng = np.random.default_rng(43)
    v, t = meshes[0]
    v = v.astype(np.float64)
    pick = t[rng.integers(0, len(t), 600)]
    # a third aimed at vertices, a third at edge midpoints, a third just inside an edge
    w = np.zeros((600, 3))
    w[:200, 0] = 1.0
    w[200:400, :2] = 0.5
    w[400:, 0] = w[400:, 1] = 0.5 - 1e-9
    w[400:, 2] = 2e-9
    target = (v[pick] * w[:, :, None]).sum(1)
    d = rng.normal(size=(600, 3))
    d /= np.sqrt((d * d).sum(1))[:, None]
    r = np.zeros((600, 8))
    r[:, :3] = target - d * (distance + rng.uniform(0.1, 1.0, size=(600, 1)))
    r[:, 3:6] = d
    r[:, 7] = np.inf
    ts = _all_t(meshes, r)
    first = np.where(ts >= 0.0, ts, np.inf).min(1)
    # the same rays ending, and starting, exactly at the hit and one double off it
    cases = [r]
    for col in (6, 7):
        for off in (-np.inf, None, np.inf):
            x = r.copy()
            x[:, col] = first if off is None else np.nextafter(first, off)
            cases.append(x)
    for x in cases:
        inside = np.where((ts >= x[:, 6:7]) & (ts <= x[:, 7:8]), ts, np.inf)
        want = inside.min(1)
        rays = torch.from_numpy(np.ascontiguousarray(x)).cuda()
        got = unpack_hits_d(acc.intersect_d(rays))
        assert np.array_equal(got["t"].view(np.uint64), want.view(np.uint64))
        assert np.array_equal(got["prim"] >= 0, np.isfinite(want))
        assert np.array_equal(acc.intersect_test_d(rays).cpu().numpy() != 0, np.isfinite(want))
