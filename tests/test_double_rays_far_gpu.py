"""Double rays whose hits lie beyond a float's range (a coordinate over a direction's component does not fit a float): the
walk, which is in float, still reaches every leaf, and the hits are those of the reference's double test bit for bit
against brute force over all triangles."""
import numpy as np
import pytest

import scene_fixtures as sf
from skwarka_gb300.accel import Primitive, TriangleAccelerator, TriangleMesh, unpack_hits_d
from test_traversal_edges_gpu import _all_t

pytestmark = pytest.mark.gpu


def _rays(meshes, rng, n, length):
    """Rays at points inside triangles, at edges and past them, a scene's size away."""
    v = np.concatenate([v.astype(np.float64)[t] for v, t in meshes])
    pick = v[rng.integers(0, len(v), n)]
    w = rng.dirichlet((1.0, 1.0, 1.0), size=n)
    w[: n // 4] = (0.5, 0.5, 0.0)
    w[n // 4: n // 3] = (0.6, 0.6, -0.2)
    d = rng.normal(size=(n, 3))
    d /= np.sqrt((d * d).sum(1))[:, None]
    r = np.zeros((n, 8))
    r[:, :3] = (pick * w[:, :, None]).sum(1) - d * np.abs(v).max() * rng.uniform(0.1, 0.6, size=(n, 1))
    r[:, 3:6] = d * length
    r[:, 7] = np.inf
    return r


def _check(meshes, r):
    import torch
    acc = TriangleAccelerator([Primitive(TriangleMesh(v, t)) for v, t in meshes])
    ts = _all_t(meshes, r)
    first = np.where(ts >= 0.0, ts, np.inf).min(1)
    assert np.isfinite(first).sum() > len(r) // 2
    past = r.copy()
    past[:, 6] = np.nextafter(first, np.inf)  # from just past the first hit
    for x in (r, past):
        want = np.where((ts >= x[:, 6:7]) & (ts <= x[:, 7:8]), ts, np.inf).min(1)
        rays = torch.from_numpy(np.ascontiguousarray(x)).cuda()
        got = unpack_hits_d(acc.intersect_d(rays))
        assert np.array_equal(got["t"].view(np.uint64), want.view(np.uint64))
        assert np.array_equal(acc.intersect_test_d(rays).cpu().numpy() != 0, np.isfinite(want))


def _scaled(scale):
    return [((v.astype(np.float64) * scale).astype(np.float32), t) for v, t in sf.small_query_scene()]


@pytest.mark.parametrize("scale,length", [(1e5, 1e-36), (1e8, 1e-33), (1e10, 1e-30), (1e12, 1e-27)])
def test_beyond_a_float(gpu, scale, length):
    meshes = _scaled(scale)
    _check(meshes, _rays(meshes, np.random.default_rng(53), 400, length))
