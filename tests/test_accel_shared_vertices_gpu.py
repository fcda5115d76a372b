"""The GPU build over meshes that are parts of one vertex array: the host build's tree, and what the build copies follows
the triangles, not the array."""
import time

import numpy as np
import pytest

from skwarka_gb300 import scenes
from skwarka_gb300.accel import Context, Primitive, TriangleAccelerator, TriangleMesh, build_flat_tree

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(gpu):
    return Context(0)


# vertices per triangle on both sides of where a mesh gives only its own, parts smaller and larger than a copy of its own
@pytest.mark.parametrize("parts,triangles,vertices", [(3, 40, 1280), (3, 40, 1311), (3, 40, 1312), (3, 40, 5000),
                                                      (2, 9000, 288_000), (2, 9000, 288_032), (2, 9000, 400_000)])
@pytest.mark.parametrize("matrix", [False, True])
def test_trees(ctx, parts, triangles, vertices, matrix):
    rng = np.random.default_rng(vertices)
    pool = rng.uniform(-1.0, 1.0, size=(vertices, 3)).astype(np.float32)
    prims = []
    for k in range(parts):
        # neighbouring vertices, some triangles dropped: out of range, negative or repeated
        t = rng.integers(0, vertices - 3, size=(triangles, 1)) + rng.permuted(np.tile([0, 1, 2], (triangles, 1)), axis=1)
        bad = rng.integers(0, 12, size=triangles)
        t[bad == 0, 0] = vertices
        t[bad == 1, 1] = -1
        t[bad == 2, 2] = t[bad == 2, 0]
        t[bad == 3] = np.iinfo(np.int32).min
        m = np.eye(4)
        m[:3] += rng.uniform(-0.5, 0.5, (3, 4))
        prims.append(Primitive(TriangleMesh(pool, t.astype(np.int32)), m if matrix else None))
    host = build_flat_tree(prims)
    dev = build_flat_tree(prims, device=ctx, min_device_triangles=0)
    assert dev["on_device"]
    for k in ("nodes", "tris", "tri_prim", "tri_index"):
        a, b = (np.ascontiguousarray(x[k]).view(np.uint32) for x in (host, dev))
        assert np.array_equal(a, b), k


def test_cost_follows_the_triangles(ctx):
    """400 parts of 50 triangles of one array of 3,000,000 vertices: within five times the time of the same parts with
    arrays of their own (copying the array for each part is 14 GB, a hundred times)."""
    v, t = scenes.random_triangles(1_000_000, 0.02, 0.0, 1.0, 5)
    shared = [Primitive(TriangleMesh(v, np.ascontiguousarray(t[50 * k:50 * k + 50]))) for k in range(400)]
    own = [Primitive(TriangleMesh(np.ascontiguousarray(v[150 * k:150 * k + 150]), np.ascontiguousarray(t[:50])))
           for k in range(400)]

    def seconds(prims):
        best = np.inf
        for _ in range(4):
            t0 = time.perf_counter()
            a = TriangleAccelerator(prims, ctx)
            best = min(best, time.perf_counter() - t0)
            assert a.info["built_on_device"] and a.info["n_triangles"] == 20_000
        return best

    assert seconds(shared) < 5.0 * seconds(own)
