"""What the GPU build reads and leaves behind: the meshes' triangles collected on the device (small arrays copied
together, large ones by themselves; dropped triangles; matrices with and without a perspective row) and the flattened
tree as the accelerator exports it, all bit for bit those of the host build."""
import numpy as np
import pytest

from skwarka_gb300 import scenes
from skwarka_gb300.accel import Context, Primitive, TriangleAccelerator, TriangleMesh, build_flat_tree

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(gpu):
    return Context(0)


def _bits(a):
    return a.view(np.uint32) if a.dtype == np.float32 else a


def _same(prims, ctx):
    host = build_flat_tree(prims)
    dev = build_flat_tree(prims, device=ctx, min_device_triangles=0)
    assert dev["on_device"]
    for k in ("nodes", "tris", "tri_prim", "tri_index"):
        assert host[k].shape == dev[k].shape and np.array_equal(_bits(host[k]), _bits(dev[k])), k
    assert host["max_depth"] == dev["max_depth"]
    return host


def _matrix(kind, rng):
    m = np.eye(4)
    m[:3] += rng.uniform(-0.7, 0.7, (3, 4))
    if kind == "w":
        m[3] = rng.uniform(0.1, 0.4, 4)
    if kind == "w0":  # w vanishes: infinite and undefined points
        m[3] = 0.0
    return m


# 5,461 triangles or 5,461 vertices of 12 bytes are just below 64 KB, 5,462 above
@pytest.mark.parametrize("sizes", [(1,), (5461,), (5462,), (5461, 1, 5462, 3, 20000), tuple(range(1, 200))])
@pytest.mark.parametrize("kind", [None, "affine", "w", "w0"])
def test_meshes(ctx, sizes, kind):
    rng = np.random.default_rng(len(sizes))
    prims = []
    for k, n in enumerate(sizes):
        v, t = scenes.random_triangles(n, 0.05, -1.0, 1.0, k + 1)
        prims.append(Primitive(TriangleMesh(v, t), None if kind is None else _matrix(kind, rng)))
    _same(prims, ctx)


@pytest.mark.parametrize("n", [300, 30_000])
def test_dropped_triangles(ctx, n):
    rng = np.random.default_rng(n)
    prims = []
    for k in range(4):
        v, t = scenes.random_triangles(n, 0.05, -1.0, 1.0, k + 1)
        t = t.copy()
        if k == 0:
            t[:, 2] = t[:, 0]  # nothing kept
        else:
            bad = rng.integers(0, 8, n)
            t[bad == 0, 0] = -1
            t[bad == 1, 1] = len(v)
            t[bad == 2, 2] = t[bad == 2, 1]
            t[bad == 3, 1] = t[bad == 3, 0]
            t[bad == 4, 2] = np.iinfo(np.int32).max
        prims.append(Primitive(TriangleMesh(v, t)))
    prims.append(Primitive(TriangleMesh(v, np.zeros((0, 3), np.int32))))
    _same(prims, ctx)


@pytest.mark.parametrize("n,kept", [(16383, 16383), (16384, 16384), (20_000, 16_383), (20_000, 16_384), (300_000, 300_000)])
def test_export(ctx, n, kept):
    """Around the size from which the accelerator builds on the GPU, counted in kept triangles."""
    v, t = scenes.random_triangles(n, 0.02, -1.0, 1.0, 9)
    t = t.copy()
    t[kept:, 1] = t[kept:, 0]
    prims = [Primitive(TriangleMesh(v, t))]
    host = build_flat_tree(prims)
    a = TriangleAccelerator(prims, ctx)
    assert a.info["built_on_device"] == (1 if kept >= 16384 else 0)
    nodes, prim, index = a.export()
    assert np.array_equal(nodes.reshape(-1), host["nodes"].view(np.uint32).reshape(-1))
    assert np.array_equal(prim, host["tri_prim"]) and np.array_equal(index, host["tri_index"])
    assert np.array_equal(a.info["bounds"], host["nodes"].view(np.float32).reshape(-1, 8)[0, :6])
    assert a.info["max_depth"] == host["max_depth"] and a.info["n_triangles"] == kept


def test_export_while_another_stream_captures(ctx):
    import torch
    v, t = scenes.random_triangles(500, 0.02, -1.0, 1.0, 9)
    a = TriangleAccelerator([Primitive(TriangleMesh(v, t))], ctx)
    want = a.export()
    x = torch.zeros(8, device="cuda")
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        x += 1
        got = a.export()
    g.replay()
    torch.cuda.synchronize()
    assert all(np.array_equal(p, q) for p, q in zip(want, got)) and x[0].item() == 1
