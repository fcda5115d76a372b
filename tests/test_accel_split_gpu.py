"""The GPU build's split search at the sizes where it changes hands (one warp up to 32 triangles, one block per axis
up to 4,096, chunks of 4,096 above) and on boxes whose float costs decide nothing: the tree is the host build's node
for node."""
import numpy as np
import pytest

from skwarka_gb300 import scenes
from skwarka_gb300.accel import Context, Primitive, TriangleMesh, build_flat_tree

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(gpu):
    return Context(0)


def _same(v, t, ctx):
    prims = [Primitive(TriangleMesh(v, t))]
    host = build_flat_tree(prims)
    dev = build_flat_tree(prims, device=ctx, min_device_triangles=0)
    assert dev["on_device"]
    for k in ("nodes", "tri_prim", "tri_index"):
        assert np.array_equal(host[k], dev[k]), k
    assert host["max_depth"] == dev["max_depth"]


@pytest.mark.parametrize("n", [5, 31, 32, 33, 64, 99, 100, 101, 4095, 4096, 4097, 8192, 8193, 20001])
@pytest.mark.parametrize("edge", [0.002, 0.7])
def test_sizes(ctx, n, edge):
    _same(*scenes.random_triangles(n, edge, 0.0, 1.0, n), ctx)


@pytest.mark.parametrize("n", [24, 33, 5000])
@pytest.mark.parametrize("scale", [1e-22, 1e-12, 1.0, 1e12, 1e22])
def test_extents(ctx, n, scale):
    """Areas that underflow or overflow in float."""
    v, t = scenes.random_triangles(n, 0.05, -1.0, 1.0, n + 1)
    _same((v.astype(np.float64) * scale).astype(np.float32), t, ctx)


@pytest.mark.parametrize("n", [32, 300, 6000])
def test_ties_and_flat_boxes(ctx, n):
    """Copies of a few boxes (equal costs on many planes and axes), points, axis-parallel lines and flat triangles."""
    rng = np.random.default_rng(n)
    grid = rng.integers(0, 4, size=(n, 1, 3)).astype(np.float32)
    tri = grid + np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float32)
    kind = np.arange(n) % 5
    tri[kind == 1] = grid[kind == 1]                       # points
    tri[kind == 2, 2] = tri[kind == 2, 1]                  # lines along x
    tri[kind == 3, :, 2] = 0.0                             # in the plane z = 0
    tri[kind == 4] = np.array([[0, 0, 0], [4, 0, 0], [0, 4, 4]], np.float32)  # one wide box
    _same(tri.reshape(-1, 3).copy(), np.arange(3 * n, dtype=np.int32).reshape(n, 3), ctx)


def test_not_a_number(ctx):
    """Triangles with NaN and infinite vertices take part as on the host."""
    v, t = scenes.random_triangles(3000, 0.05, -1.0, 1.0, 3)
    v[::97, 1] = np.nan
    v[50::211] = np.inf
    v[51::307, 2] = -np.inf
    _same(v, t, ctx)
