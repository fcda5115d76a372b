"""Scenes with next to no extent on one axis, where the split search's planes per unit of length overflow a float: a
box that reaches through the node then lies on both sides of every plane.  The GPU build's tree is the host build's,
node for node, at every size of its split search."""
import numpy as np
import pytest

from skwarka_gb300.accel import Context, Primitive, TriangleMesh, build_flat_tree

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(gpu):
    return Context(0)


@pytest.mark.parametrize("n", [5, 6, 9, 17, 31, 32, 33, 300, 5000])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("extent", [1e-44, 1e-38, 1e-37, 2e-36])
def test_thin_axis(ctx, n, axis, extent):
    for seed in range(12 if n < 100 else 4):
        rng = np.random.default_rng([n, axis, seed])
        tri = rng.uniform(0.0, 0.05, size=(n, 3, 3))
        # from scenes spread over the other axes to copies of one triangle, which no plane across these parts
        tri += rng.uniform(0.0, (0.0, 0.01, 1.0)[seed % 3], size=(n, 1, 3))
        if seed % 4 == 3:
            tri[:] = tri[0]
        # flat at either end, reaching through, or anywhere between; every fourth scene all reach through
        kind = rng.integers(0, 4, size=n) if seed % 4 != 3 else np.full(n, 2)
        tri[:, :, axis] = np.where(kind[:, None] == 0, 0.0, np.where(kind[:, None] == 1, extent, np.where(
            kind[:, None] == 2, extent * np.array([0.0, 1.0, 0.5]), extent * rng.uniform(size=(n, 3)))))
        prims = [Primitive(TriangleMesh(tri.reshape(-1, 3).astype(np.float32),
                                        np.arange(3 * n, dtype=np.int32).reshape(n, 3)))]
        host = build_flat_tree(prims)
        dev = build_flat_tree(prims, device=ctx, min_device_triangles=0)
        assert dev["on_device"]
        for k in ("nodes", "tri_prim", "tri_index"):
            assert np.array_equal(host[k], dev[k]), (k, seed)
