"""Reading an accelerator's tree back disturbs nothing: it waits for no other work on the GPU, whatever the size of the
tree, and writes all of the caller's buffers and nothing besides."""
import numpy as np
import pytest

from skwarka_gb300 import _lib, scenes
from skwarka_gb300.accel import Primitive, TriangleAccelerator, TriangleMesh, build_flat_tree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 500, 16383, 16384, 200_000])
def test_export_waits_for_nothing_else(gpu, n):
    import torch
    prims = [Primitive(TriangleMesh(*scenes.random_triangles(n, 0.02, -1.0, 1.0, 9)))]
    a = TriangleAccelerator(prims)
    a.export()
    busy, done = torch.cuda.Stream(), torch.cuda.Event()
    torch.cuda.synchronize()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(1_000_000_000)  # one thread for half a second
        done.record()
    nodes, prim, index = a.export()
    assert not done.query()
    torch.cuda.synchronize()
    host = build_flat_tree(prims)
    assert np.array_equal(nodes.reshape(-1), host["nodes"].view(np.uint32).reshape(-1))
    assert np.array_equal(prim, host["tri_prim"]) and np.array_equal(index, host["tri_index"])


@pytest.mark.parametrize("n", [0, 3, 700, 300_000])
@pytest.mark.parametrize("which", range(8))
def test_buffers(gpu, n, which):
    """Any of the three buffers may be null."""
    a = TriangleAccelerator([Primitive(TriangleMesh(*scenes.random_triangles(max(n, 1), 0.02, -1.0, 1.0, 9)))] if n
                            else [])
    want = a.export()
    got = [np.full(x.size + 2, 0x5A5A5A5A, x.dtype) for x in want]
    _lib.check(_lib.load().skw_accel_export(a.handle, *(g[1:].ctypes.data if which >> k & 1 else None
                                                        for k, g in enumerate(got))), a.ctx.handle)
    for k, (g, x) in enumerate(zip(got, want)):
        assert g[0] == g[-1] == 0x5A5A5A5A
        assert np.array_equal(g[1:-1], x.reshape(-1)) if which >> k & 1 else (g == 0x5A5A5A5A).all()
