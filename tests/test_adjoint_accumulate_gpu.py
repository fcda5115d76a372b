"""skw_render_direct_adjoint adds to the caller's gradients: into buffers that already hold something, and from calls
queued on several streams at once, as for the views of one loss.

All terms are positive, so a float sum of n of them is within n u (u = 2^-24) of its value: an entry has at most 12 views
x 48 x 36 pixels x 4 samples x 2 terms in the sum over the views (1e-2 in the worst order, which a spread over thousands
of triangles is far from) and 13,824 in one view (8.2e-4).  The bound is 2e-3, two such sums of one view; a lost call
takes all that its view adds to a triangle.
"""
import ctypes as C

import numpy as np
import pytest

from skwarka_gb300 import _lib, scenes
from skwarka_gb300.accel import TriangleMesh
from skwarka_gb300.adjoint import DirectLighting
from skwarka_gb300.render import Camera, Material, RenderPrimitive, RenderScene, c_camera

pytestmark = pytest.mark.gpu

VIEWS, STREAMS = 12, 4


@pytest.fixture(scope="module")
def views(gpu):
    """A finely divided ball (65,536 triangles: the gradient's own pass over them takes many blocks) seen from
    VIEWS sides."""
    import torch
    v, t = scenes.sphere_mesh(7)
    lv = np.array([[-0.8, -0.8, 2.5], [0.8, -0.8, 2.5], [0.8, 0.8, 2.5], [-0.8, 0.8, 2.5]], np.float32)
    scene = RenderScene([RenderPrimitive(TriangleMesh(v.astype(np.float32), t[:, [0, 2, 1]]), 0),
                         RenderPrimitive(TriangleMesh(lv, np.array([[0, 2, 1], [0, 3, 2]], np.int32)), 1,
                                         emission=(4.0, 3.0, 2.0))],
                        [Material(kd=(0.5, 0.5, 0.5)), Material(kd=(0.0, 0.0, 0.0))])
    cams = [Camera.look_at((3.0 * np.cos(a), 3.0 * np.sin(a), 1.5), (0.0, 0.0, 0.3), (0, 0, 1), 0.8, 48, 36)
            for a in np.linspace(0.0, 6.0, VIEWS)]
    renders = [DirectLighting(scene, c, 2, 2, 1, seed=k) for k, c in enumerate(cams)]
    albedo = torch.full((renders[0].scene.n_triangles, 3), 0.6, device="cuda")
    weight = torch.rand((36, 48, 3), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda") + 0.5
    alone = [r.adjoint(albedo, 1.0, weight) for r in renders]  # (leaves the albedo set)
    torch.cuda.synchronize()
    return renders, weight, alone


def _add(render, weight, g_albedo, g_emission, stream):
    cam = c_camera(render.camera)
    _lib.check(_lib.load().skw_render_direct_adjoint(render.scene.handle, C.byref(cam), C.byref(render.params),
                                                     weight.data_ptr(), g_albedo.data_ptr(), g_emission.data_ptr(),
                                                     stream.cuda_stream), render.scene.ctx.handle)


def _close(got, want):
    assert float(want.max()) > 0.0
    assert bool(((got - want).abs() <= 2e-3 * want).all())


def test_into_a_non_zero_buffer(views):
    import torch
    renders, weight, alone = views
    start = torch.rand((renders[0].scene.n_triangles, 3), device="cuda")
    g, e = start.clone(), torch.full((1,), 7.0, dtype=torch.float64, device="cuda")
    _add(renders[0], weight, g, e, torch.cuda.current_stream())
    torch.cuda.synchronize()
    _close(g.double(), start.double() + alone[0][0].double())
    _close(e, 7.0 + alone[0][1])


def test_from_several_streams(views):
    import torch
    renders, weight, alone = views
    g = torch.zeros((renders[0].scene.n_triangles, 3), device="cuda")
    e = torch.zeros(1, dtype=torch.float64, device="cuda")
    streams = [torch.cuda.Stream() for _ in range(STREAMS)]
    torch.cuda.synchronize()
    for k, r in enumerate(renders):
        _add(r, weight, g, e, streams[k % STREAMS])
    torch.cuda.synchronize()
    _close(g.double(), torch.stack([a[0] for a in alone]).double().sum(0))
    _close(e, torch.stack([a[1] for a in alone]).sum(0))
