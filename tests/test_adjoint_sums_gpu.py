"""The adjoint's gradient sums at the sizes where they can go wrong: films whose entries do not fill a warp, one
triangle shared by every lane, triangles of a lane each, and both at once.  For matte surfaces the estimator is linear
in the albedo, so the directional derivative along a step equals the central difference of the forward render up to
float rounding: the images' rounding (1e-7 of the loss) over a loss change of about 5 % of it is 2e-6; 1e-4 leaves
room for the sums of both."""
import numpy as np
import pytest

from skwarka_gb300 import scenes
from skwarka_gb300.accel import TriangleMesh
from skwarka_gb300.adjoint import DirectLighting
from skwarka_gb300.render import Camera, Material, RenderPrimitive, RenderScene

pytestmark = pytest.mark.gpu


def _scene(kind):
    q = 3.0
    floor = TriangleMesh(np.array([[-q, -q, 0], [q, -q, 0], [q, q, 0], [-q, q, 0]], np.float32),
                         np.array([[0, 1, 2], [0, 2, 3]], np.int32))
    v, t = scenes.sphere_mesh(5)
    ball = TriangleMesh((v * 0.5 + np.array([0.0, 0.0, 0.5])).astype(np.float32), t[:, [0, 2, 1]])
    lv = np.array([[-0.5, -0.5, 2.5], [0.5, -0.5, 2.5], [0.5, 0.5, 2.5], [-0.5, 0.5, 2.5]], np.float32)
    light = RenderPrimitive(TriangleMesh(lv, np.array([[0, 2, 1], [0, 3, 2]], np.int32)), 1, emission=(4.0, 3.0, 2.0))
    prims = {"floor": [RenderPrimitive(floor, 0)], "ball": [RenderPrimitive(ball, 0)],
             "both": [RenderPrimitive(floor, 0), RenderPrimitive(ball, 0)]}[kind]
    return RenderScene(prims + [light], [Material(kd=(0.5, 0.5, 0.5)), Material(kd=(0.0, 0.0, 0.0))])


@pytest.mark.parametrize("kind", ["floor", "ball", "both"])
@pytest.mark.parametrize("size", [(1, 1), (5, 7), (40, 23)])
def test_directional_derivative(gpu, kind, size):
    import torch
    cam = Camera.look_at((0.2, -1.6, 1.7), (0.0, 0.0, 0.45), (0, 0, 1), 0.5, *size)
    r = DirectLighting(_scene(kind), cam, 3, 3, 1, seed=4)
    rng = np.random.default_rng(5)
    n = r.scene.n_triangles
    albedo = torch.tensor(rng.uniform(0.3, 0.7, size=(n, 3)), dtype=torch.float32, device="cuda")
    step = torch.tensor(rng.uniform(0.0, 0.1, size=(n, 3)), dtype=torch.float32, device="cuda")
    weight = torch.tensor(rng.uniform(0.5, 1.5, size=(size[1], size[0], 3)), dtype=torch.float32, device="cuda")

    def loss(a, s):
        return float((r.forward_image(a, s).double() * weight.double()).sum())

    g_albedo, g_em = r.adjoint(albedo, 1.0, weight)
    assert loss(albedo, 1.0) > 0.0
    want = (loss(albedo + step, 1.0) - loss(albedo - step, 1.0)) / 2.0
    got = float((g_albedo.double() * step.double()).sum())
    want_em = (loss(albedo, 1.5) - loss(albedo, 0.5))
    print(f"{kind} {size}: albedo {got:.6e} {want:.6e}, emission {float(g_em):.6e} {want_em:.6e}")
    assert abs(got - want) <= 1e-4 * abs(want)
    assert abs(float(g_em) - want_em) <= 1e-4 * abs(want_em)
