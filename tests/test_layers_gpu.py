"""A diffuse one-layer surface is shaded by code of its own; the other kinds go through the layers.  A surface made so
that the layers give the same values -- a mix of a matte surface with itself, an uber one with its diffuse part alone --
renders the same image, with one light and with several, by light and by BSDF samples.

Tolerance: the densities are the same floats (p + p is exact) and the sampled directions too; a value f carries three
more roundings (two scales and their sum) and the pixel is a sum of at most 2 x 2 x 16 positive terms, each addition
rounded once more at most: (3 + 64) 2^-24 = 4e-6."""
import numpy as np
import pytest

from skwarka_gb300 import scenes
from skwarka_gb300.accel import TriangleMesh
from skwarka_gb300.render import MIX, UBER, Camera, Material, PointLight, RenderPrimitive, RenderScene

pytestmark = pytest.mark.gpu
BLACK = Material(kd=(0.0, 0.0, 0.0))


def _scene(mats, lights):
    q = 0.4
    patch = TriangleMesh(np.array([[-q, -q, 0], [q, -q, 0.1], [q, q, -0.2], [-q, q, 0]], np.float32),
                         np.array([[0, 1, 2], [0, 2, 3]], np.int32))
    v, t = scenes._box_inward()
    walls = [TriangleMesh(v, f) for f in (t.reshape(6, 2, 3)[:lights] if lights > 1 else [t])]
    prims = [RenderPrimitive(patch, 0)] + [
        RenderPrimitive(w, len(mats), emission=(2.0, 1.0, 0.5 + k)) for k, w in enumerate(walls)]
    return RenderScene(prims, mats + [BLACK], [PointLight((0.1, 0.2, 0.8), (0.3, 0.2, 0.1))])


@pytest.mark.parametrize("lights", [1, 2, 6])
@pytest.mark.parametrize("sigma", [0.0, 0.35])
def test_same_surface(gpu, lights, sigma):
    matte = Material(kd=(0.5, 0.25, 0.75), sigma=sigma)
    others = [[Material(kind=MIX, mix=(1, 2), mix_scale=(0.25, 0.5, 0.3)), matte, matte]]
    if sigma == 0.0:
        others.append([Material(kind=UBER, kd=(0.5, 0.25, 0.75), ks=(0.0, 0.0, 0.0), kr=(0.0, 0.0, 0.0))])
    cam = Camera.look_at((0.1, -0.3, 0.7), (0, 0, 0), (0, 1, 0), 0.5, 48, 48)
    want = _scene([matte], lights).render_direct(cam, 4, 4, 2, seed=9).cpu().numpy()
    assert want.mean() > 0.1
    for mats in others:
        got = _scene(mats, lights).render_direct(cam, 4, 4, 2, seed=9).cpu().numpy()
        rel = np.abs(got - want) / np.maximum(want, 1e-3)
        print(f"lights={lights} sigma={sigma}: {rel.max():.2e}")
        assert rel.max() <= 4e-6
