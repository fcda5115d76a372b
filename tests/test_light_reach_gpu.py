"""BSDF-sampled rays that cannot reach an area light are not traced.  A white
furnace shows that none that can is lost: a Lambertian patch inside emitting
walls of radiance L reflects albedo x L exactly, and multiple importance
sampling takes a good part of that from BSDF samples.

Tolerance: a sample's relative deviation is about 1 and 65,536 samples are
averaged, so the mean's is 0.4 %; 3 % is over seven of them, and the walls of
one face missing would take 7 % or more."""
import numpy as np
import pytest

from skwarka_gb300 import scenes
from skwarka_gb300.accel import TriangleMesh
from skwarka_gb300.render import PLASTIC, Camera, Material, RenderPrimitive, RenderScene

pytestmark = pytest.mark.gpu


def _walls(split, turn):
    """The inward box as one light, or each face as a flat light of its own; turned about x by `turn` radians."""
    v, t = scenes._box_inward()
    c, s = np.cos(turn), np.sin(turn)
    v = (v.astype(np.float64) @ np.array([[1, 0, 0], [0, c, s], [0, -s, c]])).astype(np.float32)
    return [TriangleMesh(v, f) for f in (t.reshape(6, 2, 3) if split else [t])]


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("turn", [0.0, 0.4])
@pytest.mark.parametrize("offset", [0.0, 300.0])
def test_furnace(gpu, split, turn, offset):
    shift = np.array([offset, 0.0, -offset], np.float32)
    q = 0.05
    patch = TriangleMesh(np.array([[-q, -q, 0], [q, -q, 0], [q, q, 0], [-q, q, 0]], np.float32) + shift,
                         np.array([[0, 1, 2], [0, 2, 3]], np.int32))
    prims = [RenderPrimitive(patch, 0)] + [
        RenderPrimitive(TriangleMesh(w.vertices + shift, w.triangles), 1, emission=(2.0, 2.0, 2.0))
        for w in _walls(split, turn)]
    sc = RenderScene(prims, [Material(kd=(0.5, 0.5, 0.5)), Material(kd=(0.0, 0.0, 0.0))])
    cam = Camera.look_at(tuple(np.array([0.0, 0.0, 0.5]) + shift), tuple(shift.astype(float)), (0, 1, 0), 0.1, 64, 64)
    img = sc.render_direct(cam, 4, 4, 1, seed=5).cpu().numpy()
    print(f"split={split} turn={turn} offset={offset}: mean {img.mean():.5f} (1.0)")
    assert abs(img.mean() - 1.0) <= 0.03


def test_light_out_of_reach(gpu):
    """A glossy patch that faces away from its only light stays black, and one facing it does not."""
    q = 0.5
    lv = np.array([[-q, -q, 2], [q, -q, 2], [q, q, 2], [-q, q, 2]], np.float32)
    light = RenderPrimitive(TriangleMesh(lv, np.array([[0, 2, 1], [0, 3, 2]], np.int32)), 1, emission=(3.0, 3.0, 3.0))
    pv = np.array([[-2, -2, 0], [2, -2, 0], [2, 2, 0], [-2, 2, 0]], np.float32)
    mats = [Material(kind=PLASTIC, kd=(0.2, 0.2, 0.2), ks=(0.5, 0.5, 0.5), roughness=0.05), Material(kd=(0, 0, 0))]
    for up in (True, False):
        tri = np.array([[0, 1, 2], [0, 2, 3]] if up else [[0, 2, 1], [0, 3, 2]], np.int32)
        sc = RenderScene([RenderPrimitive(TriangleMesh(pv, tri), 0), light], mats)
        z = 1.0 if up else -1.0
        cam = Camera.look_at((0.3, 0.1, z), (0, 0, 0), (0, 1, 0), 0.6, 32, 32)
        img = sc.render_direct(cam, 2, 2, 2, seed=6).cpu().numpy()
        assert (img.mean() > 0.05) if up else not img.any()
