"""Double rays where single products of the float triangle test fall below a float's normal range: scenes far smaller
and larger than one, and directions far from unit length.  Their hits are those of the reference's double test all the
same, bit for bit against brute force over all triangles."""
import numpy as np
import pytest

from test_double_rays_far_gpu import _check, _rays, _scaled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-30, 1e-20, 1e-15, 1e-14, 1e-13, 1e-12, 1e-11, 1e-6, 1e6, 1e10, 1e12])
def test_scene_size(gpu, scale):
    meshes = _scaled(scale)
    _check(meshes, _rays(meshes, np.random.default_rng(51), 800, 1.0))


@pytest.mark.parametrize("length", [1e-300, 1e-44, 1e-39, 1e-38, 1e-37, 1e-36, 1e-34, 1e-30, 1e-12, 1e12, 1e30, 1e36])
def test_direction_length(gpu, length):
    meshes = _scaled(0.5)
    _check(meshes, _rays(meshes, np.random.default_rng(52), 800, length))


def test_small_scene_and_short_directions(gpu):
    for scale, length in ((1e-8, 1e-20), (1e-12, 1e-10), (1e-5, 1e-25), (1e5, 1e-36), (1e-12, 1e20)):
        meshes = _scaled(scale)
        _check(meshes, _rays(meshes, np.random.default_rng(53), 400, length))
