"""The medium march past the 128 steps whose numbers a block makes beforehand.  A finer march of the same medium
converges to the same in-scattering: its bias is of first order in the step, at most sigma_t step / 2 = 1.25 % at step
0.05, and the noise of 36,864 samples is below 0.5 %, so 3 % holds for every pair.  Lit by point lights, of which the
step's first number chooses one: an area light's own leaf occludes it by the rounding of each step's sample, so that
in-scattering does not converge (test_medium_gpu.py compares it with the reference's renders)."""
import numpy as np
import pytest

from skwarka_gb300.accel import TriangleMesh
from skwarka_gb300.render import Camera, Material, Medium, PointLight, RenderPrimitive, RenderScene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lights", [1, 2, 5])
def test_fine_march_agrees(gpu, lights):
    v = np.array([[-0.4, -0.3, -1.2], [0.4, -0.3, -1.2], [0.0, 0.4, -1.2]], np.float32)
    prims = [RenderPrimitive(TriangleMesh(v, np.array([[0, 2, 1]], np.int32)), 0)]
    points = [PointLight((0.3 * k - 0.5, 0.8 - 0.3 * k, 0.9), (1.0 + k, 2.0, 1.0)) for k in range(lights)]
    sc = RenderScene(prims, [Material(kd=(0.0, 0.0, 0.0))], points)
    cam = Camera.look_at((1.6, 1.2, -0.4), (0.0, 0.0, -0.6), (0, 0, 1), 0.7, 96, 64)
    means = []
    for step in (0.05, 0.024, 0.012):
        sc.set_medium(Medium(lo=(-1.5,) * 3, hi=(1.5,) * 3, sigma_a=(0.1,) * 3, sigma_s=(0.4,) * 3, step=step))
        means.append(float(sc.render_direct(cam, 3, 2, 1, seed=3).mean()))
    print(lights, means)
    assert means[0] > 0.0
    for m in means[1:]:
        assert abs(m / means[0] - 1.0) <= 0.03
