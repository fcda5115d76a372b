"""What a call copies to the GPU has arrived before its kernels read it, however busy the GPU is: photon maps made and
rendered again and again by several processes at once all give the same images."""
import hashlib
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu


def images(n):
    """The digests of n maps and renders, the distinct ones."""
    from skwarka_gb300 import scenes
    from skwarka_gb300.photon import PhotonMap, render_photon
    from skwarka_gb300.render import RenderScene
    prims, mats, cam = scenes.direct_lighting_box()
    found = set()
    for _ in range(n):
        sc = RenderScene(prims, mats)
        pm = PhotonMap.shoot(sc, 200_000, seed=5)
        img = render_photon(sc, pm, cam(48, 48), 2, 2, gather_samples=9, seed=9).cpu().numpy()
        found.add(hashlib.sha1(img.tobytes()).hexdigest())
    return found


def test_maps_at_once(gpu):
    root = Path(__file__).resolve().parent
    code = ("import sys; sys.path[:0] = [%r, %r]; import test_uploads_gpu as t; print('images', *t.images(20))"
            % (str(root.parent), str(root)))
    runs = [subprocess.Popen([sys.executable, "-c", code], stdout=subprocess.PIPE, text=True) for _ in range(4)]
    out = [r.communicate(timeout=240)[0] for r in runs]
    assert all(r.returncode == 0 for r in runs)
    found = {w for o in out for line in o.splitlines() if line.startswith("images") for w in line.split()[1:]}
    assert len(found) == 1, found
