"""Lookups of k > 128, whose heaps are in global memory, around the size from which lanes no longer wait for one another:
the oracle's answers."""
import numpy as np
import pytest

from skwarka_gb300.kdtree import PhotonKDTree, compress_directions

pytestmark = pytest.mark.gpu


def _sphere(n, seed):
    v = np.random.default_rng(seed).normal(size=(n, 3))
    return v / np.linalg.norm(v, axis=1, keepdims=True)


@pytest.mark.parametrize("nq", [116_737, 233_472, 233_473])
@pytest.mark.parametrize("k,radius", [(129, 0.15), (200, 0.5)])
def test_answers(gpu, oracle, nq, k, radius):
    import torch
    pos = _sphere(4000, 1).astype(np.float32)
    nid = compress_directions(pos.astype(np.float64))
    q = _sphere(nq, 2)
    dq = torch.from_numpy(q).cuda()
    got = PhotonKDTree(pos, nid).get_nearest_points(dq, dq, k, radius, 0.9)
    some = np.r_[:1500, nq // 2:nq // 2 + 500, nq - 1500:nq]
    ref = oracle.kdtree(pos, nid).knn(q[some], q[some], k, radius, 0.9)
    for key in ("count", "idx", "d2"):
        assert np.array_equal(got[key][torch.from_numpy(some).cuda()].cpu().numpy(), ref[key]), key
