"""Lookups of large heaps whose warps just fit the GPU, or just do not: the oracle's answers, and no time lost to a second
round of blocks."""
import numpy as np
import pytest

from skwarka_gb300.kdtree import PhotonKDTree, compress_directions

pytestmark = pytest.mark.gpu


def _sphere(n, seed):
    v = np.random.default_rng(seed).normal(size=(n, 3))
    return v / np.linalg.norm(v, axis=1, keepdims=True)


@pytest.mark.parametrize("k", [101, 112, 128])
@pytest.mark.parametrize("nq", [1672, 1673, 20_000, 53_504, 53_505])
def test_answers(gpu, oracle, k, nq):
    import torch
    pos = _sphere(4000, 1).astype(np.float32)
    nid = compress_directions(pos.astype(np.float64))
    q = _sphere(nq, 2)
    got = PhotonKDTree(pos, nid).get_nearest_points(torch.from_numpy(q).cuda(), torch.from_numpy(q).cuda(), k, 0.4, 0.9)
    ref = oracle.kdtree(pos, nid).knn(q, q, k, 0.4, 0.9)
    for key in ("count", "idx", "d2"):
        assert np.array_equal(got[key].cpu().numpy(), ref[key]), key


def test_time_follows_the_queries(gpu):
    """50,000 lookups of k = 128 that do not fill their heaps take no longer than 5 / 4 of those of k = 100, whose heaps
    all fit at once."""
    import torch
    pos = _sphere(6000, 3).astype(np.float32)
    tree = PhotonKDTree(pos, compress_directions(pos.astype(np.float64)))
    q = torch.from_numpy(_sphere(50_000, 4)).cuda()

    def us(k):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        best = np.inf
        for _ in range(8):
            a.record()
            for _ in range(5):
                tree.get_nearest_points(q, None, k, 0.16, -1.0)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 200.0)
        return best

    few, many = us(100), us(128)
    assert many < 1.25 * few, (few, many)
