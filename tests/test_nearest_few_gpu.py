"""Nearest points of few queries over few points, whose walks are given up for a look at every point: the oracle's
answers where some queries of a warp walk far and others do not, and no more time than a launch of one query more,
which walks throughout, where the walks are short."""
import numpy as np
import pytest

from skwarka_gb300.kdtree import PhotonKDTree, compress_directions

pytestmark = pytest.mark.gpu


def _sphere(n, seed):
    v = np.random.default_rng(seed).normal(size=(n, 3))
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, np.float64)).cuda()


# no walks from 16 to 2,048 queries over at most 2,048 points; else they are given up after some 24 to 536 nodes
@pytest.mark.parametrize("n", [20, 127, 129, 2048, 2049, 4000, 8192])
@pytest.mark.parametrize("nq", [1, 15, 16, 2048, 2049, 6200, 16384])
def test_mixed_warps(gpu, oracle, n, nq):
    pos = _sphere(n, n).astype(np.float32)
    nid = compress_directions(pos.astype(np.float64))
    q = _sphere(nq, 3)
    qn = q.copy()
    far = np.random.default_rng(4).random(nq) < 0.3
    qn[far] = -qn[far]  # the nearest points that pass lie on the other side
    want = oracle.kdtree(pos, nid)
    tree = PhotonKDTree(pos, nid)
    for cos, radius in ((0.9, np.inf), (0.9, 0.3), (0.9999, np.inf), (-1.0, np.inf)):
        got = tree.get_nearest_point(_dev(q), _dev(qn), radius, cos).cpu().numpy()
        assert np.array_equal(got, want.nearest(q, qn, radius, cos))


@pytest.mark.parametrize("n", [100, 2000, 8192])
@pytest.mark.parametrize("radius", [1e-3, np.inf])
@pytest.mark.parametrize("cos", [-1.0, 0.87])
def test_short_walks_stay_short(gpu, n, radius, cos):
    import torch
    pos = _sphere(n, n).astype(np.float32)
    tree = PhotonKDTree(pos, compress_directions(pos.astype(np.float64)))
    q = _dev(_sphere(16385, 5))

    def us(nq):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        best = np.inf
        for _ in range(6):
            a.record()
            for _ in range(20):
                tree.get_nearest_point(q[:nq], q[:nq], radius, cos)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 50.0)
        return best

    few, more = us(16384), us(16385)
    assert few < 1.5 * more, (few, more)
