"""Photon lookups where their code changes hands, against the oracle bit for bit: heaps of one word per entry up to
k = 128 (local and global sizes on both sides), launches spread over the warps (fewer queries than full warps fill the
GPU), nearest points by scan and by walk, and points with equal distances, whose order the reference's comparisons
decide."""
import numpy as np
import pytest

from skwarka_gb300.kdtree import PhotonKDTree, compress_directions

pytestmark = pytest.mark.gpu


def _points(n, seed, lattice):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(-1, 1, size=(n, 3))
    if lattice:
        pos = np.round(pos * 6.0) / 6.0
    nrm = rng.normal(size=(n, 3))
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    return pos.astype(np.float32), compress_directions(nrm)


def _queries(n, seed, lattice):
    rng = np.random.default_rng(seed)
    q = rng.uniform(-1, 1, size=(n, 3))
    if lattice:
        q[::2] = np.round(q[::2] * 12.0) / 12.0
    qn = rng.normal(size=(n, 3))
    return q, qn / np.linalg.norm(qn, axis=1, keepdims=True)


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, np.float64)).cuda()


@pytest.fixture(scope="module")
def trees(gpu, oracle):
    made = {}

    def get(n, lattice):
        if (n, lattice) not in made:
            pos, nid = _points(n, n, lattice)
            made[n, lattice] = PhotonKDTree(pos, nid), oracle.kdtree(pos, nid)
        return made[n, lattice]
    return get


def _check_knn(trees, n, lattice, nq, k, radius, cos):
    tree, want = trees(n, lattice)
    q, qn = _queries(nq, nq + k, lattice)
    got = tree.get_nearest_points(_dev(q), _dev(qn), k, radius, cos)
    ref = want.knn(q, qn, k, radius, cos)
    for key in ("count", "idx", "d2"):
        assert np.array_equal(got[key].cpu().numpy(), ref[key]), key


@pytest.mark.parametrize("k", [1, 2, 3, 31, 32, 33, 100, 127, 128, 129, 300])
@pytest.mark.parametrize("lattice", [False, True])
@pytest.mark.parametrize("cos", [-1.0, 0.3])
def test_heap_sizes(trees, k, lattice, cos):
    _check_knn(trees, 6000, lattice, 700, k, 0.6, cos)


@pytest.mark.parametrize("nq", [1, 31, 2048, 2049, 4097, 65535, 65537])
def test_spread_launches(trees, nq):
    _check_knn(trees, 6000, False, nq, 20, 0.2, 0.3)


def _check_nearest(trees, n, lattice, nq, radius, cos):
    tree, want = trees(n, lattice)
    q, qn = _queries(nq, nq + 1, lattice)
    got = tree.get_nearest_point(_dev(q), _dev(qn), radius, cos).cpu().numpy()
    assert np.array_equal(got, want.nearest(q, qn, radius, cos))


@pytest.mark.parametrize("n", [1, 33, 129, 2048, 2049, 8192, 8193])
@pytest.mark.parametrize("nq", [1, 63, 64, 5000])
@pytest.mark.parametrize("lattice", [False, True])
def test_nearest_sizes(trees, n, nq, lattice):
    for cos, radius in ((-1.0, np.inf), (0.9, np.inf), (0.3, 0.25)):
        _check_nearest(trees, n, lattice, nq, radius, cos)


@pytest.mark.parametrize("nq", [16384, 16385])
def test_nearest_many(trees, nq):
    for cos in (-1.0, 0.9):
        _check_nearest(trees, 8192, False, nq, np.inf, cos)


def test_radius_at_a_point(trees):
    """The radius is exclusive: points at exactly max_dist are left out, by scan and by walk."""
    for n in (1000, 20000):
        tree, want = trees(n, True)
        q, qn = _queries(300, 9, True)
        for radius in (1.0 / 12.0, 1.0 / 6.0, 0.5):
            got = tree.get_nearest_point(_dev(q), _dev(qn), radius, -1.0).cpu().numpy()
            assert np.array_equal(got, want.nearest(q, qn, radius, -1.0))
            _check_knn(trees, n, True, 300, 40, radius, -1.0)


@pytest.mark.parametrize("k,radius", [(48, 0.25), (49, 0.25), (64, 0.2), (128, 0.45), (129, 0.35)])
@pytest.mark.parametrize("lattice", [False, True])
def test_full_warps(trees, k, radius, lattice):
    """From 63,489 queries on the warps are full and lanes wait for one another at their heaps (k > 48): with heaps
    that some queries of a warp fill and others do not, with the filter and without, and a last warp in part."""
    _check_knn(trees, 6000, lattice, 63_489 + k, k, radius, 0.3 if k % 2 else -1.0)


def test_far_from_the_origin(trees, oracle):
    """Coordinates whose float spacing is large against the distances: what float cannot tell apart is decided in
    double."""
    pos, nid = _points(4000, 3, False)
    for shift in (1e3, 3e7):
        p = (pos.astype(np.float64) + shift).astype(np.float32)
        tree, want = PhotonKDTree(p, nid), oracle.kdtree(p, nid)
        q, qn = _queries(500, 4, False)
        q = q + shift
        for k, cos in ((10, 0.3), (60, -1.0)):
            got = tree.get_nearest_points(_dev(q), _dev(qn), k, 2.0 if shift < 1e6 else 40.0, cos)
            ref = want.knn(q, qn, k, 2.0 if shift < 1e6 else 40.0, cos)
            for key in ("count", "idx", "d2"):
                assert np.array_equal(got[key].cpu().numpy(), ref[key]), (shift, k, key)
