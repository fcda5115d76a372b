"""The tree builds' scans at the sizes where they change hands -- one tile of 2,048 values, several, and so many that
the tiles' totals are scanned by themselves (more than 8,192) -- seen through photon trees, whose sort scans three
values a point: the trees are the host build's."""
import numpy as np
import pytest

from skwarka_gb300.kdtree import build_device, build_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 682, 683, 1365, 1366, 2048, 2049, 4096, 100_003, 5_700_001])
def test_photon_tree(gpu, n):
    pos = np.random.default_rng(n).uniform(-1, 1, size=(n, 3)).astype(np.float32)
    perm, nodes, _ = build_device(pos)
    want_perm, want_nodes = build_host(pos)
    assert np.array_equal(perm, want_perm) and np.array_equal(nodes, want_nodes)
