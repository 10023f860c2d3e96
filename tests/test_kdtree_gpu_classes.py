"""The device builder's split-search classes (one warp, one block, globally
sorted keys) against the host builder: roots at the class edges, planes at
exactly zero, cost parameters that switch the FP32 filter off, and
axis-aligned Gaussians that share interval ends."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

sc = importlib.import_module("3dgrt_kdtree_gb300.scenes")


def _same(a, b):
    np.testing.assert_array_equal(a.nodes, b.nodes)
    np.testing.assert_array_equal(a.offsets, b.offsets)
    np.testing.assert_array_equal(a.valid, b.valid)
    assert (a.depth, a.n_leaves, a.max_leaf) == (b.depth, b.n_leaves, b.max_leaf)


@pytest.mark.parametrize("n", [16, 17, 63, 64, 65, 255, 256, 257, 1023, 1024, 1025, 2500])
@pytest.mark.parametrize("flags", [dict(), dict(sah_mode=0, force_split=0), dict(sah_mode=4), dict(sah_mode=7),
                                   dict(isect_cost=-1.0), dict(max_level=3)])
def test_class_edges(pkg, cuda, n, flags):
    rec = sc.uniform_cube(n, seed=n, scale=0.05)
    rec[:, 3] = np.maximum(rec[:, 3], 0.1)  # every Gaussian has a proxy: the root holds n IDs
    _same(pkg.kdtree.build(rec, device="cuda", **flags), pkg.kdtree.build(rec, **flags))


@pytest.mark.parametrize("n", [50, 200, 900, 3000])
def test_shared_interval_ends(pkg, cuda, n):
    """Equal unrotated Gaussians on a lattice through the origin: interval
    ends coincide, and mirrored ones put edges at zero of either sign."""
    rec = sc.uniform_cube(n, seed=7, scale=0.02)
    side = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    rec[:, 0:3] = ((g - side // 2) * 0.125).astype(np.float32)
    rec[:, 3] = 0.5
    rec[:, 4:7] = np.float32(0.0625)
    rec[:, 8:12] = (1.0, 0.0, 0.0, 0.0)
    _same(pkg.kdtree.build(rec, device="cuda"), pkg.kdtree.build(rec))
