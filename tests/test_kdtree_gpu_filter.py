"""Where the device builder's FP32 scores must not decide, against the host
builder: costs that switch the filter off."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

sc = importlib.import_module("3dgrt_kdtree_gb300.scenes")


def _same(a, b):
    np.testing.assert_array_equal(a.nodes, b.nodes)
    np.testing.assert_array_equal(a.offsets, b.offsets)


def _records(n):
    """Unrotated Gaussians without extent at the origin."""
    rec = sc.uniform_cube(n, seed=1, scale=0.05)
    rec[:, 0:3] = 0.0
    rec[:, 3] = 0.9
    rec[:, 4:7] = 0.0
    rec[:, 8:12] = (1.0, 0.0, 0.0, 0.0)
    return rec


def test_last_position_close_to_the_leaf_cost(pkg, cuda):
    """Seventeen equal needles along x and two points on the scene box: the
    splits forced by the triangle count end in a node with one position left,
    and with a negative intersection cost its score crosses the leaf's at one
    cost parameter.  On both sides of that value, float by float, the host's
    FP64 comparison decides."""
    rec = _records(19)
    rec[:17, 4] = 1.0
    rec[17:, 0] = pkg.kdtree.build(rec).aabb[3]
    rec[17:, 1:3] = 1.0
    flags = dict(sah_mode=0, force_split=300)

    def host(bits):
        return pkg.kdtree.build(rec, isect_cost=float(np.uint32(bits).view(np.float32)), **flags)

    few, many = (int(np.float32(c).view(np.uint32)) for c in (-0.3, -1.0))
    assert host(few).n_leaves == 3 and host(many).n_leaves == 4
    while many - few > 1:
        mid = (few + many) // 2
        few, many = (mid, many) if host(mid).n_leaves == 3 else (few, mid)
    for bits in [few - 9, few - 3, few - 1, few, many, many + 1, many + 9]:
        cost = float(np.uint32(bits).view(np.float32))
        _same(pkg.kdtree.build(rec, device="cuda", isect_cost=cost, **flags), host(bits))


@pytest.mark.parametrize("n,cost,free", [(1000, 10, 8), (3000, 40, 30)])
@pytest.mark.parametrize("thin", [2e-39, 5e-39, 1e-38, 1e-33, 1e-30, 1e-26])
def test_thin_scenes(pkg, cuda, n, cost, free, thin):
    """Points along x whose SAH costs are equal to 1e-7 by construction (the
    position of the k-th solves k p + (n - k)(1 - p) = cost), in a box `thin`
    wide on the other axes: 4e-6 of FP32 slack is not enough where the half
    area is a denormal's size."""
    k = np.arange(n - cost + 1, n - cost + 1 + free)
    x = np.concatenate([np.zeros(n - cost), (cost - n + k) / (2.0 * k - n), np.ones(cost - free)])
    rec = _records(n)
    rec[:, 0] = x.astype(np.float32)
    rec[-1, 1:3] = np.float32(thin)
    flags = dict(sah_mode=0)
    _same(pkg.kdtree.build(rec, device="cuda", **flags), pkg.kdtree.build(rec, **flags))
