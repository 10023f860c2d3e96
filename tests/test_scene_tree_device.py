"""The device side of a scene upload: trees shallower and deeper than its
breadth-first top and than one batch of levels, odd and empty leaves, nodes
nothing refers to, and malformed trees, against the plain kernel (which reads
the tree as given) and against the host check."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

K = importlib.import_module("3dgrt_kdtree_gb300.kdtree")
sc = importlib.import_module("3dgrt_kdtree_gb300.scenes")


def _chain(n, levels, spare=0):
    """A comb along x over n Gaussians sorted by x: level i cuts off one slab
    (leaves of 0, 1 or 2 IDs), the last child holds the rest; `spare` nodes
    at the end that no node refers to."""
    nodes = np.zeros((2 * levels + 1 + spare, 2), np.uint32)
    planes = np.linspace(-0.45, 0.45, levels + 2)[1:-1].astype(np.float32)
    offsets = []
    at = 0
    for i in range(levels):
        c = 1 + 2 * i
        nodes[at] = (c << 3, planes[i:i + 1].view(np.uint32)[0])
        ids = [(2 * i + k) % n for k in range(i % 3)]
        nodes[c] = (len(ids) << 3 | 3, len(offsets))
        offsets += ids
        at = c + 1
    nodes[at] = (n << 3 | 3, len(offsets))
    offsets += list(range(n))
    nodes[2 * levels + 1:] = (3, 0)
    return K.KdTree(nodes, np.array(offsets, np.uint32), np.array([-0.6] * 3 + [0.6] * 3, np.float32))


@pytest.mark.parametrize("levels,spare", [(0, 0), (1, 0), (9, 3), (10, 0), (11, 0), (25, 1), (26, 0), (140, 5)])
def test_comb_trees(pkg, cuda, levels, spare):
    rec = sc.uniform_cube(33, seed=levels, scale=0.05)
    tree = _chain(33, levels, spare)
    F = pkg.renderer
    scene = F.Scene(tree, rec, forms=F.FORM_EXACT | F.FORM_FAST | F.FORM_PACKED)
    info = scene.info()
    assert info["depth"] == levels and info["n_leaves"] == levels + 1 + spare and info["max_leaf"] == 33
    assert info["top_nodes"] == 1 + 2 * min(levels, 10)
    w, h = 40, 24
    cam = sc.look_at((0.3, 0.2, 1.5), aspect=w / h)
    out = [torch.zeros(w * h * 3, device=cuda) for _ in range(3)]
    scene.render(cam, w, h, out[0])
    scene.render_fast(cam, w, h, out[1])
    scene.render_fast(cam, w, h, out[2], precision=1)
    torch.cuda.synchronize()
    assert scene.status() == 0
    # the fast forms agree with the plain one to their stated RMSE
    for o in out[1:]:
        assert float((o - out[0]).square().mean().sqrt()) <= 1e-3
    assert float(out[0].abs().sum()) > 0


@pytest.mark.parametrize("fault", ["child", "twice", "axis", "leaf", "id"])
@pytest.mark.parametrize("level", [1, 5, 12, 30])
def test_malformed_trees_are_refused(pkg, cuda, fault, level):
    rec = sc.uniform_cube(33, seed=1)
    tree = _chain(33, 40)
    at = 2 * level  # the comb's inner node of that level
    if fault == "child":
        tree.nodes[at, 0] = tree.n_nodes << 3
    elif fault == "twice":
        tree.nodes[at, 0] = 1 << 3
    elif fault == "axis":
        tree.nodes[at, 0] |= 4
    elif fault == "leaf":
        tree.nodes[2 * level + 1] = (8 << 3 | 3, tree.offsets.size - 3)
    else:
        tree.offsets[-1] = 33
    with pytest.raises(pkg.capi.KdgrError) as host:
        K.validate(tree, 33)
    with pytest.raises(pkg.capi.KdgrError) as dev:
        pkg.renderer.Scene(tree, rec)
    assert str(host.value).split(":", 1)[-1].strip().split(": ")[-1] in str(dev.value)
