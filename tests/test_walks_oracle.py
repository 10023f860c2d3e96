"""The plain form's filtered walks and the uploaded tree behind them against
the CPU oracle, which shares nothing with them: images of every walk and the
traces, for records at the edges of the filter's bound (needles, scales beyond
its range, quaternions off unit length or zero) and for comb trees deeper than
the breadth-first top of the relaid tree."""
import importlib

import numpy as np
import pytest
import torch

from gpu_util import TRACE_BYTES, oracle_image
from test_scene_tree_device import _chain

pytestmark = pytest.mark.gpu

sc = importlib.import_module("3dgrt_kdtree_gb300.scenes")


def _check(pkg, O, dev, scene, tree, rec, cam, w, h):
    """Plain frame, traced frame and trace records of one camera."""
    rgb, alpha, depth, trace = oracle_image(O, tree, rec, cam, w, h)
    traced = torch.zeros(w * h * TRACE_BYTES, dtype=torch.uint8, device=dev)
    for tr in (None, traced):
        out = [torch.full((w * h * k,), -1.0, device=dev) for k in (3, 1, 1)]
        if tr is None:
            scene.render(cam, w, h, *out)
        else:
            scene.render_trace(cam, w, h, *out, tr)
        torch.cuda.synchronize()
        assert scene.status() == 0
        for got, want in zip(out, (rgb, alpha, depth)):
            np.testing.assert_array_equal(got.cpu().numpy().view(np.uint32), want.reshape(-1).view(np.uint32))
    np.testing.assert_array_equal(np.frombuffer(traced.cpu().numpy().tobytes(), dtype=O.TRACE_DTYPE), trace)
    return alpha


@pytest.fixture(scope="module", params=["few", "many"])
def edge_scene(pkg, cuda, request):
    if request.param == "few":
        rec = sc.cluster_shell(4000, seed=13, n_clusters=5)
    else:
        rec = sc.uniform_cube(2500, seed=14, scale=0.12)
    rng = np.random.default_rng(15)
    pick = rng.permutation(len(rec))
    rec[pick[:200], 8:12] *= np.float32(1.5)
    rec[pick[200:300], 8:12] *= np.float32(1) + np.linspace(-2e-6, 2e-6, 100, dtype=np.float32)[:, None]
    rec[pick[300:350], 8:12] = 0.0
    rec[pick[350:450], 4] = np.float32(1e-5)
    rec[pick[350:360], 4] = np.float32(1e-9)
    rec[pick[350:450], 5] = np.float32(0.8)
    rec[pick[450:500], 4:7] = np.float32(0.8) * np.float32([1.0, 1 / 4000, 1 / 4000])
    tree = pkg.kdtree.build(rec)
    assert (tree.offsets.size > 64 * len(rec)) == (request.param == "many")
    F = pkg.renderer
    return rec, tree, F.Scene(tree, rec, forms=F.FORM_EXACT)


@pytest.mark.parametrize("w,h", [(33, 21), (251, 161), (331, 243), (731, 503), (1043, 991)])
def test_edge_records(pkg, O, cuda, edge_scene, w, h):
    rec, tree, scene = edge_scene
    cam = sc.look_at((0.7, 0.4, 1.9), target=(0.02, 0.01, 0.0), aspect=w / h)
    assert _check(pkg, O, cuda, scene, tree, rec, cam, w, h).max() > 0.5


@pytest.mark.parametrize("levels,spare", [(0, 0), (1, 0), (10, 0), (11, 0), (26, 0), (140, 5)])
def test_comb_trees(pkg, O, cuda, levels, spare):
    rec = sc.uniform_cube(33, seed=levels, scale=0.05)
    tree = _chain(33, levels, spare)
    F = pkg.renderer
    scene = F.Scene(tree, rec, forms=F.FORM_EXACT)
    for w, h in ((40, 24), (400, 251)):
        cam = sc.look_at((0.3, 0.2, 1.5), aspect=w / h)
        assert _check(pkg, O, cuda, scene, tree, rec, cam, w, h).max() > 0.0


def test_full_frame_over_overlapping_gaussians(pkg, cuda):
    """From 3M rays on such scenes are walked as packets over their leaf
    copies; their traces never use those."""
    rec = sc.uniform_cube(2500, seed=14, scale=0.12)
    tree = pkg.kdtree.build(rec)
    assert tree.offsets.size > 64 * len(rec)
    scene = pkg.renderer.Scene(tree, rec, forms=pkg.renderer.FORM_EXACT)
    w, h = 2051, 1471
    cam = sc.look_at((0.7, 0.4, 1.9), target=(0.02, 0.01, 0.0), aspect=w / h)
    out = [[torch.full((w * h * k,), v, device=cuda) for k in (3, 1, 1)] for v in (-1.0, -2.0)]
    scene.render(cam, w, h, *out[0])
    scene.render_trace(cam, w, h, *out[1], torch.zeros(w * h * TRACE_BYTES, dtype=torch.uint8, device=cuda))
    torch.cuda.synchronize()
    assert scene.status() == 0
    for a, b in zip(*out):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
