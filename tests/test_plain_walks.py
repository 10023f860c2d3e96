"""The plain form's walks (lanes sharing rays, independent rays, packets,
records gathered by ID) against the per-ray trace kernel, bit for bit: image
sizes on both sides of every line of the launch rule, on a scene whose
Gaussians sit in few leaves and on one where they sit in many, with needles,
quaternions off unit length and extreme scales among the records."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

sc = importlib.import_module("3dgrt_kdtree_gb300.scenes")


@pytest.fixture(scope="module", params=["few", "many"])
def walk_scene(pkg, cuda, request):
    if request.param == "few":
        rec = sc.cluster_shell(4000, seed=3, n_clusters=5)
    else:
        rec = sc.uniform_cube(2500, seed=4, scale=0.12)
    rng = np.random.default_rng(5)
    rec[rng.choice(len(rec), 200, False), 8:12] *= np.float32(1.5)
    rec[rng.choice(len(rec), 50, False), 8:12] = 0.0
    thin = rng.choice(len(rec), 100, False)
    rec[thin, 4] = np.float32(1e-5)
    rec[thin[:10], 4] = np.float32(1e-9)
    rec[thin, 5] = np.float32(0.8)
    tree = pkg.kdtree.build(rec)
    assert (tree.offsets.size > 64 * len(rec)) == (request.param == "many")
    F = pkg.renderer
    return request.param, F.Scene(tree, rec, forms=F.FORM_EXACT), F.Scene(tree, rec)


@pytest.mark.parametrize("w,h", [(1, 1), (9, 5), (191, 188), (251, 161), (331, 239), (331, 243), (641, 479), (701, 501), (1013, 991)])
def test_walks_match_the_trace_kernel(pkg, cuda, walk_scene, w, h):
    name, exact_only, both = walk_scene
    if name == "many" and w * h > 200_000:
        pytest.skip("one walk for all larger frames")
    cam = sc.look_at((0.7, 0.4, 1.9), target=(0.02, 0.01, 0.0), aspect=w / h)
    want = [torch.zeros(w * h * k, device=cuda) for k in (3, 1, 1)]
    trace = torch.zeros(w * h * 56, dtype=torch.uint8, device=cuda)
    exact_only.render_trace(cam, w, h, *want, trace)
    for scene in (exact_only, both):
        got = [torch.full_like(o, -1.0) for o in want]
        scene.render(cam, w, h, *got)
        torch.cuda.synchronize()
        assert scene.status() == 0
        for a, b in zip(got, want):
            assert torch.equal(a.view(torch.int32), b.view(torch.int32))
