"""Small default launches (four-ray packets, independent rays) give the pixels
of the walk a caller asks for explicitly, in both forms, through every entry
point, at ray counts on both sides of the lines of the rule."""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu

sc = importlib.import_module("3dgrt_kdtree_gb300.scenes")


@pytest.fixture(scope="module", params=["few", "mid", "many"])
def scene(pkg, cuda, request):
    rec = (sc.cluster_shell(6000, seed=8, n_clusters=6) if request.param == "few"
           else sc.uniform_cube(2500, seed=9, scale=0.12 if request.param == "many" else 0.027))
    tree = pkg.kdtree.build(rec)
    dup = tree.offsets.size / len(rec)
    assert {"few": dup < 14, "mid": 18 < dup < 50, "many": dup > 64}[request.param]
    F = pkg.renderer
    return rec, tree, F.Scene(tree, rec, forms=F.FORM_FAST | F.FORM_PACKED)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("sizes", [[(1, 1)], [(7, 3)], [(199, 149)], [(203, 151)], [(499, 499)], [(503, 509)], [(773, 773), (71, 9)], [(787, 781)],
                                   [(64, 48)] * 9, [(160, 120), (33, 17), (250, 190)],
                                   # groups of 2x2 and 2x4 blocks
                                   [(1203, 701)], [(1920, 1088), (17, 3), (331, 77), (1919, 1089)]])
def test_default_equals_explicit(pkg, cuda, scene, precision, sizes):
    rec, tree, S = scene
    F = pkg.renderer
    cams = [(sc.look_at((0.6 + 0.1 * i, 0.3, 1.8), aspect=w / h), w, h) for i, (w, h) in enumerate(sizes)]
    views, total, _ = F.make_views(cams)

    def planes():
        return [torch.full((total * k,), -1.0, device=cuda) for k in (3, 1, 1)]

    explicit = F.BatchConfig.default()
    explicit.precision = precision
    explicit.blocks_per_sm = 8  # not the default: the packet walk as it is
    want = planes()
    S.render_batch(views, len(cams), *want, cfg=explicit)
    cfg = F.BatchConfig.default()
    cfg.precision = precision
    got = planes()
    S.render_batch(views, len(cams), *got, cfg=cfg)
    graph = planes()
    B = F.Batch(S, views, len(cams), *graph, cfg=cfg)
    B.run()
    torch.cuda.synchronize()
    assert S.status() == 0
    for a, b, c in zip(want, got, graph):
        assert torch.equal(a, b) and torch.equal(a, c)
    srv = F.Server(hbm_budget_bytes=2 << 30, arena_bytes=128 << 20, precision=precision)
    slot = srv.add_scene(tree, rec)
    out = torch.full((total * 3,), -1.0).pin_memory()
    assert srv.wait(srv.submit(slot, views, len(cams), out))[0] == 0
    srv.close()
    assert torch.equal(out, want[0].cpu())
