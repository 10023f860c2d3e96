"""The secondary-ray kernel against the oracle, bit for bit: meshes of one, part
of and several groups of triangles, triangles too large for a group to be
skipped, and image sizes on both sides of the line between its walks."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

sc = importlib.import_module("3dgrt_kdtree_gb300.scenes")


def _ball(n, radius, at):
    """n triangles around a sphere (a latitude strip triangulation)."""
    k = np.arange(n)
    a, b = 2.399963 * k, np.arccos(1 - 2 * (k + 0.5) / n)
    c = np.stack([np.sin(b) * np.cos(a), np.cos(b), np.sin(b) * np.sin(a)], 1)
    u = np.cross(c, np.roll(c, 1, 1))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    v = np.cross(c, u)
    s = 2.2 / np.sqrt(n)
    t = np.stack([c + s * u, c + s * v, c - s * (u + v)], 1)
    return (t * radius + np.asarray(at)).reshape(-1, 9).astype(np.float32)


@pytest.mark.parametrize("mesh", ["none", "one", "ball8", "ball9", "ball64", "ball65", "ball330", "mid_ball65", "wall"])
@pytest.mark.parametrize("w,h", [(120, 90), (643, 479), (1011, 601)])
def test_hybrid_matches_oracle(pkg, O, cuda, mesh, w, h):
    F = pkg.renderer
    if mesh not in ("ball330", "mid_ball65")[:2 if w < 900 else 1] and w > 200:
        pytest.skip("one mesh at the larger size")
    mid = mesh.startswith("mid_")  # more than 16 leaves per Gaussian: small frames walk the tree as given
    rec = sc.uniform_cube(2500, seed=9, scale=0.025) if mid else sc.cluster_shell(2500, seed=6, n_clusters=5)
    tree = pkg.kdtree.build(rec)
    assert (tree.offsets.size > 16 * len(rec)) == mid
    mesh = mesh.removeprefix("mid_")
    tris = {"none": np.zeros((0, 9), np.float32), "one": _ball(8, 0.5, (0, 0, 0.3))[:1],
            "wall": np.array([[-9, -9, -0.5, 9, -9, -0.5, 9, 9, -0.5], [-9, -9, -0.5, 9, 9, -0.5, -9, 9, -0.5]],
                             np.float32)}.get(mesh)
    if tris is None:
        tris = _ball(int(mesh[4:]), 0.45, (0.1, -0.05, 0.2))
    mat = F.material(F.MIRROR, 0.8, 1.0, (0.9, 0.8, 0.7))
    spheres = F.demo_spheres() + [F.sphere((-0.5, 0.1, 0.9), 0.15, F.material(F.OPAQUE, 0.0, 1.0, (0.2, 0.5, 0.9)))]
    cam = sc.look_at((0.5, 0.3, 2.4), aspect=w / h)
    scene = F.Scene(tree, rec)
    out = torch.full((w * h * 3,), -1.0, device=cuda)
    scene.render_hybrid(cam, w, h, F.Secondary(spheres, tris, mat), out)
    assert scene.status() == 0
    S = O.OracleScene(tree.nodes, tree.offsets, tree.aabb, O.invert_scales(rec))

    def words(m):
        return (m.material, m.reflectivity, m.ior, tuple(m.color))

    want = O.render_hybrid(S, cam, w, h,
                           spheres=[(tuple(s.center), s.radius, *words(s.material)) for s in spheres],
                           tris=tris, tri_material=words(mat))
    np.testing.assert_array_equal(out.cpu().numpy().reshape(h, w, 3), O.to_image(want, w, h))
