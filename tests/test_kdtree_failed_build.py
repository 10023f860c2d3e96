"""A tree build that fails leaves the caller's tree as it was (host and device
builder; refused before any device work, so no GPU is needed)."""
import ctypes
import importlib

import pytest

sc = importlib.import_module("3dgrt_kdtree_gb300.scenes")


@pytest.mark.parametrize("fn", ["kdgr_build_tree", "kdgr_build_tree_gpu"])
def test_failed_build_leaves_the_tree(pkg, fn):
    L = pkg.capi.lib()
    rec = sc.uniform_cube(40, seed=5)
    t = pkg.capi.Tree()
    assert L.kdgr_build_tree(rec.ctypes.data, len(rec), None, ctypes.byref(t), None) == 0
    before = bytes(t)
    rec[:, 3] = 0.001  # every Gaussian below the opacity cut
    assert getattr(L, fn)(rec.ctypes.data, len(rec), None, ctypes.byref(t), None) != 0
    assert bytes(t) == before
    L.kdgr_tree_free(ctypes.byref(t))
