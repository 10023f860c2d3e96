"""bench.py's issue-rate roofline counts the instructions of the kernel it
timed: the committed capture is of the groups deal that the default
configuration runs, and another configuration has no capture."""
import importlib

import pytest

bench = importlib.import_module("bench")


class _Config:
    def __init__(self, **kw):
        self._d = {"schedule": 2, "min_blocks": 8, "blocks_per_sm": 0, "chunk": 1, "precision": 0, "hit_buffer": 4,
                   "traversal": 0, "tile_shape": 0, "rays_per_warp": 32, **kw}
        self.precision = self._d["precision"]

    def as_dict(self):
        return dict(self._d)


def test_capture_is_of_the_default_kernel():
    cap = bench.load_capture(bench.capture_key("scale", _Config(), _Config()))
    schedule = cap["kernel"].split("<")[1].split(",")[1]
    assert schedule == "4"  # kSchedGroups in render_packet.cuh


@pytest.mark.parametrize("change", [dict(schedule=3), dict(traversal=1), dict(hit_buffer=8), dict(rays_per_warp=8)])
def test_other_configurations_have_no_fraction(change):
    key = bench.capture_key("scale", _Config(**change), _Config())
    r = bench.roofline(key, 1.7, {"sm_mhz": 2070}, 152, 1e9, 1 << 20)
    assert r["achieved"] is None and r["frac"] is None and r["memory"]["dram_bytes_per_launch"] is None


def test_precision_has_its_own_key():
    assert bench.capture_key("precision", _Config(precision=1), _Config()) == "precision:packed"
