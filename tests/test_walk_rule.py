"""The batched launch's walk rule on the host (no GPU): a configuration whose
zeros stand for the default values is the default one; any other runs as it is
written."""
import subprocess

from test_failures import link


def test_equal_configurations_run_the_same(pkg, tmp_path):
    exe = link("walk_rule.cpp", tmp_path / "walk_rule")
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
