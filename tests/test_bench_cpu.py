"""bench.py where the reference's C transport is not built: the reference arm says
so on its line and exits 0."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_without_the_reference(tmp_path):
    code = ("import sys; from oracle import pyoracle as po; "
            f"po.REF_SO = {{k: {str(tmp_path)!r} + '/missing_' + k for k in po.REF_SO}}; "
            "sys.argv = ['bench.py', '--impl', 'reference', '--steps', '2', '--warmup', '1']; "
            "import bench; bench.main()")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout)
    assert set(line) == {"impl", "unavailable"} and line["impl"] == "reference"
    assert "\n" not in line["unavailable"] and "not built" in line["unavailable"]
