"""Point location through the prefix table against a scan of all leaves (CPU)."""
import subprocess
from pathlib import Path

HERE = Path(__file__).resolve().parent


def test_locator_equals_scan(tmp_path):
    exe = tmp_path / "forest_check"
    subprocess.run(["g++", "-O2", "-std=c++17", str(HERE / "forest_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
