"""The bound on build memory that contexts keep (CPU)."""
import subprocess
from pathlib import Path

HERE = Path(__file__).resolve().parent


def test_owners_stay_below_the_cap(tmp_path):
    exe = tmp_path / "budget_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", str(HERE / "budget_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
