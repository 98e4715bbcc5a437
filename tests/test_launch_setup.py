"""The launchers' per-device setup (CPU: the device numbers are the test's own)."""
import subprocess
from pathlib import Path

HERE = Path(__file__).resolve().parent


def test_setup_is_kept_per_device(tmp_path):
    exe = tmp_path / "launch_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", str(HERE / "launch_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    # no launcher keeps its setup once for the process
    csrc = HERE.parent / "forestclaw_b200" / "csrc"
    for f in sorted(csrc.glob("fcb_*.cu*")):
        for k, line in enumerate(f.read_text().splitlines(), 1):
            assert not line.strip().startswith(("static bool", "static int ", "static std::atomic<int>")) or "(" in line, f"{f.name}:{k}: {line}"
