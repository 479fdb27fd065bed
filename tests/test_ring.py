"""The step kernels' column ring, past 2^32 claims of one launch (host code)."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_ring_claims(tmp_path):
    exe = tmp_path / "ring_host"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", str(ROOT / "tests" / "cpp" / "ring_host.cpp"),
                    "-o", str(exe)], check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "ring ok" in r.stdout, r.stdout + r.stderr
