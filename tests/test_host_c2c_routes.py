"""CPU: the C2C routes of the host runtime (which kernel a candidate runs, the one-pass cluster kernels
and their failures) with a fake device seam that has the kernels of the product."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "ascend-fft_b200" / "csrc"


@pytest.mark.skipif(not shutil.which("g++"), reason="g++ required")
def test_c2c_routes(tmp_path):
    exe = tmp_path / "routes"
    host = ROOT / "tests" / "host"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-I", str(ROOT / "include"), "-I", str(CSRC),
                        "-I", str(host), str(host / "test_c2c_routes.cpp"), str(host / "direct_backend.cpp"),
                        str(CSRC / "plan.cpp"), str(CSRC / "acceptance.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe), str(ROOT / "ascend-fft_b200" / "config")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "all checks passed" in r.stdout
