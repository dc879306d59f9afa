"""CPU: one plan used by several threads through the C ABI, under the thread sanitizer."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "ascend-fft_b200" / "csrc"
HOST = ROOT / "tests" / "host"


@pytest.mark.skipif(not shutil.which("g++"), reason="g++ required")
def test_threads_share_a_plan(tmp_path):
    probe = tmp_path / "probe.cpp"
    probe.write_text("int main() {}\n")
    build = ["g++", "-std=c++17", "-O1", "-g", "-fsanitize=thread"]
    r = subprocess.run([*build, str(probe), "-o", str(tmp_path / "probe")], capture_output=True)
    if r.returncode or subprocess.run([str(tmp_path / "probe")], capture_output=True).returncode:
        pytest.skip("no thread sanitizer here")
    exe = tmp_path / "threads"
    r = subprocess.run([*build, "-Wall", "-Wextra", "-I", str(ROOT / "include"), "-I", str(CSRC),
                        str(HOST / "test_plan_threads.cpp"), str(HOST / "fake_backend.cpp"), str(CSRC / "plan.cpp"),
                        str(CSRC / "acceptance.cpp"), str(CSRC / "capi.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe), str(ROOT / "ascend-fft_b200" / "config")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr[-4000:]
    assert "all checks passed" in r.stdout
