"""The host conversions' threads (cubokit_b200/csrc/host_ranges.h): an allocation that fails while they are started neither
ends the process nor leaves items out."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_every_item_is_taken_once_when_memory_for_threads_runs_out(tmp_path):
    exe = tmp_path / "host_ranges"
    gxx = "/usr/bin/g++" if Path("/usr/bin/g++").exists() else "g++"
    subprocess.run([gxx, "-std=c++17", "-O1", "-pthread", "-I", str(ROOT / "cubokit_b200" / "csrc"),
                    str(ROOT / "tests" / "cpp" / "host_ranges.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
