"""The staging memory of the object and probe transfers (cubokit_b200/csrc/host_staging.h): a plan's transfers share one
allocation, gradients included, and go through pageable memory where none can be page-locked."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_one_allocation_serves_a_plan_and_pageable_memory_stands_in(tmp_path):
    exe = tmp_path / "host_staging"
    gxx = "/usr/bin/g++" if Path("/usr/bin/g++").exists() else "g++"
    subprocess.run([gxx, "-std=c++17", "-O1", "-fsanitize=address", "-I", str(ROOT / "cubokit_b200" / "csrc"),
                    str(ROOT / "tests" / "cpp" / "host_staging.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)

