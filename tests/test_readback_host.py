"""Read-backs into pageable memory on the host (CPU): tests/cpp/readback_host.cpp
drives tspeed_b200/csrc/tsp_readback.h over a stand-in for the CUDA runtime,
under AddressSanitizer and UndefinedBehaviorSanitizer."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INCLUDE = os.path.join(os.path.dirname(os.path.dirname(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc")), "include")


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")),
                    reason="g++ or the CUDA headers not available")
def test_read_back_over_a_stand_in_runtime(tmp_path):
    exe = str(tmp_path / "readback_host")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-pthread", "-fsanitize=address,undefined",
                    "-fno-sanitize-recover=all", "-I" + os.path.join(ROOT, "tspeed_b200", "csrc"), "-I" + CUDA_INCLUDE,
                    os.path.join(ROOT, "tests", "cpp", "readback_host.cpp"), "-o", exe], check=True, timeout=300)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "read-back checks passed" in r.stdout
