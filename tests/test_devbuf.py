"""The owned device buffers after a failed allocation (tests/devbuf_check.cpp, compiled here with g++ against
stand-ins of the CUDA runtime): a buffer that could not be allocated is empty and claims nothing, so that the
call that allocates it on first use does so again instead of launching on a null pointer."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_a_failed_allocation_leaves_the_buffer_empty(tmp_path):
    gxx = shutil.which("g++")
    cuda = Path("/usr/local/cuda/include")
    if gxx is None or not (cuda / "cuda_runtime_api.h").exists():
        pytest.skip("g++ or the CUDA headers not available")
    exe = tmp_path / "devbuf_check"
    subprocess.run([gxx, "-std=c++17", "-I", str(ROOT / "ablate_b200" / "csrc"), "-I", str(ROOT / "include"), "-I", str(cuda),
                    str(ROOT / "tests" / "devbuf_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
