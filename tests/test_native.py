"""Host-side parts of the CUDA sources, compiled into small programs that need no GPU (tests/native)."""
import os
import subprocess

import pytest

from afmm2d_b200.build import nvcc

NATIVE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native")


@pytest.mark.parametrize("name", ["arena_test"])
def test_native_program(name, tmp_path):
    exe = tmp_path / name
    subprocess.run([nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I",
                    os.path.join(NATIVE, "..", "..", "include"), os.path.join(NATIVE, name + ".cu"), "-o", str(exe)],
                   check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
