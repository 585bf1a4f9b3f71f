"""The atlas lookups' octahedral mapping has the bits of the mapping with
divisions (tests/native/oct_check.cu, 67 M directions on the GPU)."""
import os
import subprocess

import pytest

from vulkanexp_gb300 import build

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_oct_map_has_the_bits_of_divisions(gpu_lib, tmp_path):
    exe = str(tmp_path / "oct_check")
    subprocess.check_call([build.nvcc()] + build.ARCH + ["-O3", "-std=c++17", "--expt-relaxed-constexpr", "-o", exe,
                                                         os.path.join(ROOT, "tests/native/oct_check.cu")])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "all ok" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]
