"""The kernels' short forms of sqrtf, rsqrtf, floorf and __fdividef give the
functions' bits over the whole ranges that they are used on (every float)."""
import os
import shutil
import subprocess

import pytest

from lc2registration_gb300 import build as lbuild

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_short_forms_equal_the_functions(tmp_path):
    if shutil.which(lbuild.nvcc()) is None:
        pytest.skip("nvcc missing")
    exe = str(tmp_path / "device_math")
    subprocess.run([lbuild.nvcc(), *lbuild.ARCH, "-O3", "-std=c++17", "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cpp", "device_math.cu"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    assert out.split() == "sqrt 0 rsqrt 0 floor 0 div 0 divscale 0".split()
