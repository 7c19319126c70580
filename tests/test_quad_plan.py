"""Launch plans and groups of the quad kernels (lc2_quad_plan.hpp): the same as
the full search over pairs of chunk sizes, at a fraction of its host time,
which every launch outside a graph pays."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_plans_equal_the_full_search(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ missing")
    exe = str(tmp_path / "quad_plan")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", os.path.join(ROOT, "tests", "cpp", "quad_plan.cpp"),
                    "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    bad, two, searched, planned = re.match(
        r"(\d+) wrong, (\d+) with two launches, ([\d.]+) us searched, ([\d.]+) us planned", out).groups()
    assert int(bad) == 0, out
    assert int(two) > 1000, out
    assert float(planned) * 4 < float(searched), out


def test_padded_layout_covers_every_read(tmp_path):
    """Borders shared by neighbouring rows, slices and images: a read outside the
    grid finds a zero, inside the allocation."""
    if shutil.which("g++") is None:
        pytest.skip("g++ missing")
    exe = str(tmp_path / "pad_layout")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", os.path.join(ROOT, "tests", "cpp", "pad_layout.cpp"),
                    "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    assert re.match(r"0 wrong of \d{7,}", out), out
