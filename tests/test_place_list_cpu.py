"""The rasterizer's list of failed pixel tests: its counter goes on when the list is full, and
however many tests ask, none past the list's length is handed a place."""

import os
import subprocess

import facade_build

CSRC = os.path.join(facade_build.ROOT, "otmap_b200", "csrc")


def test_a_full_list_stays_full(tmp_path):
    exe = str(tmp_path / "place_list")
    subprocess.run([facade_build.cxx(), "-std=c++17", "-O2", "-I", CSRC,
                    os.path.join(facade_build.ROOT, "tests", "cpp", "place_list.cpp"), "-o", exe], check=True)
    assert int(subprocess.run([exe], check=True, capture_output=True, text=True).stdout) == 65536
