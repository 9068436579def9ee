"""The point locator pools the face lists of a warp's 32 points: their entries are numbered through
in windows that keep the numbers within an int, however long the lists are."""

import os
import subprocess

import facade_build
import pytest

CSRC = os.path.join(facade_build.ROOT, "otmap_b200", "csrc")


@pytest.mark.parametrize("counts", [(0,), (7, 0, 200), (2**26 - 1,), (2**26,), (2**28, 0, 5), (2**31 - 1,)])
def test_numbers_stay_within_an_int(tmp_path, counts):
    exe = str(tmp_path / "pool_window")
    subprocess.run([facade_build.cxx(), "-std=c++17", "-O2", "-I", CSRC,
                    os.path.join(facade_build.ROOT, "tests", "cpp", "pool_window.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe, *map(str, counts)], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["1", "1"]
