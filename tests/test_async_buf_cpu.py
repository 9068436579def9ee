"""A buffer that one stream fills and another reads is freed on its readers' stream: a free on
the filling stream could hand the memory on under a kernel that still reads it."""

import os
import subprocess

import facade_build

CSRC = os.path.join(facade_build.ROOT, "otmap_b200", "csrc")


def test_freed_on_the_readers_stream(tmp_path):
    from otmap_b200 import build

    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    exe = str(tmp_path / "async_buf")
    subprocess.run([facade_build.cxx(), "-std=c++17", "-O1", "-I", CSRC, "-isystem", cuda,
                    os.path.join(facade_build.ROOT, "tests", "cpp", "async_buf.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["m1", "m2", "f1", "m2", "f1", "f1"]


def test_the_locator_names_its_readers_stream():
    """The one buffer that is filled beside the context's stream, in the locator's build."""
    with open(os.path.join(CSRC, "locate.cu")) as f:
        text = f.read()
    build = text[text.index("static void build_locator"):]
    build = build[:build.index("\n}")]
    beside = [line for line in build.splitlines() if ".reserve(" in line and " bs," in line]
    assert beside and all(line.rstrip().endswith("ctx->pool, st);") for line in beside)
