"""The device code of the 3D clip, run on the host by 32 lanes in step (warp_on_host.h), where what it holds between its cuts can
be looked at: every vertex's links, whatever ties the seeds bring, and its place in a cell far smaller than the box."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "sdot-ffi_b200", "csrc")


@pytest.fixture(scope="module")
def clip3(tmp_path_factory):
    d = tmp_path_factory.mktemp("clip3")
    src = open(os.path.join(CSRC, "cells3d.cu")).read()
    (d / "clip3.inc").write_text(src[src.index("constexpr unsigned FULL3"):src.index("constexpr int WALK_STACK3")])
    exe = str(d / "clip3")
    # (an index past a fixed array ends the program)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fsanitize=bounds", "-fno-sanitize-recover", "-I", str(d), "-I", HERE, "-I", CSRC,
                    "-I", "/usr/local/cuda/include", os.path.join(HERE, "clip3_on_host.cpp"), "-o", exe], check=True)
    return lambda *args: [float(x) for x in subprocess.run([exe, *map(str, args)], check=True, capture_output=True, text=True).stdout.split()]


def test_links_after_every_cut(clip3):
    """seeds tied to the rounding of their coordinates, whose cuts now and then leave a boundary that is not one cycle: after every
    cut each link of a cell is to a vertex of the cell that holds the reversed edge and links back, or there is none"""
    cuts, wrong, unlinked = clip3("links", 2000)
    assert cuts > 20000 and unlinked > 0
    assert wrong == 0


@pytest.mark.parametrize("h", [1e-3, 1e-5, 1e-6, 1e-7, 1e-8, 1e-9])
def test_cells_far_smaller_than_the_box(clip3, h):
    """clusters of extent h: the volume of a cell, against its faces cut one by one in 80 bits.  Planes and vertices are exact to a few
    eps of h and the angles' condition (under 1e2); a vertex kept within the tie band (under 1e-14 of the box) costs its cube: 1e-13"""
    worst, = clip3("volume", h, 60)
    assert worst < 1e-13
