"""What the transform's feeding warps hand one another about an atom
(csrc/feed_extent.cuh), built for the host (tests/host_feed.cpp): the taking
warp gets its atom's values in every order in which the others may already be at
the next one. No GPU needed."""
import os
import subprocess

from conftest import ROOT


def test_extent_in_every_order(tmp_path):
    exe = str(tmp_path / "host_feed")
    subprocess.run(["g++", "-O1", "-std=c++17", "-w", "-I", os.path.join(ROOT, "volume-compressor_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "host_feed.cpp"), "-o", exe], check=True)
    wrong, checked = map(int, subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split())
    assert checked > 1000 and wrong == 0
