"""Streams staged in shared memory (stage_fits, built for the host): every length
up to 2^32 - 1 against the room, the zero bytes after it counted. A payload of
nearly 4 GiB, in an archive larger than that, is not taken for a short one. No GPU
needed."""
import os
import subprocess

from conftest import ROOT


def test_stage_fits(tmp_path):
    exe = str(tmp_path / "host_stage")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-w", "-I", os.path.join(ROOT, "volume-compressor_gb300", "csrc"),
                           os.path.join(ROOT, "tests", "host_stage.cpp"), "-o", exe])
    out = subprocess.check_output([exe], text=True)
    assert out == "10800 tried\n"
