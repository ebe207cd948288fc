"""A wait that runs out inside the tensor-core inverse transform ends the kernel
with its fail word set, whichever role of the CTA is late (tests/give_up.cu, with
a limit of four milliseconds on the waits): no role stays behind at a barrier."""
import os
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def build(exe):
    csrc = os.path.join(ROOT, "volume-compressor_gb300", "csrc")
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-DVCG_WAIT_TRIES=1024u",
                    "-I", csrc, os.path.join(ROOT, "tests", "give_up.cu"), "-o", exe], check=True)


def test_every_role_late(tmp_path, gpu):
    exe = str(tmp_path / "give_up")
    build(exe)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
    rows = [tuple(map(int, line.split())) for line in r.stdout.splitlines()]
    assert rows == [(0, 0, 0), (1, 0, 1), (2, 0, 1), (3, 0, 1), (4, 0, 1)]
