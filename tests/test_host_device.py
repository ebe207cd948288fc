"""The device runtime's decode call (csrc/vc_device.cu) built for the host over
stand-ins for the CUDA runtime and the launches (tests/host_device.cpp): a wait
that ran out in the inverse transform fails the call (VC_ERR_IO) whichever way its
output leaves, in one copy or in slabs, and also where a malformed atom ends the
slabs. No GPU needed."""
import os
import subprocess

import pytest

from conftest import ROOT

VC_OK, VC_ERR_FORMAT, VC_ERR_IO = 0, 1, 4


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("host_device") / "host_device")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-w", "-I", os.path.join(ROOT, "volume-compressor_gb300", "csrc"),
                        "-I", os.path.join(cuda, "include"), os.path.join(ROOT, "tests", "host_device.cpp"),
                        "-o", exe, "-lpthread"], capture_output=True, text=True)
    if r.returncode:
        pytest.fail(r.stderr[-2000:])
    return exe


@pytest.mark.parametrize("mib,slabs", [(8, False), (128, True)])
@pytest.mark.parametrize("malformed,gave_up,status", [(-1, 0, VC_OK), (-1, 1, VC_ERR_IO), (5, 0, VC_ERR_FORMAT),
                                                      (5, 1, VC_ERR_IO)])
def test_wait_that_ran_out_fails_the_call(harness, mib, slabs, malformed, gave_up, status):
    r = subprocess.run([harness, str(malformed), str(gave_up), str(mib)], capture_output=True, text=True, check=True)
    got, transforms = map(int, r.stdout.split())
    assert got == status
    assert (transforms > 1) == (slabs and malformed < 0)
