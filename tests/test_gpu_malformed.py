"""Malformed payloads whose escape prefix shows far from every end (the EOB some
hundred positions on, stream bytes to spare), in the per-lane decoder's kernels:
every atom of the box, or one, which then ends last in its warp. The call
returns VC_ERR_FORMAT, as the one-atom decoders' does, and the library goes on."""
import struct

import numpy as np
import pytest

from test_gpu_decode import _slot_offset
from test_gpu_lane_rounds import encoded
from test_host_lanes import crafted

pytestmark = pytest.mark.gpu


def patched(data, atoms, which, eob, ones, rng):
    """`which` atoms' payloads replaced in place, their lengths kept."""
    data = bytearray(data)
    n = 0
    for az in range(atoms[2]):
        for ay in range(atoms[1]):
            for ax in range(atoms[0]):
                if not which(ax, ay, az):
                    continue
                off, ln = struct.unpack_from("<QI", data, _slot_offset(data, 0, az, ay, ax))
                bad = bytes([100]) + crafted(eob, [0, 2, 0, 14], ones, b"")
                if ln < len(bad) + 32:
                    continue
                data[off:off + len(bad)] = bad
                data[off + len(bad):off + ln] = rng.integers(0, 256, ln - len(bad)).astype(np.uint8).tobytes()
                n += 1
    return bytes(data), n


# solo warps beside the lanes (609 atoms, policy 0), the lanes alone (20,480)
@pytest.mark.parametrize("atoms,q,policy", [((29, 7, 3), 0.3, 0), ((32, 32, 20), 1.3, -1)])
@pytest.mark.parametrize("every", [True, False])
@pytest.mark.parametrize("eob", [200, 30000])
def test_overlong_prefix_is_refused(vc, gpu, atoms, q, policy, every, eob):
    data, dims = encoded(vc, atoms, q)
    last = (atoms[0] - 1, atoms[1] // 2, atoms[2] - 1)
    bad, n = patched(data, atoms, lambda *a: every or a == last, eob, 40, np.random.default_rng(eob))
    assert n >= (atoms[0] * atoms[1] * atoms[2] // 2 if every else 1)
    out = vc.DeviceBuffer(dims[0] * dims[1] * dims[2])
    vc.lib().vcg_set_rc_scalar_warps(policy)
    try:
        a = vc.Archive(bad)
        assert a.decode_region_device(0, (0, 0, 0) + dims, out) == vc.VC_ERR_FORMAT
        _, st = a.decode_regions([(0, (0, 0, 0) + dims)], [np.zeros(dims[::-1], np.uint8)])
        assert list(st) == [vc.VC_ERR_FORMAT]
        a.close()
        b = vc.Archive(data)
        assert b.decode_region_device(0, (0, 0, 0) + dims, out) == 0
        b.close()
    finally:
        vc.lib().vcg_set_rc_scalar_warps(-1)
        out.free()
