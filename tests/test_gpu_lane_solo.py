"""The longest atoms of a per-lane decode run alone, a warp each, while at most
one warp of lanes fills a sub-partition: the bytes and statuses of the scalar
decoder (policy 64, in slabs of fewer atoms) where all but one atom run alone
and their streams are longer than the shared-memory stage, at the last count
with solo warps and past it, and for a malformed stream."""
import struct

import numpy as np
import pytest

from rcstream import hostile_payload
from test_gpu_decode import _slot_offset
from test_gpu_lane_rounds import decoded, encoded

pytestmark = pytest.mark.gpu


def noise(vc, atoms):
    dims = tuple(32 * a for a in atoms)
    vol = np.random.default_rng(9).integers(0, 256, dims[::-1], dtype=np.uint8)
    s, data = vc.encode_q(vol, 10.0, [0.05] * 8)
    assert s == 0
    return data, dims


@pytest.mark.parametrize("atoms,q", [((29, 7, 3), 0.0), ((32, 32, 19), 13.5), ((32, 32, 20), 13.5)])
def test_solo_edges(vc, gpu, atoms, q):
    data, dims = encoded(vc, atoms, q) if q else noise(vc, atoms)
    if not q:
        off, ln = struct.unpack_from("<QI", data, _slot_offset(data, 0, 1, 2, 3))
        assert ln > 22 * 1024   # the stage
    assert (decoded(vc, data, dims, 0, dims[2]) == decoded(vc, data, dims, 64, 32)).all()


def test_solo_malformed(vc, gpu):
    data, dims = encoded(vc, (29, 7, 3), 0.3)
    data = bytearray(data)
    so = _slot_offset(data, 0, 1, 2, 3)
    off, ln = struct.unpack_from("<QI", data, so)
    bad = hostile_payload()
    assert ln >= len(bad)
    data[off:off + len(bad)] = bad
    data[off + len(bad):off + ln] = bytes(ln - len(bad))   # its length, and so its place in the order, stays
    a = vc.Archive(bytes(data))
    out = vc.DeviceBuffer(dims[0] * dims[1] * dims[2])
    got = []
    for policy in (0, 64):
        vc.lib().vcg_set_rc_scalar_warps(policy)
        try:
            got.append(a.decode_region_device(0, (0, 0, 0) + dims, out))
        finally:
            vc.lib().vcg_set_rc_scalar_warps(-1)
    assert got == [vc.VC_ERR_FORMAT] * 2


@pytest.mark.parametrize("rows", [26, 27])   # 4,160 and 4,320 atoms: below and above 28 an SM
def test_long_streams_change_over(vc, gpu, rows):
    """Streams too long to be staged: a warp each below the line, a lane each above it."""
    data, dims = encoded(vc, (32, rows, 5), 0.3)
    assert (decoded(vc, data, dims, -1, dims[2]) == decoded(vc, data, dims, 64, dims[2])).all()
