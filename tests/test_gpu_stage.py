"""One-atom range decoder on streams staged in shared memory: payload lengths
around a staged word and around the staging limits (one atom alone stages any
stream; a full sub-partition's worth of long streams does not fit and is read
from global memory). Crafted payload lengths come from cutting coded atoms short
(bytes past the end read as zero), so the oracle's status and bytes are the bar;
they are exact."""
import numpy as np
import pytest

from conftest import load_archive
from test_gpu_decode import _slot_offset

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cut", [2, 3, 4, 5, 6, 7, 8, 9, 12, 13, 17, 100, 1001, 1002, 1003])
def test_short_streams(vc, oracle, gpu, golden, cut):
    data = bytearray(load_archive(golden["synth_prime_97x131x65_t20"]))
    for az, ay, ax in ((0, 0, 0), (1, 2, 1)):
        at = _slot_offset(data, 0, az, ay, ax)
        data[at + 8:at + 12] = cut.to_bytes(4, "little")   # payload length
    data = bytes(data)
    a, o = vc.Archive(data), oracle.Archive(data)
    for az, ay, ax in ((0, 0, 0), (1, 2, 1)):
        s1, g = a.decode_atom(0, ax, ay, az)
        s2, r = o.decode_atom(0, ax, ay, az)
        assert s1 == s2 and (g == r).all()
    s1, g = a.decode_lod(0)
    s2, r = o.decode_lod(0)
    assert s1 == s2 and (s1 or (g == r).all())


@pytest.mark.parametrize("atoms", [1, 152, 153, 608, 609, 1216])
def test_long_streams(vc, oracle, gpu, atoms):
    """Noise at the finest q: payloads of about 40 KB, of which one SM stages at most five."""
    rng = np.random.default_rng(atoms)
    vol = rng.integers(0, 256, (32, 32, 32 * atoms), dtype=np.uint8)
    s, data = vc.encode_q(vol, 10.0, [0.05] * 8)
    assert s == 0
    a, o = vc.Archive(data), oracle.Archive(data)
    s, got = a.decode_lod(0)
    s2, want = o.decode_lod(0, threads=8)
    assert s == s2 == 0 and (got == want).all()
