"""Atoms with more coder bytes than a slot of sums holds (white noise at the
finest quantiser), among atoms that fit, in every form of the coder: groups of
one, two and three atoms, a lane per atom, and one to several of them a warp
where they are coded from their lists, in LOD0 and in the coarser LODs at once.
Archives are the oracle's, byte for byte."""
import hashlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def volume(nx, ny, nz, every):
    """White noise, `every`-th slab of atoms along x smooth instead."""
    v = np.random.default_rng(nx + every).integers(0, 256, (nz, ny, nx), dtype=np.uint8)
    if every:
        z, y, x = np.ogrid[:nz, :ny, :nx]
        smooth = (120 + 50 * np.sin(x / 9.0) * np.cos(y / 13.0 + z / 29.0)).astype(np.uint8)
        pick = ((np.arange(nx) // 32) % every) == every - 1
        v[:, :, pick] = smooth[:, :, pick]
    return v


@pytest.mark.parametrize("dims,every,q,coarse", [
    ((160, 160, 160), 0, 0.05, 0.05),    # 125 and 35 atoms, all long
    ((288, 288, 288), 0, 0.05, 4.0),     # 729, all long: groups of two, and two a warp from their lists
    ((352, 352, 352), 2, 0.1, 4.0),      # 1331: groups of three
    ((544, 544, 544), 3, 0.05, 4.0),     # 4913: a lane each; their lists tell which are long, six a warp from them
    ((544, 544, 544), 3, 0.2, 4.0),      # just too long, which their lists don't tell
    ((544, 544, 544), 0, 0.05, 0.05),    # every atom of every LOD
])
def test_long_atoms_match_the_oracle(vc, oracle, gpu, dims, every, q, coarse):
    qs = [q] + [coarse] * 7
    vol = volume(*dims, every)
    s1, got = vc.encode_q(vol, 10.0, qs)
    s2, want = oracle.encode_fixed_q(vol, 10.0, qs)
    assert s1 == s2 == 0
    assert len(got) == len(want)
    assert hashlib.sha256(bytes(got)).digest() == hashlib.sha256(bytes(want)).digest()


def test_appended_long_atoms(vc, gpu, tmp_path):
    """Long atoms through the writer: the payloads of the whole-volume encoder at the same quantiser."""
    dims = (96, 96, 64)
    vol = volume(*dims, 3)
    s, want = vc.encode_q(vol, 10.0, [0.05] * 8)
    assert s == 0
    path = str(tmp_path / "long.vca")
    with vc.Writer(path, dims, 10.0) as w:
        assert w.set_base_q(0, 0.05) == 0
        assert w.append_box(0, (0, 0, 0) + dims, vol) == 0
    with open(path, "rb") as f:
        got = f.read()
    a, b = vc.Archive(want), vc.Archive(got)
    for az in range(2):
        for ay in range(3):
            for ax in range(3):
                _, o1, n1 = a.payload_range(0, az, ay, ax)
                _, o2, n2 = b.payload_range(0, az, ay, ax)
                assert want[o1:o1 + n1] == got[o2:o2 + n2]
                assert (n1 > 32768) == (ax != 2)
