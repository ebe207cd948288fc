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


@pytest.mark.parametrize("dims,every,coarse", [
    ((160, 160, 160), 0, 0.05),    # 125 and 35 atoms, all long
    ((288, 288, 288), 0, 4.0),     # 729, all long: groups of two, and two a warp from their lists
    ((352, 352, 352), 2, 4.0),     # 1331: groups of three
    ((544, 544, 544), 3, 4.0),     # 4913: a lane each, six a warp from their lists
])
def test_long_atoms_match_the_oracle(vc, oracle, gpu, dims, every, coarse):
    qs = [0.05] + [coarse] * 7
    vol = volume(*dims, every)
    s1, got = vc.encode_q(vol, 10.0, qs)
    s2, want = oracle.encode_fixed_q(vol, 10.0, qs)
    assert s1 == s2 == 0
    assert len(got) == len(want)
    assert hashlib.sha256(bytes(got)).digest() == hashlib.sha256(bytes(want)).digest()
