"""The coder's passes over carry-free sums (csrc/rc_encode.cuh) and the resolve
that makes bytes of them: archives byte-identical to the oracle's where a launch
is one group of one atom per SM sub-partition (two producers a group), of two, of
three (a producer with one atom), a lane per atom, and where an atom has more
bytes than its slot of sums holds (white noise at the finest quantiser). And the
lengths from costs that rate control goes by: 24 passes whose totals choose the
quantiser, of which a few leave atoms in doubt that the coder then sizes."""
import hashlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def volume(nx, ny, nz, noise):
    rng = np.random.default_rng(nx * ny * nz)
    if noise:
        return rng.integers(0, 256, (nz, ny, nx)).astype(np.uint8)
    # smooth everywhere, empty in places (zero atoms), rough in some slabs
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij", sparse=True)
    v = 110 + 60 * np.sin(x / 11.0) * np.cos(y / 17.0) + 30 * np.sin(z / 5.0 + x / 40.0)
    v[(z // 64 + y // 96 + x // 128) % 5 == 0] = 0
    k = (z // 32) % 7 == 3
    v = np.where(k, v + rng.normal(0, 12, (nz, ny, 1)), v)
    return np.clip(v, 0, 255).astype(np.uint8)


@pytest.mark.parametrize("dims,qs,noise", [
    ((70, 45, 90), [0.05] * 8, True),             # LOD0: 18 atoms, more bytes than a slot holds
    ((33, 1, 1), [1.3] * 8, False),               # 2 atoms, lists of a few entries
    ((289, 288, 320), [1.3 * 0.6 ** k for k in range(8)], False),    # 900 atoms: groups of two
    ((320, 320, 512), [2.6 * 0.6 ** k for k in range(8)], False),    # 1600: of three
    ((544, 544, 544), [6.5 * 0.6 ** k for k in range(8)], False),    # 4913: a lane each
])
def test_archives_match_the_oracle(vc, oracle, gpu, dims, qs, noise):
    qs = [max(0.05, q) for q in qs]
    vol = volume(*dims, noise)
    s1, got = vc.encode_q(vol, 10.0, qs)
    s2, want = oracle.encode_fixed_q(vol, 10.0, qs)
    assert s1 == s2 == 0
    assert len(got) == len(want)
    assert hashlib.sha256(bytes(got)).digest() == hashlib.sha256(bytes(want)).digest()


@pytest.mark.parametrize("dims,target", [((289, 160, 170), 10.0), ((96, 64, 65), 2.0), ((64, 64, 64), 1000.0)])
def test_rate_control_matches_the_oracle(vc, oracle, gpu, dims, target):
    vol = volume(*dims, False)
    s1, got = vc.encode(vol, target)
    s2, want = oracle.encode(vol, target)
    assert s1 == s2 == 0
    assert len(got) == len(want)
    assert hashlib.sha256(bytes(got)).digest() == hashlib.sha256(bytes(want)).digest()
