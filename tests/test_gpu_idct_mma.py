"""Inverse transform on the tensor cores (decodes of at least four atoms per SM):
contents and quantisers on both sides of the coefficient norm up to which its
sums are exact, levels that end at every tile of four kz, zero atoms between, and
boxes that cut atoms on every side. The bytes are the oracle's (integers: no
tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ATOMS = (29, 7, 3)   # x, y, z: 609, the first count above four per SM on 152 SMs
DIMS = tuple(32 * n for n in ATOMS)


def volume(kind, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nz = DIMS
    if kind == "binary":   # noise of 0 and 255: coefficient norm 23,000 an atom
        return (rng.integers(0, 2, (nz, ny, nx)) * 255).astype(np.uint8)
    if kind == "halves":   # the largest norms: half of an atom 0, half 255, split along x, y or z
        z, y, x = np.ogrid[:nz, :ny, :nx]
        which = rng.integers(0, 3, (ATOMS[2], ATOMS[1], ATOMS[0]))
        w = which.repeat(32, 0).repeat(32, 1).repeat(32, 2)
        v = np.where(w == 0, (x // 16) % 2, np.where(w == 1, (y // 16) % 2, (z // 16) % 2))
        return (v * 255).astype(np.uint8)
    # bands along z: atom i keeps frequencies up to i mod 33, every third atom is zero
    v = np.zeros((nz, ny, nx), np.uint8)
    zz = np.arange(32)
    for i in range(ATOMS[0] * ATOMS[1] * ATOMS[2]):
        if i % 3 == 2:
            continue
        az, ay, ax = i // (ATOMS[0] * ATOMS[1]), (i // ATOMS[0]) % ATOMS[1], i % ATOMS[0]
        f = i % 33
        wave = 128 + 100 * np.cos(np.pi * f * (2 * zz + 1) / 64)
        v[az * 32:az * 32 + 32, ay * 32:ay * 32 + 32, ax * 32:ax * 32 + 32] = wave.astype(np.uint8)[:, None, None]
    return v


@pytest.mark.parametrize("kind,q", [("binary", 0.5), ("binary", 60.0), ("binary", 900.0), ("binary", 4096.0),
                                    ("halves", 0.05), ("halves", 2000.0), ("bands", 0.3), ("bands", 40.0)])
def test_inverse_matches_oracle(vc, oracle, gpu, kind, q):
    vol = volume(kind, int(q * 100))
    s, data = vc.encode_q(vol, 10.0, [q] * 8)
    assert s == 0
    s, want = oracle.Archive(data).decode_lod(0, threads=8)
    assert s == 0
    a = vc.Archive(data)
    s, got = a.decode_lod(0)
    assert s == 0 and (got == want).all()
    for box in ((0, 0, 0) + DIMS, (1, 0, 0) + DIMS, (5, 3, 7, DIMS[0] - 1, DIMS[1] - 9, DIMS[2] - 30),
                (0, 16, 31, DIMS[0], DIMS[1] - 1, DIMS[2] - 31)):
        x0, y0, z0, x1, y1, z1 = box
        s, got = a.decode_region(0, box)
        assert s == 0 and (got.reshape(z1 - z0, y1 - y0, x1 - x0) == want[z0:z1, y0:y1, x0:x1]).all()
