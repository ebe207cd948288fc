"""Per-lane range decoder at the edges of its work split: 32 atoms a warp, four
warps per SM before a sub-partition takes a second one, eight warps per SM before
a second CTA; payloads on both sides of the length from which a round takes no
zeros at once. The decoded bytes must be those of the scalar decoder (policy 64,
in slabs of fewer atoms), and the oracle's where the volume is small. Bytes are exact,
so there is no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def encoded(vc, atoms, q):
    dims = (32 * atoms[0], 32 * atoms[1], 32 * atoms[2])
    vol = vc.synth_device(*dims, vc.config_seed(77) + sum(atoms))
    s, data = vc.encode_q(vol, 10.0, [max(0.05, q * 0.6 ** l) for l in range(8)], on_device=dims)
    vol.free()
    assert s == 0
    return data, dims


def decoded(vc, data, dims, policy, slab):
    """LOD0 by region decodes of `slab` voxel layers each (a whole number of atoms)."""
    nx, ny, nz = dims
    a = vc.Archive(data)
    got = []
    vc.lib().vcg_set_rc_scalar_warps(policy)
    try:
        for z in range(0, nz, slab):
            z1 = min(nz, z + slab)
            out = vc.DeviceBuffer(nx * ny * (z1 - z))
            assert a.decode_region_device(0, (0, 0, z, nx, ny, z1), out) == 0
            got.append(out.download())
            out.free()
    finally:
        vc.lib().vcg_set_rc_scalar_warps(-1)
    a.close()
    return np.concatenate(got)


# atoms: 609 (the first count above one per sub-partition), one lane more and one
# fewer than a full warp, a warp more than one per sub-partition, more than eight
# warps per SM (a second CTA)
@pytest.mark.parametrize("atoms,q", [((29, 7, 3), 0.3), ((29, 7, 3), 6.5), ((11, 19, 3), 2.5), ((13, 17, 3), 2.5),
                                     ((9, 83, 26), 6.5), ((60, 25, 26), 13.5)])
def test_lane_decoder_edges(vc, oracle, gpu, atoms, q):
    data, dims = encoded(vc, atoms, q)
    got = decoded(vc, data, dims, 0, dims[2])
    assert (got == decoded(vc, data, dims, 64, 8 * 32)).all()
    if got.size <= 700 * 32768:
        s, want = oracle.Archive(data).decode_lod(0)
        assert s == 0 and (got == want.reshape(-1)).all()
