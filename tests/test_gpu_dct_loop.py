"""The butterfly form with more atoms than SMs, where a CTA holds the next atom's
rows, or has them on their way into L2, while it transforms one: the oracle's
coefficients and voxels bit for bit, on volumes of one atom less, as many, one
more and twice as many and one."""
import numpy as np
import pytest

from test_gpu_dct import oracle_fdct, oracle_idct, run_forward

pytestmark = pytest.mark.gpu

SMS = 152


@pytest.mark.parametrize("atoms", [SMS - 1, SMS, SMS + 1, 2 * SMS + 1])
def test_butterfly_over_several_atoms_a_cta(vc, oracle, gpu, atoms):
    dims = (32 * atoms, 32, 32)
    vol = np.random.default_rng(atoms).integers(0, 256, dims[::-1], dtype=np.uint8)
    want, dcs = oracle_fdct(vol, -1)
    got, got_dcs = run_forward(vc, vol, -1, vc.DCT_BUTTERFLY)
    assert (got_dcs == dcs).all()
    assert (got == want).all()
    dcoef = vc.DeviceBuffer(got.nbytes)
    dcoef.upload(got)
    ddc = vc.DeviceBuffer(dcs.size)
    ddc.upload(dcs)
    back = vc.DeviceBuffer(vol.size)
    s, redone = vc.dct_inverse(dcoef, dims, vc.DCT_ATOM_DC, vc.DCT_BUTTERFLY, back, ddc)
    assert s == vc.VC_OK and redone == 0
    assert (back.download(vol.size).reshape(vol.shape) == oracle_idct(want, dims, -1, dcs)).all()
