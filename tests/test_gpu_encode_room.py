"""Encodes when the archive's own allocation fails: what the call holds for speed
alone (the kept transform, the coder's sums) is given back for it, so the call
succeeds as it does without them. vcg_debug_fail_alloc(n) makes the n-th
allocation of a call fail."""
import pytest

from test_gpu_oom import LIMIT, in_thread, sha

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,qs", [((96, 80, 72), None), ((96, 80, 72), [1.3] * 8), ((33, 20, 30), [1.3] * 8)])
def test_archive_allocation_has_a_way_out(vc, gpu, dims, qs):
    vol = vc.synth(*dims, 0x0A110E)

    def op():
        return vc.encode_q(vol, 10.0, qs) if qs else vc.encode(vol, 10.0)

    (s, want), _ = in_thread(vc, op)
    assert s == vc.VC_OK
    failed = 0
    for n in range(1, LIMIT):
        vc.lib().vcg_debug_fail_alloc(n)
        try:
            (s, got), err = in_thread(vc, op)
        finally:
            hit = vc.lib().vcg_debug_fail_alloc(0) == -1
        if not hit:
            break
        assert s in (vc.VC_OK, vc.VC_ERR_OOM)
        assert s == vc.VC_ERR_OOM or sha(got) == sha(want)
        if s == vc.VC_ERR_OOM:
            failed += 1
            assert "archive" not in err, err
    assert n > failed + 1   # the run without a failure, and the allocations with a way out


def test_lists_of_three_quantisers_have_a_way_out(vc, gpu):
    """Rate control of few atoms holds the lists of three quantisers at once: where they
    have no room, one at a time."""
    vol = vc.synth(96, 80, 72, 0x0A110E)

    def op():
        return vc.encode(vol, 10.0)

    (s, want), _ = in_thread(vc, op)
    assert s == vc.VC_OK
    errs = []
    for n in range(1, LIMIT):
        vc.lib().vcg_debug_fail_alloc(n)
        try:
            (s, got), err = in_thread(vc, op)
        finally:
            hit = vc.lib().vcg_debug_fail_alloc(0) == -1
        if not hit:
            break
        assert s in (vc.VC_OK, vc.VC_ERR_OOM)
        assert s == vc.VC_ERR_OOM or sha(got) == sha(want)
        errs += [err] if s == vc.VC_ERR_OOM else []
    assert errs and not any("coefficient lists" in e for e in errs), errs
