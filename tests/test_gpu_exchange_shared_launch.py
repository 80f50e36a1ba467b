"""Exchange calls that one launch plays for several ranks: how the ranks share the SMs, and the results of each way."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _call(cp, entries, dim, dtype=torch.bfloat16, calls=2):
    """Runs the fused combine for ``entries`` rows per rank; returns the launch it took, having checked what it returned."""
    import helix_a2a_b200 as helix
    from helix_a2a_b200.ops import reference_math as rm
    from helix_a2a_b200.ops._ext import ext
    ext()
    gen = torch.Generator(device="cuda").manual_seed(entries * 10 + cp)
    ws = helix.allocate_workspace(cp, 0)
    helix.init_workspace_all_rows(ws, cp)
    o = torch.randn(cp, entries, cp, dim, device="cuda", generator=gen).to(dtype)
    lse = torch.randn(cp, entries, cp, device="cuda", generator=gen) * 3
    for _ in range(calls):      # the second call goes on where the first one left the rings
        got, glse = torch.ops.helix_a2a_b200.alltoall_combine(o, lse, ws, 0, cp, 0, True, False, 0, True, 0, 0)
    want, wlse = rm.head_scatter_combine_reference(o, lse, return_lse=True)
    # One rounding to the 16-bit result is at most 2^-8 (fp16 2^-11) of it.  Either side's fp32 sum of `cp` weighted values under 6,
    # with some twenty roundings and two-ulp exponentials each, is within cp * 6 * 2^-20.
    half_ulp = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    assert ((got.float() - want).abs() <= want.abs() * half_ulp + cp * 6 * 2.0 ** -20).all()
    assert ((glse - wlse).abs() <= 1e-5 * (1 + wlse.abs())).all()
    for r in range(cp):
        assert helix.check_status(ws, r, cp)["code"] == 0
    return ext().last_launch_info()


@pytest.mark.parametrize("cp,entries,dim", [(5, 512, 512), (6, 362, 512), (3, 256, 1024), (5, 362, 2048)])
def test_small_ctas_that_share_an_sm_keep_their_channels(native_built, cp, entries, dim):
    """Two small CTAs fit an SM: a plan of larger ones, with half of the channels, has to shorten a warp's chain of messages."""
    info = _call(cp, entries, dim)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert sms < info["channels"] * cp <= 2 * sms, info


@pytest.mark.parametrize("cp,entries,dim,recv", [(8, 91, 1024, 3), (7, 256, 1024, 7)])
def test_larger_ctas_where_they_shorten_the_chain(native_built, cp, entries, dim, recv):
    info = _call(cp, entries, dim)
    assert info["channels"] * cp <= torch.cuda.get_device_properties(0).multi_processor_count and info["recv_warps"] == recv, info


# on 148 SMs: messages of the peers per channel below and from 8 (rows of 128), entries per channel below and from 64 (rows of 256),
# entries per channel times ranks times lines below and from 2304 (rows of 512, 9 lines, and of 704, 12 lines)
@pytest.mark.parametrize("cp,entries,dim,ctas", [
    (2, 32, 128, 1), (8, 16, 128, 1), (4, 64, 128, 1), (2, 591, 128, 1), (2, 592, 128, 2), (8, 36, 128, 2),
    (2, 4735, 256, 1), (2, 4736, 256, 2), (8, 1152, 256, 2),
    (2, 5920, 512, 1), (2, 9472, 512, 2), (3, 3136, 512, 1), (4, 2367, 512, 1), (4, 2368, 512, 2), (8, 576, 512, 2),
    (3, 3087, 704, 1), (3, 3136, 704, 2)])
def test_two_ctas_per_sm_where_a_channel_has_enough_to_do(native_built, cp, entries, dim, ctas):
    assert _call(cp, entries, dim)["ctas_per_sm"] == ctas


# Rows of one, two and three iterations on two CTAs per SM.  Messages of 3, 5 and 9 lines: 342 entries a channel of rows of 128, 206 of
# rows of 256 and 115 of rows of 512 are more than half a ring of 2048, so receivers publish within the call, and three calls go
# round the ring.
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("cp,entries,dim", [
    (2, 148 * 345 + 3, 128), (4, 74 * 345 + 3, 128), (8, 37 * 345 + 3, 128),
    (2, 148 * 210 + 5, 256), (4, 37 * 64, 256), (8, 18 * 70 + 1, 256), (3, 98 * 210 + 1, 240),
    (2, 74 * 230 + 7, 512), (4, 37 * 66, 512)])
def test_bulk_calls_on_two_ctas_per_sm(native_built, dtype, cp, entries, dim):
    info = _call(cp, entries, dim, dtype, calls=3)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert info["ctas_per_sm"] == 2 and info["channels"] * cp > sms, info
    assert info["recv_warps"] > 8 and info["send_warps"] + info["recv_warps"] <= 16, info      # the bulk split of a CTA's warps
