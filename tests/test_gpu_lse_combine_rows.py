"""Stand-alone LSE combine (``csrc/lse_combine.cu``): half a warp or a warp per row, ranks below, at and above the lanes of a row."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# rows that end inside a warp and a block; both sides of the 16-chunk rule (128 elements) and of 2048 rows for one or two ranks
@pytest.mark.parametrize("n,rows,dim", [(1, 1, 8), (1, 5, 8), (1, 2100, 128), (2, 7, 64), (3, 17, 128), (8, 33, 128), (9, 5, 136), (16, 8, 120), (17, 4, 128),
                                        (33, 3, 128), (40, 9, 512), (4, 2, 520), (2, 2047, 128), (2, 2048, 128), (2, 2049, 72)])
@pytest.mark.parametrize("layout", ["NBHD", "BHND"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_combine_rows(native_built, n, rows, dim, layout, dtype):
    import helix_a2a_b200 as helix
    gen = torch.Generator(device="cuda").manual_seed(n * 1000 + dim)
    o = torch.randn(n, rows, dim, device="cuda", generator=gen).to(dtype)
    lse = torch.randn(n, rows, device="cuda", generator=gen) * 3
    lse[0, 0], lse[n // 2, rows - 1], lse[-1, rows // 2] = float("-inf"), float("nan"), float("inf")
    dead = torch.isfinite(lse).logical_not()
    o[dead] = float("nan")                               # rows without a weight are not even read
    l64 = lse.double().masked_fill(dead, float("-inf"))
    top = l64.max(0).values
    w = torch.where(top.isinf(), torch.zeros_like(l64), (l64 - top).exp())
    s = w.sum(0)
    want = (w.unsqueeze(-1) * o.double().nan_to_num(0.0)).sum(0) / s.clamp_min(1e-300).unsqueeze(-1)
    want_lse = torch.where(s > 0, top + s.log(), torch.full_like(s, float("-inf")))
    args = (o, lse) if layout == "NBHD" else (o.transpose(0, 1).contiguous(), lse.transpose(0, 1).contiguous())
    got, g = helix.lse_combine(*args, layout=layout, return_lse=True)
    # One rounding to the 16-bit result is at most 2^-8 (fp16 2^-11) of it.  The fp32 sum of n weighted values under 5.5 has n
    # roundings of 2^-24, and the weights' arguments (under 32) and exponentials some 60 more.
    bound = want.abs() * 2.0 ** (-8 if dtype == torch.bfloat16 else -11) + 5.5 * (n + 60) * 2.0 ** -24
    assert ((got.double() - want).abs() <= bound).all(), ((got.double() - want).abs() - bound).max()
    live = s > 0
    assert torch.equal(g[~live], want_lse[~live].float()) and ((g[live] - want_lse[live]).abs() < 1e-5 * (1 + want_lse[live].abs())).all()
