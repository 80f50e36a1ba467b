"""MLA decode attention on clusters of two CTAs (``csrc/decode_attn_mla_pair.cu``) against the fp32 oracle."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(seq_lens, page, seed=0, std=0.5):
    from helix_a2a_b200.ops import reference_math as rm
    gen = torch.Generator(device="cuda").manual_seed(seed)
    B = len(seq_lens)
    blocks = max((s + page - 1) // page for s in seq_lens) + 1
    pages = B * blocks + 2
    bt = torch.randperm(pages, generator=gen, device="cuda")[:B * blocks].view(B, blocks).int()
    ckv, scales = rm.quantize_fp8_blockscaled(torch.randn(pages, page, 512, device="cuda", generator=gen), 128)
    kpe = torch.randn(pages, page, 64, device="cuda", generator=gen).bfloat16()
    qn = (torch.randn(B, 128, 512, device="cuda", generator=gen) * std).bfloat16()
    qp = (torch.randn(B, 128, 64, device="cuda", generator=gen) * std).bfloat16()
    return qn, qp, ckv, scales, kpe, bt, torch.tensor(seq_lens, dtype=torch.int32, device="cuda")


def _check(seq_lens, page, ctas, scale, base2=False, std=0.5, poison=False):
    from helix_a2a_b200.ops import attention, reference_math as rm
    from helix_a2a_b200.ops.oproj import check_compute_status
    qn, qp, ckv, scales, kpe, bt, sl = _case(seq_lens, page, seed=len(seq_lens) + page, std=std)
    if poison:       # whatever lies behind a sequence's last token in its page must not reach the result
        for b, n in enumerate(seq_lens):
            if n % page:
                pg = int(bt[b, n // page])
                ckv.view(torch.uint8)[pg, n % page:] = 0x7F
                kpe[pg, n % page:] = float("nan")
                scales[pg, n % page:] = float("inf")
    o, lse = attention.mla_decode(qn, qp, ckv, scales, kpe, bt, sl, scale=scale, ctas=ctas, lse_base2=base2,
                                  max_seq_len=max(seq_lens))
    torch.cuda.synchronize()
    check_compute_status(qn)
    lat = rm.dequantize_fp8_blockscaled(ckv, scales, 128)
    for b, n in enumerate(seq_lens):
        if n == 0:
            assert (o[b] == 0).all() and (lse[b] == float("-inf")).all()
            continue
        idx = bt[b, :(n + page - 1) // page].long()
        o_ref, l_ref = rm.mla_partial_attention(qn[b:b + 1].float(), qp[b:b + 1].float(), lat[idx].reshape(-1, 512)[:n],
                                                kpe[idx].reshape(-1, 64)[:n].float(), scale, base2)
        # Dequantised values carry two bf16 roundings (scale, product), probabilities one, the result one: 4 x 2^-9 of
        # values that are at most about 4.5.  A score is off by at most 2^-8 of the sum of its four blocks' |q . k|, each
        # 0.5 * sqrt(128) / sqrt(192) = 0.41 in the standard deviation and under three of them: 2^-8 * 4 * 3 * 0.41 = 0.019.
        # That is also the bound of the LSE with a few tokens.  From 64 on their errors, which have either sign, average
        # out to less than a quarter of it: 5e-3, where a systematic error of the scores would show.
        assert (o[b].float() - o_ref[0]).abs().max() < 3e-2, (b, n)
        assert (lse[b] - l_ref[0]).abs().max() < (1.9e-2 if n < 64 else 5e-3) * (1.45 if base2 else 1), (b, n)


# edges of the 64-token tile and of the 16-token unit, one to several tiles a piece, more sequences than clusters, empty
# sequences, pieces whose boundaries fall inside and between sequences, every shape of the fold (by batch size)
@pytest.mark.parametrize("seq_lens,page,ctas", [
    ([1], 16, 0), ([64], 16, 0), ([15, 16, 17, 63, 64, 65], 16, 2), ([127, 0, 128, 129], 32, 4), ([300, 1, 700], 48, 6),
    ([1024], 64, 2), ([1000], 64, 32), ([5, 0, 64] * 70, 16, 0), ([2049, 640, 4096], 32, 10), ([20000], 16, 0),
    ([2000] * 6, 16, 0), ([300, 900] * 10, 32, 0), ([700] * 40, 16, 0),
    # more sequences than clusters (the fold goes by what the clusters noted), more than the table in shared memory holds
    ([200, 0, 16] * 50, 16, 0), ([64] * 75, 16, 0), ([9000] + [40] * 80, 16, 0), ([130, 0, 64, 1] * 150, 16, 0),
    ([500, 70, 900], 16, 2), ([33, 700, 20, 0, 260], 16, 4)])
def test_pair_kernel_matches_fp32_reference(native_built, seq_lens, page, ctas):
    _check(seq_lens, page, ctas, 1.0 / math.sqrt(192))


def test_pair_kernel_options(native_built):
    _check([70, 513], 16, 4, 1.0 / math.sqrt(192), base2=True, poison=True)
    _check([70, 513], 16, 4, -1.0 / math.sqrt(192))          # a negative scale turns maxima into minima


def test_pair_kernel_rescales_and_agrees_with_one_piece(native_built):
    """Scores that keep growing along the sequence force the running maximum to be re-applied many times."""
    from helix_a2a_b200.ops import attention, reference_math as rm
    n, page = 1024, 16
    qn, qp, ckv, scales, kpe, bt, sl = _case([n], page, seed=3)
    qp[:] = 1.0
    rows = bt[0, :n // page].long()
    kpe[rows] = (torch.arange(n, device="cuda").float() / n * 6).view(n // page, page, 1).bfloat16()     # up to 384
    lat = rm.dequantize_fp8_blockscaled(ckv, scales, 128)[rows].reshape(-1, 512)
    o_ref, l_ref = rm.mla_partial_attention(qn.float(), qp.float(), lat, kpe[rows].reshape(-1, 64).float(), 0.25)
    for ctas in (2, 0):
        o, lse = attention.mla_decode(qn, qp, ckv, scales, kpe, bt, sl, scale=0.25, ctas=ctas, max_seq_len=n)
        torch.cuda.synchronize()
        assert (lse - l_ref).abs().max() < 5e-2
        # scores here are off by up to 0.25 * 0.5 * 2^-8 * sqrt(512) = 0.011, so weights by 1.1 %
        assert (o.float() - o_ref).abs().max() < 0.1


def test_unaligned_queries_keep_a_kernel_that_takes_them(native_built):
    """A contiguous q_nope that starts 4 bytes off a 16-byte boundary (a view into a larger buffer)."""
    from helix_a2a_b200.ops import attention
    qn, qp, ckv, scales, kpe, bt, sl = _case([200, 33], 16, seed=9)
    shifted = torch.empty(qn.numel() + 8, dtype=qn.dtype, device="cuda")[2:2 + qn.numel()].view_as(qn).copy_(qn)
    assert shifted.data_ptr() % 16 == 4 and shifted.is_contiguous()
    want, got = (attention.mla_decode(q, qp, ckv, scales, kpe, bt, sl, scale=0.07, max_seq_len=200) for q in (qn, shifted))
    # two kernels of the same precision: one bf16 rounding of values up to about 4.5 apart, and of the probabilities
    assert (want[0].float() - got[0].float()).abs().max() < 3e-2 and (want[1] - got[1]).abs().max() < 1e-3


def _shift(t, elements):
    """The same contiguous tensor, ``elements`` behind the start of its storage."""
    flat = torch.empty(t.numel() + 16, dtype=t.dtype, device=t.device)[elements:elements + t.numel()]
    flat.copy_(t.reshape(-1))
    return flat.view(t.shape)


# q_nope and q_pe each 0, 2, 4 or 8 bytes off a 16-byte boundary: every kernel either reads them there or gets a copy
@pytest.mark.parametrize("variant", ["pair", "ws", "lockstep"])
@pytest.mark.parametrize("off_nope,off_pe", [(0, 1), (0, 2), (0, 4), (1, 0), (2, 2), (1, 1), (4, 4)])
def test_queries_may_start_anywhere(native_built, monkeypatch, variant, off_nope, off_pe):
    from helix_a2a_b200.ops import attention
    monkeypatch.setenv("HELIX_A2A_MLA_VARIANT", variant)
    qn, qp, ckv, scales, kpe, bt, sl = _case([200, 33], 16, seed=9)
    want = attention.mla_decode(qn, qp, ckv, scales, kpe, bt, sl, scale=0.07, max_seq_len=200)
    a, b = _shift(qn, off_nope), _shift(qp, off_pe)
    assert a.data_ptr() % 16 == 2 * off_nope and b.data_ptr() % 16 == 2 * off_pe
    got = attention.mla_decode(a, b, ckv, scales, kpe, bt, sl, scale=0.07, max_seq_len=200)
    # as in the test above where another kernel of the same precision may have run, to the bit elsewhere
    if variant == "pair" and off_nope in (2, 4):
        assert (want[0].float() - got[0].float()).abs().max() < 3e-2 and (want[1] - got[1]).abs().max() < 1e-3
    else:
        assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1])


def test_a_cache_off_its_boundary_is_refused(native_built, monkeypatch):
    from helix_a2a_b200.ops import attention
    qn, qp, ckv, scales, kpe, bt, sl = _case([200, 33], 16, seed=9)
    call = lambda c, s, k: attention.mla_decode(qn, qp, c, s, k, bt, sl, scale=0.07, max_seq_len=200)   # noqa: E731
    want = call(ckv, scales, kpe)
    with pytest.raises(RuntimeError, match="16-byte boundary"):
        call(_shift(ckv.view(torch.uint8), 8).view(ckv.dtype), scales, kpe)
    with pytest.raises(RuntimeError, match="16-byte boundary"):
        call(ckv, scales, _shift(kpe, 2))
    got = call(ckv, _shift(scales, 1), kpe)              # 4 bytes at a time in the pair kernel
    assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1])
    monkeypatch.setenv("HELIX_A2A_MLA_VARIANT", "ws")
    with pytest.raises(RuntimeError, match="16-byte boundary"):
        call(ckv, _shift(scales, 1), kpe)
