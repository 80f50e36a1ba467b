"""GQA decode attention: unsplit short sequences and the fold kernel, against the fp32 oracle and each other."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(lens, hkv, group, page, layout, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    blocks = max(1, max((n + page - 1) // page for n in lens))
    pages = len(lens) * blocks + 3
    bt = torch.randperm(pages, generator=gen, device="cuda")[:len(lens) * blocks].view(len(lens), blocks).int()
    shape = (pages, hkv, page, 128) if layout == "HND" else (pages, page, hkv, 128)
    k, v = (torch.empty(shape, device="cuda").normal_(generator=gen).bfloat16() for _ in range(2))
    q = torch.empty(len(lens), hkv * group, 128, device="cuda").normal_(generator=gen).bfloat16()
    return q, k, v, bt, torch.tensor(lens, dtype=torch.int32, device="cuda")


# around one 16-token block, empty sequences, few and many pairs, groups of one to eight heads; both sides of the longest
# unsplit sequence on 148 SMs: 41 blocks (656 tokens) with 8 pairs, 96 blocks (1536 tokens) from 173 pairs on; splits = 0 leaves
# the form to the library, the others force shares and the fold
@pytest.mark.parametrize("lens,hkv,group,page,layout", [
    ([1], 1, 1, 16, "HND"), ([15, 16, 17, 0], 8, 8, 16, "NHD"), ([300], 8, 8, 16, "HND"), ([511, 512, 64], 2, 4, 32, "NHD"),
    ([513, 3], 8, 3, 16, "HND"), ([100] * 40 + [0, 1], 8, 8, 64, "HND"), ([2000, 0, 90, 7000], 4, 8, 16, "HND"),
    ([40, 600] * 150, 2, 8, 16, "HND"), ([20000], 8, 8, 16, "NHD"), ([656], 8, 8, 16, "HND"), ([657], 8, 8, 16, "HND"),
    ([1536, 5, 900, 0] * 25, 4, 2, 16, "HND"), ([1537, 5, 900, 0] * 25, 4, 2, 16, "NHD")])
def test_forms_agree_with_the_oracle(native_built, lens, hkv, group, page, layout):
    from helix_a2a_b200.ops import attention, reference_math as rm
    from helix_a2a_b200.ops.oproj import check_compute_status
    q, k, v, bt, sl = _case(lens, hkv, group, page, layout, len(lens) + hkv)
    kc, vc = (t if layout == "HND" else t.permute(0, 2, 1, 3) for t in (k, v))
    o_ref, l_ref = rm.paged_decode_attention_reference(q.cpu(), kc.cpu(), vc.cpu(), bt.cpu(), sl.cpu(), 1 / math.sqrt(128), False)
    for splits in (0, 1, 3):
        for _ in range(2):      # the second call also shows that the first one left counters and pools as it found them
            o, lse = attention.gqa_decode(q, k, v, bt, sl, layout=layout, splits=splits, max_seq_len=max(lens))
        torch.cuda.synchronize()
        check_compute_status(q)
        live = (sl > 0).cpu()
        # probabilities and the result carry one bf16 rounding each: 2 x 2^-9 of values up to about 4.5
        assert (o.cpu().float() - o_ref.float()).abs().max() < 2e-2, splits
        assert (lse.cpu()[live] - l_ref[live]).abs().max() < 1e-3, splits
        assert torch.isneginf(lse.cpu()[~live]).all()


# 1024 unsplit pairs are more CTAs than any split launch has; 2 x 20000 tokens are split
@pytest.mark.parametrize("lens,hkv", [([40, 17, 0, 300] * 32, 8), ([20000, 700], 8)])
def test_time_stamps_have_a_row_for_every_cta(native_built, monkeypatch, lens, hkv):
    from helix_a2a_b200.ops import attention
    from helix_a2a_b200.ops._ext import ext, ops
    q, k, v, bt, sl = _case(lens, hkv, 8, 16, "HND", 5)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    ctas = len(lens) * hkv if max(lens) < 1000 else ext().gqa_pick_ctas(len(lens), hkv, max(lens), sms)
    monkeypatch.setenv("HELIX_A2A_ATTN_DYN_PCT", "0")            # fixed shares: who streams what does not change from call to call
    want = attention.gqa_decode(q, k, v, bt, sl, max_seq_len=max(lens))
    monkeypatch.setenv("HELIX_A2A_ATTN_TRACE", "1")
    got = attention.gqa_decode(q, k, v, bt, sl, max_seq_len=max(lens))
    stamps = ops().attn_trace(q).view(-1, 8)
    assert stamps.shape[0] >= ctas and (stamps[:ctas, 3] >= stamps[:ctas, 0]).all() and (stamps[:ctas, 0] > 0).all()
    assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1])


# Batches around the sizes where planning changes: lanes take runs of sequences above 16, pools end above 256, the fold finds
# its pairs through the CTAs that start them above 64 pairs.  A bound below the real lengths makes the pools want more
# chunks than there are slots; one far above them keeps short sequences in shares.
@pytest.mark.parametrize("B,hkv,top,bound", [(16, 4, 3000, 3000), (17, 4, 3000, 3000), (33, 2, 6000, 6000), (20, 8, 5000, 1600),
                                             (40, 8, 900, 131072), (200, 2, 1500, 131072), (256, 1, 2500, 2500),
                                             (257, 1, 2500, 2500), (300, 2, 700, 131072), (70, 1, 9000, 2000)])
def test_many_sequences_in_shares_and_pools(native_built, monkeypatch, B, hkv, top, bound):
    from helix_a2a_b200.ops import attention, reference_math as rm
    from helix_a2a_b200.ops.oproj import check_compute_status
    lens = [(i * 7919 + 13) % top for i in range(B)]
    lens[B // 2], lens[-1], lens[0] = top, 0, top
    q, k, v, bt, sl = _case(lens, hkv, 4, 16, "HND", B)
    o_ref, l_ref = rm.paged_decode_attention_reference(q, k, v, bt, sl, 1 / math.sqrt(128), False)
    live = sl > 0
    for pct, chunk, least in (("30", "4", "8"), ("0", "4", "8"), (None, None, None)):
        for name, val in (("PCT", pct), ("CHUNK", chunk), ("MIN_BLOCKS", least)):
            if val is None:
                monkeypatch.delenv("HELIX_A2A_ATTN_DYN_" + name, raising=False)
            else:
                monkeypatch.setenv("HELIX_A2A_ATTN_DYN_" + name, val)
        for _ in range(2):
            o, lse = attention.gqa_decode(q, k, v, bt, sl, max_seq_len=bound)
        torch.cuda.synchronize()
        check_compute_status(q)
        assert (o.float() - o_ref.float()).abs().max() < 2e-2, pct
        assert (lse[live] - l_ref[live]).abs().max() < 1e-3, pct
        assert torch.isneginf(lse[~live]).all()
