"""Attention and o_proj calls chained by programmatic launch, eagerly and in a graph: they all meet in the same scratch."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_two_launch_calls_back_to_back_under_programmatic_launch(native_built, monkeypatch):
    """MLA decode (main kernel and fold) -> split o_proj (kernel and sum) -> GQA decode (shares and fold) -> plain o_proj, three
    rounds without a synchronisation: no launch may touch partials or counters before the one that uses them is done."""
    from helix_a2a_b200.ops import attention, oproj as O, reference_math as rm
    monkeypatch.setenv("HELIX_A2A_ENABLE_PDL", "1")
    monkeypatch.setenv("HELIX_A2A_ATTN_DYN_PCT", "0")          # fixed shares: the results repeat to the bit
    gen = torch.Generator(device="cuda").manual_seed(4)
    n, lens = [1500, 700], [9000, 40]
    pages = [(t + 15) // 16 for t in n]
    bt_m = torch.randperm(2 * max(pages), generator=gen, device="cuda").view(2, -1).int()
    ckv, scales = rm.quantize_fp8_blockscaled(torch.randn(2 * max(pages), 16, 512, device="cuda", generator=gen), 128)
    kpe = torch.randn(2 * max(pages), 16, 64, device="cuda", generator=gen).bfloat16()
    qp = torch.randn(2, 128, 64, device="cuda", generator=gen).bfloat16()
    sl_m = torch.tensor(n, dtype=torch.int32, device="cuda")
    blocks = (max(lens) + 15) // 16
    bt_g = torch.randperm(2 * blocks, generator=gen, device="cuda").view(2, -1).int()
    k, v = (torch.randn(2 * blocks, 8, 16, 128, device="cuda", generator=gen).bfloat16() for _ in range(2))
    sl_g = torch.tensor(lens, dtype=torch.int32, device="cuda")
    w1 = O.prepack_weight((torch.randn(2048, 4096, device="cuda", generator=gen) * 0.02).bfloat16())
    w2 = O.prepack_weight((torch.randn(8192, 8192, device="cuda", generator=gen) * 0.02).bfloat16())

    def chain(qn):
        o, lse = attention.mla_decode(qn, qp, ckv, scales, kpe, bt_m, sl_m, scale=1 / math.sqrt(192), max_seq_len=max(n))
        y = O.oproj(o.view(32, 4096), w1)                       # 32 tokens: split K and the sum of the partials
        q = y.view(-1)[:2 * 64 * 128].view(2, 64, 128)
        g, lse_g = attention.gqa_decode(q, k, v, bt_g, sl_g, max_seq_len=max(lens))
        return lse, y, g, lse_g, O.oproj(g.view(2, 8192), w2)

    inputs = [torch.randn(2, 128, 512, device="cuda", generator=gen).bfloat16() for _ in range(3)]
    monkeypatch.setenv("HELIX_A2A_ENABLE_PDL", "0")
    want = []
    for x in inputs:
        want.append([t.clone() for t in chain(x)])
        torch.cuda.synchronize()
    lat = rm.dequantize_fp8_blockscaled(ckv, scales, 128)
    for i, x in enumerate(inputs):                              # the unchained results are right to begin with
        for b in range(2):
            rows = bt_m[b, :pages[b]].long()
            _, l_ref = rm.mla_partial_attention(x[b:b + 1].float(), qp[b:b + 1].float(), lat[rows].reshape(-1, 512)[:n[b]],
                                                kpe[rows].reshape(-1, 64)[:n[b]].float(), 1 / math.sqrt(192))
            assert (want[i][0][b] - l_ref[0]).abs().max() < 1e-2
    monkeypatch.setenv("HELIX_A2A_ENABLE_PDL", "1")
    for _ in range(3):
        got = [chain(x) for x in inputs]
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for w, g in zip(want, got) for a, b in zip(w, g))
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        res = [chain(x) for x in inputs]
    for _ in range(3):
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for w, g in zip(want, res) for a, b in zip(w, g))
    O.check_compute_status(qp)
