"""Threads that share a stream: a call of two launches (a streaming kernel and the fold of its partials) is one unit."""
import math
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _gqa(seed, lens):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    blocks = max((n + 15) // 16 for n in lens)
    bt = torch.randperm(len(lens) * blocks, generator=gen, device="cuda").view(len(lens), blocks).int()
    k, v = (torch.empty(len(lens) * blocks, 8, 16, 128, device="cuda").normal_(generator=gen).bfloat16() for _ in range(2))
    q = torch.empty(len(lens), 64, 128, device="cuda").normal_(generator=gen).bfloat16()
    return q, k, v, bt, torch.tensor(lens, dtype=torch.int32, device="cuda")


def _mla(seed, n):
    from helix_a2a_b200.ops import reference_math as rm
    gen = torch.Generator(device="cuda").manual_seed(seed)
    pages = (n + 15) // 16
    bt = torch.randperm(pages, generator=gen, device="cuda").view(1, pages).int()
    ckv, scales = rm.quantize_fp8_blockscaled(torch.randn(pages, 16, 512, device="cuda", generator=gen), 128)
    kpe = torch.randn(pages, 16, 64, device="cuda", generator=gen).bfloat16()
    qn, qp = (torch.randn(1, 128, d, device="cuda", generator=gen).bfloat16() for d in (512, 64))
    return qn, qp, ckv, scales, kpe, bt, torch.tensor([n], dtype=torch.int32, device="cuda")


def _calls(monkeypatch):
    """Calls of every form that is two launches, each with inputs of its own; their results do not change from run to run."""
    from helix_a2a_b200.ops import attention, oproj as O
    monkeypatch.setenv("HELIX_A2A_ATTN_DYN_PCT", "0")
    gen = torch.Generator(device="cuda").manual_seed(1)
    out = []
    for seed, lens in ((1, [9000, 300]), (2, [5000] * 3)):
        q, k, v, bt, sl = _gqa(seed, lens)
        out.append(lambda a=(q, k, v, bt, sl), m=max(lens): attention.gqa_decode(*a, max_seq_len=m))
    for seed, n in ((3, 3000), (4, 1100)):
        a = _mla(seed, n)
        out.append(lambda a=a, n=n: attention.mla_decode(*a, scale=0.07, max_seq_len=n))
    for hidden, K, tokens in ((2048, 4096, 64), (1024, 8192, 100)):
        w = (torch.randn(hidden, K, device="cuda", generator=gen) * 0.02).bfloat16()
        x = torch.randn(tokens, K, device="cuda", generator=gen).bfloat16()
        out.append(lambda x=x, w=w: (O.oproj(x, w, library=False),))
    return out


def _run_threads(work):
    errors = []

    def body(f):
        try:
            f()
        except Exception as e:  # noqa: BLE001 - handed to the test
            errors.append(e)
    threads = [threading.Thread(target=body, args=(f,)) for f in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_threads_and_graph_replays_on_one_stream(native_built, monkeypatch):
    from helix_a2a_b200.ops.oproj import check_compute_status
    calls = _calls(monkeypatch)
    want = [[t.clone() for t in c()] for c in calls]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graphs = []
    for c in calls:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            res = c()
        graphs.append((g, res))
    torch.cuda.synchronize()
    rounds = 40
    got = [[] for _ in calls]
    replayed = [[] for _ in calls]

    def eager(i):
        for _ in range(rounds):
            got[i].append(calls[i]())

    def replay():
        for r in range(rounds):
            for i, (g, res) in enumerate(graphs):
                g.replay()
                replayed[i].append([t.clone() for t in res])
    # every thread's current stream is the device's default stream
    _run_threads([lambda i=i: eager(i) for i in range(len(calls))] + [replay])
    torch.cuda.synchronize()
    check_compute_status(want[0][0])
    for i in range(len(calls)):
        for res in got[i] + replayed[i]:
            assert all(torch.equal(a, b) for a, b in zip(want[i], res)), i


def test_threads_call_the_allocation_free_entry_point_on_one_stream(native_built):
    import ctypes
    import glob
    import os

    from helix_a2a_b200.ops import attention
    from helix_a2a_b200.ops._ext import ext
    ext()
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    fn = ctypes.CDLL(glob.glob(os.path.join(root, "helix_a2a_b200", "_C*.so"))[0]).helix_gqa_decode_noalloc
    P, L, I = ctypes.c_void_p, ctypes.c_int64, ctypes.c_int  # noqa: E741
    fn.restype = I
    fn.argtypes = [P, L, L, P, P, L, L, L, L, P, L, P, P, P, I, I, I, I, I, ctypes.c_float, I, P]
    lens = ([9000, 300], [5000] * 3, [20000])
    cases = [_gqa(10 + i, n) for i, n in enumerate(lens)]
    want = [attention.gqa_decode(*c, max_seq_len=max(n)) for c, n in zip(cases, lens)]
    rounds = 40
    outs = [[(torch.zeros_like(o), torch.zeros_like(l)) for _ in range(rounds)] for o, l in want]
    torch.cuda.synchronize()

    def body(i):
        q, k, v, bt, sl = cases[i]
        torch.cuda.synchronize()            # makes the device's context current in this thread, as its program would
        for o, l in outs[i]:
            rc = fn(q.data_ptr(), q.stride(0), q.stride(1), k.data_ptr(), v.data_ptr(), k.shape[0], k.stride(0), k.stride(1),
                    k.stride(2), bt.data_ptr(), bt.stride(0), sl.data_ptr(), o.data_ptr(), l.data_ptr(), q.shape[0], 64, 8, 16,
                    max(lens[i]), 1 / math.sqrt(128), 0, 0)
            assert rc == 0
    _run_threads([lambda i=i: body(i) for i in range(len(cases))])
    torch.cuda.synchronize()
    for i, (o_ref, l_ref) in enumerate(want):
        for o, l in outs[i]:
            # other shares than the regular call: bf16 rounding of values up to about 4.5, fp32 sums in another order
            assert (o.float() - o_ref.float()).abs().max() < 2e-2 and (l - l_ref).abs().max() < 1e-4
