"""The decode work that a program has this library do, as cases that can be timed.

Every case is one call (one decode step for ``step``) of a public entry point on one GPU:

* ``gqa``      ``ops.attention.gqa_decode``: paged split-KV attention, bf16 cache
* ``mla``      ``ops.attention.mla_decode``: latent attention, block-scaled fp8 cache
* ``oproj``    ``ops.oproj.oproj``: the output projection, plain or packed weights
* ``combine``  ``lse_combine``: partial outputs that are already on this rank
* ``exchange`` exchange + LSE combine of all ranks of a group, played by one launch over one
  single-process workspace (the form in which the exchange runs on a single GPU)
* ``step``     ``models.llama_decode.HelixDecodeStack.decode_step_host``: a captured decode step
"""
from __future__ import annotations

import math
import os

import torch

import helix_a2a_b200 as helix
from helix_a2a_b200.models.llama_decode import HelixDecodeStack, LlamaDecodeConfig
from helix_a2a_b200.ops import attention, oproj as oproj_mod, reference_math as rm
from helix_a2a_b200.ops._ext import ops


def listed():
    return [
        # one short chat: nothing but latency
        dict(name="gqa short", op="gqa", batch=1, ctx=300, ragged=False, q_heads=64, kv_heads=8, page=16, layout="HND"),
        # a mixed serving batch: every sequence another length, the NHD cache and base-2 LSE that vLLM's backends use,
        # four query heads per KV head
        dict(name="gqa ragged batch", op="gqa", batch=24, ctx=9000, ragged=True, q_heads=32, kv_heads=8, page=32,
             layout="NHD"),
        # one layer of the headline model with one 128K sequence
        dict(name="gqa 128k", op="gqa", batch=1, ctx=131072, ragged=False, q_heads=64, kv_heads=8, page=16, layout="HND"),
        # MLA: a small interactive batch, a mixed batch, and a full batch of long contexts (bound by the tensor cores)
        dict(name="mla short", op="mla", batch=2, ctx=1500, ragged=False, page=16),
        dict(name="mla ragged batch", op="mla", batch=16, ctx=17000, ragged=True, page=64),
        dict(name="mla large", op="mla", batch=32, ctx=32768, ragged=False, page=16),
        # o_proj: one rank's K-slice of eight as a strided view of the full matrix; the whole layer with weights packed
        # at load time at a decode batch; and a large batch of an MLA layer's slice
        dict(name="oproj slice", op="oproj", tokens=3, hidden=8192, k=1024, packed=False),
        dict(name="oproj decode", op="oproj", tokens=8, hidden=8192, k=8192, packed=True),
        dict(name="oproj large batch", op="oproj", tokens=200, hidden=7168, k=8192, packed=True),
        # what an NCCL all-to-all of eight ranks leaves to be combined
        dict(name="combine", op="combine", ranks=8, rows=2048, dim=512, layout="NBHD", return_lse=True),
        # the exchange itself, four ranks, latent rows of 512
        dict(name="exchange", op="exchange", cp=4, batch=32, heads=128, dim=512),
        # decode steps of the attention stack end to end, from pinned host queries to the host result, as CUDA graphs
        dict(name="decode step", op="step", layers=16, batch=1, ctx=32768),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["gqa", "gqa", "mla", "mla", "oproj", "oproj", "combine", "exchange", "step"])
    if op == "gqa":
        batch = _log(rng, 1, 64)
        kv_heads, group = rng.choice([(8, 8), (8, 4), (4, 8), (2, 8), (8, 1)])
        return dict(op=op, batch=batch, ctx=_log(rng, 16, 131072 // batch), ragged=rng.random() < 0.6,
                    q_heads=kv_heads * group, kv_heads=kv_heads, page=rng.choice([16, 32, 64]),
                    layout=rng.choice(["HND", "NHD"]))
    if op == "mla":
        batch = _log(rng, 1, 64)
        return dict(op=op, batch=batch, ctx=_log(rng, 16, min(131072, (1 << 20) // batch)), ragged=rng.random() < 0.6,
                    page=rng.choice([16, 32, 64]))
    if op == "oproj":
        return dict(op=op, tokens=_log(rng, 1, 256), hidden=rng.choice([1024, 2048, 4096, 7168, 8192]),
                    k=rng.choice([832, 1024, 2048, 4096, 8192]), packed=rng.random() < 0.6)
    if op == "combine":
        return dict(op=op, ranks=rng.choice([2, 3, 4, 8]), rows=_log(rng, 16, 16384), dim=rng.choice([128, 512]),
                    layout=rng.choice(["NBHD", "BHND"]), return_lse=rng.random() < 0.5)
    if op == "exchange":
        heads, dim = rng.choice([(128, 512), (64, 128)])
        return dict(op=op, cp=rng.choice([2, 4, 8]), batch=_log(rng, 1, 128), heads=heads, dim=dim)
    return dict(op=op, layers=rng.randint(4, 12), batch=rng.randint(1, 4), ctx=_log(rng, 512, 8192))


def _lens(case):
    """Tokens of each sequence: all alike, or spread over the range (the same lengths whatever the seed)."""
    b, ctx = case["batch"], case["ctx"]
    if not case["ragged"]:
        return [ctx] * b
    return [max(1, int(ctx * ((0.137 + i * 0.6180339887) % 1.0))) for i in range(b)]


def _pages(lens, page, gen):
    """Block table with the pages of all sequences scattered over a pool, as a paged allocator leaves them."""
    counts = [-(-n // page) for n in lens]
    pool = sum(counts) + 3
    ids = torch.randperm(pool, generator=gen, device="cuda").int()
    table = torch.zeros(len(lens), max(counts), dtype=torch.int32, device="cuda")
    at = 0
    for i, c in enumerate(counts):
        table[i, :c] = ids[at:at + c]
        at += c
    return table, pool


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, std=1.0, dtype=torch.bfloat16):
        return torch.empty(*shape, dtype=dtype, device="cuda").normal_(0, std, generator=gen)

    op = case["op"]
    if op in ("gqa", "mla"):
        lens = _lens(case)
        order = torch.randperm(len(lens), generator=torch.Generator().manual_seed(seed)).tolist()
        lens = [lens[i] for i in order]
        page, batch = case["page"], case["batch"]
        table, pool = _pages(lens, page, gen)
        state = dict(op=op, table=table, max_len=max(lens),
                     lens=torch.tensor(lens, dtype=torch.int32, device="cuda"))
        if op == "gqa":
            h, hnd = case["kv_heads"], case["layout"] == "HND"
            shape = (pool, h, page, 128) if hnd else (pool, page, h, 128)
            state.update(q=normal(batch, case["q_heads"], 128), k=normal(*shape), v=normal(*shape),
                         layout=case["layout"], base2=not hnd)
            return state
        ckv = torch.empty(pool, page, 512, dtype=torch.float8_e4m3fn, device="cuda")
        scales = torch.empty(pool, page, 4, dtype=torch.float32, device="cuda")
        slab = max(1, (1 << 17) // page)            # bounds the fp32 temporaries of the quantiser
        for p0 in range(0, pool, slab):
            n = min(slab, pool - p0)
            ckv[p0:p0 + n], scales[p0:p0 + n] = rm.quantize_fp8_blockscaled(normal(n, page, 512, dtype=torch.float32), 128)
        state.update(q_nope=normal(batch, 128, 512, std=0.5), q_pe=normal(batch, 128, 64, std=0.5), ckv=ckv, scales=scales,
                     kpe=normal(pool, page, 64), scale=1.0 / math.sqrt(128 + 64))
        return state
    if op == "oproj":
        tokens, hidden, k = case["tokens"], case["hidden"], case["k"]
        # a context-parallel rank's weight is a column slice of the layer's matrix
        w = normal(hidden, 2 * k, std=0.02)[:, k // 64 * 32:][:, :k]
        return dict(op=op, x=normal(tokens, k), w=oproj_mod.prepack_weight(w) if case["packed"] else w)
    if op == "combine":
        n, rows, d = case["ranks"], case["rows"], case["dim"]
        shape = (n, rows, d) if case["layout"] == "NBHD" else (rows, n, d)
        return dict(op=op, o=normal(*shape), lse=normal(*shape[:-1], std=2.0, dtype=torch.float32),
                    layout=case["layout"], return_lse=case["return_lse"])
    if op == "exchange":
        cp, b, h, d = case["cp"], case["batch"], case["heads"], case["dim"]
        ws = helix.allocate_workspace(cp, 0)
        helix.init_workspace_all_rows(ws, cp)
        return dict(op=op, cp=cp, ws=ws, o=normal(cp, b, h, d), lse=normal(cp, b, h, std=2.0, dtype=torch.float32))
    cfg = LlamaDecodeConfig.llama3_70b(n_layers=case["layers"])
    stack = HelixDecodeStack(cfg, batch=case["batch"], local_ctx=case["ctx"], seed=seed)
    q = normal(cfg.n_layers, case["batch"], cfg.n_q_heads, cfg.head_dim)
    # the kernels of a captured step are chained by programmatic dependent launch, as bench.py has it
    before = os.environ.get("HELIX_A2A_ENABLE_PDL")
    os.environ["HELIX_A2A_ENABLE_PDL"] = "1"
    try:
        stack.capture(q)
    finally:
        if before is None:
            del os.environ["HELIX_A2A_ENABLE_PDL"]
        else:
            os.environ["HELIX_A2A_ENABLE_PDL"] = before
    return dict(op=op, stack=stack, q=q.cpu().pin_memory(),
                y=torch.empty(case["batch"], cfg.hidden, dtype=torch.bfloat16).pin_memory())


def run(s):
    op = s["op"]
    if op == "gqa":
        return attention.gqa_decode(s["q"], s["k"], s["v"], s["table"], s["lens"], layout=s["layout"],
                                    lse_base2=s["base2"], max_seq_len=s["max_len"])
    if op == "mla":
        return attention.mla_decode(s["q_nope"], s["q_pe"], s["ckv"], s["scales"], s["kpe"], s["table"], s["lens"],
                                    scale=s["scale"], max_seq_len=s["max_len"])
    if op == "oproj":
        return oproj_mod.oproj(s["x"], s["w"])
    if op == "combine":
        return helix.lse_combine(s["o"], s["lse"], layout=s["layout"], return_lse=s["return_lse"])
    if op == "exchange":
        return ops().alltoall_combine(s["o"], s["lse"], s["ws"], 0, s["cp"], 0, True, False, 0, True, 0, 0)
    return s["stack"].decode_step_host(s["q"], s["y"])


def work(case):
    op = case["op"]
    if op == "gqa":
        n, hq, b = sum(_lens(case)), case["q_heads"], case["batch"]
        return dict(bytes=n * case["kv_heads"] * 512 + b * hq * (512 + 4), flops=4 * 128 * hq * n)
    if op == "mla":
        n, b = sum(_lens(case)), case["batch"]
        return dict(bytes=n * 656 + b * 128 * (2 * 576 + 2 * 512 + 4), flops=2 * 128 * (576 + 512) * n)
    if op == "oproj":
        t, h, k = case["tokens"], case["hidden"], case["k"]
        return dict(bytes=2 * (h * k + t * k + t * h), flops=2 * t * h * k)
    if op == "combine":
        n, r, d = case["ranks"], case["rows"], case["dim"]
        return dict(bytes=r * (n + 1) * 2 * d + 4 * r * (n + (1 if case["return_lse"] else 0)), flops=2 * n * r * d)
    if op == "exchange":
        cp, rows, d = case["cp"], case["batch"] * case["heads"], case["dim"]
        return dict(bytes=rows * (cp * (2 * d + 4) + 2 * d + 4), flops=2 * cp * rows * d)
    layers, b, n = case["layers"], case["batch"], case["batch"] * case["ctx"]
    return dict(bytes=layers * (n * 8 * 512 + 8192 * 8192 * 2 + b * 4 * 8192), flops=layers * (4 * 8192 * n + 2 * b * 8192 * 8192))


def tolerance(case):
    # 2-norm errors seen against the same arithmetic in float64; about four times that is stated
    return {"gqa": {"rel": 1e-2}, "mla": {"rel": 1.2e-2}, "oproj": {"rel": 7e-3}, "combine": {"rel": 7e-3},
            "exchange": {"rel": 7e-3}, "step": {"rel": 1.2e-2}}[case["op"]]


def _combine64(o, lse):
    """LSE-weighted sum over the leading dimension, and the LSE of the whole."""
    o, lse = o.double(), lse.double()
    return (torch.softmax(lse, 0).unsqueeze(-1) * o).sum(0), torch.logsumexp(lse, 0)


def _gqa64(q, k, v, rows, n, scale):
    """One sequence: ``q [Hq, d]``, ``k`` / ``v`` ``[pages, page, Hkv, d]``, ``rows`` its pages, ``n`` its tokens."""
    k, v = (t[rows].flatten(0, 1)[:n].double().transpose(0, 1) for t in (k, v))           # [Hkv, n, d]
    s = q.double().view(k.shape[0], -1, q.shape[-1]) @ k.transpose(1, 2) * scale
    return (torch.softmax(s, -1) @ v).reshape(q.shape), torch.logsumexp(s, -1).reshape(-1)


def exact(case, seed):
    """What ``run`` returns, from plain torch in float64."""
    s = prepare(case, seed)
    op = case["op"]
    if op == "gqa":
        k, v = (t.transpose(1, 2) if s["layout"] == "HND" else t for t in (s["k"], s["v"]))
        each = [_gqa64(s["q"][b], k, v, s["table"][b, :-(-n // case["page"])].long(), n, 1.0 / math.sqrt(128))
                for b, n in enumerate(s["lens"].tolist())]
        o, lse = (torch.stack(t) for t in zip(*each))
        return o, lse / math.log(2.0) if s["base2"] else lse
    if op == "mla":
        outs, lses = [], []
        for b, n in enumerate(s["lens"].tolist()):
            rows = s["table"][b, :-(-n // case["page"])].long()
            c = s["ckv"][rows].flatten(0, 1)[:n].double().view(n, 4, 128)
            c = (c * s["scales"][rows].flatten(0, 1)[:n].double().unsqueeze(-1)).view(n, 512)
            kpe = s["kpe"][rows].flatten(0, 1)[:n].double()
            x = (s["q_nope"][b].double() @ c.t() + s["q_pe"][b].double() @ kpe.t()) * s["scale"]
            outs.append(torch.softmax(x, -1) @ c)
            lses.append(torch.logsumexp(x, -1))
        return torch.stack(outs), torch.stack(lses)
    if op == "oproj":
        w = prepare(dict(case, packed=False), seed)["w"]
        return s["x"].double() @ w.double().t()
    if op == "combine":
        o, lse = (s["o"], s["lse"]) if s["layout"] == "NBHD" else (s["o"].transpose(0, 1), s["lse"].transpose(0, 1))
        out, g = _combine64(o, lse)
        return (out, g) if s["return_lse"] else out
    if op == "exchange":
        out, g = _combine64(s["o"], s["lse"])                       # rank r keeps the r-th part of the heads
        return tuple(torch.stack(t.chunk(s["cp"], dim=1)) for t in (out, g))
    stack = s["stack"]                                              # the step returns its last layer's output
    k, v = stack.k_cache[-1].transpose(1, 2), stack.v_cache[-1].transpose(1, 2)
    o = torch.stack([_gqa64(q, k, v, stack.block_table[b].long(), case["ctx"], 1.0 / math.sqrt(128))[0]
                     for b, q in enumerate(s["q"][-1].cuda())])
    return (o.flatten(1) @ stack.w_o[-1].double().t()).cpu()
