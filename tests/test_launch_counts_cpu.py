"""How many kernels a call launches, as the library's own rules have it (no GPU needed)."""

def test_launches_of_attention_and_oproj(native_built):
    from helix_a2a_b200.ops._ext import ext
    e = ext()
    assert e.gqa_launches(1, 8, 300, 148) == 1                 # one CTA per (sequence, kv head) pair
    assert e.gqa_launches(1, 8, 131072, 148) == 2              # shares and the fold of their pieces
    assert e.gqa_launches(0, 8, 300, 148) == 0
    assert e.oproj_launches(8, 8192, 8192, True, 148) == 1
    assert e.oproj_launches(200, 7168, 8192, True, 148) == 2   # split K and the sum of the partials
    assert e.oproj_launches(456, 7168, 8192, True, 148) == 4   # 256 tokens a slice
    assert e.oproj_launches(0, 7168, 8192, True, 148) == 0


def test_kernels_per_step_counts_every_launch(native_built):
    from helix_a2a_b200.models.llama_decode import HelixDecodeStack, LlamaDecodeConfig
    cfg = LlamaDecodeConfig.tiny(hidden=256)
    stack = HelixDecodeStack(cfg, batch=1, local_ctx=64, device="cpu")
    assert stack.kernels_per_step() == cfg.n_layers * 2
    stack.local_ctx = 131072                                   # a split attention call is two kernels
    assert stack.kernels_per_step() == cfg.n_layers * 3
    stack.cp_size = 2
    assert stack.kernels_per_step() == cfg.n_layers * 4
    stack.fuse_oproj = True
    assert stack.kernels_per_step() == cfg.n_layers * 3


def test_oproj_keeps_one_launch_where_the_split_kernels_are_slower(native_built):
    from helix_a2a_b200.ops._ext import ext
    one = lambda hidden, K, tokens: ext().oproj_launches(tokens, hidden, K, True, 148) == 1   # noqa: E731
    for hidden, K in ((3072, 4096), (4096, 4096), (5120, 5120), (6144, 4096), (8192, 8192)):
        assert one(hidden, K, 1) and one(hidden, K, 8)
    assert not one(1024, 4096, 1) and not one(2048, 8192, 8)              # few slabs: finer splits pay from the first token
    assert not one(4096, 4096, 9) and not one(5120, 5120, 9) and one(8192, 8192, 16)
    # no split to begin with: the second launch has to earn itself
    for hidden, K, tokens in ((10240, 2048, 32), (5120, 1024, 64), (16384, 5120, 128), (16384, 8192, 256), (4096, 1024, 48)):
        assert one(hidden, K, tokens), (hidden, K, tokens)
    assert not one(10240, 8192, 32) and not one(16384, 16384, 64) and not one(1024, 2048, 17)
