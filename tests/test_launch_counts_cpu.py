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
