"""The o_proj split counts picked for at most 8 tokens, and the plain grid where stream-K was near, against fp32 matmuls."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# both sides of each line of the rule: blocks of 256 that fill K, that leave a remainder, that do not split evenly (nine
# and twenty-five of them); few, middling and many slabs; 8 and 9 tokens; 112 and 114 plain CTAs at up to 16, 17 and 32 tokens
@pytest.mark.parametrize("hidden,K,tokens", [
    (1024, 1792, 8), (1024, 1856, 8), (2048, 2048, 1), (2048, 2048, 9), (2304, 2560, 8), (4096, 2048, 8), (4736, 2048, 8),
    (4096, 2112, 3), (6272, 2048, 8), (6400, 2048, 8), (8192, 2048, 1), (8192, 2304, 8), (7168, 8192, 8), (7168, 8192, 17),
    (4864, 8192, 16), (4864, 8256, 32), (1024, 2304, 8), (2048, 2112, 1), (2304, 6400, 8)])
@pytest.mark.parametrize("packed", [False, True])
def test_few_tokens_match_fp32(native_built, hidden, K, tokens, packed):
    from helix_a2a_b200.ops import oproj as O
    gen = torch.Generator(device="cuda").manual_seed(hidden + K + tokens)
    w = torch.empty(hidden, K, device="cuda").normal_(0, 0.02, generator=gen).bfloat16()
    x = torch.empty(tokens, K, device="cuda").normal_(generator=gen).bfloat16()
    for _ in range(2):          # the second call runs on the scratch the first one left
        y = O.oproj(x, O.prepack_weight(w) if packed else w, library=False)
    ref = x.float() @ w.float().t()
    # one bf16 rounding of the result (at most 2^-8 of it), and fp32 sums of K products of about 0.02 in any order
    bound = ref.abs() * 2.0 ** -8 + 0.02 * K ** 0.5 * 2.0 ** -15
    assert ((y.float() - ref).abs() <= bound).all(), ((y.float() - ref).abs() - bound).max()
    O.check_compute_status(x)
