"""The split o_proj kernels (one or two slabs per CTA, partials summed by a second kernel) against fp32 matmuls."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(y, x, w):
    ref = x.float() @ w.float().t()
    # one bf16 rounding of the result (2^-9), and fp32 sums of K products of about 0.02 in any order
    bound = ref.abs() * 2.0 ** -8 + 0.02 * x.shape[1] ** 0.5 * 2.0 ** -15
    assert ((y.float() - ref).abs() <= bound).all(), ((y.float() - ref).abs() - bound).max()


# one and two slabs per CTA, an odd number of slabs, one K atom, atoms that do not fill the last stage, token counts
# around the padding to 16 and above one launch's 256
@pytest.mark.parametrize("hidden,K,tokens", [
    (128, 64, 40), (256, 64, 256), (384, 832, 100), (1024, 832, 33), (2048, 8192, 16), (2048, 8192, 65), (4096, 1024, 47),
    (4096, 4096, 129), (7168, 2048, 200), (8192, 1024, 255), (1024, 2048, 300)])
@pytest.mark.parametrize("packed", [False, True])
def test_split_kernels_match_fp32(native_built, hidden, K, tokens, packed):
    from helix_a2a_b200.ops import oproj as O
    gen = torch.Generator(device="cuda").manual_seed(hidden + K + tokens)
    w = torch.empty(hidden, 2 * K, device="cuda").normal_(0, 0.02, generator=gen).bfloat16()[:, K:]      # a column slice
    x = torch.empty(tokens, K + 8, device="cuda").normal_(generator=gen).bfloat16()[:, :K]               # padded rows
    for _ in range(2):          # the second call runs on the scratch the first one left
        y = O.oproj(x, O.prepack_weight(w) if packed else w, library=False)
    _check(y, x, w)
    O.check_compute_status(x)
