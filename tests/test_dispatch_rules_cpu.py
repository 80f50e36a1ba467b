"""Which kernel and split a call takes, as the library's own rules have it (no GPU needed)."""


def test_lse_combine_rows_that_take_half_a_warp(native_built):
    from helix_a2a_b200.ops._ext import ext
    half = ext().lse_combine_half_warps                    # (rows, ranks, bytes of a row)
    for ranks in (1, 2):
        assert not any(half(rows, ranks, 256) for rows in (1, 16, 256, 2047))
        assert half(2048, ranks, 256) and half(65536, ranks, 16)
    assert all(half(rows, 3, 256) for rows in (1, 2047, 2048))
    assert not half(65536, 2, 272) and not half(65536, 8, 1024)      # longer rows fill a warp


def test_oproj_splits_of_few_tokens_all_have_work(native_built):
    from helix_a2a_b200.ops._ext import ext
    few = ext().oproj_pick_splits_few                      # (hidden, K, SMs); a split takes whole blocks of 256
    for hidden in range(128, 16384 + 128, 128):
        for K in range(64, 16384 + 64, 64):
            splits, blocks = few(hidden, K, 148), -(-K // 256)
            assert 1 <= splits <= max(blocks, 1) and (splits - 1) * -(-blocks // splits) < blocks, (hidden, K, splits)
    assert few(1024, 2304, 148) == 3 and few(2048, 2112, 148) == 3           # nine blocks: three each
    assert few(1024, 2048, 148) == 4 and few(1024, 2560, 148) == 4 and few(4096, 2048, 148) == 4 and few(8192, 2048, 148) == 1
