"""Which kernel and split a call takes, as the library's own rules have it (no GPU needed)."""


def test_lse_combine_rows_that_take_half_a_warp(native_built):
    from helix_a2a_b200.ops._ext import ext
    half = ext().lse_combine_half_warps                    # (rows, ranks, bytes of a row)
    for ranks in (1, 2):
        assert not any(half(rows, ranks, 256) for rows in (1, 16, 256, 2047))
        assert half(2048, ranks, 256) and half(65536, ranks, 16)
    assert all(half(rows, 3, 256) for rows in (1, 2047, 2048))
    assert not half(65536, 2, 272) and not half(65536, 8, 1024)      # longer rows fill a warp
