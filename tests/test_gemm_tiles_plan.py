"""The tiles of the two-SM product, planned on the host."""

from oxr_inference_b200 import ops


def test_every_plan_is_a_valid_launch():
    for m in (512, 513, 700, 1000, 1421, 1562, 2011, 2048, 5000):
        for n, k in ((576, 4096), (4096, 4096), (6144, 4096), (24576, 4096), (4096, 12288), (32768, 2048), (8192, 64)):
            for gated in (False, True):
                tile, across = ops._gemm_pair_tiles(m, n, k, gated)
                assert tile % 32 == 0 and 64 <= tile <= 256 and across in (0, 1)


def test_rows_that_fill_tiles_badly_lie_across():
    assert ops._gemm_pair_tiles(1562, 24576, 4096) == (160, 1)      # 10 x 160 rows instead of 7 x 256
    assert ops._gemm_pair_tiles(1421, 4096, 12288) == (160, 1)
    assert ops._gemm_pair_tiles(1024, 24576, 4096)[1] == 0           # four tiles of 256 rows exactly
    assert ops._gemm_pair_tiles(1000, 8192, 2048)[1] == 0            # so short a k that the epilogue would not be hidden
    # promises that measured slower: a few per cent, and gated products whose epilogue is the dearer one
    assert ops._gemm_pair_tiles(1912, 2048, 4096)[1] == 0
    assert ops._gemm_pair_tiles(1340, 12352, 4096, True)[1] == ops._gemm_pair_tiles(1430, 4096, 4096, True)[1] == 0
    assert ops._gemm_pair_tiles(1599, 24576, 8192, True)[1] == 1


def test_32_bit_plans_without_rows_and_without_clusters(monkeypatch):
    assert ops._gemm_f32_plan.__wrapped__(0, 2048, 4096) == (16, False)
    monkeypatch.setattr(ops, "_f32_clusters", lambda segments: 0)           # what the library answers where no cluster can be launched
    for m, n, k in ((1, 2048, 8192), (333, 16384, 2048), (5000, 300, 64)):
        tile, shared = ops._gemm_f32_plan.__wrapped__(m, n, k)
        assert tile % 16 == 0 and 16 <= tile <= ops.F32_MAX_TILE and not shared


def test_32_bit_products_bound_their_scratch():
    for m, k in ((1, 64), (333, 2048), (2048, 8192), (8192, 12288), (100000, 2047), (300, 1 << 20)):
        rows = ops._gemm_f32_rows(m, k)
        assert 0 < rows <= m and (rows == m or rows % ops.F32_MAX_TILE == 0)
        assert rows <= ops.F32_MAX_TILE or 6 * rows * (-(-k // 8) * 8) <= ops.F32_PARTS_BYTES
    assert ops._gemm_f32_rows(2048, 8192) == 2048
