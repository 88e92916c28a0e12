"""Which kernel's tiles a masked mixer asks for: the rule of ``masked_long_rows`` over head sizes, pages, groups, biases and scales."""

import pytest
import torch

from oxr_inference_b200 import ops

BF = torch.bfloat16


@pytest.mark.parametrize("D", [16, 48, 64, 80, 96, 128, 192, 224, 256])
@pytest.mark.parametrize("page", [1, 4, 8, 16, 24, 64, 128])
@pytest.mark.parametrize("shared", [False, True])
def test_rows_by_size(D, page, shared):
    tma = D % 64 == 0 and page >= 8 and page & (page - 1) == 0
    want = 64 if not tma else 256 if D <= 128 else 128 if shared else 64
    assert ops.masked_long_rows(8, 2, D, BF, page, shared=shared) == want
    assert ops.masked_long_rows(8, 2, D, BF, page, shared=shared, scale=0.0) == 64      # a scale that is not positive: the general kernel
    assert ops.masked_long_rows(8, 2, D, BF, page, shared=shared, scale=-1.0) == 64
    assert ops.masked_long_rows(8, 2, D, torch.float32, page, shared=shared) == 64
    if D > 128:
        assert ops.masked_long_rows(8, 2, D, BF, page, shared=shared, bias_rows=9) == 64
    short, long_ = ops.masked_tile_specs(8, 2, D, BF, page, shared=shared)
    assert short == ops.attention_tile_specs(8, 2, D, BF)[0] and long_ == (want // 4, ops.SHORT_MAX_TOKENS + 1, 1 << 30)
    assert ops.masked_tile_specs(8, 2, D, torch.float32, page, shared=shared) == ops.attention_tile_specs(8, 2, D, torch.float32)


def test_a_bias_table_has_to_fit():
    fits = lambda rows, group: ops.masked_long_rows(group, 1, 128, BF, 16, bias_rows=rows) == 256
    assert fits(513, 4) and fits(2, 32) and not fits(513, 32)
    for group in (1, 2, 3, 4, 8, 16, 32):
        most = max(r for r in range(1, 9000) if fits(r, group))
        # the table's rows, 127 distances of padding on each side, a pitch of 8 modulo 32 words
        assert all(fits(r, group) for r in range(1, most)) and 4 * group * (most + 254) <= ops.LONG_MASK_BYTES < 4 * group * (most + 254 + 64)
