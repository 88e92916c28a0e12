"""fp32 attention: blocks of four and of eight warps give a row the same bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, PAGE = "cuda", 16


@pytest.mark.parametrize("dim", [16, 48, 64, 80, 128])
@pytest.mark.parametrize("window", [0, 100])
def test_rows_of_a_long_prompt_and_of_a_short_portion(dim, window):
    """900 tokens are more blocks than three an SM, their last 37 fewer."""
    from oxr_inference_b200 import ops

    heads, kv, n = 16, 4, 900
    g = torch.Generator(device=DEV).manual_seed(dim)
    q = torch.randn(n, heads, dim, device=DEV, generator=g)
    k, v = (torch.randn(-(-n // PAGE), PAGE, kv, dim, device=DEV, generator=g) for _ in range(2))
    table = torch.arange(k.shape[0], dtype=torch.int32, device=DEV).view(1, -1)
    (spec,) = ops.attention_tile_specs(heads, kv, dim, torch.float32)
    status = ops.new_status(DEV)

    def rows(last):
        starts = list(range(0, last, spec[0]))
        tiles = {spec: (torch.zeros(len(starts), dtype=torch.int32, device=DEV), torch.tensor(starts, dtype=torch.int32, device=DEV), len(starts))}
        return ops.paged_attention(q[n - last:].contiguous(), k, v, tiles=tiles, cu_q=torch.tensor([0, last], dtype=torch.int32, device=DEV),
                                   ctx_lens=torch.tensor([n], dtype=torch.int32, device=DEV), block_table=table, page_size=PAGE, scale=dim ** -0.5, window=window,
                                   kv_len_bound=n, status=status)

    whole = rows(n)
    assert torch.equal(whole[-37:], rows(37))
    ops.check_status(status)
    back = torch.arange(n, device=DEV)[:, None] - torch.arange(n, device=DEV)[None, :]
    seen = (back >= 0) & (back < window if window else True)
    for h in (0, 5, 15):
        s = (q[:, h].double() @ k.view(-1, kv, dim)[:n, h // 4].double().T) * dim ** -0.5
        want = torch.softmax(s.masked_fill(~seen, -torch.inf), -1) @ v.view(-1, kv, dim)[:n, h // 4].double()
        # n and dim roundings of 2^-24 of values of at most 5
        assert (whole[:, h].double() - want).abs().max() <= 5 * (n + dim) * 2 ** -24
