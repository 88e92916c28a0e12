"""Long tiles of masked attention, and of attention whose keys are the values, on the tcgen05 kernels: every mask and extra at head sizes, page sizes,
group sizes and lengths around the kernels' tiles and blocks, against the formula in 64 bits. Cache rows that no query may see hold NaN."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    from oxr_inference_b200 import ops

    return ops


def formula(q, k, v, positions, scale, window, chunk, keep_first, bias, sink):
    """q [n, H, D], k, v [ctx, KV, D] in 64 bits -> [n, H, D]."""
    n, H, D = q.shape
    G = H // k.shape[1]
    pos = torch.tensor(positions, device=q.device)[:, None]
    j = torch.arange(k.shape[0], device=q.device)[None, :]
    seen = j <= pos
    if window:
        seen &= (j > pos - window) | (j < keep_first)
    if chunk:
        seen &= j // chunk == pos // chunk
    s = torch.einsum("nhd,khd->hnk", q, k.repeat_interleave(G, 1)) * scale
    if bias is not None:
        s = s + bias[(pos - j).clamp(0, bias.shape[0] - 1)].permute(2, 0, 1)
    s = s.masked_fill(~seen[None], -torch.inf)
    if sink is not None:
        s = torch.cat((s, sink[:, None, None].expand(H, n, 1)), -1)
    p = torch.softmax(s, -1)[..., :k.shape[0]]
    return torch.einsum("hnk,khd->nhd", p, v.repeat_interleave(G, 1))


MASKS = {"plain": {}, "window": {"window": 37}, "sink": {"sink": True}, "chunk_bias": {"chunk": 96, "bias": 41}, "bias_short": {"bias": 2}, "bias_long": {"bias": 515},
         "kept": {"window": 50, "keep_first": 21}, "kept_block": {"window": 9, "keep_first": 130, "sink": True}, "chunk_window": {"chunk": 200, "window": 33}}
SHAPES = [(8, 2, 128, 16, False), (32, 8, 128, 8, False), (3, 1, 64, 64, False), (5, 5, 128, 128, False), (32, 1, 256, 16, True), (6, 2, 256, 8, True), (3, 1, 192, 32, True),
          (16, 1, 128, 16, True)]


@pytest.mark.parametrize("mask", sorted(MASKS))
@pytest.mark.parametrize("H,KV,D,P,shared", SHAPES)
def test_against_the_formula(ops, H, KV, D, P, shared, mask):
    m = MASKS[mask]
    window, chunk, keep_first, scale = m.get("window", 0), m.get("chunk", 0), m.get("keep_first", 0), 0.11
    if mask == "plain" and not shared:
        pytest.skip("plain attention over separate keys and values has kv_maps")
    g = torch.Generator(device=DEV).manual_seed(3)
    bias = torch.randn(m["bias"], H, generator=g, device=DEV) if "bias" in m else None
    sink = torch.randn(H, generator=g, device=DEV) * 3 if m.get("sink") else None
    rows = ops.masked_long_rows(H, KV, D, torch.bfloat16, P, shared=shared, bias_rows=m.get("bias", 0), scale=scale)
    if D > 128:
        assert rows == (64 if bias is not None else 128)
    else:
        assert rows == (64 if bias is not None and not ops._attn_lib(D).oxr_attn_bias_fits(m["bias"], H // KV) else 256)
    # (tokens in the cache after the step, tokens of this step): less than a tile, a tile, odd portions behind a context, beside short ones
    sizes = [(9, 9), (128, 128), (300, 300), (517, 131), (70, 1), (401, 67), (64, 8)]
    pages = [-(-c // P) for c, _ in sizes]
    order = torch.randperm(sum(pages) + 2, generator=g, device=DEV).tolist()
    k_pool = torch.full((2, sum(pages) + 2, P, KV, D), torch.nan, dtype=torch.bfloat16, device=DEV)
    v_pool = k_pool if shared else torch.full_like(k_pool, torch.nan)
    table = torch.full((len(sizes), max(pages)), -1, dtype=torch.int32, device=DEV)
    qs, wants, cu = [], [], [0]
    specs = ops.masked_tile_specs(H, KV, D, torch.bfloat16, P, shared=shared, bias_rows=m.get("bias", 0), scale=scale)
    cut = {spec: ([], []) for spec in specs}
    for r, (c, n) in enumerate(sizes):
        k = torch.randn(c, KV, D, generator=g, device=DEV).bfloat16()
        v = k if shared else torch.randn(c, KV, D, generator=g, device=DEV).bfloat16()
        first = max(0, c - n)
        lowest = max(max(0, first - window + 1) if window else 0, first // chunk * chunk if chunk else 0)
        for i in range(pages[r]):
            page, here = order.pop(), slice(i * P, min((i + 1) * P, c))
            table[r, i] = page
            k_pool[1, page, :here.stop - here.start], v_pool[1, page, :here.stop - here.start] = k[here], v[here]
        for j in range(lowest):   # behind every mask: what is left of other requests
            if j >= keep_first:
                k_pool[1, int(table[r, j // P]), j % P] = torch.nan
                v_pool[1, int(table[r, j // P]), j % P] = torch.nan
        q = torch.randn(n, H, D, generator=g, device=DEV).bfloat16()
        qs.append(q)
        cu.append(cu[-1] + n)
        wants.append(formula(q.double(), k.double(), v.double(), list(range(c - n, c)), scale, window, chunk, keep_first,
                             None if bias is None else bias.double(), None if sink is None else sink.double()))
        for spec in specs:
            if spec[1] <= n <= spec[2]:
                for t in range(0, n, spec[0]):
                    cut[spec][0].append(r)
                    cut[spec][1].append(t)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    tiles = {spec: (i32(a or [0]), i32(b or [0]), len(a)) for spec, (a, b) in cut.items()}
    status = ops.new_status(DEV)
    maps = ops.make_kv_maps(k_pool, v_pool, P)
    got = ops.paged_attention(torch.cat(qs), k_pool[1], k_pool[1] if shared else v_pool[1], tiles=tiles, cu_q=i32(cu), ctx_lens=i32([c for c, _ in sizes]), block_table=table,
                              page_size=P, scale=scale, window=window, kv_len_bound=max(c for c, _ in sizes), status=status, chunk=chunk, dist_bias=bias,
                              sink=sink, keep_first=keep_first, long_maps=maps, layer_in_pool=1)
    ops.check_status(status)
    want = torch.cat(wants)
    # probabilities and the output are rounded to bf16 once each (2^-9 relative), the sums are fp32: 2^-8 of the values, which reach about 4
    err = (got.double() - want).abs().max().item()
    assert err < 4 * 2 ** -8 * 1.5, f"off by {err:.2e}"
    rel = ((got.double() - want).norm() / want.norm()).item()
    assert rel < 2 ** -8, f"relative error {rel:.2e}"
