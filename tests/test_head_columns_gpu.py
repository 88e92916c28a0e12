"""Maps per head and latent rows from columns of a wider product."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    from oxr_inference_b200 import ops

    return ops


def randn(*shape, seed):
    return torch.randn(*shape, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV)


@pytest.mark.parametrize("n", [5, 40])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_head_maps_and_latent_rows_from_columns_of_a_wider_product(ops, n, dtype):
    """The same bits from columns of a wider product as from a copy of them."""
    H, D, R, L = 3, 32, 16, 48
    both = randn(n, H * (D + R) + 24, seed=13).to(dtype)
    apart = both[:, 8:8 + H * (D + R)].unflatten(1, (H, D + R))
    w, c = randn(H, D, L, seed=14).to(dtype), randn(n, R // 2, seed=15)
    down, norm = randn(n, L + R, seed=16).to(dtype), randn(L, seed=17)
    slots, status = torch.arange(n, dtype=torch.int32, device=DEV), ops.new_status(DEV)
    results = []
    for q in (apart, apart.contiguous()):
        out, pool = torch.zeros(n, H, L + R, dtype=dtype, device=DEV), torch.zeros(4, 16, 1, L + R, dtype=dtype, device=DEV)
        ops.latent_prep(pool, down, L, R, norm, 1e-6, q, H, D + R, D, out, L + R, L, c.cos(), c.sin(), slots, status)
        ops.head_linear(out, 0, q, 0, w)
        results.append((out, pool))
    ops.check_status(status)
    assert all(torch.equal(a, b) for a, b in zip(*results))
    with pytest.raises(ops.KernelError):
        ops.head_linear(torch.zeros(n, H, L + R, dtype=dtype, device=DEV), 0, apart.transpose(1, 2), 0, w)
