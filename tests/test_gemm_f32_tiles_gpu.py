"""The 32-bit product at the edges of its tiles: every tile shape that the launcher chooses, rows and columns that fill none of them, k that is no multiple of
the depth of a stage or of a 16-byte word."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [17, 31, 48, 65, 130, 333])
@pytest.mark.parametrize("N,K", [(1, 16), (95, 20), (700, 33), (2048, 68), (5000, 77), (16390, 16), (40000, 4)])
def test_every_row_as_if_alone(M, N, K):
    from oxr_inference_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(M * N + K)
    x = torch.randn(M, K, device="cuda", generator=g)
    w = torch.randn(N, K, device="cuda", generator=g)
    got = ops.linear(x, w)
    # K products and K roundings of partial sums that stay below a few sqrt(K): 2^-24 K sqrt(K), with room
    torch.testing.assert_close(got.double(), x.double() @ w.double().T, atol=2 ** -22 * K ** 1.5, rtol=0)
    # one order of summation, whatever the tile: the rows one by one (the kernel for few rows) give the same bits
    rows = [0, M // 2, M - 1]
    assert torch.equal(torch.cat([ops.linear(x[r:r + 1].contiguous(), w) for r in rows]), got[rows])
