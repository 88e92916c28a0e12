"""32-bit products of short rows, summed in 64 bits, at the edges of their tiles and of the rule that picks them."""

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


@pytest.mark.parametrize("M", [1, 15, 17, 64, 65, 333, 1000])
@pytest.mark.parametrize("N,K", [(1, 1), (33, 2), (2048, 16), (4097, 13), (120, 33), (64, 64), (40, 101), (16, 256), (17, 240)])
def test_one_rounding_and_rows_as_if_alone(ops, M, N, K):
    assert ops._lib().oxr_gemm_f32_is_short(N, K)
    wide = randn(M, K + 1, seed=1)
    for x in (randn(M, K, seed=2), wide.view(-1)[1:1 + M * K].view(M, K)):        # whole 16-byte words, and a base that is none
        w = randn(N, K, seed=3)
        want = x.double() @ w.double().T
        got = ops.linear(x, w)
        # one rounding to 32 bits (2^-24 of the result), K of 64 bits (2^-53 of the magnitudes' sum each)
        assert ((got.double() - want).abs() <= 2 ** -24 * want.abs() + (K + 1) * 2 ** -53 * (x.double().abs() @ w.double().abs().T) + 2.0 ** -150).all()
        for r in {0, M // 2, M - 1}:
            assert torch.equal(ops.linear(x[r:r + 1].contiguous(), w)[0], got[r])


def test_infinities_nan_and_the_smallest_numbers(ops):
    x, w = randn(20, 40, seed=4), randn(50, 40, seed=5)
    x[3, 5], x[4, 7], x[6], x[7] = float("inf"), float("nan"), 3e38, x[7] * 2.0 ** -146
    w[10, 5], w[11, 9] = 0.0, -float("inf")
    got, want = ops.linear(x, w), (x.double() @ w.double().T).float()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    there = want.isfinite()
    assert ((got[there].double() - want[there].double()).abs() <= 2 ** -23 * want[there].double().abs() + 2.0 ** -149).all()


def test_the_rule_looks_at_the_weight_alone(ops):
    short = ops._lib().oxr_gemm_f32_is_short
    assert short(100000, 16) and not short(2048, 17) and short(240, 17) and short(64, 64) and not short(65, 64) and short(16, 256) and not short(1, 257)
