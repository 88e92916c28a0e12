"""The 32-bit product on parts of eight bits, at the sizes where it can go wrong."""

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


@pytest.mark.parametrize("widened", [False, True], ids=["24bit", "widened"])
@pytest.mark.parametrize("K", [60, 64, 1028, 2048, 4100, 8190])
def test_sums_in_segments_are_the_same_however_dealt_out(ops, K, widened):
    """One, two and four segments of k, whole and ragged chunks, rows of whole 16-byte words and others; blocks that take one segment and blocks that take
    all, tiles of every width. W of 24-bit numbers, of bf16 numbers, and with a few 24-bit numbers among these (a chunk then takes all six products)."""
    x, w = randn(130, K, seed=1), randn(300, K, seed=2)
    if widened:
        w = w.bfloat16().float()
        w[70, K // 2] += 2 ** -20
        w[299, K - 1] = 1 / 3
    want = x.double() @ w.double().T
    lib, status = ops._lib(), ops.new_status(DEV)
    got = []
    for tile in (16, 48, 112, 128):
        for shared in (0, 1):
            out = torch.full((130, 300), float("nan"), device=DEV)
            parts = torch.empty(3, 130, -(-K // 8) * 8, dtype=torch.bfloat16, device=DEV)
            assert lib.oxr_gemm_f32_nt(out.data_ptr(), x.data_ptr(), w.data_ptr(), parts.data_ptr(), 130, 300, K, tile, shared, status.data_ptr(), ops._stream()) == 0
            got.append(out)
    ops.check_status(status)
    # a chunk's four times sixteen products, each time at most 2^-23 of what is there, and the parts left out; then K / 64 + 4 roundings of 2^-24
    assert ((got[0].double() - want).abs() <= (16 + K / 64) * 2 ** -24 * (x.double().abs() @ w.double().abs().T)).all()
    assert all(torch.equal(got[0], other) for other in got[1:])
    assert torch.equal(ops.linear(x[7:8].contiguous(), w), got[0][7:8])


def test_infinities_and_what_rounds_to_one(ops):
    x, w = randn(20, 300, seed=3), randn(140, 300, seed=4)
    x[3, 5], x[4, 7], x[6, 20] = float("inf"), float("nan"), 3.4e38
    w[10, 5], w[11, 9], w[12, 20] = 0.0, -float("inf"), 0.5
    got, want = ops.linear(x, w), (x.double() @ w.double().T).float()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    assert torch.equal(got[got.isinf()], want[want.isinf()])
    assert got[6, 12].isfinite() and abs(got[6, 12] / want[6, 12] - 1) < 1e-6


@pytest.mark.parametrize("K", [300, 2050, 4100])
@pytest.mark.parametrize("power", [-100, -112, -116, -120, -126, -130, -140, -146])
def test_small_operands_keep_their_bits(ops, K, power):
    """One, two and four segments; small rows of x and small rows of W, down to where an operand has three bits left; products that are themselves among the smallest numbers."""
    small = (randn(40, K, seed=21).double() * 2.0 ** power).float()        # rounded to what fp32 has there
    other = randn(150, K, seed=22)
    lib, status = ops._lib(), ops.new_status(DEV)
    for x, w in ((small, other * 2.0 ** 60), (other * 2.0 ** 60, small), (small, other)):
        want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
        # as for operands of ordinary size; and half of the smallest number where the result is rounded to a multiple of it
        room = (16 + K / 64) * 2 ** -24 * size + 2.0 ** -150
        for shared in (0, 1):
            out = torch.full(want.shape, float("nan"), device=DEV)
            parts = torch.empty(3, x.shape[0], -(-K // 8) * 8, dtype=torch.bfloat16, device=DEV)
            assert lib.oxr_gemm_f32_nt(out.data_ptr(), x.data_ptr(), w.data_ptr(), parts.data_ptr(), *want.shape, K, 48, shared, status.data_ptr(), ops._stream()) == 0
            assert ((out.double() - want).abs() <= room).all()
            if w.abs().max() > 1e3 or x.abs().max() > 1e3:                 # normal results: the error of ordinary operands
                assert (out.double() - want).norm() <= 3e-7 * want.norm()
    ops.check_status(status)


@pytest.mark.parametrize("M,N", [(0, 40), (3, 0), (0, 0)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_products_without_rows_or_columns_are_empty(ops, M, N, dtype):
    got = ops.linear(torch.empty(M, 2048, device=DEV, dtype=dtype), torch.empty(N, 2048, device=DEV))
    assert got.shape == (M, N) and got.dtype == dtype
    given = torch.empty(M, N, device=DEV, dtype=dtype)
    assert ops.linear(torch.empty(M, 2048, device=DEV, dtype=dtype), torch.empty(N, 2048, device=DEV), out=given) is given


def test_products_cut_by_rows_keep_their_bits(ops, monkeypatch):
    x, w = randn(700, 2052, seed=31), randn(96, 2052, seed=32)
    whole = ops.linear(x, w)
    monkeypatch.setattr(ops, "F32_PARTS_BYTES", 1)
    before = ops.launch_count
    assert ops._gemm_f32_rows(700, 2052) == 128 and torch.equal(ops.linear(x, w), whole)
    assert ops.launch_count - before == 12          # six pieces of two kernels
    given = torch.empty_like(whole)
    assert ops.linear(x, w, out=given) is given and torch.equal(given, whole)
