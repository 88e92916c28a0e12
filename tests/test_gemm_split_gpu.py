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
    small = (randn(240, K, seed=21).double() * 2.0 ** power).float()        # rounded to what fp32 has there
    other = randn(300, K, seed=22)
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


# Relative errors against 64 bits (2-norms) of products of normal numbers: 1.1e-7 at 2,048 k, 1.3e-7 at 8,192. Without the parts w0 a2, w1 a1 and w2 a0 they are 4.4e-6,
# without W's lower parts 2e-3: a lost or stale part shows at every K.
@pytest.mark.parametrize("K", [300, 1028, 2048, 4100, 8190])
@pytest.mark.parametrize("shared", [0, 1])
def test_no_part_is_lost(ops, K, shared):
    """Random 24-bit W; and a W of bf16 numbers with a few large 24-bit numbers in chunks of either stage, chunks of bf16 numbers alone behind them."""
    x, w = randn(130, K, seed=41), randn(300, K, seed=42)
    mixed = w.bfloat16().float()
    rows = {70: (5,), 299: (K - 1,), 17: (64 + 3,), 130: (128 + 60, K // 2), 200: (K // 3, 2 * K // 3, K - 40)}
    for row, places in rows.items():
        for k in places:
            mixed[row, k] = 64 / 3 if row % 2 else -100 / 7
    lib, status = ops._lib(), ops.new_status(DEV)
    parts = torch.empty(3, 130, -(-K // 8) * 8, dtype=torch.bfloat16, device=DEV)
    for weight in (w, mixed):
        out = torch.full((130, 300), float("nan"), device=DEV)
        assert lib.oxr_gemm_f32_nt(out.data_ptr(), x.data_ptr(), weight.data_ptr(), parts.data_ptr(), 130, 300, K, 112, shared, status.data_ptr(), ops._stream()) == 0
        want = x.double() @ weight.double().T
        off = out.double() - want
        assert off.norm() <= 3e-7 * want.norm()
        # column by column: the second part of 64 / 3 is 0.04 and the third 8e-5, times a column of x of norm 11; a column of the product has norm 11 sqrt(K)
        assert (off.norm(dim=0) <= 6e-7 * want.norm(dim=0)).all()
    ops.check_status(status)


@pytest.mark.parametrize("K", [300, 2050, 4100])
@pytest.mark.parametrize("shared", [0, 1])
def test_what_is_not_finite_in_any_segment(ops, K, shared):
    """Infinities, NaN and operands that the scale takes out of range in the first, a middle and the last segment, added up in one block and across a cluster;
    sums that leave the range in one segment only and come back in another."""
    x, w = randn(40, K, seed=43), randn(300, K, seed=44)
    for i, k in enumerate((3, K // 2, K - 2)):
        x[3 * i, k], x[3 * i + 1, k], x[3 * i + 2, k] = float("inf"), float("nan"), 3.4e38
        w[10 + i, k], w[20 + i, k], w[30 + i, k] = 0.0, -float("inf"), 0.5
        x[20 + i, k], w[40 + i, k] = 2.0 ** 60, 2.0 ** 50
    x[30, 1], x[30, K - 1], w[50, 1], w[50, K - 1] = 2.0 ** 100, 2.0 ** 100, 1.0, -1.0
    lib, status = ops._lib(), ops.new_status(DEV)
    parts = torch.empty(3, 40, -(-K // 8) * 8, dtype=torch.bfloat16, device=DEV)
    out = torch.full((40, 300), 7.0, device=DEV)
    assert lib.oxr_gemm_f32_nt(out.data_ptr(), x.data_ptr(), w.data_ptr(), parts.data_ptr(), 40, 300, K, 48, shared, status.data_ptr(), ops._stream()) == 0
    ops.check_status(status)
    exact, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    want = torch.zeros_like(out)      # as it is defined: fused multiply-adds in the order of k (3.4e38 times 2 is infinite before the -inf of a later k)
    for k in range(K):
        want = (x[:, k:k + 1].double() * w[None, :, k].double() + want.double()).float()
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.isinf(), want.isinf()) and torch.equal(out[out.isinf()], want[want.isinf()])
    there = want.isfinite()
    # K multiply-adds one after the other where the scale does not reach, each rounding at most 2^-24 of the magnitudes' sum
    assert ((out.double() - exact).abs()[there] <= (K + 16) * 2 ** -24 * size[there]).all()


def test_more_columns_than_a_grid_has_rows(ops):
    """8.4 million columns in tiles of 128: cut by columns."""
    N, K = 65536 * 128 + 40, 24
    x, w = randn(3, K, seed=51), randn(N, K, seed=52)
    got = ops.linear(x, w)
    some = torch.tensor([0, 127, 128, 65535 * 128 - 1, 65535 * 128, N - 41, N - 1], device=DEV)
    want, size = x.double() @ w[some].double().T, x.double().abs() @ w[some].double().abs().T
    assert ((got[:, some].double() - want).abs() <= (16 + K / 64) * 2 ** -24 * size).all()
