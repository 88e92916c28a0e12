"""Grouped products: tiles of no group, and the activation behind the product."""

import threading

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


@pytest.mark.parametrize("groups", [[0, 0, 2, -1, 1, -1, -1], [-1, -1], [3], [1, 1, 1, 0] + [-1] * 40])
def test_grouped_product_with_tiles_of_no_group(ops, groups):
    """Tiles of no group at the end (the usual case) and between others; none used at all."""
    m, n, k = 128 * len(groups), 272, 136
    x, w = randn(m, k, seed=9).bfloat16(), (randn(4 * n, k, seed=10) * 0.1).bfloat16()
    status = ops.new_status(DEV)
    got = ops.grouped_linear(x, w, torch.tensor(groups, dtype=torch.int32, device=DEV), n, torch.float32)
    ops.check_status(status)
    for i, g in enumerate(groups):
        if g >= 0:
            rows = slice(128 * i, 128 * i + 128)
            torch.testing.assert_close(got[rows], x[rows].float() @ w[g * n:(g + 1) * n].float().T, atol=1e-4, rtol=1e-5)


@pytest.mark.parametrize("ff", [16, 136, 200])
@pytest.mark.parametrize("kind", ["silu", "clamped"])
def test_grouped_product_with_the_activation_behind_it(ops, ff, kind):
    """Gates' rows first, then the ups': halves of a tile that reach beyond the gates and beyond the matrix."""
    groups, k = [2, 0, 0, -1, 1, -1], 136
    m, n = 128 * len(groups), 2 * ff
    x, w = randn(m, k, seed=11).bfloat16(), (randn(3 * n, k, seed=12) * 0.1).bfloat16()
    status = ops.new_status(DEV)
    got = ops.grouped_gated_linear(x, w, torch.tensor(groups, dtype=torch.int32, device=DEV), n, kind=kind, alpha=1.7, limit=1.5)
    ops.check_status(status)
    assert got.shape == (m, ff) and got.dtype == torch.bfloat16
    for i, e in enumerate(groups):
        if e >= 0:
            rows = slice(128 * i, 128 * i + 128)
            g, u = (x[rows].float() @ w[e * n:(e + 1) * n].float().T).split(ff, 1)
            if kind == "silu":
                want = torch.nn.functional.silu(g) * u
            else:
                g = g.clamp(max=1.5)
                want = g * torch.sigmoid(1.7 * g) * (u.clamp(-1.5, 1.5) + 1)
            # one rounding to 16 bits, the fast exponential's and division's few steps of 32 bits, sums in another order
            torch.testing.assert_close(got[rows].float(), want, rtol=2 ** -7, atol=1e-3)


@pytest.mark.parametrize("grouped", [False, True])
def test_another_thread_does_not_change_the_activation(ops, grouped):
    """A second engine asks for its own form between this thread's two calls."""
    m, n, k = 256, 64, 72
    x, w = randn(m, k, seed=13).bfloat16(), (randn(2 * n, k, seed=14) * 0.1).bfloat16()
    groups, lib, status = torch.tensor([1, 0], dtype=torch.int32, device=DEV), ops._lib(), ops.new_status(DEV)

    def product(other):
        out = torch.empty(m, n // 2, dtype=torch.bfloat16, device=DEV)
        lib.oxr_set_gate_form(0, 1.0, 0.0)
        if other:
            t = threading.Thread(target=lib.oxr_set_gate_form, args=(1, 1.7, 0.01))
            t.start()
            t.join()
        if grouped:
            code = lib.oxr_gemm_tcgen05_grouped_gated_bf16(out.data_ptr(), x.data_ptr(), w.data_ptr(), m, n, k, 2, groups.data_ptr(), 64, status.data_ptr(), ops._stream())
        else:
            code = lib.oxr_gemm_tcgen05_gated_bf16(out.data_ptr(), x.data_ptr(), w.data_ptr(), m, n, k, 64, status.data_ptr(), ops._stream())
        assert code == 0
        ops.check_status(status)
        return out

    assert torch.equal(product(True), product(False))


@pytest.mark.parametrize("spread", [True, False], ids=["evenly", "all the same"])
def test_a_layer_of_experts_at_its_real_size(ops, spread):
    """1,421 tokens of ordinary size, 4 of 16 experts: some 355 rows each, or all tokens on the same four. Forty tokens against 64 bits."""
    tokens, hidden, ff, experts, top = 1421, 4096, 1536, 16, 4
    h = randn(tokens, hidden, seed=21).bfloat16()
    up, down = (randn(experts * 2 * ff, hidden, seed=22) * 0.02).bfloat16(), (randn(experts * hidden, ff, seed=23) * 0.02).bfloat16()
    ids = randn(tokens, experts, seed=24).topk(top).indices.int() if spread else torch.tensor([[3, 7, 8, 15]], dtype=torch.int32, device=DEV).repeat(tokens, 1)
    weights = torch.softmax(randn(tokens, top, seed=25), -1)
    status = ops.new_status(DEV)
    _, order, place, tile_group = ops.expert_sort(ids, experts, pad=ops.GROUP_TILE_ROWS)
    a = ops.grouped_gated_linear(ops.gather_rows(h, order, top), up, tile_group, 2 * ff)
    got = ops.combine_rows(ops.grouped_linear(a, down, tile_group, hidden), place, weights)
    ops.check_status(status)
    for t in range(0, tokens, 36):
        want = torch.zeros(hidden, dtype=torch.float64, device=DEV)
        for e, share in zip(ids[t].tolist(), weights[t].double()):
            g, u = (up[e * 2 * ff:(e + 1) * 2 * ff].double() @ h[t].double()).split(ff)
            want += share * (down[e * hidden:(e + 1) * hidden].double() @ (torch.nn.functional.silu(g) * u))
        # three roundings to 16 bits (activation, each expert's row, their sum), 2^-9 of a value each and of either sign
        assert (got[t].double() - want).norm() <= 3 * 2 ** -9 * want.norm()
