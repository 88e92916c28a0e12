"""The two-SM product with W along its long side, at the sizes where it can go wrong."""

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


@pytest.mark.parametrize("M,tile", [(96, 32), (200, 64), (300, 256), (513, 128), (255, 96), (500, 160), (37, 224), (256, 256), (1, 192)])
@pytest.mark.parametrize("N,K", [(256, 64), (600, 200), (16, 72), (1040, 1032)])
def test_w_along_the_long_side(ops, M, N, K, tile):
    """Tiles of 256 columns by `tile` rows: all columns ragged, rows that fill no tile, more tiles than pairs and fewer; plain to both
    types, with an activation, and gated."""
    x, w = randn(M, K, seed=5).bfloat16(), (randn(N, K, seed=6) * 0.1).bfloat16()
    want = x.float() @ w.float().T
    lib, status, stream = ops._lib(), ops.new_status(DEV), ops._stream()

    def run(dtype, act, gated=False):
        out = torch.full((M, N // 2 if gated else N), float("nan"), dtype=dtype, device=DEV)
        if gated:
            lib.oxr_set_gate_form(0, 1.0, 0.0)
            code = lib.oxr_gemm_tcgen05_pair_gated_bf16(out.data_ptr(), x.data_ptr(), w.data_ptr(), M, N, K, tile, 1, status.data_ptr(), stream)
        else:
            code = lib.oxr_gemm_tcgen05_pair_bf16(out.data_ptr(), x.data_ptr(), w.data_ptr(), M, N, K, ops._DT[dtype], tile, 1, act, status.data_ptr(), stream)
        assert code == 0
        ops.check_status(status)
        return out.float()

    # 32-bit sums in another order: 2^-24 K of the magnitudes' sum at most, K below 2^11; 16-bit results one rounding more
    room = 2 ** -13 * (x.float().abs() @ w.float().abs().T)
    assert ((run(torch.float32, 0) - want).abs() <= room).all()
    assert ((run(torch.bfloat16, 0) - want).abs() <= room + 2 ** -8 * want.abs()).all()
    squared = want.relu().square()
    assert ((run(torch.bfloat16, 1) - squared).abs() <= 2 * room * (want.abs() + room) + 2 ** -8 * squared).all()
    if N % 16 == 0:
        pairs = want.view(M, N // 16, 2, 8)
        gated = (torch.nn.functional.silu(pairs[:, :, 0]) * pairs[:, :, 1]).reshape(M, N // 2)
        # silu's slope is at most 1.1; one rounding to 16 bits and the fast division's two
        slack = room.view(M, N // 16, 2, 8)
        allowed = (1.1 * slack[:, :, 0] * (pairs[:, :, 1].abs() + slack[:, :, 1]) + pairs[:, :, 0].abs() * slack[:, :, 1]).reshape(M, N // 2)
        assert ((run(torch.bfloat16, 0, True) - gated).abs() <= allowed + 2 ** -7 * gated.abs()).all()


def test_tiles_that_do_not_fit_are_refused(ops):
    x, w = randn(300, 64, seed=7).bfloat16(), randn(256, 64, seed=8).bfloat16()
    out, status = torch.empty(300, 256, dtype=torch.bfloat16, device=DEV), ops.new_status(DEV)
    for tile, across in [(48, 1), (288, 1), (16, 1), (288, 0), (0, 1)]:
        assert ops._lib().oxr_gemm_tcgen05_pair_bf16(out.data_ptr(), x.data_ptr(), w.data_ptr(), 300, 256, 64, 1, tile, across, 0, status.data_ptr(), ops._stream()) != 0


@pytest.mark.parametrize("M,N,K", [(700, 1040, 1032), (1144, 4096, 512), (513, 16, 72)])
@pytest.mark.parametrize("kind,alpha,limit", [(0, 1.0, 0.0), (1, 1.702, 1.5), (3, 1.0, 0.0)], ids=["silu", "clamped", "gelu"])
def test_both_forms_give_the_same_bits(ops, M, N, K, kind, alpha, limit):
    """Every activation of the gated product, and the plain product with and without its own: a plan that turns a product over changes no answer."""
    x, w = randn(M, K, seed=9).bfloat16(), (randn(N, K, seed=10) * K ** -0.5).bfloat16()
    lib, status, stream = ops._lib(), ops.new_status(DEV), ops._stream()
    for dtype, act in ((None, 0), (torch.bfloat16, 0), (torch.bfloat16, 1), (torch.float32, 0), (torch.float32, 1)):
        outs = []
        for tile, across in ((256, 0), (96, 0), (256, 1), (160, 1), (32, 1)):
            if dtype is None:
                out = torch.full((M, N // 2), float("nan"), dtype=torch.bfloat16, device=DEV)
                lib.oxr_set_gate_form(kind, alpha, limit)
                code = lib.oxr_gemm_tcgen05_pair_gated_bf16(out.data_ptr(), x.data_ptr(), w.data_ptr(), M, N, K, tile, across, status.data_ptr(), stream)
            else:
                out = torch.full((M, N), float("nan"), dtype=dtype, device=DEV)
                code = lib.oxr_gemm_tcgen05_pair_bf16(out.data_ptr(), x.data_ptr(), w.data_ptr(), M, N, K, ops._DT[dtype], tile, across, act, status.data_ptr(), stream)
            assert code == 0
            outs.append(out)
        ops.check_status(status)
        assert all(torch.equal(outs[0], other) for other in outs[1:])
    if kind:
        pairs = (x.double() @ w.double().T).view(M, N // 16, 2, 8)
        g, u = pairs[:, :, 0], pairs[:, :, 1]
        want = g.clamp(max=limit) * torch.sigmoid(alpha * g.clamp(max=limit)) * (u.clamp(-limit, limit) + 1) if kind == 1 else torch.nn.functional.gelu(g, approximate="tanh") * u
        lib.oxr_set_gate_form(kind, alpha, limit)
        out = torch.empty(M, N // 2, dtype=torch.bfloat16, device=DEV)
        assert lib.oxr_gemm_tcgen05_pair_gated_bf16(out.data_ptr(), x.data_ptr(), w.data_ptr(), M, N, K, 160, 1, status.data_ptr(), stream) == 0
        # gates and ups of at most 6, each off by 2^-24 K times the magnitudes' sum of at most 30 (2e-3 for K = 1,032), the forms' slopes below 8; one rounding to 16 bits
        assert ((out.double() - want.reshape(M, N // 2)).abs() <= 2 ** -8 * want.reshape(M, N // 2).abs() + 1.6e-2).all()
