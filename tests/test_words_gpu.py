"""The 16-byte forms of Mamba's convolution and gated norm, of the stream's norm and of the embedding's widening, and the per-head map of few tokens: edges of runs,
words and rows, beside sizes that the general kernels take, against the formula in 64 bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    from oxr_inference_b200 import ops

    return ops


def near(got, want, steps):
    """Within `steps` roundings to bf16 (2^-8 of a value at most each) and a 32-bit sum's error."""
    assert ((got.double() - want).abs() <= want.abs() * 2 ** -8 * steps + 1e-5).all()


@pytest.mark.parametrize("lengths", [[17], [16, 1], [1, 15, 1, 33, 2], [64], [3, 3, 3]])
@pytest.mark.parametrize("channels,taps", [(8, 4), (24, 4), (2056, 4), (20, 4), (24, 3)])
def test_mamba_conv(ops, lengths, channels, taps):
    torch.manual_seed(1)
    n, col0 = sum(lengths), 16
    proj = torch.randn(n, 48 + channels, device=DEV).bfloat16()
    w, b = torch.randn(channels, taps, device=DEV), torch.randn(channels, device=DEV)
    state = torch.randn(len(lengths) + 1, channels * (taps - 1) + 4, device=DEV)
    before = state.clone()
    cu = torch.tensor([0, *torch.tensor(lengths).cumsum(0).tolist()], dtype=torch.int32, device=DEV)
    req = torch.repeat_interleave(torch.arange(len(lengths)), torch.tensor(lengths)).to(DEV, torch.int32)
    slots = torch.arange(len(lengths), 0, -1, dtype=torch.int32, device=DEV)
    got = ops.mamba_conv(proj, col0, channels, w, b, state, req_of_token=req, cu_q=cu, state_slots=slots, n_requests=len(lengths))
    for r, slot in enumerate(slots.tolist()):
        tail = before[slot, :channels * (taps - 1)].view(channels, taps - 1).double()
        x = torch.cat((tail, proj[cu[r]:cu[r + 1], col0:col0 + channels].double().T), 1)
        z = torch.nn.functional.conv1d(x[None], w.double()[:, None], b.double(), groups=channels)[0].T
        near(got[cu[r]:cu[r + 1]], z * torch.sigmoid(z), 1)
        assert torch.equal(state[slot, :channels * (taps - 1)].view(channels, taps - 1), x[:, -(taps - 1):].float())


@pytest.mark.parametrize("lengths,channels", [([1, 15, 1, 33, 2, 1500], 2056), ([1] * 40 + [1461], 2056), ([300, 1, 17, 16], 10248), ([293, 1], 10240)])
def test_mamba_conv_of_many_tokens(ops, lengths, channels):
    """From three million entries behind the requests' first tokens on the 16-byte form takes the step; below, the general one."""
    test_mamba_conv(ops, lengths, channels, 4)


@pytest.mark.parametrize("n", [1, 19])
@pytest.mark.parametrize("inner,parts", [(8, 1), (1032, 3), (8192, 8), (16384, 1), (60, 3), (8192, 1), (8184, 1), (8200, 1)])
def test_gated_group_norm(ops, n, inner, parts):
    torch.manual_seed(2)
    y, w = torch.randn(n, inner, device=DEV), torch.rand(inner, device=DEV) + 0.5
    proj = torch.randn(n, 16 + inner, device=DEV).bfloat16()
    z = proj[:, 8:8 + inner].double()
    v = (y.double() * z * torch.sigmoid(z)).view(n, parts, -1)
    want = (v * torch.rsqrt(v.square().mean(-1, keepdim=True) + 1e-5)).view(n, inner) * w.double()
    near(ops.gated_group_norm(y, proj, 8, w, parts, 1e-5), want, 1)


@pytest.mark.parametrize("hidden", [8, 264, 4096, 4104, 16392, 32768, 32776, 90])
def test_stream_norm_and_embedding(ops, hidden):
    torch.manual_seed(3)
    x, w = torch.randn(5, hidden, device=DEV) * 3, torch.rand(hidden, device=DEV) + 0.5
    rows = torch.tensor([4, 0, 0], dtype=torch.int32, device=DEV)
    want = x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-6) * w.double()
    near(ops.stream_rms_norm(x, w, 1e-6, torch.bfloat16), want, 1)
    near(ops.stream_rms_norm(x, w, 1e-6, torch.bfloat16, rows=rows), want[rows.long()], 1)
    table, status = torch.randn(7, hidden, device=DEV).bfloat16(), ops.new_status(DEV)
    got = ops.embedding(torch.tensor([6, 0, 3], dtype=torch.int32, device=DEV), table, torch.float32, status, 0.7)
    assert torch.equal(got, table[[6, 0, 3]].float() * torch.tensor(0.7, dtype=torch.float32))
    ops.check_status(status)
    assert (ops.embedding(torch.tensor([7, -1], dtype=torch.int32, device=DEV), table, torch.float32, status, 1.0) == 0).all()
    with pytest.raises(ops.KernelError, match="token id"):
        ops.check_status(status)


@pytest.mark.parametrize("n", [1, 8, 9, 16])
@pytest.mark.parametrize("n_in,n_out", [(16, 2), (128, 192), (144, 66), (192, 128), (256, 64), (272, 64), (20, 64)])
def test_head_linear_of_few_tokens(ops, n, n_in, n_out):
    torch.manual_seed(4)
    heads = 3
    x, w = torch.randn(n, heads, n_in + 8, device=DEV).bfloat16(), (torch.randn(heads, n_in, n_out, device=DEV) * n_in ** -0.5).bfloat16()
    out = torch.full((n, heads, n_out + 4), 7.0, device=DEV).bfloat16()
    ops.head_linear(out, 2, x, 8, w)
    want = torch.einsum("thi,hio->tho", x[:, :, 8:].double(), w.double())
    near(out[:, :, 2:2 + n_out], want, 1)
    assert (out[:, :, :2] == 7).all() and (out[:, :, 2 + n_out:] == 7).all()


@pytest.mark.parametrize("n,heads", [(17, 2), (64, 3), (65, 2), (1300, 40), (700, 300)])
@pytest.mark.parametrize("n_in,n_out,x0", [(16, 16, 8), (128, 192, 0), (192, 128, 8), (48, 80, 0), (256, 256, 0), (32, 48, 3)])
def test_head_linear_of_many_tokens(ops, n, heads, n_in, n_out, x0):
    torch.manual_seed(5)
    x, w = torch.randn(n, heads, n_in + 8, device=DEV).bfloat16(), (torch.randn(heads, n_in, n_out, device=DEV) * n_in ** -0.5).bfloat16()
    out = torch.full((n, heads, n_out + 8), 7.0, device=DEV).bfloat16()
    ops.head_linear(out, 4, x, x0, w)
    near(out[:, :, 4:4 + n_out], torch.einsum("thi,hio->tho", x[:, :, x0:x0 + n_in].double(), w.double()), 1)
    assert (out[:, :, :4] == 7).all() and (out[:, :, 4 + n_out:] == 7).all()


@pytest.mark.parametrize("n,top,width", [(1, 1, 8), (5, 4, 4096), (300, 3, 2056), (40, 9, 264), (40, 2, 90)])
@pytest.mark.parametrize("kept", [False, True])
def test_combine_rows(ops, n, top, width, kept):
    torch.manual_seed(6)
    y = torch.randn(n * top + 3, width, device=DEV).bfloat16()
    place = torch.randperm(n * top + 3, device=DEV)[:n * top].int()
    place[::5] = -1
    weights = torch.rand(n, top, device=DEV)
    x, share = (torch.randn(n, width, device=DEV).bfloat16(), torch.rand(n, device=DEV)) if kept else (None, None)
    got = ops.combine_rows(y, place, weights, x, share)
    rows = y.double()[place.clamp(min=0).long()].view(n, top, width) * (place >= 0).view(n, top, 1)
    want = (rows * weights.double()[:, :, None]).sum(1) + (x.double() * share.double()[:, None] if kept else 0)
    near(got, want, 1)
