"""Recurrences of steps with many tokens per request: the kernel whose threads hold several columns of the state, against the formula in 64 bits, at
its key sizes, with requests shorter and longer than its tiles, and the other kernels' sizes through the same entry."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
LENGTHS = [[1], [8], [37], [2, 1, 19, 40, 16], [9] * 33]


@pytest.fixture(scope="module")
def ops():
    from oxr_inference_b200 import ops

    return ops


def split(lengths):
    cu = [0]
    for n in lengths:
        cu.append(cu[-1] + n)
    return cu, torch.tensor(cu, dtype=torch.int32, device=DEV), torch.randperm(len(lengths) + 1, device=DEV)[:len(lengths)].int()


def close(got, want):
    # sums of at most 256 products in fp32, and a state whose decay is below one: a few hundred roundings of 2^-24 of the largest partial sums
    assert ((got.double() - want).norm() / want.norm()).item() < 2e-6


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lengths", LENGTHS, ids=lambda x: f"{len(x)}x{x[-1]}")
@pytest.mark.parametrize("H,DK,DV", [(3, 64, 72), (2, 128, 256), (2, 256, 40), (2, 48, 64), (1, 128, 36)])
def test_decay_per_key_entry(ops, H, DK, DV, lengths, dtype):
    torch.manual_seed(1)
    cu, cu_q, slots = split(lengths)
    n = cu[-1]
    proj = torch.randn(n, H * (2 * DK + DV), device=DEV).to(dtype)
    z, bias = torch.randn(n, H * DK, device=DEV) * 2, torch.randn(H * DK, device=DEV)
    state = torch.randn(len(lengths) + 1, H * DK * DV + 4, device=DEV)
    left = state.clone()
    got = ops.gla_scan(proj, 0, H * DK, 2 * H * DK, z, bias, heads=H, key_dim=DK, value_dim=DV, tau=4.0, q_scale=0.3, state=left, cu_q=cu_q, state_slots=slots,
                       n_requests=len(lengths))
    q, k, v = (t.view(n, H, -1) for t in proj.double().split((H * DK, H * DK, H * DV), 1))
    a = torch.sigmoid(z.double() + bias.double()).pow(0.25).view(n, H, DK)
    want, after = torch.empty(n, H, DV, dtype=torch.float64, device=DEV), state.double()
    for r, slot in enumerate(slots.tolist()):
        S = after[slot, :H * DK * DV].view(H, DK, DV)
        for t in range(cu[r], cu[r + 1]):
            S.mul_(a[t][:, :, None]).add_(k[t][:, :, None] * v[t][:, None, :])
            want[t] = torch.einsum("hkv,hk->hv", S, q[t]) * 0.3
    close(got, want.view(n, -1))
    close(left, after)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lengths", LENGTHS, ids=lambda x: f"{len(x)}x{x[-1]}")
@pytest.mark.parametrize("H,N,P,G", [(4, 64, 72, 2), (3, 128, 64, 1), (2, 256, 40, 2), (2, 40, 64, 1), (1, 128, 36, 1)])
def test_decay_per_token(ops, H, N, P, G, lengths, dtype):
    torch.manual_seed(2)
    cu, cu_q, slots = split(lengths)
    n = cu[-1]
    xbc = torch.randn(n, H * P + 2 * G * N, device=DEV).to(dtype)
    proj = torch.randn(n, 16 + H, device=DEV).to(dtype)
    dt_bias, a_log, skip = torch.randn(H, device=DEV), torch.randn(H, device=DEV) * 0.5 - 2, torch.randn(H, device=DEV)
    state = torch.randn(len(lengths) + 1, H * N * P + 4, device=DEV)
    left = state.clone()
    got = ops.mamba_scan(xbc, proj, 16, heads=H, vdim=P, state=N, groups=G, dt_bias=dt_bias, a_log=a_log, d_skip=skip, ssm=left, cu_q=cu_q, state_slots=slots,
                         n_requests=len(lengths))
    x, b, c = xbc.double().split((H * P, G * N, G * N), 1)
    x, b, c = x.view(n, H, P), b.view(n, G, N).repeat_interleave(H // G, 1), c.view(n, G, N).repeat_interleave(H // G, 1)
    dt = torch.nn.functional.softplus(proj[:, 16:].double() + dt_bias.double())
    decay = torch.exp(-torch.exp(a_log.double()) * dt)
    want, after = torch.empty(n, H, P, dtype=torch.float64, device=DEV), state.double()
    for r, slot in enumerate(slots.tolist()):
        S = after[slot, :H * N * P].view(H, N, P)
        for t in range(cu[r], cu[r + 1]):
            S.mul_(decay[t][:, None, None]).add_((b[t] * dt[t][:, None])[:, :, None] * x[t][:, None, :])
            want[t] = torch.einsum("hnp,hn->hp", S, c[t]) + skip.double()[:, None] * x[t]
    close(got, want.view(n, -1))
    close(left, after)


def tokens_of(kind, n, H, DK, DV, dtype, g):
    """One request's inputs, a row per token."""
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    if kind == "entry":
        return rnd(n, H * (2 * DK + DV)).to(dtype), rnd(n, H * DK) * 2
    return rnd(n, H * DV + 2 * 2 * DK).to(dtype), rnd(n, 8 + H).to(dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("kind,H,DK,DV", [("entry", 16, 128, 128), ("entry", 64, 64, 72), ("entry", 2, 256, 40), ("entry", 2, 48, 64), ("entry", 3, 16, 24), ("entry", 1, 20, 8),
                                          ("token", 32, 128, 64), ("token", 64, 64, 72), ("token", 2, 256, 40), ("token", 2, 40, 64), ("token", 4, 100, 36)])
def test_same_bits_however_cut_and_whatever_else_is_in_the_batch(ops, kind, H, DK, DV, dtype):
    """One sequence in a step of its own, in portions with single tokens between, and beside others: few requests and many (from 2,048 warps of eight
    entries on, a lane of the kernel for many tokens holds eight entries instead of four), single tokens and portions."""
    g = torch.Generator(device=DEV).manual_seed(7)
    per_head = torch.randn(3, H * (DK if kind == "entry" else 1), generator=g, device=DEV) * 0.5
    mine = tokens_of(kind, 61, H, DK, DV, dtype, g)
    start = torch.randn(H * DK * DV, generator=g, device=DEV)

    def step(requests, state, slots, named=False):
        cu, cu_q, _ = split([len(r[0]) for r in requests])
        rows, extra = (torch.cat([r[i] for r in requests]) for i in (0, 1))
        common = dict(heads=H, cu_q=cu_q, state_slots=torch.tensor(slots, dtype=torch.int32, device=DEV), n_requests=len(requests),
                      q_lens=[len(r[0]) for r in requests] if named else None)
        if kind == "entry":
            return ops.gla_scan(rows, 0, H * DK, 2 * H * DK, extra, per_head[0], key_dim=DK, value_dim=DV, tau=4.0, q_scale=0.3, state=state, **common), cu
        return ops.mamba_scan(rows, extra, 8, vdim=DV, state=DK, groups=2, dt_bias=per_head[0], a_log=per_head[1] - 2, d_skip=per_head[2],
                              ssm=state, **common), cu

    alone = start.repeat(1, 1)
    want, _ = step([mine], alone, [0])
    cut, rows, at = start.repeat(1, 1), [], 0
    for n in (1, 2, 1, 5, 17, 3, 1, 1, 30):
        rows.append(step([[t[at:at + n] for t in mine]], cut, [0])[0])
        at += n
    assert at == 61 and torch.equal(torch.cat(rows), want) and torch.equal(cut, alone)
    # without and with the lengths on the host, which name the requests of the kernel for many tokens (up to 32 of them); 40 such requests; 70 single tokens
    for others, named in [(o, named) for o in ([1], [1] * 8, [40, 1, 3, 70, 1, 1, 9, 2], [1] * 70, [18, 1] * 40) for named in (False, True)]:
        states = torch.randn(len(others) + 1, H * DK * DV, generator=g, device=DEV)
        states[len(others) // 2] = start
        step_of = [tokens_of(kind, n, H, DK, DV, dtype, g) for n in others]
        step_of.insert(len(others) // 2, mine)
        got, cu = step(step_of, states, list(range(len(others) + 1)), named)
        first = cu[len(others) // 2]
        assert torch.equal(got[first:first + 61], want) and torch.equal(states[len(others) // 2], alone[0])
