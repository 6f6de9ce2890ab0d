"""The 16-byte forms of the short convolution and of the gated norm over groups against their general forms, which rows
off the 16-byte grid still take."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DTYPES = [torch.float32, torch.bfloat16]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("channels", [8, 264, 1096])
@pytest.mark.parametrize("lens", [(1, 1, 1), (700,), (2, 1, 35, 17, 1), (16, 3, 16)])
@pytest.mark.parametrize("bias", [False, True])
def test_convolution_in_runs_gives_the_same_bits(dtype, taps, channels, lens, bias):
    from gllm_b200.ops import stateful

    g = torch.Generator().manual_seed(taps * channels)
    n, R = sum(lens), len(lens)
    wide = torch.randn(n, channels + 16, generator=g).to(dtype).cuda()
    w = torch.randn(channels, taps, generator=g).cuda()
    b = torch.randn(channels, generator=g).cuda() if bias else None
    state = torch.randn(R + 2, taps - 1, channels, generator=g).cuda()
    rows = torch.randperm(R + 2, generator=g)[:R].to(torch.int32)
    starts = torch.tensor([0, 5, 1, 0, 7][:R])
    pos = torch.cat([s + torch.arange(m) for s, m in zip(starts, lens)]).to(torch.int32).cuda()
    row = rows.repeat_interleave(torch.tensor(lens)).cuda()
    aligned = wide[:, 8:8 + channels]
    off = torch.empty(n, channels + 1, dtype=dtype, device="cuda")[:, 1:]     # rows off the 16-byte grid
    off.copy_(aligned)
    a = stateful.conv_silu(aligned, w, b, state, pos, row)
    assert torch.equal(a, stateful.conv_silu(off, w, b, state, pos, row))
    # and a request's tokens do not depend on what lies around them
    at = n - lens[-1]
    assert torch.equal(a[at:], stateful.conv_silu(aligned[at:], w, b, state, pos[at:].contiguous(), row[at:].contiguous()))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n,groups,width", [(1, 1, 8), (3, 2, 264), (700, 1, 4096), (2, 1, 4104), (5, 1, 16384), (40, 4, 1000)])
@pytest.mark.parametrize("skip", [False, True])
def test_gated_norm_keeps_its_columns(dtype, n, groups, width, skip):
    from gllm_b200.ops import stateful

    g = torch.Generator().manual_seed(n + width)
    total, heads = groups * width, groups * width // 8
    y, w = torch.randn(n, total, generator=g).cuda(), torch.randn(total, generator=g).cuda()
    zx = torch.randn(n, 2 * total, generator=g).to(dtype).cuda()
    z, x = zx[:, :total], zx[:, total:]
    D = torch.randn(heads, generator=g).cuda() if skip else None
    args = dict(skip=D, x=x, head_width=8) if skip else {}
    got = stateful.gated_group_norm(y, z, w, groups, 1e-5, **args)
    z_off = torch.empty(n, total + 1, dtype=dtype, device="cuda")[:, 1:]
    z_off.copy_(z)
    general = stateful.gated_group_norm(y, z_off, w, groups, 1e-5, **args)
    u = y.double() + (D.double().repeat_interleave(8) * x.double() if skip else 0.0)
    u = (u * torch.nn.functional.silu(z.double())).view(n, groups, width)
    want = (u / torch.sqrt(u.square().mean(-1, keepdim=True) + 1e-5)).reshape(n, total) * w.double()
    # a handful of roundings and one of the result's type
    rtol = 2e-6 if dtype == torch.float32 else 2.0 ** -8
    torch.testing.assert_close(got.double(), want, rtol=rtol, atol=2e-6)
    torch.testing.assert_close(general.double(), want, rtol=rtol, atol=2e-6)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n,heads,dv", [(1, 1, 4), (5, 3, 36), (130, 16, 128), (7, 2, 200), (3, 2, 512)])
@pytest.mark.parametrize("gate", [None, "sigmoid", "silu"])
@pytest.mark.parametrize("shared", [False, True])
def test_head_norm_keeps_its_columns(dtype, n, heads, dv, gate, shared):
    from gllm_b200.ops import stateful

    g = torch.Generator().manual_seed(n + dv)
    o, w = torch.randn(n, heads * dv, generator=g).cuda(), torch.randn(dv if shared else heads * dv, generator=g).cuda()
    wide = torch.randn(n, heads * dv + 4, generator=g).to(dtype).cuda()
    z = wide[:, 4:]
    off = torch.empty(n, heads * dv + 1, dtype=dtype, device="cuda")[:, 1:]
    off.copy_(z)
    run = lambda t: stateful.head_norm(o, heads, dv, w, 1e-5, dtype, gate=t if gate else None, gate_kind=gate or "sigmoid")  # noqa: E731
    x = o.double().view(n, heads, dv)
    want = (x / torch.sqrt(x.square().mean(-1, keepdim=True) + 1e-5)).reshape(n, -1) * (w.double().repeat(heads) if shared else w.double())
    if gate:
        want = want * (torch.sigmoid(z.double()) if gate == "sigmoid" else torch.nn.functional.silu(z.double()))
    rtol = 2e-6 if dtype == torch.float32 else 2.0 ** -8
    torch.testing.assert_close(run(z).double(), want, rtol=rtol, atol=2e-6)
    torch.testing.assert_close(run(off).double(), want, rtol=rtol, atol=2e-6)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,kv_heads,dk,dv", [(16, 16, 64, 128), (4, 2, 32, 24), (2, 1, 128, 8), (4, 4, 8, 40)])
@pytest.mark.parametrize("taps", [2, 4])
@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("lens", [(600,), (2, 1, 35, 17, 1)])
def test_delta_preparation_in_runs(dtype, heads, kv_heads, dk, dv, taps, per_head, lens):
    from gllm_b200.ops import stateful

    g = torch.Generator().manual_seed(heads + dk + taps)
    n, R, channels = sum(lens), len(lens), 2 * kv_heads * dk + heads * dv
    wide = torch.randn(n, channels + 8, generator=g).to(dtype).cuda()
    off = torch.empty(n, channels + 9, dtype=dtype, device="cuda")[:, 1:]
    off.copy_(wide)
    conv = torch.randn(channels, taps, generator=g).cuda()
    state = torch.randn(R + 1, taps - 1, channels, generator=g).cuda()
    width = heads * (1 if per_head else dk)
    raw, bias = torch.randn(n, width, generator=g).cuda(), torch.randn(width, generator=g).cuda()
    A_log, b_raw = torch.randn(heads, generator=g).cuda(), torch.randn(n, heads, generator=g).cuda()
    rows = torch.randperm(R + 1, generator=g)[:R].to(torch.int32)
    starts = torch.tensor([0, 5, 1, 0, 7][:R])
    pos = torch.cat([s + torch.arange(m) for s, m in zip(starts, lens)]).to(torch.int32).cuda()
    row, cu = rows.repeat_interleave(torch.tensor(lens)).cuda(), torch.tensor([0, *lens]).cumsum(0).to(torch.int32).cuda()

    def run(x):
        s = state.clone()
        return stateful.delta_prep(x, conv, s, pos, row, cu, rows.cuda(), R, raw, bias, A_log, b_raw, heads, kv_heads, dk, dv,
                                   1e-6, dk ** -0.5, max_q_len=max(lens)), s

    (qk, v, loss, beta), after = run(wide)
    (qk2, v2, loss2, beta2), after2 = run(off)          # rows off the 16-byte grid: the general form
    for a, b in ((v, v2), (loss, loss2), (beta, beta2), (after, after2)):
        assert torch.equal(a, b)
    # the squares of a head are added in another order: dk roundings of 2^-24 at most, halved by the root
    torch.testing.assert_close(qk, qk2, rtol=dk * 2.0 ** -25 + 4 * 2.0 ** -24, atol=0)
