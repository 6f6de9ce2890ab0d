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
