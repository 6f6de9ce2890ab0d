"""The grouped product on pairs of CTAs (tiles of 256 rows) against the one on single CTAs and against 64 bits: groups
that end at a tile's edges, groups without rows, widths that end inside a tile, row factors and the gate's limits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(256, 256), (1, 0, 255, 257), (128, 129, 0, 513, 2), (700,)])
@pytest.mark.parametrize("n,k", [(256, 64), (384, 200), (128, 1024), (640, 72)])
@pytest.mark.parametrize("gated,scaled", [(False, False), (True, False), (True, True)])
def test_pair_tiles_give_what_single_tiles_give(counts, n, k, gated, scaled):
    from gllm_b200.ops import gemm_bf16, moe
    from gllm_b200 import ops

    g = torch.Generator().manual_seed(n + k)
    E, pairs = len(counts), sum(counts)
    ids = torch.cat([torch.full((c,), e) for e, c in enumerate(counts)])[torch.randperm(pairs, generator=g)].to(torch.int32)
    x = torch.randn(pairs, k, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(E, n, k, generator=g) * k ** -0.5).to(torch.bfloat16).cuda()
    factor = torch.rand(pairs, generator=g).cuda() if scaled else None
    got = {}
    for tile in (128, 256):
        _, tile_group, num_tiles, row_of_pair = moe.align(ids.cuda()[:, None], E, tile, want_rows=True)
        rows = tile_group.numel() * tile
        if scaled:
            xs, scale = moe.gather_rows(x, 1, row_of_pair, rows, factor[:, None])
        else:
            xs, scale = moe.gather_rows(x, 1, row_of_pair, rows), None
        out = gemm_bf16.linear_grouped(xs, w, tile_group, num_tiles, gated=gated, wide=n % 256 == 0, act=(1.2, 2.0, 0.5),
                                       row_scale=scale, tile_rows=tile)
        got[tile] = out[row_of_pair.long()]
    ops.check_status()
    assert torch.equal(got[128], got[256])                  # the same sums in the same order
    want = torch.einsum("pk,pnk->pn", x.double(), w.double()[ids.long().cuda()])
    if gated:
        gate, up = (t.reshape(pairs, -1) for t in want.view(pairs, n // 128, 2, 64).unbind(2))
        if scaled:
            gate, up = gate * factor.double()[:, None], up * factor.double()[:, None]
        gate, up = gate.clamp(max=2.0), up.clamp(-2.0, 2.0)
        want = gate * torch.sigmoid(1.2 * gate) * (up + 0.5)
    # k products of unit scale summed in 32 bits, and one rounding to bfloat16 in the gated form
    torch.testing.assert_close(got[256].double(), want, rtol=2.0 ** -8 if gated else 1e-4, atol=2e-3 if gated else 1e-4)
