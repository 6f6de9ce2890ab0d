"""Unsummed parts: their sum on both sides of the size from which four elements a thread add them, and as the shared
expert's result inside the kernel that adds the experts'."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DTYPES = [torch.float32, torch.bfloat16]


def _in_order(parts):
    total = torch.zeros_like(parts[0])
    for p in parts:
        total = total + p
    return total


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("count", [1, 4, 5, 9])
@pytest.mark.parametrize("more", [-4, -1, 0, 1, 2, 4])
def test_sum_of_parts_around_the_wide_kernels_size(dtype, count, more):
    from gllm_b200 import ops

    n = 2 * 1024 * torch.cuda.get_device_properties(0).multi_processor_count + more
    parts = torch.randn(count, 1, n, generator=torch.Generator().manual_seed(count)).cuda()
    assert torch.equal(ops.SplitSum(parts, dtype).tensor(), _in_order(parts).to(dtype))
    shifted = torch.empty(count * n + 1, device="cuda")[1:].view(count, 1, n)            # off the 16-byte grid
    shifted.copy_(parts)
    assert torch.equal(ops.SplitSum(shifted, dtype).tensor(), _in_order(parts).to(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width", [64, 66, 1028])
@pytest.mark.parametrize("count", [1, 5])
@pytest.mark.parametrize("tokens", [3, 70])
@pytest.mark.parametrize("gate", [False, True])
@pytest.mark.parametrize("gap", [0, 1, 4])
def test_shared_parts_join_the_experts_as_their_sum_does(dtype, width, count, tokens, gate, gap):
    from gllm_b200 import ops
    from gllm_b200.ops import moe

    g = torch.Generator().manual_seed(width + count)
    top = 2
    y, weights = torch.randn(tokens * top, width, generator=g).cuda(), torch.rand(tokens, top, generator=g).cuda()
    stride = tokens * width + gap
    parts = torch.randn(count * stride, generator=g).cuda().as_strided((count, tokens, width), (stride, width, 1))
    logits = torch.randn(tokens, 3, generator=g).cuda()[:, 1] if gate else None
    split = ops.SplitSum(parts, dtype)
    got = moe.combine(y, weights, split, dtype, shared_gate=logits)
    assert torch.equal(got, moe.combine(y, weights, split.tensor(), dtype, shared_gate=logits))
    shared = _in_order(parts).to(dtype).double()
    want = torch.einsum("ts,tsc->tc", weights.double(), y.double().view(tokens, top, width))
    want = want + (torch.sigmoid(logits.double())[:, None] if gate else 1.0) * shared
    # three products of numbers of a few units, then one rounding to the type
    torch.testing.assert_close(got.double(), want, rtol=2.0 ** -8 if dtype == torch.bfloat16 else 1e-6, atol=2e-6)


@pytest.mark.parametrize("top", [1, 2, 3, 5])
@pytest.mark.parametrize("parts", [1, 2, 3])
@pytest.mark.parametrize("width", [66, 1028])
@pytest.mark.parametrize("rows", [False, True])
def test_sum_over_slots(top, parts, width, rows):
    """Parts in ascending order, then slots in ascending order by fused multiply-adds; a token's only slot has a kernel of its own."""
    from gllm_b200.ops import moe

    g = torch.Generator().manual_seed(top)
    tokens = 70
    y, weights = torch.randn(parts, tokens * top, width, generator=g).cuda(), torch.rand(tokens, top, generator=g).cuda()
    at = torch.randperm(tokens * top, generator=g) if rows else torch.arange(tokens * top)
    got = moe.combine(y, weights, None, torch.float32, row_of_pair=at.int().cuda() if rows else None)
    each = _in_order(y)[at.cuda()].view(tokens, top, width)
    want = torch.zeros(tokens, width, device="cuda", dtype=torch.float64)
    size = torch.zeros_like(want)
    for s in range(top):
        want += weights[:, s:s + 1].double() * each[:, s].double()
        size += (weights[:, s:s + 1] * each[:, s]).abs().double()
    # one rounding a slot, of a sum no larger than the magnitudes'
    assert bool(((got.double() - want).abs() <= top * 2.0 ** -24 * size + 1e-37).all())
