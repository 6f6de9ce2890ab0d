"""The 32-bit product on the tensor cores (three bfloat16 parts a number): widths of its token tiles, ends of blocks, chunks and
ranges of K, magnitudes, and operands that are not finite."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _bound(a, b):
    """Per element: the leading accumulator truncates at most 16 times a chunk of 256, a chunk's and a range's sum round once
    each, what the cut leaves out is under 2^-24 of a product, and the smaller products' accumulator is 2^-7 of the leading one
    with up to 640 truncations (2,048 of K, five products of 16 a time)."""
    k = a.shape[1]
    steps = 2.0 * (16 + 640 / 128) + (k / 256 + k / 2048 + 4)
    return steps * 2.0 ** -24 * (a.double().abs() @ b.double().abs().T) + 1e-37


@pytest.mark.parametrize("m", [1, 16, 17, 33, 64, 65, 97, 200])
@pytest.mark.parametrize("n,k", [(1, 32), (127, 36), (129, 256), (300, 260), (2048, 2080), (257, 4100)])
def test_sizes(m, n, k):
    from gllm_b200 import ops

    g = torch.Generator().manual_seed(m * n + k)
    a, b = torch.randn(m, k, generator=g).cuda(), torch.randn(n, k, generator=g).cuda()
    got = ops.linear(a, b)
    want = a.double() @ b.double().T
    assert bool(((got.double() - want).abs() <= _bound(a, b)).all())
    assert torch.equal(ops.linear(a[m // 2:m // 2 + 1].contiguous(), b)[0], got[m // 2])
    assert int(ops.status_word(a.device)[0]) == 0


@pytest.mark.parametrize("scale_a,scale_b", [(1e30, 1e-30), (1e-18, 1e-12), (1e18, 1e18), (3e-30, 1.0)])
def test_magnitudes(scale_a, scale_b):
    from gllm_b200 import ops

    g = torch.Generator().manual_seed(3)
    a = (torch.randn(70, 520, generator=g) * scale_a).cuda()
    b = (torch.randn(130, 520, generator=g) * scale_b).cuda()
    a[:, ::7] *= 1e-6                                    # very different numbers in one row
    got = ops.linear(a, b)
    want = a.double() @ b.double().T
    assert bool(((got.double() - want).abs() <= _bound(a, b)).all())


@pytest.mark.parametrize("m", [3, 90, 200])
def test_not_finite(m):
    """As the sum of 32-bit products has it: an infinity stays one, and what does not meet it stays as it is."""
    from gllm_b200 import ops

    g = torch.Generator().manual_seed(m)
    a, b = torch.randn(m, 2100, generator=g).cuda(), torch.randn(260, 2100, generator=g).cuda()
    clean = ops.linear(a, b)
    a[1, 2099], a[2, 5] = float("inf"), float("nan")
    a[0, 7] = 3.4e38                                     # finite, and an infinity once rounded to bfloat16
    b[200, 40] = float("-inf")
    b[:, 7] = 0.25
    got, want = ops.linear(a, b), a.double() @ b.double().T
    finite = want.isfinite() & (want.abs() < 3.4e38)
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got[~finite & ~want.isnan()].double(), want[~finite & ~want.isnan()])
    assert bool(((got.double() - want).abs()[finite] <= (1.1 * 2100 * 2.0 ** -24 * (a.double().abs() @ b.double().abs().T))[finite]).all())
    rows = torch.arange(m, device="cuda") > 2
    cols = torch.arange(260, device="cuda") != 200
    b2 = b.clone()
    assert torch.equal(ops.linear(a[rows], b2)[:, cols], got[rows][:, cols])
    assert clean.isfinite().all()


@pytest.mark.parametrize("m", [3, 90])
@pytest.mark.parametrize("k", [64, 600])
def test_weight_that_the_kernel_before_writes(m, k):
    """Either operand may be the result of the product right before, in memory that held another one's: nothing waits in between."""
    from gllm_b200 import ops

    g = torch.Generator().manual_seed(m)
    a, b, x = (torch.randn(*shape, generator=g).cuda() for shape in ((200, k), (600, k), (m, 600)))
    held = torch.empty(200, 600, device="cuda")
    for factor in (1.0, -1.0, 2.0, 0.0, 0.5):
        first = factor * a
        torch.cuda.synchronize()
        y = ops.linear(first, b, out=held)
        of_weight, of_both = ops.linear(x, y), ops.linear(y, y)
        torch.cuda.synchronize()
        want = first.double() @ b.double().T
        for got, right in ((y, want), (of_weight, x.double() @ want.T), (of_both, want @ want.T)):
            assert bool(((got.double() - right).abs() <= 1e-5 * right.abs().max()).all())


def _off(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


@pytest.mark.parametrize("k", [32, 64, 96, 128, 256, 384, 512, 516, 640, 1024, 1280, 1792, 2048, 4096])
@pytest.mark.parametrize("signs", ["both", "one"])
def test_no_further_from_64_bits_than_multiply_adds(k, signs):
    """Rows off 16-byte boundaries run plain 32-bit multiply-adds, two sums a result; the others may not err by more.  (Each error is
    a norm over 100,000 results, good to a few parts in a thousand.)"""
    from gllm_b200 import ops

    g = torch.Generator().manual_seed(k)
    wide, b = torch.randn(200, k + 1, generator=g).cuda(), torch.randn(512, k, generator=g).cuda()
    if signs == "one":
        wide, b = wide.abs(), b.abs()
    a = wide[:, :k]
    want = a.double() @ b.double().T
    assert _off(ops.linear(a.contiguous(), b), want) <= 1.03 * _off(ops.linear(a, b), want)


@pytest.mark.parametrize("scale_a,scale_b", [(1e-33, 1e30), (1e-35, 1e30), (1e-36, 1e30), (1e-37, 1e33), (1e30, 1e-37), (1e-39, 1e33)])
@pytest.mark.parametrize("k", [260, 1032])
def test_smallest_numbers_keep_their_bits(scale_a, scale_b, k):
    """Operands down to the subnormal ones are what they are: the errors of 32-bit sums, relative to the result."""
    from gllm_b200 import ops

    g = torch.Generator().manual_seed(5)
    a, b = (torch.randn(70, k, generator=g) * scale_a).cuda(), (torch.randn(130, k, generator=g) * scale_b).cuda()
    want = a.double() @ b.double().T
    # (5.7e-7 is what multiply-adds leave at K = 2,048; without the third part it would be 4e-6)
    assert _off(ops.linear(a, b), want) <= 6e-7


@pytest.mark.parametrize("m", [70, 300])
def test_subnormal_results(m):
    """They come from 32-bit multiply-adds, each of which rounds by up to half a unit of the smallest number here; and are the same in a
    batch as alone."""
    from gllm_b200 import ops

    g = torch.Generator().manual_seed(m)
    a, b = (torch.randn(m, 4100, generator=g) * 1e-21).cuda(), (torch.randn(2048, 4100, generator=g) * 1e-21).cuda()
    got = ops.linear(a, b)
    want = a.double() @ b.double().T
    assert bool(((got.double() - want).abs() <= a.shape[1] * 2.0 ** -150).all())
    for row in (0, m - 1):
        assert torch.equal(ops.linear(a[row:row + 1].contiguous(), b)[0], got[row])


@pytest.mark.parametrize("m", [1, 17, 90])
@pytest.mark.parametrize("n,k", [(10001, 600), (2050, 2100), (700, 1100)])
def test_broken_rows_of_either_operand(m, n, k):
    """Results that are not finite, in tiles with a range each and with all: as multiply-adds have them; the others do not change."""
    from gllm_b200 import ops

    g = torch.Generator().manual_seed(m + n)
    a, b = torch.randn(m, k, generator=g).cuda(), torch.randn(n, k, generator=g).cuda()
    clean = ops.linear(a, b)
    x, w = a.clone(), b.clone()
    x[m - 1, k - 1], w[n - 1, 3], w[5, 0] = float("nan"), float("inf"), float("nan")
    got, want = ops.linear(x, w), x.double() @ w.double().T
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    assert torch.equal(got[want.isinf()].double(), want[want.isinf()])
    assert torch.equal(got[want.isfinite()], clean[want.isfinite()])
    big = ops.linear(a * 1e34, b)                         # finite, and beyond what the parts' sums hold
    assert _off(big / 1e34, a.double() @ b.double().T) <= 1e-6


@pytest.mark.parametrize("m", [1, 33, 97])
@pytest.mark.parametrize("n,k", [(127, 516), (300, 1292), (257, 4100), (2048, 2080), (9700, 2080)])
def test_every_part_everywhere(m, n, k):
    """The whole sum, and the sums of some of k alone, are as close to 64 bits as 32-bit sums are: 2.4e-7 measured; what two parts a
    number leave is 4.4e-6 whatever K is."""
    from gllm_b200 import ops

    g = torch.Generator().manual_seed(m + n + k)
    a, b = torch.randn(m, k, generator=g).cuda(), torch.randn(n, k, generator=g).cuda()
    for low, high in ((0, k), (0, 32), (256, 512), (k // 2 - 128, k // 2 + 128), (k - 256, k), (k - 4, k)):
        only = torch.zeros_like(a)
        only[:, low:high] = a[:, low:high]
        want = only.double() @ b.double().T
        assert _off(ops.linear(only, b), want) <= 6e-7
