"""Where the 32-bit product cuts its sums: by the sizes of weight and sum alone, whatever GPU there is (here none)."""

from ctypes import c_int

import pytest


@pytest.mark.parametrize("n,k,blocks", [
    (64, 544, 9), (128, 2048, 8), (1024, 1024, 8), (2048, 2048, 11), (2048, 8192, 43), (2816, 2048, 11), (2944, 2048, 13),
    (3072, 2048, 13), (3328, 2048, 13), (4096, 2048, 16), (5632, 2048, 22), (8192, 2048, 32), (9472, 2048, 32), (9600, 2048, 64),
    (16384, 2048, 64), (16384, 8192, 64), (128256, 4096, 64), (128256, 65536, 128),
])
def test_ranges_follow_the_sizes(n, k, blocks):
    from gllm_b200.ops.build import load_module

    f = load_module("gemm_fp32").gllm_gemm_f32_range_blocks
    f.argtypes, f.restype = [c_int, c_int], c_int
    assert f(n, k) == blocks
