"""Calls between 193 and 1024 rows that take CTA pairs or one-CTA tiles by size: every row of the result is the same, bit for
bit, as in a call of at most 128 rows, which is always one-CTA (K is whole in both, its blocks in the same order)."""

import pytest
import torch

from rk_b200 import _lib

pytestmark = pytest.mark.gpu
DEVICE = torch.device("cuda:0")


def both(linear, pack, m, n, k, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    x = torch.randn(m, k, generator=gen, device=DEVICE).bfloat16()
    w = pack((torch.randn(n, k, generator=gen, device=DEVICE) * 0.05).bfloat16())
    bias = torch.randn(n, generator=gen, device=DEVICE).bfloat16()
    whole = linear(pack(x), w, bias)
    parts = torch.cat([linear(pack(x[r:r + 128]), w, bias) for r in range(0, m, 128)])
    assert whole.shape == (m, n) and torch.equal(whole.view(torch.int16), parts.view(torch.int16))
    assert _lib.read_status(_lib.workspace(DEVICE, _lib.WORKSPACE_HEADER)) == 0


# one row more than the limits; few tiles and many; padding above and below a quarter with K on both sides of 4096; ragged columns
@pytest.mark.parametrize("m,n,k", [(193, 520, 256), (193, 16384, 256), (264, 4096, 2048), (384, 8192, 512), (385, 8192, 512),
                                   (500, 2056, 1024), (511, 16384, 128)])
@pytest.mark.parametrize("kind", ["mxfp8", "nvfp4"])
def test_block_scaled_rows_do_not_depend_on_the_route(m, n, k, kind):
    from rk_b200 import fp4_linear as P4
    from rk_b200 import fp8_linear as P8

    if kind == "mxfp8":
        both(lambda a, b, bias: P8.mxfp8_linear(*a, *b, bias), P8.mxfp8_pack, m, n, k, m + n)
    else:
        both(lambda a, b, bias: P4.linear_forward_packed_gemm_bf16(*a, None, *b, None, bias, k), P4.pack_nvfp4, m, n, k, m + n)


@pytest.mark.parametrize("m,n,k", [(320, 16384, 256), (321, 16384, 256), (384, 9608, 384), (560, 10248, 4096), (560, 8192, 4224),
                                   (576, 8192, 4224), (816, 2048, 512), (816, 16400, 384), (1024, 6144, 128), (1000, 8200, 640)])
@pytest.mark.parametrize("kind", ["int8", "fp8"])
def test_w8a8_and_fp8_rows_do_not_depend_on_the_route(m, n, k, kind):
    from rk_b200 import fp8_linear as P8
    from rk_b200.integer import integer_gemm

    if kind == "int8":
        pack = lambda t: ((t * 20).round().clamp(-127, 127).to(torch.int8), t.float().abs().amax(1) * 0.01)
        both(lambda a, b, bias: integer_gemm(*a, *b, bias, 8, 0), pack, m, n, k, m + n)
    else:
        one = torch.full((1,), 0.03125, device=DEVICE)
        both(lambda a, b, bias: P8.linear_forward_packed(*a, *b, bias), lambda t: (t.to(torch.float8_e4m3fn), one), m, n, k, m + n)
