"""The streaming W4A16 kernel of one to sixteen activation rows, at the edges of its fragments, shares of K and loads.

Reference: the packed integers and bf16 scales multiplied in 64 bits.  Bound of an output: its bf16 rounding (2^-8 of the
value at most) plus fp32 accumulation, k * 2^-23 of the sum of magnitudes (the tensor cores may truncate)."""

import pytest
import torch

from rk_b200 import _lib
from rk_b200.w4a16_linear import linear_w4a16, pack_weight

pytestmark = pytest.mark.gpu
DEVICE = torch.device("cuda:0")


def reference(x, packed, scales, bias):
    lo, hi = (packed & 15).to(torch.int16), (packed >> 4).to(torch.int16)
    n, half = packed.shape
    nibbles = torch.cat(((lo - 16 * (lo > 7)).view(n, -1, 4), (hi - 16 * (hi > 7)).view(n, -1, 4)), -1).reshape(n, 2 * half)
    w = nibbles.double() * scales.double().t().repeat_interleave(128, 1)
    out, magnitude = x.double() @ w.t(), x.double().abs() @ w.abs().t()
    return (out if bias is None else out + bias.double()), magnitude


@pytest.mark.parametrize("n,k", [
    (8, 128),       # half a channel tile, one group: no share of K
    (24, 384),      # a tile and a half, three groups in two shares
    (40, 1152),     # nine groups in eight shares: one has two
    (1024, 1024),   # a group per warp
    (136, 2176),    # seventeen groups in sixteen shares
    (2048, 4480),   # 35 groups: batches end inside a share
    (16392, 256),   # several tiles per CTA, the last CTA not full
])
@pytest.mark.parametrize("m", [1, 2, 7, 8, 9, 15, 16])
def test_few_rows_match_the_exact_product(n, k, m):
    gen = torch.Generator(device=DEVICE).manual_seed(n + k + m)
    r = lambda *s: torch.randn(s, generator=gen, device=DEVICE)
    packed, scales = pack_weight((r(n, k) * 0.02).bfloat16())
    x = r(m, k).bfloat16()
    bias = (r(n) * 0.1).bfloat16() if (m + n) % 2 else None
    buf = torch.full((m + 2, n), 7.0, dtype=torch.bfloat16, device=DEVICE)
    ws = _lib.gemm_workspace(_lib.OP_W4A16, DEVICE, m, n, k)
    code = _lib.load().rk_gemm_w4a16_g128(_lib.ptr(x), _lib.ptr(packed), _lib.ptr(scales), _lib.ptr(bias), _lib.ptr(buf[1:m + 1]), m, n, k,
                                          0, _lib.ptr(ws), ws.numel(), _lib.stream_ptr(DEVICE))
    _lib.check(code, "rk_gemm_w4a16_g128")
    assert _lib.read_status(ws) == 0
    assert (buf[0] == 7.0).all() and (buf[m + 1] == 7.0).all()
    want, magnitude = reference(x, packed, scales, bias)
    bound = 2.0 ** -8 * want.abs() + k * 2.0 ** -23 * magnitude
    assert ((buf[1:m + 1].double() - want).abs() <= bound).all()


@pytest.mark.parametrize("m,k", [(1, 32768), (4, 16384), (8, 12288), (16, 4096)])
def test_long_rows_with_and_without_room_for_the_activations(m, k):
    gen = torch.Generator(device=DEVICE).manual_seed(k)
    packed, scales = pack_weight((torch.randn(64, k, generator=gen, device=DEVICE) * 0.02).bfloat16())
    x = torch.randn(m, k, generator=gen, device=DEVICE).bfloat16()
    want, magnitude = reference(x, packed, scales, None)
    bound = 2.0 ** -8 * want.abs() + k * 2.0 ** -23 * magnitude
    assert ((linear_w4a16(x, packed, scales).double() - want).abs() <= bound).all()


def test_rows_do_not_reach_each_other():
    """Infinities and NaN stay in their row; a row of zeros gives zeros."""
    gen = torch.Generator(device=DEVICE).manual_seed(5)
    packed, scales = pack_weight((torch.randn(32, 256, generator=gen, device=DEVICE) * 0.02).bfloat16())
    x = torch.randn(9, 256, generator=gen, device=DEVICE).bfloat16()
    clean = linear_w4a16(x, packed, scales)
    x[3, 5], x[8, 250], x[4] = float("inf"), float("nan"), 0.0
    got = linear_w4a16(x, packed, scales)
    same = [0, 1, 2, 5, 6, 7]
    assert torch.equal(got[same], clean[same]) and (got[4] == 0).all()
    assert not torch.isfinite(got[3]).any() and torch.isnan(got[8]).all()


@pytest.mark.parametrize("m,n,k", [
    (129, 1000, 128),    # narrow tiles: two row tiles, the last of one row, one group
    (256, 2048, 2048),   # narrow, eight CTAs to a tile
    (257, 2568, 640),    # three row tiles, an odd group at the end
    (384, 4736, 256),    # 111 narrow tiles
    (1000, 2368, 128),   # 152: wide ones
    (160, 4096, 4096),   # eight group pairs to a CTA, the most
    (300, 2048, 8192),   # eleven: wide
])
def test_row_tiles_above_128_rows_match_the_folded_product(m, n, k):
    """The scale folded into bf16 weights, then products and sums in 64 bits; bounds as above."""
    gen = torch.Generator(device=DEVICE).manual_seed(n + k + m)
    r = lambda *s: torch.randn(s, generator=gen, device=DEVICE)
    packed, scales = pack_weight((r(n, k) * 0.02).bfloat16())
    x, bias = r(m, k).bfloat16(), (r(n) * 0.1).bfloat16()
    eye, _ = reference(torch.eye(k, device=DEVICE), packed, torch.ones_like(scales), None)  # [k, n] integers
    w = (eye.bfloat16() * scales.repeat_interleave(128, 0)).double()
    want, magnitude = x.double() @ w + bias.double(), x.double().abs() @ w.abs()
    got = linear_w4a16(x, packed, scales, bias)
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + k * 2.0 ** -23 * magnitude).all()
    assert _lib.read_status(_lib.workspace(DEVICE, _lib.WORKSPACE_HEADER)) == 0
