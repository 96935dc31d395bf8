"""The order in which CTA pairs take their tiles (equal groups of at most eight row tiles, column by column inside a group)
and the 256-column tiles of the re-packing epilogues."""

import numpy as np
import pytest
import torch

from rk_b200 import _lib
from rk_b200.integer import integer_gemm

pytestmark = pytest.mark.gpu
DEVICE = torch.device("cuda:0")


@pytest.mark.parametrize("m,n,k", [
    (1025, 264, 128),    # five row tiles, one group, the last tile with one row
    (2049, 1032, 256),   # nine: groups of five and four
    (4400, 520, 128),    # eighteen: three groups of six
    (6400, 4104, 128),   # 25: groups of seven, seven, seven and four; several tiles per pair
])
def test_every_tile_of_every_group_is_computed_once(m, n, k):
    gen = torch.Generator(device=DEVICE).manual_seed(m)
    a, b = (torch.randint(-127, 128, (r, k), generator=gen, device=DEVICE, dtype=torch.int8) for r in (m, n))
    one = torch.ones(max(m, n), device=DEVICE)
    got = integer_gemm(a, one[:m], b, one[:n], None, 8, 0)
    want = a.double() @ b.double().T  # whole numbers below 2^22: exact
    assert torch.equal(got, want.float().bfloat16())


@pytest.mark.parametrize("m,n,k", [
    (1100, 1024, 128),   # at most 74 tiles: row tiles outermost
    (1025, 128, 128),    # one column of five tiles
    (2048, 9480, 128),   # eight row tiles, more tiles than pairs: columns outermost
    (1281, 16392, 128),  # six: a factor that does not divide 2^32
    (20000, 136, 128),   # 79 row tiles, weights of a few KB: row tiles outermost
    (2304, 8200, 640),   # nine row tiles, weights above 4 MB: groups of five and four
    (2304, 8200, 384),   # below: row tiles outermost
])
def test_every_tile_of_every_order_is_computed_once(m, n, k):
    test_every_tile_of_every_group_is_computed_once(m, n, k)


@pytest.mark.parametrize("m,n", [(64, 128), (200, 1024), (129, 25600), (257, 20480)])
def test_one_and_two_row_tiles_of_the_repacking_gemm(m, n):
    """One row tile with one, few and more column tiles than pairs; two row tiles with more than pairs."""
    from rk_b200 import fp4_linear as P4

    k, inter = 256, n // 2
    gen = torch.Generator(device=DEVICE).manual_seed(m + n)
    x = torch.randn(m, k, generator=gen, device=DEVICE).bfloat16()
    qa, sfa = P4.pack_nvfp4(x)
    qi, sfi = P4.pack_nvfp4(P4.interleave_gate_up_rows((torch.randn(n, k, generator=gen, device=DEVICE) * 0.05).bfloat16(), inter))
    plain = P4.linear_forward_packed_gemm_bf16(qa, sfa, None, qi, sfi, None, None, k)
    want_q, want_sf = P4.pack_swiglu_nvfp4(plain, inter, interleaved=True)
    got_q, got_sf = P4.linear_swiglu_packed_gemm(qa, sfa, None, qi, sfi, None, k)
    assert torch.equal(got_q, want_q) and torch.equal(got_sf, want_sf)


@pytest.mark.parametrize("m,n,k", [(600, 8192, 256), (600, 8192, 1024), (816, 4096, 2048), (1300, 4096, 256), (1300, 8192, 512)])
def test_repacking_tile_widths_by_the_longer_of_loop_and_epilogue(m, n, k):
    """Either side of the rule: short loops in tiles of 128 columns, long ones of 256, for the three epilogues."""
    from rk_b200 import fp4_linear as P4
    from rk_b200 import fp8_linear as P8
    from rk_b200 import mxfp8_swiglu as MS
    from rk_b200.cute_mxfp8_swiglu import cutlass_swiglu_mxfp8_packed

    inter = n // 2
    gen = torch.Generator(device=DEVICE).manual_seed(m + n + k)
    x = torch.randn(m, k, generator=gen, device=DEVICE).bfloat16()
    w = (torch.randn(n, k, generator=gen, device=DEVICE) * 0.05).bfloat16()
    wi = P4.interleave_gate_up_rows(w, inter)
    qa, sfa = P4.pack_nvfp4(x)
    qi, sfi = P4.pack_nvfp4(wi)
    plain = P4.linear_forward_packed_gemm_bf16(qa, sfa, None, qi, sfi, None, None, k)
    want_q, want_sf = P4.pack_swiglu_nvfp4(plain, inter, interleaved=True)
    got_q, got_sf = P4.linear_swiglu_packed_gemm(qa, sfa, None, qi, sfi, None, k)
    assert torch.equal(got_q, want_q) and torch.equal(got_sf, want_sf)
    # the activation by table, and its scale
    table = MS.make_bf16_silu_table(DEVICE)
    blocks = plain.view(m, inter // 64, 2, 64)  # 64 up, 64 gate
    up, gate = (blocks[:, :, i].reshape(m, inter) for i in (0, 1))
    want = (table.view(-1)[gate.contiguous().view(torch.int16).to(torch.int32) & 0xFFFF].float() * up.float()).bfloat16()
    out, scale = torch.empty_like(want), torch.zeros(1, device=DEVICE)
    ws = _lib.workspace(DEVICE, _lib.WORKSPACE_HEADER)
    P = _lib.ptr
    code = _lib.load().rk_gemm_nvfp4_gated_act(P(qa), P(sfa), None, P(qi), P(sfi), None, P(table), 448.0, P(out), P(scale), m, n, k, 0,
                                               P(ws), ws.numel(), _lib.stream_ptr(DEVICE))
    _lib.check(code, "rk_gemm_nvfp4_gated_act")
    assert torch.equal(out.view(torch.int16), want.view(torch.int16))
    assert scale.item() == np.float32(want.float().abs().max().item()) / np.float32(448.0)  # the IEEE quotient
    a, sa = P8.mxfp8_pack(x)
    b, sb = P8.mxfp8_pack(w)
    bi, sbi = P8.mxfp8_pack(wi)
    want_q, want_sf = MS.silu_mul_pack_mxfp8(P8.mxfp8_linear(a, sa, b, sb), inter, table)
    q, sf = cutlass_swiglu_mxfp8_packed(a, sa, bi, sbi, table)
    assert torch.equal(q.view(torch.uint8), want_q.view(torch.uint8)) and torch.equal(sf, want_sf)
    assert _lib.read_status(ws) == 0


@pytest.mark.parametrize("m,n", [(1300, 4992), (816, 16512), (2100, 4992)])
def test_repacking_epilogues_in_256_column_tiles(m, n):
    """Sizes whose tiles are 256 columns wide (2048-wide rows, several rounds of the pairs), 128 of them in the last tile for NVFP4:
    the bytes of the plain GEMM and the packing producer."""
    from rk_b200 import fp4_linear as P4
    from rk_b200 import fp8_linear as P8
    from rk_b200 import mxfp8_swiglu as MS
    from rk_b200.cute_mxfp8_swiglu import cutlass_swiglu_mxfp8_packed

    k, inter = 2048, n // 2
    gen = torch.Generator(device=DEVICE).manual_seed(m)
    x = torch.randn(m, k, generator=gen, device=DEVICE).bfloat16()
    w = (torch.randn(n, k, generator=gen, device=DEVICE) * 0.05).bfloat16()  # rows: gate (inter), then up (inter)
    wi = P4.interleave_gate_up_rows(w, inter)
    qa, sfa = P4.pack_nvfp4(x)
    qi, sfi = P4.pack_nvfp4(wi)
    plain = P4.linear_forward_packed_gemm_bf16(qa, sfa, None, qi, sfi, None, None, k)
    want_q, want_sf = P4.pack_swiglu_nvfp4(plain, inter, interleaved=True)
    got_q, got_sf = P4.linear_swiglu_packed_gemm(qa, sfa, None, qi, sfi, None, k)
    assert torch.equal(got_q, want_q) and torch.equal(got_sf, want_sf)
    if n % 256 == 0:
        table = MS.make_bf16_silu_table(DEVICE)
        a, sa = P8.mxfp8_pack(x)
        b, sb = P8.mxfp8_pack(w)
        bi, sbi = P8.mxfp8_pack(wi)
        want_q, want_sf = MS.silu_mul_pack_mxfp8(P8.mxfp8_linear(a, sa, b, sb), inter, table)
        q, sf = cutlass_swiglu_mxfp8_packed(a, sa, bi, sbi, table)
        assert torch.equal(q.view(torch.uint8), want_q.view(torch.uint8)) and torch.equal(sf, want_sf)
    assert _lib.read_status(_lib.workspace(DEVICE, _lib.WORKSPACE_HEADER)) == 0
