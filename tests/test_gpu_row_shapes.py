"""The row kernels pick threads and vectors per row by the number of rows and their length.  The choice must never show in
a result: rows of a tall matrix (64 threads each) equal the same rows quantized alone (256 threads), bit for bit.  The small
launches are held to the oracle by the other tests."""

import numpy as np
import pytest
import torch

from rk_b200 import _lib

pytestmark = pytest.mark.gpu
TALL, FEW = 2400, 48  # multiples of the 48 rows that share one modulation vector


def _randn(gen, *shape, std=1.0):
    return (torch.randn(*shape, generator=gen, device="cuda") * std).bfloat16()


def _bits(tensors, rows):
    return [t[rows].contiguous().view(torch.uint8) for t in tensors]


@pytest.mark.parametrize("k", [8, 250, 333, 512, 1000, 1032, 2048, 2056, 4096, 4100, 8192])
@pytest.mark.parametrize("bits", [8, 4])
def test_the_shape_of_a_launch_never_changes_a_row(k, bits):
    lib, dev, ptr = _lib.load(), torch.device("cuda:0"), _lib.ptr
    gen = torch.Generator(device=dev).manual_seed(k)
    x_all, y_all = _randn(gen, TALL, k), _randn(gen, TALL, k)
    scale_all, shift_all, gate_all = (_randn(gen, TALL // 48, k, std=0.1) for _ in range(3))
    x_all[1] = 0.0
    x_all[2, 0], x_all[3, 0], x_all[4, 0] = float("inf"), float("nan"), 3e38
    table = torch.nn.functional.gelu(torch.arange(65536, device=dev, dtype=torch.int32).to(torch.int16).view(torch.bfloat16))
    ws = torch.zeros(_lib.WORKSPACE_HEADER, device=dev, dtype=torch.uint8)
    width = (k + 127) // 128 * 128 * bits // 8

    def run(first, rows):
        part = slice(first, first + rows)
        vectors = slice(first // 48, (first + rows) // 48)
        x, y = x_all[part].clone(), y_all[part].clone()  # at aligned addresses, whatever k
        scale, shift, gate = (t[vectors].clone() for t in (scale_all, shift_all, gate_all))
        q, s = torch.zeros(rows, width, device=dev, dtype=torch.uint8), torch.zeros(rows, device=dev)
        stream, results = _lib.stream_ptr(dev), []
        for mode in (_lib.ACT_PLAIN, _lib.ACT_LUT_MUL, _lib.ACT_LUT):
            _lib.check(lib.rk_quant_rows(ptr(x), rows, k, k, ptr(y), k, ptr(table), mode, bits, ptr(q), ptr(s), stream), "rows")
            results += [q.clone(), s.clone()]
        for norm in (0, 1):
            res = torch.zeros(rows, k, device=dev, dtype=torch.bfloat16)
            _lib.check(lib.rk_quant_rows_modulated(ptr(x), ptr(scale), ptr(shift), rows, k, 48, norm, 1e-6, ptr(y), ptr(gate),
                                                   ptr(res), bits, ptr(q), ptr(s), stream), "modulated")
            results += [q.clone(), s.clone(), res]
        res, normed = (torch.zeros(rows, k, device=dev, dtype=torch.bfloat16) for _ in range(2))
        _lib.check(lib.rk_gated_rmsnorm_quant_rows(ptr(x), ptr(y), ptr(gate), ptr(scale), ptr(shift), 48, rows, k, 1e-6, bits,
                                                   ptr(res), ptr(normed), ptr(q), ptr(s), stream), "rmsnorm")
        results += [q.clone(), s.clone(), res, normed]
        if bits == 8:
            res, normed, one = torch.zeros_like(res), torch.zeros_like(normed), torch.zeros(1, device=dev)
            _lib.check(lib.rk_rmsnorm_tensor_scale(ptr(x), ptr(y), ptr(scale_all), None, 0, rows, k, 1e-6, 2688.0, ptr(res),
                                                   ptr(normed), ptr(one), ptr(ws), ws.numel(), stream), "tensor scale")
            finite = normed.float()[torch.isfinite(normed)].abs().max().item()
            assert one.item() == max(np.float32(finite) / np.float32(2688.0), np.float32(1e-12))  # the IEEE quotient
            results += [res, normed]
        return results

    all_rows = run(0, TALL)
    for first in (0, TALL - FEW):  # rows that a CTA takes first and rows it comes to last
        for tall, few in zip(_bits(all_rows, slice(first, first + FEW)), _bits(run(first, FEW), slice(FEW))):
            assert torch.equal(tall, few)


@pytest.mark.parametrize("rows,k", [(1200, 2048), (331, 4100), (160, 8190), (1181, 2056), (150, 8192)])
@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("strided", [False, True])
def test_table_on_chip_equals_the_gathered_table(rows, k, bits, strided):
    """Enough elements for the table in shared memory: rows equal the same rows in small launches (table through L1), for dense
    and strided inputs, with groups of threads that run out of rows."""
    lib, dev, ptr = _lib.load(), torch.device("cuda:0"), _lib.ptr
    gen = torch.Generator(device=dev).manual_seed(rows + k)
    pitch = k + 24 if strided else k
    x, up = _randn(gen, rows, pitch)[:, :k], _randn(gen, rows, pitch)[:, :k]
    table = _randn(gen, 65536)
    table[0x4000:0x4010] = float("nan")
    width = (k + 127) // 128 * 128 * bits // 8
    ws = torch.zeros(_lib.WORKSPACE_HEADER, device=dev, dtype=torch.uint8)

    def quantized(mode, first, count):
        q, s = torch.full((count, width), 9, device=dev, dtype=torch.uint8), torch.zeros(count, device=dev)
        _lib.check(lib.rk_quant_rows(ptr(x[first:]), count, k, pitch, ptr(up[first:]), pitch, ptr(table), mode, bits, ptr(q),
                                     ptr(s), _lib.stream_ptr(dev)), "rows")
        return q, s

    for mode in (_lib.ACT_LUT_MUL, _lib.ACT_LUT):
        q, s = quantized(mode, 0, rows)
        for first in (0, rows // 2, rows - 20):
            few_q, few_s = quantized(mode, first, 20)
            assert torch.equal(q[first:first + 20], few_q) and torch.equal(s[first:first + 20], few_s)
    if k % 8 == 0 and pitch % 8 == 0:
        out, one = torch.zeros(rows, k, device=dev, dtype=torch.bfloat16), torch.zeros(1, device=dev)
        _lib.check(lib.rk_lut_mul_tensor_scale(ptr(x), pitch, ptr(up), pitch, ptr(table), rows, k, 2688.0, ptr(out), ptr(one),
                                               ptr(ws), ws.numel(), _lib.stream_ptr(dev)), "product")
        index = x.contiguous().view(torch.int16).to(torch.int64) & 0xFFFF
        want = (table[index].float() * up.float()).bfloat16()
        assert torch.equal(torch.nan_to_num(out.float(), nan=-7.5), torch.nan_to_num(want.float(), nan=-7.5))
        finite = want.float()[torch.isfinite(want)].abs().max().item()
        assert one.item() == np.float32(finite) / np.float32(2688.0)


@pytest.mark.parametrize("k,group", [(2048, 64), (520, 64), (2056, 128), (4096, 128), (8190, 256)])
@pytest.mark.parametrize("mode", ["gelu", "gelu times up"])
def test_every_row_of_every_trip_of_the_table_kernel(k, group, mode):
    """Two full trips of 148 CTAs with 1024 / `group` rows each and a third for five rows, so every group of threads of a CTA
    (sixteen with 64 threads per row: as many as it has named barriers) takes several rows.  Every row equals the same
    row in small launches, which gather the table through L1."""
    lib, dev, ptr = _lib.load(), torch.device("cuda:0"), _lib.ptr
    rows, few = 2 * 148 * (1024 // group) + 5, 1200000 // k  # fewer elements than the table in shared memory asks for
    gen = torch.Generator(device=dev).manual_seed(k)
    # rows of very different size: a maximum taken from another row or another warp's half shows in the scale
    x = _randn(gen, rows, k) * torch.logspace(-2, 2, 31, device=dev)[torch.arange(rows, device=dev) % 31, None].bfloat16()
    up = _randn(gen, rows, k)
    table = torch.nn.functional.gelu(torch.arange(65536, device=dev, dtype=torch.int32).to(torch.int16).view(torch.bfloat16))
    act = _lib.ACT_LUT if mode == "gelu" else _lib.ACT_LUT_MUL
    width = (k + 127) // 128 * 128

    def quantized(first, count):
        q, s = torch.full((count, width), 9, device=dev, dtype=torch.int8), torch.zeros(count, device=dev)
        _lib.check(lib.rk_quant_rows(ptr(x[first:]), count, k, k, ptr(up[first:]), k, ptr(table), act, 8, ptr(q), ptr(s),
                                     _lib.stream_ptr(dev)), mode)
        return q, s

    q, s = quantized(0, rows)
    for first in range(0, rows, few):
        count = min(few, rows - first)
        few_q, few_s = quantized(first, count)
        assert torch.equal(q[first:first + count], few_q) and torch.equal(s[first:first + count], few_s)
