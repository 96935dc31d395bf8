"""W8A8 products with more rows than 128 x 148: the entry points return (CPU part, on a process that sees no device), and give the
exact product where the call does not take CTA pairs - fewer than 128 output channels, a residual (GPU part)."""

import os
import subprocess
import sys

import pytest
import torch

from rk_b200 import _lib

# arguments that pass every check; without a visible device nothing is launched and nothing reads the pointers
SCRIPT = """
import ctypes, sys
sys.path.insert(0, {package!r})
from rk_b200 import _lib
lib, buffer = _lib.load(), ctypes.create_string_buffer(1 << 16)
p = ctypes.c_void_p((ctypes.addressof(buffer) + 255) & ~255)
for m in (18944, 18945, 19584, 1 << 24):
    for n, k in ((64, 2048), (2048, 128)):
        codes = [lib.rk_gemm_int(p, p, p, p, None, p, m, n, k, 8, 0, p, 4096, None),
                 lib.rk_gemm_int_residual(p, p, p, p, None, p, None, 1, p, m, n, k, 8, 0, p, 4096, None),
                 lib.rk_gemm_int_acc(p, p, p, m, n, k, 8, 0, p, 4096, None),
                 lib.rk_gemm_int4_widened(p, p, p, p, None, p, None, 1, p, m, n, k, 0, p, 1 << 60, p, 4096, None)]
        assert all(c != _lib.RK_EINVAL and c != _lib.RK_OK for c in codes), (m, n, k, codes, _lib.last_error())
print("returned")
"""


def test_many_rows_return_a_code():
    from pathlib import Path

    script = SCRIPT.format(package=str(Path(_lib.__file__).resolve().parents[1]))
    for pairs in ("", "0"):  # RK_B200_TWO_CTA=0: every call takes the one-CTA plan
        env = {**os.environ, "CUDA_VISIBLE_DEVICES": ""}
        if pairs:
            env["RK_B200_TWO_CTA"] = pairs
        done = subprocess.run([sys.executable, "-c", script], env=env, capture_output=True, text=True, timeout=300)
        assert done.returncode == 0 and "returned" in done.stdout, (done.returncode, done.stderr[-2000:])


DEVICE = torch.device("cuda:0")


@pytest.mark.gpu
@pytest.mark.parametrize("m", [18944, 18945, 19584])
@pytest.mark.parametrize("n,bits,form", [(64, 8, "plain"), (256, 8, "gate"), (256, 8, "residual"), (256, 4, "gate")])
def test_many_rows_give_the_exact_product(m, n, bits, form):
    from rk_b200.integer import integer_gemm

    gen = torch.Generator(device=DEVICE).manual_seed(m + n + bits)
    limit, k = (127, 128) if bits == 8 else (7, 2048)
    codes = lambda rows: torch.randint(-limit, limit + 1, (rows, k), generator=gen, device=DEVICE, dtype=torch.int32)
    pack = lambda q: q.to(torch.int8) if bits == 8 else ((q[:, 0::2] & 15) | ((q[:, 1::2] & 15) << 4)).to(torch.uint8)
    a, b = codes(m), codes(n)
    sa = torch.rand(m, generator=gen, device=DEVICE) * 2.0 ** -10 + 2.0 ** -12
    sb = torch.rand(n, generator=gen, device=DEVICE) * 2.0 ** -2 + 2.0 ** -4
    y = ((a.double() @ b.double().T).float() * sa[:, None] * sb).bfloat16()  # integers below 2^24, then the epilogue's roundings
    residual = torch.randn(m, n, generator=gen, device=DEVICE).bfloat16() if form != "plain" else None
    batches = next(c for c in (8, 5, 4, 3) if m % c == 0) if form == "gate" else 0
    gate = torch.randn(batches, n, generator=gen, device=DEVICE).bfloat16() if batches else None
    got = integer_gemm(pack(a), sa, pack(b), sb, None, bits, 0, residual=residual, gate=gate)
    if gate is not None:
        y = y * gate.repeat_interleave(m // batches, 0)
    want = y if residual is None else residual + y
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    assert _lib.read_status(_lib.workspace(DEVICE, _lib.WORKSPACE_HEADER)) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(1, 64, 256), (50, 8192, 256), (128, 2568, 128), (300, 2560, 512), (816, 2056, 384), (1000, 2048, 256),
                                   (1024, 520, 128)])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("gated", [False, True])
def test_residual_rows_are_read_at_any_address(m, n, k, offset, gated):
    """Narrow, wide and ragged column tiles, one to eight row tiles; residual and gate on a 16-byte boundary or two bytes off."""
    gen = torch.Generator(device=DEVICE).manual_seed(m + n + offset)
    a, b = (torch.randint(-127, 128, (r, k), generator=gen, device=DEVICE, dtype=torch.int8) for r in (m, n))
    sa, sb = (torch.rand(r, generator=gen, device=DEVICE) * 2.0 ** -5 + 2.0 ** -8 for r in (m, n))
    at = lambda rows: torch.randn(rows * n + offset, generator=gen, device=DEVICE).bfloat16()[offset:].view(rows, n)
    batches = next(c for c in (4, 3, 2, 1) if m % c == 0)
    residual, gate = at(m), at(batches) if gated else None
    out = torch.full((m + 2, n), 7.0, device=DEVICE, dtype=torch.bfloat16)
    ws = _lib.workspace(DEVICE, _lib.WORKSPACE_HEADER)
    P = _lib.ptr
    code = _lib.load().rk_gemm_int_residual(P(a), P(sa), P(b), P(sb), None, P(residual), P(gate), m // batches if gated else 1, P(out[1:]),
                                            m, n, k, 8, 0, P(ws), ws.numel(), _lib.stream_ptr(DEVICE))
    _lib.check(code, "rk_gemm_int_residual")
    y = ((a.double() @ b.double().T).float() * sa[:, None] * sb).bfloat16()
    if gated:
        y = y * gate.repeat_interleave(m // batches, 0)
    assert torch.equal(out[1:m + 1].view(torch.int16), (residual + y).view(torch.int16))
    assert (out[0] == 7.0).all() and (out[m + 1] == 7.0).all()
    assert _lib.read_status(ws) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(64, 520, 4224), (65, 2048, 4224), (72, 72, 8192), (100, 1032, 4352), (128, 2048, 4224), (129, 264, 4224)])
@pytest.mark.parametrize("with_residual", [False, True])
def test_two_row_tiles_of_a_long_loop(m, n, k, with_residual):
    """65 to 128 rows and more than 32 K blocks: two row tiles, even and odd; the rows on either side of the range."""
    from rk_b200.integer import integer_gemm

    gen = torch.Generator(device=DEVICE).manual_seed(m + n + k)
    a, b = (torch.randint(-15, 16, (r, k), generator=gen, device=DEVICE, dtype=torch.int8) for r in (m, n))
    sa, sb = (torch.rand(r, generator=gen, device=DEVICE) * 2.0 ** -5 + 2.0 ** -8 for r in (m, n))
    residual = torch.randn(m, n, generator=gen, device=DEVICE).bfloat16() if with_residual else None
    y = ((a.double() @ b.double().T).float() * sa[:, None] * sb).bfloat16()  # whole numbers below 2^21
    got = integer_gemm(a, sa, b, sb, None, 8, 0, residual=residual)
    assert torch.equal(got.view(torch.int16), (y if residual is None else residual + y).view(torch.int16))
    assert _lib.read_status(_lib.workspace(DEVICE, _lib.WORKSPACE_HEADER)) == 0
