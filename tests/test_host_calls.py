"""The native callers of the eager linears: what is not a plain call is left to the general path (CPU part), a plain call gives
the general path's result in every form that it accepts (GPU part)."""

import pytest
import torch

from rk_b200 import _lib
from rk_b200.integer import IntegerLinear, integer_gemm, prepare_activation
from rk_b200.w4a16_linear import W4A16Linear, linear_w4a16


def cpu_state(kind):
    packed = torch.zeros(8, 128, dtype=torch.int8) if kind == "integer" else torch.zeros(8, 64, dtype=torch.uint8)
    scale = torch.ones(8) if kind == "integer" else torch.ones(1, 8, dtype=torch.bfloat16)
    return {"_buffers": {"packed_weight": packed, "weight_scale": scale, "bias": None}, "in_features": 128, "out_features": 8,
            "bits": 8, "tactic": 0}


@pytest.mark.parametrize("kind", ["integer", "w4a16"])
def test_anything_but_a_plain_cuda_call_is_left_to_the_general_path(kind):
    call = getattr(_lib.host_calls(), f"{kind}_linear")
    x = torch.zeros(2, 128, dtype=torch.bfloat16)
    assert call(cpu_state(kind), x) is None
    for broken in ({}, {"_buffers": 3}, {"_buffers": {}}, {**cpu_state(kind), "tactic": "0"}, {**cpu_state(kind), "in_features": 1 << 80}):
        assert call(broken, x) is None
    for other in (None, 1, torch.nn.Linear(2, 2), torch.zeros(0, dtype=torch.bfloat16), x.to_sparse(), torch.empty(2, 128, device="meta")):
        assert call(cpu_state(kind), other) is None
    assert call(None, x) is None and call(cpu_state(kind)) is None
    assert torch.func.vmap(lambda t: torch.zeros(()) if call(cpu_state(kind), t) is None else t)(x).shape == (2,)


DEVICE = "cuda:0"


def make(kind, n, k, bias):
    gen = torch.Generator(device=DEVICE).manual_seed(n + k)
    lin = torch.nn.Linear(k, n, bias=bias, device=DEVICE, dtype=torch.bfloat16)
    with torch.no_grad():
        lin.weight.copy_(torch.randn(n, k, generator=gen, device=DEVICE) * 0.02)
    lin.requires_grad_(False)
    return IntegerLinear.from_linear(lin) if kind == "integer" else W4A16Linear.from_linear(lin)


def general(layer, x):
    flat = x.reshape(-1, layer.in_features)
    if isinstance(layer, IntegerLinear):
        p = prepare_activation(flat, 8)
        out = integer_gemm(p.data, p.scales, layer.packed_weight, layer.weight_scale, layer.bias, 8, layer.tactic)
        return out[:, :layer.out_features].reshape(*x.shape[:-1], layer.out_features)
    return linear_w4a16(flat.contiguous(), layer.packed_weight, layer.weight_scale, layer.bias).reshape(*x.shape[:-1], -1)


@pytest.mark.gpu
@pytest.mark.parametrize("kind,n,k,bias", [("integer", 64, 128, True), ("integer", 72, 250, False), ("integer", 70, 384, True),
                                           ("w4a16", 64, 128, True), ("w4a16", 264, 1024, False)])
def test_native_calls_equal_the_general_path(kind, n, k, bias):
    layer = make(kind, n, k, bias)
    call = getattr(_lib.host_calls(), f"{kind}_linear")
    _lib.workspace(torch.device(DEVICE), _lib.WORKSPACE_HEADER)
    wide = torch.randn(6, 50, k + 8, device=DEVICE).bfloat16()
    forms = {"2d": wide[0, :, :k].contiguous(), "3d": wide[..., :k].contiguous(), "row": wide[0, :1, :k].contiguous(),
             "grad": wide[1, :, :k].contiguous().requires_grad_(True), "parameter": torch.nn.Parameter(wide[2, :, :k].contiguous())}
    for name, x in forms.items():
        taken = call(layer.__dict__, x)
        assert (taken is not None) == (n % 8 == 0), name
        out = layer(x)
        assert out.shape == (*x.shape[:-1], n) and out.is_contiguous() and not out.requires_grad
        assert torch.equal(out, general(layer, x.detach())), name
    strided = wide[0, :, :k]  # rows k + 8 apart: the general path
    assert call(layer.__dict__, strided) is None
    assert torch.equal(layer(strided), general(layer, strided))
    x = forms["2d"]
    with torch.device(DEVICE):  # a torch-function mode
        assert call(layer.__dict__, x) is None and torch.equal(layer(x), general(layer, x))
    for bad in (x.float(), x[:, :-1].contiguous(), x.cpu(), x[:0]):
        assert call(layer.__dict__, bad) is None
        with pytest.raises((ValueError, RuntimeError)):
            layer(bad)
    # another stream, whose workspace the general path makes first, and a captured graph
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        first, again = layer(x), layer(x)
    torch.cuda.current_stream().wait_stream(side)
    want = general(layer, x)
    assert torch.equal(first, want) and torch.equal(again, want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        captured = layer(x)
    x.copy_(wide[3, :, :k])
    graph.replay()
    assert torch.equal(captured, general(layer, x))
    layer.packed_weight = layer.packed_weight.clone().zero_()  # a replaced buffer is the one that counts
    assert (layer(x) == (0 if layer.bias is None else layer.bias[:n])).all()


@pytest.mark.gpu
def test_a_call_that_the_gemm_refuses_queues_nothing():
    layer = make("integer", 64, 128, False)
    x = torch.randn(4, 128, device=DEVICE).bfloat16()
    assert layer(x) is not None
    layer.tactic = 9
    count = lambda: torch.cuda.memory_stats(DEVICE)["allocation.all.allocated"]  # the row codes come first
    before = count()
    assert _lib.host_calls().integer_linear(layer.__dict__, x) is None and count() == before
    with pytest.raises(RuntimeError, match="tactic"):
        layer(x)


@pytest.mark.gpu
def test_replaced_methods_stay_in_charge():
    layer = make("integer", 64, 128, False)
    x = torch.randn(4, 128, device=DEVICE).bfloat16()
    want, calls = layer(x), []
    pack = layer.pack_input
    layer.pack_input = lambda t: calls.append(1) or pack(t)
    assert torch.equal(layer(x), want) and calls == [1]

    class Sub(IntegerLinear):
        def pack_input(self, t):
            calls.append(2)
            return super().pack_input(t)

    sub = Sub(layer.packed_weight, layer.weight_scale, layer.bias, 128, 64, 8)
    assert torch.equal(sub(x), want) and calls == [1, 2]


WITHOUT_MODULE = """
import sys, warnings
sys.path.insert(0, {package!r})
sys.modules["rk_b200._host_calls"] = None  # as if the file were missing
import torch
from rk_b200.integer import IntegerLinear
from rk_b200.w4a16_linear import W4A16Linear
x = torch.zeros(2, 128, dtype=torch.bfloat16)
layers = [(IntegerLinear(torch.zeros(8, 128, dtype=torch.int8), torch.ones(8), None, 128, 8, 8), "Expected CUDA BF16 rows"),
          (IntegerLinear(torch.zeros(8, 64, dtype=torch.uint8), torch.ones(8), None, 128, 8, 4), "Expected CUDA BF16 rows"),
          (W4A16Linear(torch.zeros(8, 64, dtype=torch.uint8), torch.ones(1, 8, dtype=torch.bfloat16), None, 128, 8), "requires a contiguous CUDA")]
with warnings.catch_warnings(record=True) as told:
    warnings.simplefilter("always")
    for layer, message in layers * 2:
        try:
            layer(x)
        except ValueError as error:
            assert message in str(error), error
        else:
            raise AssertionError("no error")
assert [w.category for w in told] == [RuntimeWarning] * 2, told  # once for each kind of layer
"""


def test_without_the_native_module_the_general_path_serves_the_call():
    """On the CPU the general path says what it needs."""
    import subprocess
    import sys
    from pathlib import Path

    script = WITHOUT_MODULE.format(package=str(Path(_lib.__file__).resolve().parents[1]))
    done = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
