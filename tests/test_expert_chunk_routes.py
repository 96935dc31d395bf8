"""Calls of the action expert that its fused kernels do not take keep going through the tensor ops."""

import pytest
import torch

from rk_b200.gemma_stack import ActionExpert, GemmaAttention, GemmaConfig, kv_prefix_fill

BF16 = torch.bfloat16


@pytest.mark.parametrize("batch", [1, 2, 3])
def test_prefix_fill_leaves_a_broadcast_prefix_to_the_tensor_ops(batch):
    """One prefix for several environments (or any other pair of shapes that only broadcasting joins)."""
    prefix = torch.zeros(2, batch, 1, 8, 256, dtype=BF16)
    caches = torch.zeros(2, 2, 4, 1, 16, 256, dtype=BF16)
    assert not kv_prefix_fill(prefix, prefix, caches[0], caches[1], torch.zeros(2, 4, 1, 256, 16, dtype=BF16))


DEVICE = torch.device("cuda:0")


def small_expert(head_dim, steps=3):
    cfg = GemmaConfig(width=256, mlp_dim=512, depth=2, num_heads=2, num_kv_heads=1, head_dim=head_dim, adarms_cond_dim=256)
    return ActionExpert(cfg, chunk=50, action_dim=32, steps=steps).init_random(1).to(DEVICE).eval()


def draws(head_dim, noise_batch, prefix_batch, tokens=70):
    gen = torch.Generator(device=DEVICE).manual_seed(7)
    r = lambda *s: torch.randn(s, generator=gen, device=DEVICE)
    return r(noise_batch, 50, 32), *(r(2, prefix_batch, 1, tokens, head_dim).to(BF16) for _ in range(2))


@pytest.mark.gpu
def test_one_prefix_for_several_environments(monkeypatch):
    monkeypatch.setattr(GemmaAttention, "fused_rope", True)
    monkeypatch.setattr(GemmaAttention, "fused_attention", True)
    expert = small_expert(256)
    noise, pk, pv = draws(256, 3, 1)
    with torch.no_grad():
        shared = expert(noise, pk, pv)
        copied = expert(noise, *(t.expand(2, 3, 1, 70, 256).contiguous() for t in (pk, pv)))
    assert torch.equal(shared, copied)


def fused_step_expert():
    """An expert whose steps take the fused tail (its norms are fused with the int8 quantizers), and what undoes that."""
    from rk_b200.gemma_stack import expert_scope, fuse_norm_quantize
    from rk_b200.optimizations import quantize_linears

    expert = small_expert(128)
    context = quantize_linears(expert, "int8", scopes=("expert",), selector=expert_scope, shared_quant=True, grouped=True)
    context.__enter__()
    fuse_norm_quantize(expert.stack)
    return expert, lambda: context.__exit__(None, None, None)


def stepwise(expert, *inputs):
    """The same call with a hook in place, which keeps every step in tensor ops."""
    handle = expert.action_out_proj.register_forward_hook(lambda *a: None)
    try:
        assert not expert._fused_tail(inputs[0])
        return expert(*inputs)
    finally:
        handle.remove()


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["action_in_proj", "action_out_proj"])
def test_weights_at_any_address(name):
    """A projection whose weight is a view into a flat buffer, four bytes off."""
    expert, undo = fused_step_expert()
    inputs = draws(128, 2, 2)
    with torch.no_grad():
        assert expert._fused_tail(inputs[0])
        linear = getattr(expert, name)
        flat = torch.empty(linear.weight.numel() + 1, device=DEVICE)[1:].view_as(linear.weight)
        linear.weight.data = flat.copy_(linear.weight)
        assert linear.weight.data_ptr() % 16 and not expert._fused_tail(inputs[0])
        assert torch.equal(expert(*inputs), stepwise(expert, *inputs))
    undo()


@pytest.mark.gpu
@pytest.mark.parametrize("cached", [False, True])
def test_autocast_and_projections_cached_under_it(cached):
    """Under autocast the projections and the modulation are bf16; a projection cache filled there keeps such rows."""
    expert, undo = fused_step_expert()
    inputs = draws(128, 2, 2)
    with torch.no_grad():
        if cached:
            expert.enable_condition_caches()
        with torch.autocast("cuda", torch.bfloat16):
            assert not expert._fused_tail(inputs[0])
            assert torch.equal(expert(*inputs), stepwise(expert, *inputs))
        assert expert._fused_tail(inputs[0])
        if cached:  # bf16 rows from the cache: refused tensor by tensor
            assert expert.stack.norm.projection_cache(expert.condition(torch.ones(2, device=DEVICE), 0))[0].dtype == BF16
            assert torch.equal(expert(*inputs), stepwise(expert, *inputs))
    undo()


@pytest.mark.parametrize("odd", ["scale_type", "scale_batch", "gate_batch", "stream_type", "branch_width", "x_type", None])
def test_step_tail_leaves_other_tensors_to_the_tensor_ops(odd, monkeypatch):
    """On the CPU: what the kernel does not take is refused before the library is called; what it takes reaches the library."""
    from rk_b200 import _lib

    cfg = GemmaConfig(width=64, mlp_dim=128, depth=1, num_heads=2, num_kv_heads=1, head_dim=32, adarms_cond_dim=64)
    expert = ActionExpert(cfg, chunk=6, action_dim=8, steps=3).init_random(1).eval()
    t = lambda *s, dtype=BF16: torch.zeros(s, dtype=dtype)
    scale = t(1 if odd == "scale_batch" else 2, 1, 64, dtype=BF16 if odd == "scale_type" else torch.float32)
    monkeypatch.setattr(expert.stack.norm, "modulation", lambda cond: (scale, t(2, 1, 64, dtype=torch.float32), None))
    stream = t(2, 6, 64, dtype=torch.float32 if odd == "stream_type" else BF16)
    pending = (t(2, 6, 32 if odd == "branch_width" else 64), t(1 if odd == "gate_batch" else 2, 1, 64))
    reached = []
    monkeypatch.setattr(_lib, "load", lambda: reached.append(1) or (_ for _ in ()).throw(RuntimeError("reached")))
    monkeypatch.setattr(torch.cuda, "device", lambda device: torch.no_grad())
    call = lambda: expert._flow_step_tail(stream, pending, None, t(2, 6, 8, dtype=torch.float64 if odd == "x_type" else torch.float32), -0.1, False)
    if odd is None:
        with pytest.raises(RuntimeError, match="reached"):
            call()
        assert reached
    else:
        assert call() is None and not reached


class CountDispatch(torch.utils._python_dispatch.TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.seen = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.seen.append(func)
        return func(*args, **(kwargs or {}))


class CountFunction(torch.overrides.TorchFunctionMode):
    def __init__(self):
        super().__init__()
        self.seen = []

    def __torch_function__(self, func, types, args=(), kwargs=None):
        self.seen.append(func)
        return func(*args, **(kwargs or {}))


@pytest.mark.parametrize("mode", [CountDispatch, CountFunction])
def test_prefix_fill_leaves_modes_to_the_tensor_ops(mode):
    prefix, caches = torch.zeros(2, 4, 1, 8, 256, dtype=BF16), torch.zeros(2, 2, 4, 1, 16, 256, dtype=BF16)
    with mode():
        assert not kv_prefix_fill(prefix, prefix, caches[0], caches[1], torch.zeros(2, 4, 1, 256, 16, dtype=BF16))


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [CountDispatch, CountFunction])
def test_modes_see_every_step(mode):
    expert, undo = fused_step_expert()
    inputs = draws(128, 2, 2)
    with torch.no_grad():
        with mode() as active:
            assert not expert._fused_tail(inputs[0])
            out = expert(*inputs)
        linears = [f for f in active.seen if f in (torch.ops.aten.addmm.default, torch.nn.functional.linear)]
        assert len(linears) >= 2 * 3  # both projections of three steps
        assert torch.equal(out, stepwise(expert, *inputs))
        with torch.device(DEVICE):  # a default device is no reason
            assert expert._fused_tail(inputs[0])
    undo()
