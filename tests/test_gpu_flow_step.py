"""`rk_flow_step_tail`: update + final adaptive norm + output projection + Euler step + next input projection.

Reference: the tensor ops of the unfused step with the norm's statistics and both projections in 64 bits.  Bounds: a
normalized value on a bf16 rounding boundary may land on its neighbour (2^-8 of it, times its weight; two of the largest
products cover the handful that can), fp32 sums of n terms are off by at most n * 2^-24 of the sum of magnitudes."""

import pytest
import torch

from rk_b200 import _lib

pytestmark = pytest.mark.gpu
DEVICE = torch.device("cuda:0")


@pytest.mark.parametrize("batch,tokens,k,d,branch,gate,last", [
    (1, 50, 1024, 32, True, True, False),
    (1, 1, 256, 4, False, False, False),
    (1, 148, 1024, 32, True, False, False),  # the last size with a row per CTA
    (1, 149, 1024, 32, True, True, False),   # two rows per CTA, an odd one left
    (2, 148, 512, 12, True, True, True),
    (3, 99, 1024, 32, True, True, False),    # four rows per CTA that straddle batch entries, one left
    (8, 50, 2048, 64, True, True, False),    # the largest sizes
    (8, 50, 1028, 8, True, True, False),     # K not a multiple of the threads' share
])
def test_flow_step_tail_matches_the_tensor_ops(batch, tokens, k, d, branch, gate, last):
    gen = torch.Generator(device=DEVICE).manual_seed(k + d + tokens)
    r = lambda *s, std=1.0: torch.randn(s, generator=gen, device=DEVICE) * std
    rows, eps, dt = batch * tokens, 1e-6, -0.1
    x, y, g = r(rows, k).bfloat16(), r(rows, k).bfloat16(), r(batch, k).bfloat16()
    modulation = r(batch, 3 * k, std=0.1)
    scale, shift = modulation[:, :k], modulation[:, k:2 * k]
    if modulation.stride(0) % 4 or shift.data_ptr() % 16:
        scale, shift = scale.contiguous(), shift.contiguous()
    w_out, b_out, w_in, b_in = r(d, k, std=0.02), r(d, std=0.1), r(k, d, std=0.1), r(k, std=0.1)
    x_t = r(rows, d)
    x_next = torch.empty_like(x_t)
    out = None if last else torch.empty_like(x)
    P = _lib.ptr
    code = _lib.load().rk_flow_step_tail(
        P(x), P(y) if branch else None, P(g) if gate else None, P(scale), P(shift), scale.stride(0), tokens, rows, k, eps,
        P(w_out), P(b_out), d, P(x_t), dt, P(w_in), P(b_in), P(x_next), P(out), _lib.stream_ptr(DEVICE))
    _lib.check(code, "rk_flow_step_tail")
    rep = lambda t: t.repeat_interleave(tokens, 0)
    s = x
    if branch:
        s = x + (y * rep(g) if gate else y)
    sd = s.double()
    inv = torch.rsqrt(sd.square().mean(-1, keepdim=True).float() + eps)
    h = ((s.float() * inv) * (1.0 + rep(scale)) + rep(shift)).bfloat16().double()
    want = x_t.double() + dt * (h @ w_out.double().T + b_out.double())
    products = h[:, None, :].abs() * w_out.double().abs()
    bound = 0.1 * (2 * 2.0 ** -8 * products.amax(-1) + k * 2.0 ** -24 * products.sum(-1)) + 2.0 ** -22 * (want.abs() + x_t.abs())
    assert ((x_next.double() - want).abs() <= bound).all()
    if last:
        return
    tokens_want = x_next.double() @ w_in.double().T + b_in.double()
    magnitude = x_next.double().abs() @ w_in.double().abs().T + b_in.double().abs()
    assert ((out.double() - tokens_want).abs() <= 2.0 ** -8 * tokens_want.abs() + (d + 2) * 2.0 ** -24 * magnitude).all()


def test_flow_step_tail_refuses_bad_arguments():
    lib, t = _lib.load(), torch.zeros(4096, device=DEVICE)
    p = _lib.ptr(t)
    call = lambda **a: lib.rk_flow_step_tail(
        a.get("x", p), None, a.get("gate"), p, p, a.get("stride", 64), a.get("tokens", 2), 4, a.get("k", 64), 1e-6, p, p,
        a.get("d", 4), p, -0.1, p, p, p, p, _lib.stream_ptr(DEVICE))
    assert call(x=None) == _lib.RK_EINVAL
    assert call(gate=p) == _lib.RK_EINVAL
    assert call(tokens=3) == _lib.RK_EINVAL
    assert call(k=62) == _lib.RK_EINVAL
    assert call(stride=60) == _lib.RK_EINVAL
    assert call(d=68) == _lib.RK_EUNSUPPORTED


def test_the_last_step_needs_no_input_projection():
    """Without an output for the next step's tokens the input projection may be null; the result keeps its bits."""
    gen = torch.Generator(device=DEVICE).manual_seed(0)
    r = lambda *s: torch.randn(s, generator=gen, device=DEVICE)
    x, modulation, w_out, b_out, x_t, w_in, b_in = r(50, 1024).bfloat16(), r(2, 1024), r(32, 1024), r(32), r(50, 32), r(1024, 32), r(1024)
    P, results = _lib.ptr, []
    for tokens, w, b in ((torch.empty_like(x), w_in, b_in), (None, None, None)):
        x_next = torch.empty_like(x_t)
        code = _lib.load().rk_flow_step_tail(P(x), None, None, P(modulation[0]), P(modulation[1]), 1024, 50, 50, 1024, 1e-6, P(w_out),
                                             P(b_out), 32, P(x_t), -0.1, P(w), P(b), P(x_next), P(tokens), _lib.stream_ptr(DEVICE))
        _lib.check(code, "rk_flow_step_tail")
        results.append(x_next)
    assert torch.equal(*results)


def test_expert_loop_with_the_fused_step_tail_equals_the_stepwise_loop():
    """`ActionExpert.forward` against its own `denoise_step` loop (which a hook keeps in place), with fused norms."""
    from rk_b200.gemma_stack import ActionExpert, GemmaConfig, expert_scope, fuse_norm_quantize
    from rk_b200.optimizations import quantize_linears

    cfg = GemmaConfig(width=256, mlp_dim=512, depth=2, num_heads=4, num_kv_heads=1, head_dim=128, adarms_cond_dim=256)
    expert = ActionExpert(cfg, chunk=50, action_dim=32, steps=3).init_random(1).to(DEVICE).eval()
    gen = torch.Generator(device=DEVICE).manual_seed(3)
    noise = torch.randn(4, 50, 32, generator=gen, device=DEVICE)
    pk, pv = (torch.randn(2, 4, 1, 64, 128, generator=gen, device=DEVICE).bfloat16() for _ in range(2))
    calls = []
    with torch.no_grad(), quantize_linears(expert, "int8", scopes=("expert",), selector=expert_scope, shared_quant=True, grouped=True):
        fuse_norm_quantize(expert.stack)
        assert expert._fused_tail(noise)
        fused = expert(noise, pk, pv)
        handle = expert.action_out_proj.register_forward_hook(lambda *a: calls.append(1))
        assert not expert._fused_tail(noise)
        stepwise = expert(noise, pk, pv)
        handle.remove()
        assert len(calls) == 3
        with torch.enable_grad():
            assert not expert._fused_tail(noise)
        assert torch.equal(expert(noise, pk, pv), fused)
    # a code that moves with the order of a sum is carried through the remaining layers and steps
    assert (fused - stepwise).norm() / stepwise.norm() < 2e-2
