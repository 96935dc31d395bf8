"""GPU parity of `rk_attention_prefix` (fresh query tokens over a cached key / value prefix) and of
the transposed value cache that `rk_rope_cache_update_vt` maintains for it.

The oracle restates the reference's eager attention (models/pi05/modeling_gemma.py:247-274) with its
rounding points; the kernel follows the same points, so the only freedom is the order of fp32
accumulation inside the two matrix products.  A score that sits on a bf16 rounding boundary may
land on the neighbouring value, which moves one probability by < 1 %: the outputs are compared by
relative Frobenius error (tolerance 5e-3, written below) and by the share of elements that differ by
more than two bf16 steps."""

import numpy as np
import pytest
import torch

from oracle import attention as OA
from rk_b200 import _lib
from rk_b200.gemma_stack import attention_prefix, kv_prefix_fill, rope_cache_update, rope_tables

pytestmark = pytest.mark.gpu
DEVICE = torch.device("cuda:0")
TOL = 5e-3

# (batch, tokens, heads, kv_heads, prefix): the action-expert chunk at full size, key slices that end up
# empty, two KV heads with a ragged token count, one token
CASES = [(8, 50, 8, 1, 816), (2, 10, 8, 1, 70), (3, 33, 4, 2, 267), (1, 1, 8, 1, 300), (2, 128, 2, 2, 128)]


def make_inputs(b, t, h, kvh, prefix, seed):
    gen = torch.Generator().manual_seed(seed)
    d = 256
    kv_len = prefix + t
    pitch = (kv_len + 7) // 8 * 8
    q = torch.randn(b, t, h, d, generator=gen).to(torch.bfloat16)
    k = torch.randn(b, kvh, kv_len, d, generator=gen).to(torch.bfloat16)
    v = torch.randn(b, kvh, kv_len, d, generator=gen).to(torch.bfloat16)
    return q, k, v, kv_len, pitch


@pytest.mark.parametrize("case", CASES)
def test_attention_matches_the_eager_oracle(case):
    b, t, h, kvh, prefix = case
    q, k, v, kv_len, pitch = make_inputs(b, t, h, kvh, prefix, 21)
    rows = kv_len + 5  # the caches may be longer than what is valid
    k_all = torch.full((b, kvh, rows, 256), 3.0, dtype=torch.bfloat16)
    k_all[:, :, :kv_len] = k
    vt_all = torch.zeros((b, kvh, 256, pitch), dtype=torch.bfloat16)
    vt_all[..., :kv_len] = v.transpose(-1, -2)
    out = attention_prefix(q.to(DEVICE), k_all.to(DEVICE), vt_all.to(DEVICE), kv_len)
    ws = _lib.workspace(DEVICE, _lib.WORKSPACE_HEADER)
    assert _lib.read_status(ws) == 0
    want = OA.attention(q.permute(0, 2, 1, 3).float().numpy(), k.float().numpy(), v.float().numpy(), 256 ** -0.5)
    got = out.float().cpu().numpy()
    err = np.linalg.norm(got - want) / np.linalg.norm(want)
    assert err < TOL, f"relative Frobenius error {err}"
    step = np.maximum(np.abs(want), 2.0 ** -10) * 2.0 ** -7  # two bf16 steps
    assert (np.abs(got - want) > step).mean() < 0.01


def test_attention_matches_eager_tensor_ops_on_the_device():
    """The same comparison against the reference's four tensor ops run by torch on the GPU."""
    b, t, h, kvh, prefix = 4, 50, 8, 1, 816
    q, k, v, kv_len, pitch = make_inputs(b, t, h, kvh, prefix, 22)
    qd, kd, vd = q.to(DEVICE), k.to(DEVICE), v.to(DEVICE)
    vt_all = torch.zeros((b, kvh, 256, pitch), dtype=torch.bfloat16, device=DEVICE)
    vt_all[..., :kv_len] = vd.transpose(-1, -2)
    out = attention_prefix(qd, kd.contiguous(), vt_all, kv_len)
    qh = qd.permute(0, 2, 1, 3)
    weights = torch.matmul(qh, kd.expand(-1, h, -1, -1).transpose(2, 3)) * 256 ** -0.5
    weights = torch.nn.functional.softmax(weights, dim=-1, dtype=torch.float32).to(torch.bfloat16)
    want = torch.matmul(weights, vd.expand(-1, h, -1, -1)).transpose(1, 2).reshape(b, t, h * 256)
    err = float((out.float() - want.float()).norm() / want.float().norm())
    assert err < TOL, f"relative Frobenius error {err}"


def test_rope_kernel_maintains_the_transposed_value_cache():
    b, t, h, kvh, d, prefix = 2, 50, 8, 1, 256, 96
    gen = torch.Generator().manual_seed(23)
    width = (h + 2 * kvh) * d
    qkv = torch.randn(b, t, width, generator=gen).to(torch.bfloat16).to(DEVICE)
    q, k, v = qkv[..., :h * d], qkv[..., h * d:(h + kvh) * d], qkv[..., (h + kvh) * d:]
    positions = prefix + torch.arange(t, device=DEVICE)[None].expand(b, -1)
    cos, sin = rope_tables(positions, d, 10000.0, torch.bfloat16)
    rows = prefix + t
    pitch = (rows + 7) // 8 * 8
    k_all = torch.zeros((b, kvh, rows, d), dtype=torch.bfloat16, device=DEVICE)
    v_all = torch.zeros_like(k_all)
    vt_all = torch.full((b, kvh, d, pitch), 9.0, dtype=torch.bfloat16, device=DEVICE)
    k_plain, v_plain = torch.zeros_like(k_all), torch.zeros_like(k_all)
    q_vt = rope_cache_update(q, k, v, cos, sin, k_all, v_all, prefix, h, kvh, d, token_major=True, vt_all=vt_all)
    q_plain = rope_cache_update(q, k, v, cos, sin, k_plain, v_plain, prefix, h, kvh, d, token_major=True)
    assert torch.equal(q_vt, q_plain) and torch.equal(k_all, k_plain) and torch.equal(v_all, v_plain)
    assert torch.equal(vt_all[..., prefix:rows], v_all[:, :, prefix:rows].transpose(-1, -2))
    assert (vt_all[..., :prefix] == 9.0).all() and (vt_all[..., rows:] == 9.0).all()  # nothing else was touched


def test_attention_argument_errors():
    lib = _lib.load()
    ws = _lib.workspace(DEVICE, _lib.WORKSPACE_HEADER)
    t = torch.zeros(4096, dtype=torch.bfloat16, device=DEVICE)
    args = lambda **kw: (_lib.ptr(t), _lib.ptr(t), _lib.ptr(t), _lib.ptr(t), kw.get("batch", 1), kw.get("tokens", 4), 8, 1,
                         kw.get("dim", 256), 64, kw.get("pitch", 64), kw.get("kv_len", 64), 0.0625, _lib.ptr(ws), ws.numel(),
                         _lib.stream_ptr(DEVICE))
    assert lib.rk_attention_prefix(*args(dim=128)) == _lib.RK_EUNSUPPORTED
    assert lib.rk_attention_prefix(*args(tokens=200)) == _lib.RK_EINVAL
    assert lib.rk_attention_prefix(*args(kv_len=65)) == _lib.RK_EINVAL
    assert lib.rk_attention_prefix(*args(pitch=60)) == _lib.RK_EINVAL


@pytest.mark.parametrize("batch,prefix", [(1, 718), (1, 719), (3, 719), (4, 718), (4, 719), (5, 40)])
def test_attention_with_any_number_of_key_slices(batch, prefix):
    """Four slices up to 768 keys, eight above if that many clusters run at once (16 tiles of eight slices do not), slices
    without keys: one exchange of (maximum, sum) pairs, with a score range that makes the pairs differ widely."""
    q, k, v, kv_len, pitch = make_inputs(batch, 50, 8, 1, prefix, 23)
    k[:, :, ::7] *= 6.0  # slices and threads with very different maxima
    vt_all = torch.zeros((batch, 1, 256, pitch), dtype=torch.bfloat16)
    vt_all[..., :kv_len] = v.transpose(-1, -2)
    got = attention_prefix(q.to(DEVICE), k.to(DEVICE), vt_all.to(DEVICE), kv_len).float().cpu().numpy()
    want = OA.attention(q.permute(0, 2, 1, 3).float().numpy(), k.float().numpy(), v.float().numpy(), 256 ** -0.5)
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < TOL
    assert _lib.read_status(_lib.workspace(DEVICE, _lib.WORKSPACE_HEADER)) == 0


@pytest.mark.parametrize("batch", [1, 5])
@pytest.mark.parametrize("case", ["two shares", "last key", "every key"])
def test_attention_where_a_share_of_the_keys_weighs_nothing(case, batch):
    """Scores of -infinity and near the type's lowest value.  "two shares": with 613 keys in four slices of 160, one thread's
    keys (alternate chunks of 32 in a slice) all at -infinity, another's at -3e38.  "last key": 385 keys are slices of 128 and
    the last holds one key, at -infinity.  Such keys weigh zero and every row stays finite; a row of -infinities is NaN, as
    in the tensor ops."""
    prefix, scaling = (335, 256 ** -0.5) if case == "last key" else (563, 1.0)
    q, k, v, kv_len, pitch = make_inputs(batch, 50, 8, 1, prefix, 24)
    q *= 0.0625
    q[..., 0] = 1.0
    if case == "two shares":
        for chunk in (160 + 32, 160 + 96):
            k[:, :, chunk:chunk + 32, 0] = float("-inf")
        for chunk in (320, 320 + 64, 320 + 128):
            k[:, :, chunk:chunk + 32, 0] = -3e38
    elif case == "last key":
        k[:, :, kv_len - 1, 0] = float("-inf")
    else:
        k[..., 0] = float("-inf")
    vt_all = torch.zeros((batch, 1, 256, pitch), dtype=torch.bfloat16)
    vt_all[..., :kv_len] = v.transpose(-1, -2)
    got = attention_prefix(q.to(DEVICE), k.to(DEVICE), vt_all.to(DEVICE), kv_len, scaling).float().cpu().numpy()
    assert _lib.read_status(_lib.workspace(DEVICE, _lib.WORKSPACE_HEADER)) == 0
    if case == "every key":
        assert np.isnan(got).all()
        return
    want = OA.attention(q.permute(0, 2, 1, 3).float().numpy(), k.float().numpy(), v.float().numpy(), scaling)
    assert np.isfinite(got).all() and np.linalg.norm(got - want) / np.linalg.norm(want) < TOL


@pytest.mark.parametrize("batch,tokens,prefix,scaling", [
    (5, 52, 561, 0.0625),   # 104 rows, 160 keys in four slices: the last size whose outputs travel by bulk copies
    (5, 53, 560, 0.0625),   # 106 rows: fetched from the peers
    (5, 50, 718, 0.0625),   # 192 keys a slice, the last by bulk copies
    (5, 50, 719, 0.0625),   # 224 keys
    (10, 50, 250, 0.0625),  # two slices
    (1, 50, 816, 0.07),     # eight slices; a scale that is no power of two takes the general conversions
    (3, 64, 200, 0.0625),   # exactly 64 rows of one head
    (20, 50, 100, 0.07),    # whole rows, nothing exchanged
])
def test_attention_at_the_edges_of_its_forms(batch, tokens, prefix, scaling):
    q, k, v, kv_len, pitch = make_inputs(batch, tokens, 8, 1, prefix, 25)
    vt_all = torch.zeros((batch, 1, 256, pitch), dtype=torch.bfloat16)
    vt_all[..., :kv_len] = v.transpose(-1, -2)
    qd, kd, vd = q.to(DEVICE), k.to(DEVICE), vt_all.to(DEVICE)
    first = attention_prefix(qd, kd, vd, kv_len, scaling)
    again = attention_prefix(qd, kd, vd, kv_len, scaling)
    assert _lib.read_status(_lib.workspace(DEVICE, _lib.WORKSPACE_HEADER)) == 0
    assert torch.equal(first, again)  # fixed summation order
    want = OA.attention(q.permute(0, 2, 1, 3).float().numpy(), k.float().numpy(), v.float().numpy(), scaling)
    got = first.float().cpu().numpy()
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < TOL


@pytest.mark.parametrize("case", [
    (1, 50, 8, 1, 1450), (2, 50, 8, 1, 1450),  # eight slices: half-filled tiles only where their clusters run at once
    (8, 10, 8, 1, 1490), (2, 64, 8, 1, 1984),
    (8, 50, 8, 1, 206), (4, 50, 8, 1, 14), (8, 64, 8, 1, 1),  # two slices in place of four short ones
    (1, 50, 8, 1, 206), (3, 100, 8, 1, 156), (16, 10, 8, 1, 246),
])
def test_slices_by_keys_and_clusters(case):
    test_attention_matches_the_eager_oracle(case)


@pytest.mark.parametrize("prefix,chunk", [(1, 50), (64, 50), (70, 3), (127, 1), (128, 8), (563, 50)])
def test_prefix_fill_copies_and_transposes(prefix, chunk):
    """Whole and ragged tiles of 64 rows, a pitch that ends inside or beyond the last tile; nothing else is written."""
    gen = torch.Generator(device=DEVICE).manual_seed(prefix)
    k, v = (torch.randn(2, 3, 1, prefix, 256, generator=gen, device=DEVICE).bfloat16() for _ in range(2))
    pitch = (prefix + chunk + 7) // 8 * 8
    k_all, v_all = (torch.full((2, 3, 1, prefix + chunk, 256), 7.0, dtype=torch.bfloat16, device=DEVICE) for _ in range(2))
    vt_all = torch.full((2, 3, 1, 256, pitch), 7.0, dtype=torch.bfloat16, device=DEVICE)
    assert kv_prefix_fill(k, v, k_all, v_all, vt_all)
    assert torch.equal(k_all[:, :, :, :prefix], k) and torch.equal(v_all[:, :, :, :prefix], v)
    assert (k_all[:, :, :, prefix:] == 7.0).all() and (v_all[:, :, :, prefix:] == 7.0).all()
    assert torch.equal(vt_all[..., :prefix], v.transpose(-1, -2)) and (vt_all[..., prefix:] == 0.0).all()
    assert not kv_prefix_fill(k.transpose(0, 1), v, k_all, v_all, vt_all)
    assert not kv_prefix_fill(k.float(), v, k_all, v_all, vt_all)
