"""Rotation and cache append at the edges of the append's tiles: 32 rows a CTA, four column parts from eight rows on,
heads whose 16-byte vectors do not divide by four, several batch rows and KV heads, strided projections.

The rotation is three bf16 roundings of fp32 operations, which is what the tensor ops below do: results are equal."""

import pytest
import torch

from rk_b200.gemma_stack import rope_cache_update

pytestmark = pytest.mark.gpu
DEVICE = torch.device("cuda:0")


def rotate(x, cos, sin):
    half = x.shape[-1] // 2
    return x * cos + torch.cat((-x[..., half:], x[..., :half]), -1) * sin


@pytest.mark.parametrize("dim", [16, 48, 256, 512])
@pytest.mark.parametrize("tokens", [1, 7, 8, 31, 32, 33, 50, 65])
@pytest.mark.parametrize("token_major", [True, False])
def test_rotation_and_append_at_tile_edges(tokens, dim, token_major):
    b, h, kvh, prefix = 3, 5, 2, 9
    rows, pitch = prefix + tokens + 2, (prefix + tokens + 9) // 8 * 8
    gen = torch.Generator(device=DEVICE).manual_seed(tokens * 1000 + dim)
    draw = lambda *s: torch.randn(*s, generator=gen, device=DEVICE).to(torch.bfloat16)
    qkv = draw(b, tokens, (h + 2 * kvh) * dim + 8)  # rows of the projection, with some columns that belong to nobody
    q, k, v = (qkv[..., lo * dim:hi * dim] for lo, hi in ((0, h), (h, h + kvh), (h + kvh, h + 2 * kvh)))
    cos, sin = draw(b, tokens, dim), draw(b, tokens, dim)
    k_all, v_all = (torch.full((b, kvh, rows, dim), 5.0, dtype=torch.bfloat16, device=DEVICE) for _ in range(2))
    vt_all = torch.full((b, kvh, dim, pitch), 9.0, dtype=torch.bfloat16, device=DEVICE)
    got = rope_cache_update(q, k, v, cos, sin, k_all, v_all, prefix, h, kvh, dim, token_major=token_major, vt_all=vt_all)
    heads = lambda t, n: t.reshape(b, tokens, n, dim).transpose(1, 2)
    want = rotate(heads(q, h), cos[:, None], sin[:, None])
    assert torch.equal(got, want)
    fresh = slice(prefix, prefix + tokens)
    assert torch.equal(k_all[:, :, fresh], rotate(heads(k, kvh), cos[:, None], sin[:, None]))
    assert torch.equal(v_all[:, :, fresh], heads(v, kvh))
    assert torch.equal(vt_all[..., fresh], heads(v, kvh).transpose(-1, -2))
    for cache in (k_all, v_all):  # nothing else was touched
        assert (cache[:, :, :prefix] == 5.0).all() and (cache[:, :, prefix + tokens:] == 5.0).all()
    assert (vt_all[..., :prefix] == 9.0).all() and (vt_all[..., prefix + tokens:] == 9.0).all()
