"""The prologue's cut of a token's heads over CTAs against the formula in float64."""
import pytest
import torch

from tyr_b200 import nn as tnn

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def randn(*shape, seed=0):
    g = torch.Generator(device="cpu").manual_seed(seed)
    return torch.randn(*shape, generator=g).bfloat16()


@pytest.mark.parametrize("H,S", [(1, 1), (3, 1), (5, 33), (32, 1), (13, 40)])
@pytest.mark.parametrize("rotary", ["none", "half", "pairs"])
def test_prologue_head_chunks(H, S, rotary):
    """Heads in several CTAs (a last chunk that is not full), fewer tokens than a warp covers."""
    B, D = 2, 128
    x = randn(B, S, H, D, seed=H + S).to(DEV)
    w = torch.rand(D, generator=torch.Generator().manual_seed(1)).to(DEV) + 0.5
    ang = torch.rand(S, D // 2, generator=torch.Generator().manual_seed(2)).to(DEV) * 6.28
    cos, sin = ang.cos(), ang.sin()
    kw = {"none": {}, "half": {"cos": cos, "sin": sin},
          "pairs": {"pe": torch.stack([cos, -sin, sin, cos], -1).view(1, S, D // 2, 2, 2).contiguous()}}[rotary]
    out = torch.full((B, H, S + 1, D), 9.0, dtype=torch.bfloat16, device=DEV)
    tnn.qkPrologue(x, out, w, **kw)
    y = x.double()
    y = y / torch.sqrt(y.pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    c, s = cos.double()[None, :, None], sin.double()[None, :, None]
    if rotary == "half":
        a, b = y[..., :D // 2], y[..., D // 2:]
        y = torch.cat([a * c - b * s, a * s + b * c], -1)
    elif rotary == "pairs":
        a, b = y[..., 0::2], y[..., 1::2]
        y = torch.stack([a * c - b * s, a * s + b * c], -1).flatten(-2)
    want = y.transpose(1, 2)
    # one bf16 rounding (2^-9 relative) and fp32 arithmetic before it, whose errors scale with the two summands
    err = (out[:, :, :S].double() - want).abs()
    assert (err <= want.abs() * 2.0 ** -8 + 1e-5).all()
    assert (out[:, :, S:] == 9.0).all()


# one CTA for all heads of a token: a group's rows past 48 MB with a last group of few heads, tables past 12 MB; just
# below that, groups.  Either way a head's rows are those of a call on its own four heads, bit for bit
@pytest.mark.parametrize("B,S,H,D", [(8, 8200, 5, 64), (7, 6900, 6, 64), (1, 25000, 8, 128), (1, 24000, 9, 128), (1, 12400, 7, 256)])
def test_heads_of_many_tokens(B, S, H, D):
    g = torch.Generator(device=DEV).manual_seed(H)
    x = torch.randn(B, S, H, D, generator=g, device=DEV, dtype=torch.bfloat16)
    w = torch.rand(D, generator=g, device=DEV) + 0.5
    ang = torch.rand(S, D // 2, generator=g, device=DEV) * 6.28
    cos, sin = ang.cos(), ang.sin()
    out = torch.full((B, H, S, D), 9.0, dtype=torch.bfloat16, device=DEV)
    tnn.qkPrologue(x, out, w, cos, sin)
    for h in range(0, H, 4):
        part = torch.full_like(out[:, h:h + 4], 9.0)
        tnn.qkPrologue(x[:, :, h:h + 4], part, w, cos, sin)
        assert torch.equal(out[:, h:h + 4], part)
    y = x[:, -3:].double()
    y = y / torch.sqrt(y.pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    a, b = y[..., :D // 2], y[..., D // 2:]
    c, s = cos[-3:, None].double(), sin[-3:, None].double()
    want = torch.cat([a * c - b * s, b * c + a * s], -1).transpose(1, 2)
    assert (out[:, :, -3:].double() - want).abs().max().item() <= 2.0 ** -8 * want.abs().max().item() + 1e-3   # one bf16 rounding
