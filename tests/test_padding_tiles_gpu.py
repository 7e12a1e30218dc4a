"""The padding mask's cut of the KV tiles that are visited, against the plain formula in float64."""
import numpy as np
import pytest
import torch

from conftest import LSE_REL, O_MAX_ABS
from tyr_b200 import nn as tnn

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def randn(*shape, seed=0):
    g = torch.Generator(device="cpu").manual_seed(seed)
    return torch.randn(*shape, generator=g).bfloat16()


@pytest.fixture(autouse=True)
def _status_clean():
    yield
    assert tnn.device_status(0, True) == 0


# left and right padding over several KV tiles, a hole of whole tiles, no valid key, one valid key at either end; with 8
# batch rows and 16 heads more than two items per CTA; a group of one head (256 rows an item) and of two (two heads an item)
@pytest.mark.parametrize("Hq,Hkv", [(3, 3), (16, 8)])
@pytest.mark.parametrize("S,window", [(700, 0), (1111, 0), (1111, 300)])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D", [64, 128])
def test_padding_mask_cuts_tiles(Hq, Hkv, S, window, causal, D):
    B = 8
    q, k, v = randn(B, Hq, S, D, seed=S), randn(B, Hkv, S, D, seed=S + 1), randn(B, Hkv, S, D, seed=S + 2)
    m = torch.ones(B, S + 5, dtype=torch.uint8)
    m[0, S // 2:] = 0
    m[1, :S // 2] = 0
    m[2, 100:600] = 0
    m[3] = 0
    m[4, :S - 1] = 0
    m[5, 4:] = 0
    m[6, :300] = 0
    m[6, 430:] = 0
    mask = m[:, 3:S + 3]    # rows of no particular alignment
    o, lse = tnn.attentionFwd(q.to(DEV), k.to(DEV), v.to(DEV), is_causal=causal, window_size=window,
                              key_mask=m.to(DEV)[:, 3:S + 3])
    heads = [0, Hq - 1]     # the reference's share
    kv = [h * Hkv // Hq for h in heads]
    i, j = torch.arange(S)[:, None], torch.arange(S)[None]
    seen = (mask != 0)[:, None, None] & ((j <= i) if causal or window else (j >= 0)) & ((i - j < window) if window else (j >= 0))
    scores = (q[:, heads].double() @ k[:, kv].double().transpose(-1, -2) / D ** 0.5).masked_fill(~seen, -torch.inf)
    ro = (scores.softmax(-1) @ v[:, kv].double()).float().numpy()     # a row without a key: NaN, as from ATen
    rlse = scores.logsumexp(-1).float().numpy()
    o, lse = o[:, heads].float().cpu().numpy(), lse[:, heads].cpu().numpy()
    assert np.array_equal(np.isnan(o), np.isnan(ro))
    assert np.nanmax(np.abs(o - ro)) <= O_MAX_ABS
    some = np.isfinite(rlse)
    assert (np.abs(lse[some] - rlse[some]) / np.maximum(np.abs(rlse[some]), 1.0)).max() <= LSE_REL


# one mask for the whole batch, a window moving over one buffer, a transposed mask, a slice of a wider one: a mask of any
# strides gives the bits of its contiguous copy
@pytest.mark.parametrize("dtype", [torch.bool, torch.uint8, torch.int64, torch.float32])
@pytest.mark.parametrize("causal", [False, True])
def test_masks_of_any_strides(dtype, causal):
    B, H, S, D = 3, 4, 300, 64
    q, k, v = (randn(B, H, S, D, seed=s).to(DEV) for s in (1, 2, 3))
    bits = torch.rand(2000, generator=torch.Generator().manual_seed(4)) < 0.6
    bits[0] = bits[:S] = True       # every causal row has a key
    line = bits.to(DEV).to(dtype)
    wide = line[:B * 400].view(B, 400)
    masks = [line[40:40 + S][None].expand(B, S), line[None, :S].expand(B, -1), line.as_strided((B, S), (7, 1)),
             line[:S * B].view(S, B).t(), wide[:, :S], wide[:1, :S].expand(B, S), line[:2 * S].as_strided((B, S), (0, 2))]
    for m in masks:
        want = tnn.scaledDotProductAttentionGQAMask(q, k, v, m.ne(0).clone(memory_format=torch.contiguous_format), 0.0, causal)
        got = tnn.scaledDotProductAttentionGQAMask(q, k, v, m, 0.0, causal)
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.nan_to_num(), want.nan_to_num())
    with pytest.raises(ValueError):
        tnn.scaledDotProductAttentionGQAMask(q, k, v, line[0], 0.0, causal)
    with pytest.raises(ValueError):
        tnn.scaledDotProductAttentionGQAMask(q, k, v, line[:S], 0.0, causal)


@pytest.mark.parametrize("D", [64, 128])
def test_mask_rewritten_between_calls(D):
    # short masked launches overlap the one before them, which here writes the mask: each call sees its own mask
    B, H, S = 4, 6, 500
    q, k, v = (randn(B, H, S, D, seed=s).to(DEV) for s in (1, 2, 3))
    masks = [(torch.arange(S) < S - 60 * i).to(torch.uint8).expand(B, S).contiguous().to(DEV) for i in range(8)]
    alone = []
    for m in masks:
        alone.append(tnn.attentionFwd(q, k, v, key_mask=m))
        torch.cuda.synchronize()
    m = torch.empty_like(masks[0])
    for _ in range(5):
        got = []
        for x in masks:
            m.copy_(x)
            got.append(tnn.attentionFwd(q, k, v, key_mask=m))
        assert all(torch.equal(a, b) for x, y in zip(got, alone) for a, b in zip(x, y))
