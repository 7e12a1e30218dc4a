"""Launches with too few items for the SMs, whose CTAs split the keys of 128 query rows over both Q-tile slots, against the
oracle."""
import numpy as np
import pytest
import torch

from conftest import LSE_REL, O_MAX_ABS
from oracle import c_oracle
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


# one KV tile (slot 1 idle), two, an odd and an even number, tails of one row and one key, a second round of items on
# some CTAs (160, 200 and 264 items on 148 SMs), one query row block against several tiles; 4096 rows, which keep the
# plain form (one order of sums from 2048 on)
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Skv,causal", [
    (1, 8, 2, 129, 129, True), (1, 8, 2, 256, 256, True), (1, 4, 4, 385, 385, True), (1, 32, 8, 517, 517, True),
    (1, 25, 5, 1023, 1023, True), (2, 12, 12, 1400, 1400, True), (1, 2, 1, 4096, 4096, True), (1, 8, 8, 300, 300, False),
    (3, 6, 6, 128, 513, False), (2, 16, 8, 40, 640, False), (1, 6, 2, 700, 257, True), (1, 6, 2, 130, 900, True)])
@pytest.mark.parametrize("D", [64, 128])
def test_few_items(B, Hq, Hkv, Sq, Skv, causal, D):
    q, k, v = randn(B, Hq, Sq, D, seed=Sq), randn(B, Hkv, Skv, D, seed=Skv + 1), randn(B, Hkv, Skv, D, seed=Skv + 2)
    q[:, :, ::7] *= 6.0     # rows with a moving maximum: the accumulators are rescaled
    buf = torch.full((B, Sq, Hq, D), 7.0, dtype=torch.bfloat16, device=DEV)     # [B,S,H,D] storage
    o, lse = tnn.attentionFwd(q.to(DEV), k.to(DEV), v.to(DEV), is_causal=causal, out=buf.transpose(1, 2), workspace=False)
    ro, rlse = c_oracle.sdpa(q.float().numpy(), k.float().numpy(), v.float().numpy(), causal)
    assert np.abs(o.float().cpu().numpy() - ro).max() <= O_MAX_ABS
    assert (np.abs(lse.cpu().numpy() - rlse) / np.maximum(np.abs(rlse), 1.0)).max() <= LSE_REL


# windows shorter than a tile, of a few tiles and longer than the prompt: rows to which a slot's tiles show no key
@pytest.mark.parametrize("S,window", [(700, 1), (700, 100), (700, 256), (1023, 300), (1500, 130), (385, 1000)])
@pytest.mark.parametrize("Hq,Hkv", [(16, 4), (5, 5)])
@pytest.mark.parametrize("D", [64, 128])
def test_few_items_under_a_window(S, window, Hq, Hkv, D):
    q, k, v = randn(1, Hq, S, D, seed=S), randn(1, Hkv, S, D, seed=S + 1), randn(1, Hkv, S, D, seed=S + 2)
    o, lse = tnn.attentionFwd(q.to(DEV), k.to(DEV), v.to(DEV), window_size=window)
    ro, rlse = c_oracle.sdpa(q.float().numpy(), k.float().numpy(), v.float().numpy(), True, window=window)
    assert np.abs(o.float().cpu().numpy() - ro).max() <= O_MAX_ABS
    assert (np.abs(lse.cpu().numpy() - rlse) / np.maximum(np.abs(rlse), 1.0)).max() <= LSE_REL


# From 2048 query rows or keys on a batch element of a causal or windowed call has the bits of a call of its own, forward
# and backward, although the launch of the one has too few work items for the SMs and that of the other has not
@pytest.mark.parametrize("Sq,Skv,window", [(2048, 2048, 0), (2100, 2100, 200), (300, 2048, 0), (2048, 300, 0)])
@pytest.mark.parametrize("D", [64, 128])
def test_one_order_of_sums_for_long_calls(Sq, Skv, window, D):
    B, Hq, Hkv = 7, 4, 2
    q, d_o = randn(B, Hq, Sq, D, seed=Sq).to(DEV), randn(B, Hq, Sq, D, seed=Sq + 1).to(DEV)
    k, v = randn(B, Hkv, Skv, D, seed=Skv + 2).to(DEV), randn(B, Hkv, Skv, D, seed=Skv + 3).to(DEV)

    def both(*t):
        o, lse = tnn.attentionFwd(*t[:3], window_size=window)
        return (o, lse) + tnn.attentionBwd(*t[:3], o, lse, t[3], window_size=window)
    whole = both(q, k, v, d_o)
    for b in (0, B - 1):
        one = both(*(t[b:b + 1] for t in (q, k, v, d_o)))
        assert all(torch.equal(x[b:b + 1], y) for x, y in zip(whole, one))
