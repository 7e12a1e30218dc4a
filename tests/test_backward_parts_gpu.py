"""Backward launches whose key blocks are shared by clusters of CTAs, and gradients written over an input, against the
oracle."""
import numpy as np
import pytest
import torch

from oracle import c_oracle
from tyr_b200 import _lib, nn as tnn

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
GRAD_REL = 2e-2     # of the largest entry: the bound of the suite's other gradient tests


def randn(*shape, seed=0):
    g = torch.Generator(device="cpu").manual_seed(seed)
    return torch.randn(*shape, generator=g).bfloat16()


@pytest.fixture(autouse=True)
def _status_clean():
    yield
    assert tnn.device_status(0, True) == 0


# 8, 4 and 2 CTAs a key block on 148 SMs, parts without a pair (fewer pairs than CTAs), keys that no query sees, tails of
# one row, a window, a padding mask, more units than one wave
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Skv,causal,window,masked", [
    (1, 4, 1, 1000, 1000, True, 0, False), (1, 16, 8, 513, 513, True, 0, False), (1, 32, 8, 512, 512, False, 0, False),
    (2, 12, 12, 900, 900, True, 0, False), (1, 2, 2, 129, 1500, True, 0, False), (1, 8, 2, 200, 700, False, 0, False),
    (1, 8, 2, 1500, 1500, True, 200, False), (2, 8, 4, 600, 600, True, 0, True), (1, 40, 20, 1300, 1300, True, 0, False)])
@pytest.mark.parametrize("D", [64, 128])
def test_few_units(B, Hq, Hkv, Sq, Skv, causal, window, masked, D):
    q, d_o = randn(B, Hq, Sq, D, seed=Sq), randn(B, Hq, Sq, D, seed=Sq + 1)
    k, v = randn(B, Hkv, Skv, D, seed=Skv + 2), randn(B, Hkv, Skv, D, seed=Skv + 3)
    m = None
    if masked:
        m = torch.ones(B, Skv, dtype=torch.uint8)
        m[1, Skv // 3:] = 0
    dev = [t.to(DEV) for t in (q, k, v)]
    kw = dict(is_causal=causal, window_size=window, key_mask=None if m is None else m.to(DEV))
    o, lse = tnn.attentionFwd(*dev, **kw)
    got = tnn.attentionBwd(*dev, o, lse, d_o.to(DEV), **kw)
    want = c_oracle.sdpa_backward(*(t.float().numpy() for t in (q, k, v, d_o)), causal, window=window,
                                  key_mask=None if m is None else m.numpy())
    for g, w in zip(got, want):
        assert np.abs(g.float().cpu().numpy() - w).max() <= GRAD_REL * np.abs(w).max()
    again = tnn.attentionBwd(*dev, o, lse, d_o.to(DEV), **kw)
    assert all(torch.equal(x, y) for x, y in zip(got, again))      # no atomics: the same bits every time


@pytest.mark.parametrize("over", ["q", "d_o"])
def test_dq_written_over_an_input(over):
    # the dK/dV kernel still reads Q and dO when the dQ kernel could start: a caller that gives their memory for dQ gets
    # the gradients of a call with separate outputs
    import ctypes
    B, H, S, D = 3, 8, 700, 128
    q, k, v, d_o = (randn(B, H, S, D, seed=s).to(DEV) for s in (1, 2, 3, 4))
    o, lse = tnn.attentionFwd(q, k, v)
    want = tnn.attentionBwd(q, k, v, o, lse, d_o)
    lib = _lib.load()
    for _ in range(5):
        t = {"q": q.clone(), "k": k, "v": v, "o": o, "d_o": d_o.clone()}
        d_k, d_v = torch.empty_like(k), torch.empty_like(v)
        ws = torch.empty(lib.tyr_b200_attn_backward_workspace_bytes(B, H, S) // 4, device=DEV)
        a = _lib.BackwardArgs()
        for name, x in list(t.items()) + [("lse", lse), ("d_q", t[over]), ("d_k", d_k), ("d_v", d_v), ("workspace", ws)]:
            setattr(a, name, x.data_ptr())
        a.batch, a.n_head, a.n_kv_head, a.q_seq, a.kv_seq, a.head_dim = B, H, H, S, S, D
        for name in ("q", "k", "v", "o", "do", "dq", "dk", "dv"):
            getattr(a, name + "_stride")[:] = [H * S * D, S * D, D]
        a.dtype, a.is_causal, a.scale, a.workspace_bytes = _lib.TYR_ATTN_BF16, 1, 0.0, ws.numel() * 4
        _lib.check(lib.tyr_b200_attn_backward(ctypes.byref(a), torch.cuda.current_stream().cuda_stream))
        assert all(torch.equal(x, y) for x, y in zip((t[over], d_k, d_v), want))


@pytest.mark.parametrize("B,H,S", [(1, 4, 700), (4, 12, 1500)])     # clusters of the dK/dV kernel, and one CTA a unit
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("D", [64, 128])
def test_steps_on_one_workspace(B, H, S, masked, D):
    # a training loop: row statistics and mask change from step to step at the same addresses, and the dQ kernel runs next
    # to the dK/dV kernel; every step has the bits of a call of its own
    q, k, v = (randn(B, H, S, D, seed=s).to(DEV) for s in (1, 2, 3))
    d_o = [randn(B, H, S, D, seed=10 + i).to(DEV) * (1 + i) for i in range(6)]
    masks = [None] * 6
    if masked:
        masks = [(torch.arange(S) < S - 90 * i).to(torch.uint8).expand(B, S).contiguous().to(DEV) for i in range(6)]
    alone = []
    for g, m in zip(d_o, masks):
        o, lse = tnn.attentionFwd(q, k, v, key_mask=m)
        torch.cuda.synchronize()
        alone.append((o, lse) + tnn.attentionBwd(q, k, v, o, lse, g, key_mask=m))
        torch.cuda.synchronize()
    ws = torch.empty(_lib.load().tyr_b200_attn_backward_workspace_bytes(B, H, S) // 4, device=DEV)
    m = None if masks[0] is None else masks[0].clone()
    for _ in range(3):
        got = []
        for i, g in enumerate(d_o):
            if m is not None:
                m.copy_(masks[i])
            got.append(tnn.attentionBwd(q, k, v, alone[i][0], alone[i][1], g, workspace=ws, key_mask=m))
        for x, y in zip(got, alone):
            assert all(torch.equal(a, b) for a, b in zip(x, y[2:]))
