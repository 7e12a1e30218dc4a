"""The cuts of the decode kernel's keys (cluster merge, one chunk, workspace) and the few-row typed call, against the oracle."""
import numpy as np
import pytest
import torch

from conftest import LSE_REL, O_MAX_ABS
from oracle import c_oracle
from tyr_b200 import _lib, nn as tnn

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def randn(*shape, seed=0):
    g = torch.Generator(device="cpu").manual_seed(seed)
    return torch.randn(*shape, generator=g).bfloat16()


def check(o, lse, q, k, v):
    ro, rl = c_oracle.sdpa(q.float().numpy(), k.float().numpy(), v.float().numpy(), False)
    assert np.abs(o.float().cpu().numpy() - ro).max() <= O_MAX_ABS
    if lse is not None:
        assert (np.abs(lse.cpu().numpy() - rl) / np.maximum(np.abs(rl), 1.0)).max() <= LSE_REL


@pytest.fixture(autouse=True)
def _status_clean():
    yield
    assert tnn.device_status(0, True) == 0


# clusters of 16, 8, 7, 5, 2 CTAs, CTAs without keys, one chunk per sequence (8 and 4 warps), more than 8 query rows per
# KV head, and the workspace form next to them
@pytest.mark.parametrize("B,Hq,Hkv,L", [(1, 8, 2, 1), (1, 8, 2, 65), (1, 8, 8, 1025), (4, 8, 8, 515), (4, 36, 9, 700), (3, 16, 16, 640),
                                        (7, 16, 16, 131), (9, 16, 16, 90), (20, 16, 16, 77), (1, 40, 2, 300), (2, 24, 2, 2000),
                                        (1, 4, 1, 20000), (3, 48, 48, 1100)])
@pytest.mark.parametrize("D", [64, 128])
def test_dense_decode(B, Hq, Hkv, L, D):
    q, k, v = randn(B, Hq, 1, D, seed=L), randn(B, Hkv, L, D, seed=L + 1), randn(B, Hkv, L, D, seed=L + 2)
    o, lse = tnn.flashDecodeDense(q.to(DEV), k.to(DEV), v.to(DEV))
    check(o[:, :, None], lse[:, :, None], q, k, v)
    o = tnn.scaledDotProductAttentionGQAQKV(q.to(DEV), k.to(DEV), v.to(DEV), 0.0, False, True)
    check(o, None, q, k, v)


@pytest.mark.parametrize("D", [64, 128])
def test_clusters_over_ragged_lengths(D):
    # lengths on the device: some CTAs of a short sequence's cluster find no keys
    lens, cap = [1, 16, 17, 200, 513, 900], 900
    k, v, q = randn(6, 4, cap, D, seed=1), randn(6, 4, cap, D, seed=2), randn(6, 16, 1, D, seed=3)
    for b, n in enumerate(lens):
        k[b, :, n:] = float("nan")
        v[b, :, n:] = float("nan")
    dl = torch.tensor(lens, dtype=torch.int32, device=DEV)
    o, lse = tnn.flashDecodeDense(q.to(DEV), k.to(DEV), v.to(DEV), kv_lens=dl)
    for b, n in enumerate(lens):
        check(o[b:b + 1, :, None], lse[b:b + 1, :, None], q[b:b + 1], k[b:b + 1, :, :n], v[b:b + 1, :, :n])


# group * q_seq at and around the 8-column tiles and the limit of 16 rows; 17 rows go to the tensor-core kernel
@pytest.mark.parametrize("Hq,Hkv,Sq", [(2, 2, 7), (2, 2, 8), (2, 2, 9), (4, 2, 8), (2, 2, 16), (2, 2, 17), (6, 2, 5)])
@pytest.mark.parametrize("workspace", [None, False])
def test_few_query_rows(Hq, Hkv, Sq, workspace):
    D, L = 128, 1500
    q, k, v = randn(2, Sq, Hq, D, seed=Sq).transpose(1, 2), randn(2, Hkv, L, D, seed=5), randn(2, Hkv, L, D, seed=6)
    buf = torch.full((2, Sq, Hq, D), 7.0, dtype=torch.bfloat16, device=DEV)     # [B,S,H,D] storage on both sides
    o, lse = tnn.attentionFwd(q.to(DEV), k.to(DEV), v.to(DEV), is_causal=False, out=buf.transpose(1, 2), workspace=workspace)
    check(o, lse, q, k, v)


# calls that no workspace helps: more (sequence, KV head) pairs than one wave of CTAs has slots, long keys without a workspace
# or with one that is too small; the output starts as a value that no attention over these V gives
@pytest.mark.parametrize("B,Hq,Hkv,L,D,workspace", [
    (40, 32, 8, 1100, 128, None), (13, 24, 24, 1500, 128, None), (25, 12, 12, 3000, 64, None), (50, 6, 6, 2049, 64, None),
    (1, 32, 8, 20000, 128, False), (4, 24, 24, 2000, 128, False), (17, 32, 8, 2051, 128, False), (4, 24, 24, 2000, 128, "small")])
def test_typed_call_without_a_usable_workspace(B, Hq, Hkv, L, D, workspace):
    q, k, v = randn(B, Hq, 1, D, seed=L), randn(B, Hkv, L, D, seed=L + 1), randn(B, Hkv, L, D, seed=L + 2)
    dev = [t.to(DEV) for t in (q, k, v)]
    out = torch.full((B, Hq, 1, D), 77.0, dtype=torch.bfloat16, device=DEV)
    if workspace == "small":
        assert tnn.prefill_workspace_bytes(*dev, is_causal=False) > 256
        workspace = torch.empty(256, dtype=torch.uint8, device=DEV)
    n0 = tnn.launch_count()
    o, lse = tnn.attentionFwd(*dev, is_causal=False, out=out, workspace=workspace)
    assert tnn.launch_count() - n0 == 1
    rows = sorted({0, B // 2, B - 1})     # the oracle's share
    check(o[rows], lse[rows], q[rows], k[rows], v[rows])
    raw = torch.full_like(out, 77.0)      # the C entry that mirrors the reference's extern: it has no workspace argument
    _lib.check(_lib.load().tyr_b200_sdpa_gqa_qkv(B, Hq, Hkv, 1, L, D, *(t.data_ptr() for t in dev), raw.data_ptr(), 0.0, 0, 1,
                                                 torch.cuda.current_stream().cuda_stream))
    check(raw[rows], None, q[rows], k[rows], v[rows])
    assert not (o == 77.0).any() and not (raw == 77.0).any()


# Keys whose score is -inf (a K row with -inf where the query has a positive entry), as many as a warp's 16, a tile's 64, a
# CTA's and a chunk's share of the keys and a KV tile of 128, at the start, in the middle and at the end: such keys have no
# weight, however they are cut.  Cluster (640 keys, 5 pairs), one chunk (700 pairs), workspace (24 and 2 pairs, long).
@pytest.mark.parametrize("B,Hq,Hkv,L", [(1, 10, 5, 640), (100, 7, 7, 300), (1, 24, 24, 9000), (1, 4, 2, 20000)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dense", [False, True])
def test_scores_of_minus_infinity(B, Hq, Hkv, L, D, dense):
    q, k, v = randn(B, Hq, 1, D, seed=L), randn(B, Hkv, L, D, seed=L + 1), randn(B, Hkv, L, D, seed=L + 2)
    q[..., 0] = 1.0
    hidden = torch.zeros(L, dtype=torch.bool)
    for at, n in ((0, 128), (144, 16), (192, 64), (L // 2, L // 5), (L - 40, 40)):
        hidden[at:at + n] = True
    seen = (~hidden).nonzero()[:, 0]
    k[:, :, hidden, 0] = -torch.inf
    if dense:
        o, lse = tnn.flashDecodeDense(q.to(DEV), k.to(DEV), v.to(DEV))
        o, lse = o[:, :, None], lse[:, :, None]
    else:
        o, lse = tnn.attentionFwd(q.to(DEV), k.to(DEV), v.to(DEV), is_causal=False)
    rows = [0, B - 1]
    check(o[rows], lse[rows], q[rows], k[rows][:, :, seen], v[rows][:, :, seen])
    assert not o.isnan().any()
    # no key at all: NaN, as from ATen
    k[..., 0] = -torch.inf
    o, _ = tnn.attentionFwd(q.to(DEV), k.to(DEV), v.to(DEV), is_causal=False)
    assert o.isnan().all()
