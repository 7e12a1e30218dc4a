"""Tyr's typed attention calls, served by the sm_100a kernels.

Names and defaults follow the Lean declarations:
  scaled_dot_product_attention        Tyr/Torch.lean:663-671   (is_causal := true)
  scaledDotProductAttentionGQA        Tyr/Torch.lean:1058-1067 (enable_gqa := false)
  scaledDotProductAttentionGQAQKV     Tyr/Torch.lean:1069-1082
Each is a pure function returning a new tensor, like the `T #[b,h,s,d]` result of
the Lean call.  `attentionFwd` is the launcher-style form (caller may pass the
outputs, LSE returned) and `flashDecode` the ragged single-token decode.

Tensors are torch CUDA tensors; only their data pointers, sizes and strides cross
the C ABI, and the launch goes on torch's current stream, which is what
`torch.cuda_current_stream` returns to Tyr (cc/src/tyr.cpp:4314-4331).
"""
from __future__ import annotations

import ctypes
from typing import Optional, Sequence, Tuple

import torch

from . import _lib
from ._lib import AttnError, PrefillArgs, check


def _stream_ptr(t: torch.Tensor) -> int:
    return torch.cuda.current_stream(t.device).cuda_stream


def _require_cuda(*ts: torch.Tensor) -> None:
    # the launcher checks of Tyr/GPU/Codegen/Attribute.lean:333-336, as exceptions
    for t in ts:
        if not t.is_cuda:
            raise ValueError("tensor must be on a CUDA device")
        if t.dim() > 4:
            raise ValueError("tensor rank must be <= 4")
        if t.stride(-1) != 1:
            raise ValueError("tensor must have unit stride on the head dimension")


def _fill_prefill(q, k, v, o, lse, is_causal, scale, check_mode, window_size=0, key_mask=None) -> PrefillArgs:
    B, Hq, Sq, D = q.shape
    Bk, Hkv, Skv, Dk = k.shape
    if v.shape != k.shape or Bk != B or Dk != D or o.shape != q.shape:
        raise ValueError(f"shape mismatch: q {tuple(q.shape)} k {tuple(k.shape)} v {tuple(v.shape)}")
    if q.dtype != k.dtype or q.dtype != v.dtype or q.dtype != o.dtype:
        raise ValueError("q, k, v and out must share one dtype")
    if q.dtype == torch.bfloat16:
        dtype = _lib.TYR_ATTN_BF16
    elif q.dtype == torch.float32:
        dtype = _lib.TYR_ATTN_F32
    else:
        raise ValueError("dtype must be bfloat16 (float32 in check mode)")
    a = PrefillArgs()
    a.q, a.k, a.v, a.o = q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr()
    a.lse = lse.data_ptr() if lse is not None else None
    a.batch, a.n_head, a.n_kv_head, a.q_seq, a.kv_seq, a.head_dim = B, Hq, Hkv, Sq, Skv, D
    for name, t in (("q_stride", q), ("k_stride", k), ("v_stride", v), ("o_stride", o)):
        getattr(a, name)[:] = [t.stride(0), t.stride(1), t.stride(2)]
    a.dtype, a.is_causal, a.scale, a.check_mode = dtype, int(bool(is_causal)), float(scale or 0.0), int(bool(check_mode))
    a.window_size = int(window_size)
    if key_mask is not None:
        a.key_mask, a.key_mask_stride = key_mask.data_ptr(), key_mask.stride(0)
    else:
        a.key_mask, a.key_mask_stride = None, 0
    return a


def attentionFwd(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, is_causal: bool = True,
                 scale: Optional[float] = None, out: Optional[torch.Tensor] = None,
                 lse: Optional[torch.Tensor] = None, return_lse: bool = True,
                 check_mode: bool = False, window_size: int = 0,
                 key_mask: Optional[torch.Tensor] = None,
                 workspace=None) -> Tuple[torch.Tensor, Optional[torch.Tensor]]:
    """O = softmax(Q K^T * scale + causal) V and the per-row LSE.

    q [B,Hq,Sq,D]; k, v [B,Hkv,Skv,D] (Hq % Hkv == 0, query head h reads KV head
    h // (Hq/Hkv) as repeat_interleave does, cc/src/tyr.cpp:3931-3938).  Strided
    views are accepted (unit inner stride), e.g. the KV-cache slice of
    Tyr/Model/Qwen/Attention.lean:195-196.  `check_mode` runs the fp32-FMA kernel.
    `window_size` > 0 adds the causal sliding window of lean_torch_sdpa_gqa_window
    (cc/src/tyr.cpp:3986-3996): key j is visible to query i only if j <= i and i - j < window_size.
    `key_mask` (uint8 / bool CUDA tensor [batch, kv_seq], 0 = padding key) hides padding keys
    from every query, the key side of lean_torch_sdpa_gqa_mask (cc/src/tyr.cpp:4063-4086).
    Launcher convention of Examples/GPU/RunFlashAttn.lean:68-81: outputs may be
    pre-allocated by the caller and are written in place.
    `workspace`: a caller-kept uint8 CUDA tensor of `prefill_workspace_bytes(...)` bytes for the
    key-split of a half-empty last round, or of long keys under few query rows; when the call would use
    one, it is allocated if none is given (`workspace=False`: one launch without any).
    """
    return _lib.calls().attention_fwd(q, k, v, is_causal, scale, out, lse, return_lse, check_mode, window_size,
                                      key_mask, workspace)


def prefill_workspace_bytes(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, is_causal: bool = True) -> int:
    """Bytes of `workspace` that `attentionFwd` on these tensors would use (0: none)."""
    a = _fill_prefill(q, k, v, q, None, is_causal, None, False)  # only shapes and strides are looked at
    with torch.cuda.device(q.device):
        return max(int(_lib.load().tyr_b200_attn_prefill_workspace_bytes(ctypes.byref(a))), 0)


def attentionBwd(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, o: torch.Tensor, lse: torch.Tensor,
                 d_o: torch.Tensor, is_causal: bool = True, scale: Optional[float] = None,
                 workspace: Optional[torch.Tensor] = None, window_size: int = 0,
                 key_mask: Optional[torch.Tensor] = None
                 ) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """dQ, dK, dV of `attentionFwd` from dO, the forward's inputs, its output and its LSE.

    The gradient LibTorch autograd produces for the typed attention call in the reference
    (`autograd.backward`, Tyr/Torch.lean:742 -> cc/src/tyr.cpp:2111-2122), computed with the
    formulation of Tyr/GPU/Kernels/MhaH100.lean:196-344.  dK and dV of a KV head are summed over
    the query heads that share it.  `workspace` may be a caller-kept float32 CUDA tensor of at
    least `backward_workspace_bytes(...) / 4` elements; one is allocated otherwise.
    `window_size` and `key_mask` are those of the forward call (sliding window / padding keys).
    """
    return _lib.calls().attention_bwd(q, k, v, o, lse, d_o, is_causal, scale, workspace, window_size, key_mask)


def _sdpa(q, k, v, dropout_p, is_causal, enable_gqa):
    if dropout_p != 0.0:
        # the C ABI refuses dropout; a Tyr build keeps its LibTorch call for that case
        raise AttnError(-6)
    if not enable_gqa and q.shape[1] != k.shape[1]:
        raise AttnError(-2)
    out, _ = attentionFwd(q, k, v, is_causal=is_causal, return_lse=False)
    return out


def scaled_dot_product_attention(query, key, value, dropout_p: float = 0.0, is_causal: bool = True):
    """Tyr/Torch.lean:663-671 -> lean_torch_sdpa_4d (cc/src/tyr.cpp:2563-2589)."""
    return _sdpa(query, key, value, dropout_p, is_causal, False)


def scaledDotProductAttentionGQA(query, key, value, dropout_p: float = 0.0, is_causal: bool = True,
                                 enable_gqa: bool = False):
    """Tyr/Torch.lean:1058-1067 -> lean_torch_sdpa_gqa (cc/src/tyr.cpp:3913-3949)."""
    if query.shape[2] != key.shape[2]:
        raise ValueError("scaledDotProductAttentionGQA needs q_seq == kv_seq; use ...GQAQKV")
    return _sdpa(query, key, value, dropout_p, is_causal, enable_gqa)


def scaledDotProductAttentionGQAQKV(query, key, value, dropout_p: float = 0.0, is_causal: bool = True,
                                    enable_gqa: bool = False):
    """Tyr/Torch.lean:1069-1082 -> lean_torch_sdpa_gqa_qkv (cc/src/tyr.cpp:4100-4133)."""
    return _sdpa(query, key, value, dropout_p, is_causal, enable_gqa)


def scaledDotProductAttentionGQAWindow(query, key, value, dropout_p: float = 0.0, is_causal: bool = True,
                                       enable_gqa: bool = False, window_size: int = 1):
    """Tyr/Torch.lean:1084-1101 -> lean_torch_sdpa_gqa_window (cc/src/tyr.cpp:3953-4018).
    As in the reference, the mask is always causal | window whatever `is_causal` says."""
    if dropout_p != 0.0:
        raise AttnError(-6)
    if (not enable_gqa and query.shape[1] != key.shape[1]) or window_size <= 0:
        raise AttnError(-2)
    if query.shape[2] != key.shape[2]:
        raise ValueError("scaledDotProductAttentionGQAWindow needs q_seq == kv_seq")
    out, _ = attentionFwd(query, key, value, is_causal=True, return_lse=False, window_size=window_size)
    return out


def scaledDotProductAttentionGQAMask(query, key, value, attn_mask, dropout_p: float = 0.0,
                                     is_causal: bool = True, enable_gqa: bool = False):
    """Tyr/Torch.lean:1103-1118 -> lean_torch_sdpa_gqa_mask (cc/src/tyr.cpp:4024-4095).
    attn_mask [batch, seq]: non-zero = valid key, 0 = padding (any numeric or bool dtype)."""
    if dropout_p != 0.0:
        raise AttnError(-6)
    if not enable_gqa and query.shape[1] != key.shape[1]:
        raise AttnError(-2)
    if query.shape[2] != key.shape[2]:
        raise ValueError("scaledDotProductAttentionGQAMask needs q_seq == kv_seq")
    # one byte per key for the C ABI, the rows of a batch apart: a byte mask goes as it is, anything else (another type,
    # a mask shared by the batch through `expand`, overlapping rows) as a copy
    km = attn_mask
    if km.dtype not in (torch.bool, torch.uint8) or km.dim() != 2 or km.stride(1) != 1 or km.stride(0) < km.shape[1]:
        km = (km != 0).contiguous()
    out, _ = attentionFwd(query, key, value, is_causal=is_causal, return_lse=False, key_mask=km)
    return out


def sdpa_host(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, is_causal: bool = True,
              out: Optional[torch.Tensor] = None, lse: Optional[torch.Tensor] = None,
              device: int = 0) -> Tuple[torch.Tensor, Optional[torch.Tensor]]:
    """Host-buffer call: q/k/v/out are CPU tensors (pinned for full copy speed)."""
    for t in (q, k, v):
        if t.is_cuda or not t.is_contiguous():
            raise ValueError("sdpa_host takes contiguous CPU tensors")
    if out is None:
        out = torch.empty(q.shape, dtype=q.dtype).pin_memory()
    a = _fill_prefill(q, k, v, out, lse, is_causal, None, False)
    check(_lib.load().tyr_b200_attn_prefill_host(ctypes.byref(a), device))
    return out, lse


class DecodePlan:
    """Device-side description of a ragged KV cache for `flashDecode`.

    Holds the pointer and length arrays and the split-KV workspace so that the
    per-token call allocates nothing.  `k_list[b]`, `v_list[b]` are
    [n_kv_head, len_b, head_dim] bf16 tensors (contiguous or with a head stride).
    """

    def __init__(self, k_list: Sequence[torch.Tensor], v_list: Sequence[torch.Tensor],
                 n_head: int, max_splits: int = 64):
        if len(k_list) == 0 or len(k_list) != len(v_list):
            raise ValueError("need one K and one V tensor per sequence")
        dev = k_list[0].device
        self.device, self.batch, self.n_head = dev, len(k_list), n_head
        self.n_kv_head, _, self.head_dim = k_list[0].shape
        lens, kp, vp, hs = [], [], [], []
        for kt, vt in zip(k_list, v_list):
            _require_cuda(kt, vt)
            if kt.shape != vt.shape or kt.dtype != torch.bfloat16 or kt.stride() != vt.stride():
                raise ValueError("K and V of a sequence must match in shape, stride and be bf16")
            if kt.stride(1) != self.head_dim:
                raise ValueError("keys of one head must be contiguous rows")
            # the kernel reads rows with 16-byte copies straight from these pointers
            if kt.data_ptr() % 16 or vt.data_ptr() % 16 or kt.stride(0) % 8:
                raise ValueError("each K/V block must be 16-byte aligned with a head stride that is a multiple of 8")
            if kt.shape[1] < 1:
                raise ValueError("every sequence needs at least one cached key")
            lens.append(kt.shape[1]); kp.append(kt.data_ptr()); vp.append(vt.data_ptr()); hs.append(kt.stride(0))
        self._keep = (list(k_list), list(v_list))
        self.max_kv_seq = max(lens)
        self.lens_host = lens
        self.total_kv_len = int(sum(lens))
        self.kv_lens = torch.tensor(lens, dtype=torch.int32, device=dev)
        self.k_ptrs = torch.tensor(kp, dtype=torch.int64, device=dev)
        self.v_ptrs = torch.tensor(vp, dtype=torch.int64, device=dev)
        self.head_strides = torch.tensor(hs, dtype=torch.int64, device=dev)
        self.max_splits = max_splits
        nbytes = _lib.load().tyr_b200_attn_decode_workspace_bytes(self.batch, n_head, self.head_dim,
                                                                  self.max_kv_seq, max_splits)
        self.workspace = torch.empty(max(nbytes, 16), dtype=torch.uint8, device=dev)
        self.workspace_bytes = nbytes


def _decode_ragged(q, plan: DecodePlan, workspace, scale, out, lse, return_lse):
    """`workspace` None: the library's own array."""
    return _lib.calls().decode_ragged(
        q, plan.batch, plan.n_head, plan.n_kv_head, plan.max_kv_seq, plan.head_dim, plan.max_splits,
        plan.total_kv_len,     # the host built the plan from these lengths: the launch sizes its chunks by their sum
        plan.k_ptrs, plan.v_ptrs, plan.kv_lens, plan.head_strides, workspace, plan.workspace_bytes, scale, out, lse,
        return_lse)


def flashDecode(q: torch.Tensor, plan: DecodePlan, scale: Optional[float] = None,
                out: Optional[torch.Tensor] = None, lse: Optional[torch.Tensor] = None,
                return_lse: bool = True):
    """One query token per sequence over the ragged cache of `plan`.

    q [B, n_head, head_dim] (or [B, n_head, 1, head_dim]) bf16.  Same result as
    scaledDotProductAttentionGQAQKV(q[b:b+1], K_b, V_b, 0.0, false, true) for each b,
    the call QwenAttention.forwardStep makes (Tyr/Model/Qwen/Attention.lean:198-200).
    """
    return _decode_ragged(q, plan, plan.workspace, scale, out, lse, return_lse)


def flashDecodeStatic(q: torch.Tensor, plan: DecodePlan, scale: Optional[float] = None,
                      out: Optional[torch.Tensor] = None, lse: Optional[torch.Tensor] = None):
    """`flashDecode` for callers that may not allocate device memory while decoding.

    Some hosts of this operator cannot call cudaMalloc in their token loop: their
    memory pool already owns the device, or an allocation's device-wide
    synchronisation would stall the loop.  This call goes through
    tyr_b200_attn_decode_static, which keeps the split-KV scratch in a fixed
    16 MiB array inside the library instead of `plan.workspace`, so the library
    allocates nothing; pass `out` and `lse` to keep this wrapper allocation-free too.
    Shapes whose scratch would not fit raise AttnError (size beyond the supported
    maximum).  All calls on one device share that array: keep them on one stream.
    The first call on a device looks the array up and should come before any
    stream capture.
    """
    return _decode_ragged(q, plan, None, scale, out, lse, True)


def flashDecodeDense(q: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor,
                     kv_lens: Optional[torch.Tensor] = None, kv_len: Optional[int] = None,
                     scale: Optional[float] = None, workspace: Optional[torch.Tensor] = None,
                     max_splits: int = 64):
    """Decode over Tyr's dense KVCache layout [batch, n_kv_head, cap, head_dim]
    (Tyr/Model/Qwen/Attention.lean:54-68).  `kv_len` plays the cache's shared `seq`
    counter; `kv_lens` (int32 device tensor) makes it per sequence."""
    return _lib.calls().decode_dense(q, k_cache, v_cache, kv_lens, kv_len, scale, workspace, max_splits)


def qkPrologue(x: torch.Tensor, out: torch.Tensor, norm_weight: Optional[torch.Tensor] = None,
               cos: Optional[torch.Tensor] = None, sin: Optional[torch.Tensor] = None,
               positions: Optional[torch.Tensor] = None, position0: int = 0, eps: float = 1e-6,
               pe: Optional[torch.Tensor] = None, out_at_row0: bool = False):
    """Fused per-head RMSNorm + rotary embedding + [B,S,H,D] -> [B,H,S,D] layout change,
    written into `out` [B,H,cap,D] at rows positions[b] + s (in place: a KV-cache append
    when `out` is the cache).  One pass instead of applyHeadNorm
    (Tyr/Model/Qwen/Attention.lean:73-98), rotary.applyRotaryEmb (Tyr/Torch.lean:1043-1048),
    transpose_for_attention (Tyr/Torch.lean:589-597) and data.sliceScatter
    (Tyr/Model/Qwen/Attention.lean:189-193).  `norm_weight` [D] and `cos`/`sin`
    [max_pos, D/2] are float32 device tensors; `positions` is int32 [B].
    `pe` selects Flux's rotary form instead (flux.applyRope, Tyr/Model/Flux/RoPE.lean:71-96): a
    float32 [B or 1, max_pos, D/2, 2, 2] table of 2x2 matrices applied to interleaved pairs
    (the reference's [B, 1, S, D/2, 2, 2] `pe` with its singleton axis dropped).
    `out_at_row0`: the position selects the rotary row only and the result goes to rows 0..S-1 of
    `out` (the query of a decode step: rotated at each sequence's position, stored as row 0).
    Rows that would fall outside `out` or outside the rotary table are refused here when the
    position is known on the host (position0); with device-side `positions` the kernel skips
    them and sets the out-of-range bit of the device status word.
    """
    _lib.calls().qk_prologue(x, out, norm_weight, cos, sin, positions, position0, eps, pe, out_at_row0)
    return out


def mergePartials(o_a, lse_a, o_b, lse_b):
    """LSE merge of two partial results (Tyr/GPU/Kernels/RingAttn.lean:164-180)."""
    _require_cuda(o_a, o_b, lse_a, lse_b)
    o_a, o_b = o_a.contiguous().float(), o_b.contiguous().float()
    lse_a, lse_b = lse_a.contiguous().float(), lse_b.contiguous().float()
    out, lse = torch.empty_like(o_a), torch.empty_like(lse_a)
    with torch.cuda.device(o_a.device):
        check(_lib.load().tyr_b200_attn_merge(o_a.data_ptr(), lse_a.data_ptr(), o_b.data_ptr(),
                                              lse_b.data_ptr(), out.data_ptr(), lse.data_ptr(),
                                              lse_a.numel(), o_a.shape[-1], _stream_ptr(o_a)))
    return out, lse


def device_status(device: int = 0, clear: bool = True) -> int:
    """Status word written by the kernels' bounded waits (0 = none gave up)."""
    return int(_lib.load().tyr_b200_attn_device_status(device, int(clear)))


def device_check(device: int = 0) -> None:
    """Raise AttnError if a bounded in-kernel wait gave up or a device-side position or length
    was out of range since the last check; clears the status word."""
    check(int(_lib.load().tyr_b200_attn_device_check(device)))


def launch_count() -> int:
    return int(_lib.load().tyr_b200_attn_launch_count())
