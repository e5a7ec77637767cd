"""Python operator API of the B200 FP4 attention path.

Mirrors the reference's operator interface:

* ``sageattn(q, k, v, tensor_layout, is_causal, sm_scale, return_lse)`` - signature and semantics
  of ``sageattention/core.py:79-157`` (layouts "HND" ``[B,H,N,D]`` / "NHD" ``[B,N,H,D]``, GQA with
  ``Hq % Hkv == 0``, default scale ``D**-0.5``, optional log-sum-exp output);
* ``sageattn3_blackwell(q, k, v, ...)`` - the FP4 operator of
  ``sageattention3_blackwell/sageattn4/api.py:250-288`` without the fork's K-packing steps;
* ``sageattn4_blackwell(q, k, v, ...)`` - the same operator with the K-packing steps (15 tokens -> group
  mean + 15 residuals, ``api.py:122-177,267-274``);
* ``sageattn_varlen(q, k, v, cu_seqlens_q, cu_seqlens_k, ...)`` - ``sageattention/core.py:334-448``.

All tensor work happens in ``libsage3_b200.so`` (hand-written sm_100a CUDA behind a C ABI); this
file only allocates buffers, turns layouts into strides and passes pointers.  There is no
fallback path: without the library, or on a GPU that is not compute capability 10.x, the calls
raise.
"""
from __future__ import annotations

import contextlib
import ctypes as C
import math
import threading
from dataclasses import dataclass
from typing import Optional, Tuple

import torch

from . import _lib

_LOG2E = 1.4426950408889634


_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def _stream_ptr(device) -> int:
    if _raw_stream is not None and device.index is not None:
        return _raw_stream(device.index)                 # without building a Stream object
    return torch.cuda.current_stream(device).cuda_stream


_NOTHING = contextlib.nullcontext()


def _on_device(device):
    """Context in which `device` is the current one; nothing to do where it is already."""
    return _NOTHING if device.index == torch.cuda.current_device() else torch.cuda.device(device)


def _as_bhnd_strides(x: torch.Tensor, tensor_layout: str):
    """(B, H, N, D, stride_b, stride_h, stride_n) of a 4-D tensor in either layout."""
    if x.dim() != 4:
        raise ValueError("expected a 4-D tensor")
    if x.stride(-1) != 1:
        raise ValueError("the last dimension must be contiguous")       # core.py:274-277
    if tensor_layout == "HND":
        B, H, N, D = x.shape
        return B, H, N, D, x.stride(0), x.stride(1), x.stride(2)
    if tensor_layout == "NHD":
        B, N, H, D = x.shape
        return B, H, N, D, x.stride(0), x.stride(2), x.stride(1)
    raise ValueError(f"Unknown tensor layout: {tensor_layout}")


def _tensor_arg(x: torch.Tensor, sb, sh, sn) -> _lib.Tensor:
    return _lib.Tensor(x.data_ptr(), sb, sh, sn)


def _check_device(x: torch.Tensor):
    if not x.is_cuda:
        raise ValueError("sageattention_b200 runs on CUDA tensors only (no CPU path)")
    major, _ = torch.cuda.get_device_capability(x.device)
    if major != 10:
        raise ValueError(f"unsupported GPU: compute capability {torch.cuda.get_device_capability(x.device)}; "
                         "this build targets B200 (sm_100a) only")


def buffer_sizes(B: int, Hq: int, Hkv: int, Nq: int, Nk: int, D: int, per_block_mean: int = 1) -> _lib.Sizes:
    lib = _lib.load()
    z = _lib.Sizes()
    shape = _lib.Shape(B, Hq, Hkv, Nq, Nk, D)
    _lib.check(lib.sage3_buffer_sizes(C.byref(shape), per_block_mean, C.byref(z)), "sage3_buffer_sizes")
    return z


@dataclass
class QuantizedQKV:
    """Device buffers produced by :func:`quantize_qkv` (layouts in ``include/sage3_b200.h``)."""
    shape: Tuple[int, int, int, int, int, int]       # B, Hq, Hkv, Nq, Nk, D
    q_codes: torch.Tensor
    q_sf: torch.Tensor
    k_codes: torch.Tensor
    k_sf: torch.Tensor
    vt_codes: torch.Tensor
    vt_sf: torch.Tensor
    qm: Optional[torch.Tensor]
    km: Optional[torch.Tensor]
    delta_s: Optional[torch.Tensor]
    delta_s_rows: int
    k_lambda: Optional[torch.Tensor] = None          # K-packing mode: fp32 [B,Hkv,Tk*128]
    nk_slots: Optional[int] = None                   # K-packing mode: occupied key slots (<= Nk)
    mean_slot_first: bool = False                    # K-packing mode: the mean slot takes the first token's score


def quantize_qkv(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, tensor_layout: str = "HND",
                 per_block_mean: Optional[bool] = True, smooth_k: bool = True, with_delta_s: bool = True,
                 km: Optional[torch.Tensor] = None, qm_fp32: Optional[torch.Tensor] = None) -> QuantizedQKV:
    """Smoothing + NVFP4 quantisation of Q, K, V in one fused launch.

    Stands in for ``preprocess_qkv`` + ``scale_and_quant_fp4`` / ``_permute`` / ``_transpose`` of
    ``sageattn4/api.py:112-229``.  ``per_block_mean``: True = per-128-token Q mean, False = whole
    sequence Q mean, None = leave Q as is.  ``with_delta_s=False`` skips delta_s.  ``km`` / ``qm_fp32``
    let a caller supply the means (used by the parity tests to separate rounding of the means from
    the quantiser).
    """
    lib = _lib.load()
    _check_device(q)
    for t in (q, k, v):
        if t.dtype != torch.bfloat16:
            raise AssertionError("TODO: support inputs other than bfloat16")     # api.py:257
    B, Hq, Nq, D, qsb, qsh, qsn = _as_bhnd_strides(q, tensor_layout)
    Bk, Hkv, Nk, Dk, ksb, ksh, ksn = _as_bhnd_strides(k, tensor_layout)
    Bv, Hv, Nv, Dv, vsb, vsh, vsn = _as_bhnd_strides(v, tensor_layout)
    if not (B == Bk == Bv and D == Dk == Dv and Hkv == Hv and Nk == Nv):
        raise ValueError("q, k, v shapes do not match")
    pbm = -1 if per_block_mean is None else int(bool(per_block_mean))
    z = buffer_sizes(B, Hq, Hkv, Nq, Nk, D, pbm)
    dev = q.device
    u8 = dict(dtype=torch.uint8, device=dev)
    Tq, Tk = (Nq + 127) // 128, (Nk + 127) // 128
    out = QuantizedQKV(
        shape=(B, Hq, Hkv, Nq, Nk, D),
        q_codes=torch.empty((B, Hq, Tq, 128, D // 2), **u8), q_sf=torch.empty((B, Hq, Tq, D // 64, 512), **u8),
        k_codes=torch.empty((B, Hkv, Tk, 128, D // 2), **u8), k_sf=torch.empty((B, Hkv, Tk, D // 64, 512), **u8),
        vt_codes=torch.empty((B, Hkv, Tk, D, 64), **u8), vt_sf=torch.empty((B, Hkv, Tk, 2, 512), **u8),
        qm=None, km=None, delta_s=None, delta_s_rows=1)
    ds_rows = Tq if pbm == 1 else 1
    if pbm >= 0:
        out.qm = torch.empty((B, Hq, ds_rows, D), dtype=torch.bfloat16, device=dev)
        if with_delta_s:
            out.delta_s = torch.empty((B, Hq, ds_rows, Tk * 128), dtype=torch.bfloat16, device=dev)
            out.delta_s_rows = ds_rows
    if smooth_k:
        out.km = km.contiguous() if km is not None else torch.empty((B, Hkv, D), dtype=torch.bfloat16, device=dev)
    scratch = torch.empty(max(int(z.scratch), 256), **u8)
    a = _lib.QuantArgs()
    a.shape = _lib.Shape(B, Hq, Hkv, Nq, Nk, D)
    a.q, a.k, a.v = _tensor_arg(q, qsb, qsh, qsn), _tensor_arg(k, ksb, ksh, ksn), _tensor_arg(v, vsb, vsh, vsn)
    a.per_block_mean, a.smooth_k = pbm, int(smooth_k)
    a.km_in = out.km.data_ptr() if (smooth_k and km is not None) else None
    if qm_fp32 is not None:
        qm_fp32 = qm_fp32.to(device=dev, dtype=torch.float32).contiguous()
        a.qm_in = qm_fp32.data_ptr()
    a.q_codes, a.q_sf = out.q_codes.data_ptr(), out.q_sf.data_ptr()
    a.k_codes, a.k_sf = out.k_codes.data_ptr(), out.k_sf.data_ptr()
    a.vt_codes, a.vt_sf = out.vt_codes.data_ptr(), out.vt_sf.data_ptr()
    a.qm = out.qm.data_ptr() if out.qm is not None else None
    a.km = out.km.data_ptr() if out.km is not None else None
    a.delta_s = out.delta_s.data_ptr() if out.delta_s is not None else None
    a.scratch, a.scratch_bytes = scratch.data_ptr(), scratch.numel()
    with _on_device(dev):
        _lib.check(lib.sage3_quant_qkv(C.byref(a), _stream_ptr(dev)), "sage3_quant_qkv")
    return out


def fp4_attention(qz: QuantizedQKV, sm_scale: Optional[float] = None, is_causal: bool = False,
                  tensor_layout: str = "HND", return_lse: bool = False, check_status: bool = False,
                  sm_margin: int = 0):
    """Attention on quantised operands (``blockscaled_fp4_attn``, ``sageattn4/api.py:231-243`` ->
    ``mha_fwd``, ``blackwell/api.cpp:258``).  ``sm_margin``: SMs to leave to kernels that run at the same time
    (see :func:`sageattn3_blackwell`)."""
    lib = _lib.load()
    B, Hq, Hkv, Nq, Nk, D = qz.shape
    dev = qz.q_codes.device
    if sm_scale is None:
        sm_scale = D ** -0.5
    if tensor_layout == "HND":
        out = torch.empty((B, Hq, Nq, D), dtype=torch.bfloat16, device=dev)
        osb, osh, osn = out.stride(0), out.stride(1), out.stride(2)
    else:
        out = torch.empty((B, Nq, Hq, D), dtype=torch.bfloat16, device=dev)
        osb, osh, osn = out.stride(0), out.stride(2), out.stride(1)
    lse = torch.empty((B, Hq, Nq), dtype=torch.float32, device=dev) if return_lse else None
    status = torch.empty(1, dtype=torch.int32, device=dev)
    a = _lib.AttnArgs()
    a.shape = _lib.Shape(B, Hq, Hkv, Nq, Nk, D)
    a.q_codes, a.q_sf = qz.q_codes.data_ptr(), qz.q_sf.data_ptr()
    a.k_codes, a.k_sf = qz.k_codes.data_ptr(), qz.k_sf.data_ptr()
    a.vt_codes, a.vt_sf = qz.vt_codes.data_ptr(), qz.vt_sf.data_ptr()
    a.delta_s = qz.delta_s.data_ptr() if qz.delta_s is not None else None
    a.delta_s_rows = qz.delta_s_rows
    a.out, a.out_stride_b, a.out_stride_h, a.out_stride_n = out.data_ptr(), osb, osh, osn
    a.lse = lse.data_ptr() if lse is not None else None
    a.sm_scale, a.is_causal = float(sm_scale), int(bool(is_causal))
    a.device_status = status.data_ptr()
    a.sm_margin = int(sm_margin)
    with _on_device(dev):
        if qz.k_lambda is not None:
            a.shape = _lib.Shape(B, Hq, Hkv, Nq, int(qz.nk_slots), D)
            _lib.check(lib.sage3_attn_fwd_packed(C.byref(a), qz.k_lambda.data_ptr(), int(qz.mean_slot_first),
                                                 _stream_ptr(dev)), "sage3_attn_fwd_packed")
        else:
            _lib.check(lib.sage3_attn_fwd(C.byref(a), _stream_ptr(dev)), "sage3_attn_fwd")
        if check_status:
            _lib.check(lib.sage3_read_device_status(status.data_ptr(), _stream_ptr(dev), None), "attention kernel")
    return (out, lse) if return_lse else out


def pack_kv(k: torch.Tensor, v: torch.Tensor, tensor_layout: str = "HND", smooth_k: bool = True,
            split_first: bool = False):
    """K-packing preprocessing (``quant_pack_k`` / ``quant_pack_v`` and the K centring of
    ``sageattn4/api.py:122-177,184``): every 15 key tokens become 16 slots (FP4-rounded group mean + 15
    residuals), V gets a zero row per mean slot - or, with ``split_first`` (the reference's ``v_trick``), the
    group's first V row split into its FP4 rounding (slot 1) and the remainder (slot 0).  Returns ``(k_packed, v_packed, k_lambda, km)`` with the
    packed tensors in HND ``[B,Hkv,16*ceil(Nk/15),D]`` and ``k_lambda`` fp32 padded to a multiple of 128."""
    lib = _lib.load()
    _check_device(k)
    B, Hkv, Nk, D, ksb, ksh, ksn = _as_bhnd_strides(k, tensor_layout)
    Bv, Hv, Nv, Dv, vsb, vsh, vsn = _as_bhnd_strides(v, tensor_layout)
    if (B, Hkv, Nk, D) != (Bv, Hv, Nv, Dv):
        raise ValueError("k and v shapes do not match")
    dev = k.device
    rows = lib.sage3_packed_rows(Nk)
    kp = torch.empty((B, Hkv, rows, D), dtype=torch.bfloat16, device=dev)
    vp = torch.empty((B, Hkv, rows, D), dtype=torch.bfloat16, device=dev)
    lam = torch.empty((B, Hkv, (rows + 127) // 128 * 128), dtype=torch.float32, device=dev)
    km = torch.empty((B, Hkv, D), dtype=torch.bfloat16, device=dev) if smooth_k else None
    z = buffer_sizes(B, Hkv, Hkv, Nk, Nk, D, 1)
    scratch = torch.empty(max(int(z.scratch), 256), dtype=torch.uint8, device=dev)
    a = _lib.PackArgs()
    a.shape = _lib.Shape(B, Hkv, Hkv, Nk, Nk, D)
    a.k, a.v = _tensor_arg(k, ksb, ksh, ksn), _tensor_arg(v, vsb, vsh, vsn)
    a.smooth_k = int(smooth_k)
    a.km = km.data_ptr() if km is not None else None
    a.k_packed, a.v_packed, a.k_lambda = kp.data_ptr(), vp.data_ptr(), lam.data_ptr()
    a.scratch, a.scratch_bytes = scratch.data_ptr(), scratch.numel()
    a.split_first = int(bool(split_first))
    with _on_device(dev):
        _lib.check(lib.sage3_pack_kv(C.byref(a), _stream_ptr(dev)), "sage3_pack_kv")
    return kp, vp, lam, km


def sageattn4_blackwell(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, tensor_layout: str = "HND",
                        is_causal: bool = False, sm_scale: Optional[float] = None, per_block_mean: bool = True,
                        quant_block: int = 16, v_trick: Optional[bool] = None, attn_mask=None,
                        check_status: bool = False, **kwargs):
    """The fork's K-packing operator (``sageattn4_blackwell``, ``sageattn4/api.py:250-288``): K is centred,
    packed 15 -> 16 (group mean + residuals) and the kernel restores every score as
    ``q.residual + lambda * q.mean``.  ``per_block_mean`` selects the kernel variant as in the reference
    (``fwd_mainloop.cu:878-888``): True = per-128-token Q mean, the mean slot is masked out; False =
    whole-sequence Q mean, the mean slot takes the first token's score.  ``v_trick`` (default
    ``not per_block_mean``, ``api.py:180-181``) selects the split-first V layout.  ``quant_block`` must be 16."""
    if attn_mask is not None:
        raise NotImplementedError("attn_mask is not supported (the reference ignores it, api.py:250)")
    if quant_block != 16:
        raise AssertionError("quant_block must be 16")                                   # api.py:251
    if q.shape[-1] not in (64, 128):
        raise ValueError(f"Unsupported Headdim {q.shape[-1]}")
    if v_trick is None:
        v_trick = not per_block_mean
    if sm_scale is not None:
        sm_scale = float(sm_scale)
    key = ("packed", q.shape, k.shape, v.shape, q.stride(), k.stride(), v.stride(), q.dtype, k.dtype, v.dtype, q.device,
           tensor_layout, bool(is_causal), sm_scale, bool(per_block_mean))
    plan = _plans.get(key)
    if plan is None:
        plan = _keep_plan(key, _make_plan(q, k, v, tensor_layout, is_causal, sm_scale, per_block_mean, True, 0, packed=True))
    dev = plan.device
    out = torch.empty_like(q)
    ws = torch.empty(plan.workspace, dtype=torch.uint8, device=dev)
    status = torch.empty(1, dtype=torch.int32, device=dev) if check_status else None
    with _on_device(dev):
        stream = _stream_ptr(dev)
        st = plan.run(plan.args, int(bool(v_trick)), int(not per_block_mean), q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(),
                      ws.data_ptr(), None if status is None else status.data_ptr(), stream)
        if st:
            _lib.check(st, "sage3_attention_packed_run")
        if check_status:
            _lib.check(_lib.load().sage3_read_device_status(status.data_ptr(), stream, None), "attention kernel")
    return out


def sageattn3_blackwell(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, tensor_layout: str = "HND",
                        is_causal: bool = False, sm_scale: Optional[float] = None, per_block_mean: bool = True,
                        return_lse: bool = False, smooth_k: bool = True, attn_mask=None,
                        check_status: bool = False, sm_margin: int = 0, **kwargs):
    """FP4 attention, drop-in for ``sageattn4_blackwell`` (``sageattn4/api.py:250-288``) with the wider
    argument set of ``sageattn`` (``sageattention/core.py:79-88``).

    q ``[B,Hq,Nq,D]`` ("HND") or ``[B,Nq,Hq,D]`` ("NHD"), k/v likewise with ``Hkv`` heads
    (``Hq % Hkv == 0``), bf16, D <= 128 (head dims other than 64 and 128 are zero-padded to the next of the two,
    ``sageattention/core.py:925-937``).  Returns a tensor shaped like q (and the natural-log LSE ``[B,Hq,Nq]`` of
    ``sm_scale * q.k`` when ``return_lse``; ``-inf`` for rows that see no key).  Causal masking is bottom-right
    aligned when Nq != Nk.

    ``sm_margin`` (no counterpart in the reference): the attention kernel is persistent with one CTA per SM and a
    static work list, so a CTA whose SM is held by another kernel - a collective running beside it on another
    stream - starts late and the whole launch ends late.  With ``sm_margin = m`` it launches on ``SMs - m`` SMs
    only; the result is the same bit for bit.  It is that kernel's: the quantisation kernels, and those that take its
    place for few query rows per head, are many short CTAs which the hardware deals out to whatever SM is free.
    """
    if attn_mask is not None:
        raise NotImplementedError("attn_mask is not supported (the reference ignores it as well)")
    if sm_scale is not None:
        sm_scale = float(sm_scale)
    key = (q.shape, k.shape, v.shape, q.stride(), k.stride(), v.stride(), q.dtype, k.dtype, v.dtype, q.device, tensor_layout,
           bool(is_causal), sm_scale, bool(per_block_mean), bool(smooth_k), sm_margin)
    plan = _plans.get(key)
    if plan is None:
        plan = _keep_plan(key, _make_plan(q, k, v, tensor_layout, is_causal, sm_scale, per_block_mean, smooth_k, sm_margin))
    if plan.pad:
        # head dims that are no multiple of 8 are padded here first, as the reference does (core.py:925-937, :990)
        d_og = q.shape[-1]
        q, k, v = (torch.nn.functional.pad(t, (0, plan.pad)) for t in (q, k, v))
        res = sageattn3_blackwell(q, k, v, tensor_layout=tensor_layout, is_causal=is_causal,
                                  sm_scale=d_og ** -0.5 if sm_scale is None else sm_scale, per_block_mean=per_block_mean,
                                  return_lse=return_lse, smooth_k=smooth_k, check_status=check_status, sm_margin=sm_margin)
        return (res[0][..., :d_og].contiguous(), res[1]) if return_lse else res[..., :d_og].contiguous()
    dev = plan.device
    out = torch.empty_like(q)
    ws = torch.empty(plan.workspace, dtype=torch.uint8, device=dev)
    lse = torch.empty(plan.lse_shape, dtype=torch.float32, device=dev) if return_lse else None
    # the status word has a place in the workspace; it is only kept apart where the caller wants it read back
    status = torch.empty(1, dtype=torch.int32, device=dev) if check_status else None
    with _on_device(dev):
        stream = _stream_ptr(dev)
        st = plan.run(plan.args, q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), None if lse is None else lse.data_ptr(),
                      ws.data_ptr(), None if status is None else status.data_ptr(), stream)
        if st:
            _lib.check(st, "sage3_attention")
        if check_status:
            _lib.check(_lib.load().sage3_read_device_status(status.data_ptr(), stream, None), "attention kernel")
    return (out, lse) if return_lse else out


# What a call with given shapes, strides and options needs, worked out once: the checks, the sizes and the argument
# struct but for its pointers (a call on the smallest problems took 42 us of host time, 15 us of it this).  Read-only
# after it is made, so that threads may share it; no device memory is held.  The oldest plan makes room for a new one: in
# generation every token has another Nk, whose plan serves the layers of one step and must not take the others with it.
_MAX_PLANS = 1024
_plans = {}
_plans_lock = threading.Lock()


def _keep_plan(key, plan):
    with _plans_lock:
        while len(_plans) >= _MAX_PLANS:
            del _plans[next(iter(_plans))]
        _plans[key] = plan
    return plan


class _Plan:
    __slots__ = ("pad", "device", "workspace", "lse_shape", "struct", "args", "run")


def _check_qkv(q, k, v, tensor_layout):
    """The operator's conditions on the tensors but for where they are; their sizes and strides."""
    for t in (q, k, v):
        if t.dtype != torch.bfloat16:
            raise AssertionError("TODO: support inputs other than bfloat16")     # api.py:257
    dims = B, Hq, _, D, _, _, _ = _as_bhnd_strides(q, tensor_layout)
    dims_k = Bk, Hkv, Nk, Dk, _, _, _ = _as_bhnd_strides(k, tensor_layout)
    dims_v = Bv, Hv, Nv, Dv, _, _, _ = _as_bhnd_strides(v, tensor_layout)
    if not (B == Bk == Bv and D == Dk == Dv and Hkv == Hv and Nk == Nv):
        raise ValueError("q, k, v shapes do not match")
    if Hq % Hkv != 0:
        raise ValueError("num_qo_heads must be a multiple of num_kv_heads")
    if D > 128:
        raise ValueError(f"Unsupported head_dim: {D}")                            # core.py:937
    return dims, dims_k, dims_v


def _make_plan(q, k, v, tensor_layout, is_causal, sm_scale, per_block_mean, smooth_k, sm_margin, packed=False) -> _Plan:
    lib = _lib.load()
    _check_device(q)
    ((B, Hq, Nq, D, qsb, qsh, qsn), (_, Hkv, Nk, _, ksb, ksh, ksn),
     (_, _, _, _, vsb, vsh, vsn)) = _check_qkv(q, k, v, tensor_layout)
    # head-dim padding of sageattention/core.py:925-937: below 64 -> 64, between 64 and 128 -> 128, zeros in the
    # extra channels, default scale from the original head dim, output cut back (:990).  The kernels read rows of the
    # original width and take the rest as zero, so nothing is copied - if the width is a multiple of 8 (16-byte
    # loads); other widths are padded before the call.
    p = _Plan()
    Dp = 64 if D <= 64 else 128
    p.pad = 0 if D % 8 == 0 else Dp - D
    if p.pad:
        return p
    pbm = int(bool(per_block_mean))
    _, _, _, _, osb, osh, osn = _as_bhnd_strides(torch.empty_like(q, device="meta"), tensor_layout)
    a = p.struct = _lib.FwdArgs()
    a.shape = _lib.Shape(B, Hq, Hkv, Nq, Nk, Dp)
    a.q, a.k, a.v = _lib.Tensor(None, qsb, qsh, qsn), _lib.Tensor(None, ksb, ksh, ksn), _lib.Tensor(None, vsb, vsh, vsn)
    a.out_stride_b, a.out_stride_h, a.out_stride_n = osb, osh, osn
    a.km_out = None           # the K-mean term of the LSE is put back on the device (q . km in the quantisation kernel)
    a.sm_scale = float(sm_scale) if sm_scale is not None else 0.0
    a.is_causal, a.per_block_mean, a.smooth_k = int(bool(is_causal)), pbm, int(bool(smooth_k))
    size, p.run = ((lib.sage3_attention_packed_workspace, lib.sage3_attention_packed_run) if packed else
                   (lib.sage3_attention_workspace, lib.sage3_attention_run))
    n = C.c_size_t()
    _lib.check(size(C.byref(a.shape), pbm, C.byref(n)), "workspace size")
    workspace = n.value
    a.workspace_bytes = workspace
    a.head_dim = D if D != Dp else 0
    a.sm_margin = int(sm_margin)
    p.args = C.byref(a)
    p.device, p.workspace, p.lse_shape = q.device, workspace, (B, Hq, Nq)
    return p


def sageattn(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, tensor_layout: str = "HND", is_causal: bool = False,
             sm_scale: Optional[float] = None, return_lse: bool = False, **kwargs):
    """Automatic entry point (``sageattention/core.py:79-157``).  The reference picks a kernel family
    by GPU architecture and raises ``ValueError`` for architectures it has no kernel for; this build
    has exactly one family, the FP4 kernels for compute capability 10.x."""
    return sageattn3_blackwell(q, k, v, tensor_layout=tensor_layout, is_causal=is_causal, sm_scale=sm_scale,
                               return_lse=return_lse, **kwargs)


def sageattn_varlen(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, cu_seqlens_q: torch.Tensor,
                    cu_seqlens_k: torch.Tensor, max_seqlen_q: int, max_seqlen_k: int, is_causal: bool = False,
                    sm_scale: Optional[float] = None, smooth_k: bool = True, check_status: bool = False,
                    **kwargs) -> torch.Tensor:
    """Variable-length batch (``sageattention/core.py:334-448``): q ``[sum(len_q), Hq, D]``, k/v
    ``[sum(len_k), Hkv, D]``, ``cu_seqlens_*`` the int32 prefix sums (length batch + 1, on the device).
    One pass over the three kernels for the whole batch (``sage3_attention_varlen``); every sequence is
    smoothed, quantised and attended on its own (K means never mix sequences); sequences without keys give
    zeros.  ``max_seqlen_*`` must bound the longest sequence - they size the workspace."""
    lib = _lib.load()
    if q.dim() != 3 or k.dim() != 3 or v.dim() != 3:
        raise ValueError("varlen tensors must be [tokens, heads, head_dim]")
    _check_device(q)
    for t in (q, k, v):
        if t.dtype != torch.bfloat16:
            raise AssertionError("TODO: support inputs other than bfloat16")
        if t.stride(-1) != 1:
            raise ValueError("the head dimension must be contiguous")
    nseq = cu_seqlens_q.numel() - 1
    if cu_seqlens_k.numel() != nseq + 1 or nseq < 1:
        raise ValueError("cu_seqlens_q and cu_seqlens_k must both have batch + 1 entries")
    if max_seqlen_q <= 0 or max_seqlen_k <= 0:
        raise ValueError("max_seqlen_q and max_seqlen_k must be positive")
    dev = q.device
    cq = cu_seqlens_q.to(device=dev, dtype=torch.int32).contiguous()
    ck = cu_seqlens_k.to(device=dev, dtype=torch.int32).contiguous()
    Hq, D = q.shape[1], q.shape[2]
    Hkv = k.shape[1]
    if Hq % Hkv != 0 or v.shape != k.shape or k.shape[2] != D:
        raise ValueError("q, k, v shapes do not match")
    out = torch.empty_like(q)
    z = buffer_sizes(nseq, Hq, Hkv, int(max_seqlen_q), int(max_seqlen_k), D, 1)
    ws = torch.empty(int(z.workspace), dtype=torch.uint8, device=dev)
    status = torch.empty(1, dtype=torch.int32, device=dev)
    a = _lib.VarlenArgs()
    a.shape = _lib.Shape(nseq, Hq, Hkv, int(max_seqlen_q), int(max_seqlen_k), D)
    a.q, a.k, a.v = q.data_ptr(), k.data_ptr(), v.data_ptr()
    a.q_stride_n, a.q_stride_h = q.stride(0), q.stride(1)
    a.k_stride_n, a.k_stride_h = k.stride(0), k.stride(1)
    a.v_stride_n, a.v_stride_h = v.stride(0), v.stride(1)
    a.cu_seqlens_q, a.cu_seqlens_k = cq.data_ptr(), ck.data_ptr()
    a.out, a.out_stride_n, a.out_stride_h = out.data_ptr(), out.stride(0), out.stride(1)
    a.sm_scale = float(sm_scale) if sm_scale is not None else 0.0
    a.is_causal, a.smooth_k = int(bool(is_causal)), int(bool(smooth_k))
    a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
    a.device_status = status.data_ptr()
    with _on_device(dev):
        _lib.check(lib.sage3_attention_varlen(C.byref(a), _stream_ptr(dev)), "sage3_attention_varlen")
        if check_status:
            _lib.check(lib.sage3_read_device_status(status.data_ptr(), _stream_ptr(dev), None), "attention kernel")
    return out


_host_streams = {}


def _host_piece_bytes(total: int) -> int:
    """How much of q, k, v a piece carries: filling and draining the pipeline costs in proportion to it, the gaps between
    copies and kernels in inverse proportion, so the best size grows with the root of the whole.  Measured best for 25 /
    100 / 201 / 403 MB: 12 / 24 - 36 / 36 / 48 MB; less than 12 MB never paid."""
    return max(12 << 20, int(math.sqrt(total * 6e6)))


def _host_pieces(B: int, Hkv: int, head_bytes: int, head_chunks) -> list:
    """Pieces (first, last + 1 batch entry, first, last + 1 kv head) in which a host tensor goes through the GPU, each
    contiguous in host memory: some heads of one batch entry (a share of one in ``head_chunks`` at least), or some whole
    batch entries.  Several heads at a time ramp up from one head at the start and down to one at the end, so that the first
    kernel starts after a small copy and little is left to copy out after the last."""
    want = _host_piece_bytes(B * Hkv * head_bytes)
    if isinstance(head_chunks, (list, tuple)):
        sizes = [int(n) for n in head_chunks]                    # explicit group sizes (kv heads per group)
        if sum(sizes) != Hkv or min(sizes) < 1:
            raise ValueError(f"head_chunks {sizes} must be positive and add up to the {Hkv} kv heads")
        plan = [sizes] * B
    else:
        entries = want // max(1, Hkv * head_bytes)
        if entries >= 1 or int(head_chunks) <= 1:
            n = max(1, entries)
            return [(b, min(b + n, B), 0, Hkv) for b in range(0, B, n)]
        base = max(1, round(want / head_bytes), -(-Hkv // int(head_chunks)))
        ramp = [n for n in (1, 2, 4) if n < base]
        plan = []
        for b in range(B):
            up, down = (ramp if b == 0 else []), (ramp[::-1] if b == B - 1 else [])
            while sum(up) + sum(down) > Hkv:
                up, down = up[:-1], down[1:]
            left = Hkv - sum(up) - sum(down)
            plan.append(up + [base] * (left // base) + ([left % base] if left % base else []) + down)
    pieces = []
    for b, sizes in enumerate(plan):
        h = 0
        for n in sizes:
            pieces.append((b, b + 1, h, h + n))
            h += n
    return pieces


def sageattn_from_host(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, out: Optional[torch.Tensor] = None,
                       device=None, head_chunks=8, is_causal: bool = False, sm_scale: Optional[float] = None,
                       **kwargs) -> torch.Tensor:
    """Attention on HOST tensors (HND ``[B,H,N,D]`` bf16, ideally pinned): they go through the GPU in pieces of some kv
    heads of a batch entry, or of some whole batch entries where these are small (``head_chunks``: into how many pieces an
    entry is cut at most, not counting smaller ones at the very start and end; or a list: the kv heads per piece), and the host-to-device copy of piece ``i+1`` and the device-to-host
    copy of piece ``i-1`` run on their own streams while piece ``i`` is computed (pieces alternate between two compute
    streams so that their kernels overlap at the seams), so the
    PCIe transfers hide behind the kernels (or the other way round).  Returns the output as a host tensor
    (``out`` if given, else a new pinned tensor).  The work is ordered after the caller's current stream
    and the current stream waits for the last copy, so CUDA events recorded around the call time all of it;
    the host must still synchronise before reading ``out``."""
    if q.is_cuda or k.is_cuda or v.is_cuda:
        raise ValueError("sageattn_from_host takes host tensors; use sageattn for device tensors")
    # what the operator would refuse is refused before any copy is queued
    if kwargs.get("attn_mask") is not None:
        raise NotImplementedError("attn_mask is not supported (the reference ignores it as well)")
    if kwargs.get("return_lse"):
        raise TypeError("sageattn_from_host returns no log-sum-exp")
    (B, Hq, *_), (_, Hkv, *_), _ = _check_qkv(*(torch.empty(t.shape, dtype=t.dtype, device="meta") for t in (q, k, v)), "HND")
    g = Hq // Hkv
    pieces = _host_pieces(B, Hkv, (q.numel() + k.numel() + v.numel()) * q.element_size() // (B * Hkv), head_chunks)
    dev = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    if out is None:
        out = torch.empty_like(q).pin_memory()
    if dev not in _host_streams:
        _host_streams[dev] = tuple(torch.cuda.Stream(dev) for _ in range(4))
    s_in, s_run_a, s_run_b, s_out = streams = _host_streams[dev]
    cur = torch.cuda.current_stream(dev)
    # whole-problem buffers from the current stream's pool: everything below starts after that stream's present end and
    # it waits for everything below, so they need no further bookkeeping
    qd, kd, vd = (torch.empty(t.shape, dtype=t.dtype, device=dev) for t in (q, k, v))
    start = cur.record_event()
    for st in streams:
        st.wait_event(start)
    keep = []
    try:
        for i, (b0, b1, h0, h1) in enumerate(pieces):
            sq, sk = (slice(b0, b1), slice(h0 * g, h1 * g)), (slice(b0, b1), slice(h0, h1))
            with torch.cuda.stream(s_in):
                qd[sq].copy_(q[sq], non_blocking=True)
                kd[sk].copy_(k[sk], non_blocking=True)
                vd[sk].copy_(v[sk], non_blocking=True)
                ev_in = s_in.record_event()
            # the attention kernel is persistent (one CTA per SM): on two streams in turn, the kernels of the next piece
            # fill the SMs that the last, partly filled round of this piece leaves idle
            s_run = s_run_b if i % 2 else s_run_a
            with torch.cuda.stream(s_run):
                s_run.wait_event(ev_in)
                o = sageattn3_blackwell(qd[sq], kd[sk], vd[sk], tensor_layout="HND", is_causal=is_causal, sm_scale=sm_scale, **kwargs)
                keep.append(o)
                ev_run = s_run.record_event()
            with torch.cuda.stream(s_out):
                s_out.wait_event(ev_run)
                out[sq].copy_(o, non_blocking=True)
    finally:
        # nothing of this call may outlive the caller's next operation - also where a piece failed: copies into the buffers,
        # which the current stream's pool is about to get back, are under way then
        for st in streams:
            cur.wait_event(st.record_event())
        # the outputs came from the compute streams' pools: tell the allocator that the current stream orders their reuse
        for o in keep:
            o.record_stream(cur)
    return out
