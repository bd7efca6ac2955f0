"""Operator-level decode attention with the reference's signature
(blockgtq/kernels/fused_packed_attention.py:1541-1861).

The reference specialises its Triton kernel on one head's segment tuple and is
called once per KV head.  This wrapper accepts the same arguments, turns the
segment tuple / codebook / V LUT into a head descriptor (cached) and runs the
CUDA decode + combine kernels.  Callers that hold a whole layer should use
:mod:`blockgtq_b200.layer` directly (one launch for all heads).
"""
from __future__ import annotations

import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from . import _lib
from .layer import HD, DecodePlans, attend, growing_forms, make_decode_plan

_tables = {}          # tables by contents
_cache = {}           # the same by the full description of the tensors they were made of, with these tensors
_recent = {}          # the latest tensors seen at an address, with their tables


class _AdHocLayer(DecodePlans):
    """Minimal stand-in for LayerTables built from operator arguments."""

    def __init__(self, segments, cb, vl, v_bits, n_kv, nopack, device):
        self.n_kv = n_kv
        self.device = device
        self.desc_host = (_lib.HeadDesc * n_kv)()
        for h in range(n_kv):
            d = self.desc_host[h]
            d.n_seg = len(segments)
            d.v_bits = v_bits
            d.nopack_start, d.nopack_len = nopack
            for s, (bw, start, length, pack_off, lut_off, _ni) in enumerate(segments):
                d.seg_bw[s], d.seg_start[s], d.seg_len[s] = bw, start, length
                d.seg_pack_off[s], d.seg_lut_off[s] = pack_off, lut_off
            for i, x in enumerate(cb[:512]):
                d.codebook[i] = int(x)
            for i, x in enumerate(vl[:16]):
                d.v_lut[i] = int(x)
        self.desc_dev = torch.from_numpy(np.frombuffer(self.desc_host, dtype=np.uint8).copy()).to(device)
        self._plans = {}

    def _make_plan(self, flags):
        return make_decode_plan(self.desc_host, self.n_kv, flags, self.device)


def _version(t):
    return None if t.is_inference() else t._version


def _stamp(t):
    """What a tensor holds, as far as that can be known without reading it: where it lies, how, and how often it was
    written in place (inference tensors do not count that)."""
    return t.data_ptr(), t.dtype, t.shape, t.stride(), _version(t)


def _layer_for(segments, codebook_flat, v_lut, v_bits, n_kv, device):
    """The tables made of these arguments, kept from call to call (making them reads the tensors back to the host).  The
    caches keep the tensors they go by alive, so that no other tensor can come to lie at such an address."""
    key = (tuple(map(tuple, segments)), codebook_flat.data_ptr(), v_lut.data_ptr(), v_bits, n_kv, device)
    hit = _recent.get(key)
    if hit is not None:             # the very same tensors as in an earlier call: their versions say the rest
        cb, vl, cb_version, vl_version, lt = hit
        if cb is codebook_flat and vl is v_lut and (cb_version is None or cb_version == cb._version) and \
                (vl_version is None or vl_version == vl._version):
            return lt
    rest = (key[0], v_bits, n_kv, device)
    full = (_stamp(codebook_flat), _stamp(v_lut), rest)
    entry = _cache.get(full)
    if entry is None:
        cb, vl = (t.detach().to(torch.float16).cpu().view(torch.int16).numpy().astype(np.uint16) for t in (codebook_flat, v_lut))
        contents = (cb.tobytes(), vl.tobytes(), rest)
        lt = _tables.get(contents)
        if lt is None:
            segs = tuple(tuple(int(x) for x in s) for s in segments)
            raw = [s for s in segs if s[0] > 4 and s[2] > 0]
            nopack = (min(s[1] for s in raw), sum(s[2] for s in raw)) if raw else (HD, 0)
            lt = _AdHocLayer(segs, cb, vl, v_bits, n_kv, nopack, device)
        if len(_cache) > 4096:
            _tables.clear()
            _cache.clear()
            _recent.clear()
        _tables[contents] = lt
        entry = _cache[full] = (lt, codebook_flat, v_lut)
    lt = entry[0]
    _recent[key] = (codebook_flat, v_lut, _version(codebook_flat), _version(v_lut), lt)
    return lt


@_lib.no_grad
def fused_blockgtq_decode_attention(
        q, k_packed, k_norms, codebook_flat, lut_offset, norm_group, segments,
        v_codes, v_norms, v_lut, scale=None, block_t=64, block_m=16, t_splits=32,
        v_skip_thresh=0.0, v_norm_scale=None, onebit_fast="auto", q_pack_perm=None,
        v_bits=0, v_rotation=None, k_nibble=False, v_nibble=False, v_paired_2b=False,
        k_paired_2b=False, k_paired_4b=False, k_paired_8b=False, k_paired_1b=False,
        return_lse=False):
    """q (B, n_q, 1, 128) fp16 (already rotated for packed K) x packed cache -> (B, n_q, 1, 128) fp16.

    ``t_splits`` is honoured as the number of token splits.  Tile-shape and fast-path
    switches of the Triton kernel (``block_t``, ``block_m``, ``onebit_fast``, ``*_paired_*``,
    ``v_skip_thresh``) select between mathematically equal code paths there and are accepted and
    ignored here.  ``lut_offset`` / ``norm_group`` are unused by the reference kernel as well.
    Raw (unpacked) V codes (``v_bits=0`` without ``v_nibble``) and int4 V norms are not supported."""
    assert q.dim() == 4 and q.shape[2] == 1
    assert len(segments) <= 8
    if v_nibble:
        vb_codebook = int(round(math.log2(v_lut.numel())))
    elif v_bits and v_bits > 0:
        vb_codebook = int(v_bits)
    else:
        raise NotImplementedError("raw uint8 V codes are not supported; pack V (v_bits=1..4) or use v_nibble")
    if v_norms.dtype != torch.float16:
        raise NotImplementedError("int4 V norms are not supported")
    B, n_q, _, D = q.shape
    n_kv, T = k_packed.shape[1], k_packed.shape[2]
    if scale is None:
        scale = 1.0 / math.sqrt(D)
    if q_pack_perm is not None:
        q = q[:, :, :, q_pack_perm]
    if v_norms.dim() == 4:
        v_norms = v_norms[..., 0]
    if k_norms.dtype != torch.float16:
        k_norms = k_norms.to(torch.float16)
    dev, stored = q.device, 4 if v_nibble else vb_codebook
    lt = _layer_for(segments, codebook_flat, v_lut, vb_codebook, n_kv, dev)
    flags = (_lib.DEC_K_MIXED if k_nibble else 0) | (_lib.DEC_V_NIBBLE if v_nibble else 0)
    form, split, short = growing_forms(B, n_kv, T, dev.index, n_q // n_kv, stored)
    if form != split and not (k_packed.is_contiguous() and v_codes.is_contiguous()) and k_packed.stride(-2) + v_codes.stride(-2) > _MERGING_ROW:
        form = split
    if form and flags | form | _lib.DEC_PROGRAMMATIC not in lt._plans:
        form = _make_plans(lt, flags, form, split, short)
    flags |= form
    out, _o32, lse = attend(lt, q, k_packed, k_norms, v_codes, v_norms, 0, T, rotate=False,
                            n_splits=max(1, int(t_splits)), scale=scale, flags=flags, v_rot=_rotation(v_rotation, n_kv),
                            want_lse=return_lse)
    return (out, lse) if return_lse else out


_MERGING_ROW = 192          # bytes a token's packed K and V rows may be apart: the widest there are (padded ones leave the shares no room)


def _capturing(lt) -> bool:
    return lt.device.type == "cuda" and torch.cuda.is_current_stream_capturing()


def _make_plans(lt, flags, form, split, merging):
    """A short context's decode has two forms, each a kernel that takes a second or two to compile: the one that merges its shares
    in the launch, and the split one that takes over as the context grows.  Both are made when the first call needs either,
    side by side, so that a later call, or its capture, finds them.  Returns the form for this call: ``form``, or under a capture
    that it was not made before, the split one."""
    if _capturing(lt):
        return split
    stream = torch.cuda.current_stream(lt.device) if lt.device.type == "cuda" else None

    def make(f):
        with torch.cuda.stream(stream):         # (the caller's: what the plan's image lies in returns to that stream's pool)
            lt.plan(flags | f | _lib.DEC_PROGRAMMATIC)

    with ThreadPoolExecutor(max_workers=2) as ex:
        list(ex.map(make, {split, merging or split}))
    return form


def _rotation(v_rotation, n_kv):
    """The V rotation argument (one matrix for all heads, or one per head) as (n_kv, 128, 128) fp32."""
    if v_rotation is None:
        return None
    rot = v_rotation
    if rot.dtype != torch.float32 or not rot.is_contiguous():
        rot = rot.to(torch.float32).contiguous()
    if rot.dim() == 2 and n_kv > 1:
        rot = rot.unsqueeze(0).expand(n_kv, -1, -1).contiguous()
    return rot


@torch.no_grad()
def fused_blockgtq_prefill_attention(
        q, k_packed, k_norms, codebook_flat, lut_offset, norm_group, segments,
        v_codes, v_norms, v_lut, scale=None, block_q=64, block_t=64, v_skip_thresh=0.0,
        v_norm_scale=None, v_bits=0, v_rotation=None, is_causal=True, q_pos_offset=0,
        k_nibble=False, v_nibble=False, min_seg_for_dot=16):
    """q (B, n_q, S_q, 128) fp16 (already rotated for packed K) x packed cache -> (B, n_q, S_q, 128) fp16
    (blockgtq/kernels/fused_packed_attention.py:2597-2760).  Query i has position ``q_pos_offset + i``
    and, when ``is_causal``, attends cache tokens up to and including it.  ``block_q`` / ``block_t`` /
    ``v_skip_thresh`` / ``min_seg_for_dot`` select tile shapes and equal-valued code paths in the
    Triton kernel and are accepted and ignored; raw V codes and int4 V norms are not supported."""
    from .layer import prefill_attention
    assert q.dim() == 4 and len(segments) <= 8
    if v_nibble:
        vb_codebook = int(round(math.log2(v_lut.numel())))
    elif v_bits and v_bits > 0:
        vb_codebook = int(v_bits)
    else:
        raise NotImplementedError("raw uint8 V codes are not supported; pack V (v_bits=1..4) or use v_nibble")
    if v_norms.dtype != torch.float16:
        raise NotImplementedError("int4 V norms are not supported")
    n_kv, T = k_packed.shape[1], k_packed.shape[2]
    if v_norms.dim() == 4:
        v_norms = v_norms[..., 0]
    lt = _layer_for(segments, codebook_flat, v_lut, vb_codebook, n_kv, q.device)
    flags = (_lib.DEC_K_MIXED if k_nibble else 0) | (_lib.DEC_V_NIBBLE if v_nibble else 0)
    rot = _rotation(v_rotation, n_kv)
    q16 = q.to(torch.float16)
    if q16.stride(3) != 1:
        q16 = q16.contiguous()
    return prefill_attention(lt, q16, k_packed, k_norms.to(torch.float16), v_codes, v_norms, T,
                             q_pos_offset=int(q_pos_offset), causal=bool(is_causal), scale=scale, flags=flags,
                             v_rot=rot)
