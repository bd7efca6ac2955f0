"""Per-layer device tables and thin operator wrappers over the C ABI.

A :class:`LayerTables` owns, for the KV heads of one layer, the uploaded array
of ``BgtqHeadDesc`` records, the rotation matrices and the cached decode plans.
The functions below take torch tensors, pass raw pointers and strides to
``libbgtq.so`` and return torch tensors; they enqueue on the current stream
and never synchronise.
"""
from __future__ import annotations

import os

import ctypes as C
import functools
import math

import numpy as np
import torch

from . import _lib
from .calib import KHeadTables, VHeadTables, packed_v_bytes

HD = _lib.HD


def _fill_desc(d: _lib.HeadDesc, kt: KHeadTables, vt: VHeadTables):
    if kt.head_dim != HD:
        raise ValueError("the CUDA kernels support head_dim 128 only")
    pm = kt.pack_meta
    d.n_seg = kt.n_groups
    d.k_row_bytes = kt.total_packed_bytes
    d.v_bits = vt.bits
    d.v_row_bytes = vt.packed_bytes
    d.nopack_start, d.nopack_len = pm["nopack_start"], pm["nopack_len"]
    d.k_mixed_bytes = pm["nopack_start"] // 2 + pm["nopack_len"]
    cb16 = kt.codebook_flat.view(torch.int16).numpy().astype(np.uint16)
    for s, (bw, start, length, pack_off, lut_off, _ni) in enumerate(kt.segments):
        d.seg_bw[s], d.seg_start[s], d.seg_len[s] = bw, start, length
        d.seg_pack_off[s], d.seg_lut_off[s] = pack_off, lut_off
        d.lut_off[s] = float(kt.lut_offsets[start])
        d.lut_inv[s] = float(kt.lut_inv_scales[start])
        cents = kt.pos_centroids[start, :1 << bw]
        for i in range(1 << bw):
            d.codebook[lut_off + i] = int(cb16[lut_off + i])
            d.k_cents[lut_off + i] = float(cents[i])
        row = kt.code_lut[s].numpy()
        C.memmove(d.code_lut[s], row.ctypes.data, _lib.N_BINS)
    nc = 1 << vt.bits
    vl16 = vt.lut_f16.view(torch.int16).numpy().astype(np.uint16)
    for i in range(16):
        d.v_cents[i] = float(vt.centroids[i]) if i < nc else 0.0
        d.v_bounds[i] = float(vt.boundaries[i]) if i < nc - 1 else float("inf")
        d.v_lut[i] = int(vl16[i]) if i < nc else 0
    hp = kt.head_perm.numpy().astype(np.uint8)
    go = kt.group_of.numpy().astype(np.uint8)
    C.memmove(d.head_perm, hp.ctypes.data, HD)
    C.memmove(d.group_of, go.ctypes.data, HD)


def make_decode_plan(desc_host, n_kv: int, flags: int, device, row_strides=None):
    """Decode plan of a layer's KV heads with its lookup-table image uploaded to ``device``.
    Returns (plan, image tensor); the caller keeps the image alive as long as the plan is used.
    ``row_strides`` = (packed-K bytes, K-norm values, packed-V bytes, V-norm values) per token fixes them in
    the specialised kernel (launches with other strides or unaligned slices then run the general kernel)."""
    L = _lib.lib()
    p = _lib.DecodePlan()
    _lib.check(L.bgtq_decode_plan(C.byref(desc_host), n_kv, flags, C.byref(p)), "bgtq_decode_plan")
    n = int(L.bgtq_decode_image_bytes(C.byref(p)))
    if n <= 0:
        raise RuntimeError("bgtq_decode_image_bytes failed")
    host = np.zeros(n, dtype=np.uint8)
    _lib.check(L.bgtq_decode_build_image(C.byref(p), C.byref(desc_host), host.ctypes.data, n),
               "bgtq_decode_build_image")
    image = torch.from_numpy(host).to(device)
    _lib.check(L.bgtq_decode_plan_set_image(C.byref(p), image.data_ptr()), "bgtq_decode_plan_set_image")
    if not (flags & _lib.DEC_GENERIC) and not os.environ.get("BGTQ_DEC_NO_JIT") and torch.device(device).type == "cuda":
        if row_strides is not None:
            _lib.check(L.bgtq_decode_plan_set_row_strides(C.byref(p), *[int(x) for x in row_strides]),
                       "bgtq_decode_plan_set_row_strides")
        _specialize(p)
    return p, image


_jit_warned = False


def _specialize(plan):
    """Compile (NVRTC) and attach the decode kernel specialised for the plan's heads.  Without NVRTC the
    plan keeps using the general kernel; a compile or load failure is an error."""
    global _jit_warned
    log = C.create_string_buffer(1 << 16)
    rc = _lib.lib().bgtq_decode_plan_specialize(C.byref(plan), 0, log, len(log))
    if rc == -2:
        if not _jit_warned:
            import warnings
            warnings.warn("NVRTC not found: the packed decode runs its general kernel (" + log.value.decode() + ")")
            _jit_warned = True
        return
    if rc != 0:
        raise RuntimeError("specialising the decode kernel failed:\n" + log.value.decode(errors="replace"))


class DecodePlans:
    """The decode plans of a layer's KV heads, made by ``_make_plan(flags)`` on first use and kept for the layer's life:
    calls pass a plan's address on, and its image is device memory that launches read."""

    def plan_entry(self, flags: int):
        """(plan, image, whether the plan's decode merges its shares).  Threads may make a plan side by side (the compiler
        runs without the interpreter's lock): the first to finish is the one all of them get."""
        e = self._plans.get(flags)
        if e is None:
            p, image = self._make_plan(flags)
            e = self._plans.setdefault(flags, (p, image, _lib.lib().bgtq_decode_plan_cluster(C.byref(p)) > 0))
        return e

    def plan(self, flags: int = 0) -> _lib.DecodePlan:
        return self.plan_entry(flags)[0]


class LayerTables(DecodePlans):
    """Device-resident static tables for the KV heads of one layer."""

    def __init__(self, k_tables, v_tables, device):
        self.n_kv = len(k_tables)
        self.device = torch.device(device)
        self.k_tables, self.v_tables = list(k_tables), list(v_tables)
        self.desc_host = (_lib.HeadDesc * self.n_kv)()
        for h in range(self.n_kv):
            _fill_desc(self.desc_host[h], k_tables[h], v_tables[h])
        raw = np.frombuffer(self.desc_host, dtype=np.uint8).copy()
        self.desc_dev = torch.from_numpy(raw).to(self.device)
        self.rot_k = torch.stack([t.block_rot.T.contiguous() for t in k_tables]).contiguous().to(self.device)
        self.v_rot = torch.stack([t.rotation for t in v_tables]).contiguous().to(self.device)       # R
        self.rot_v = torch.stack([t.rotation.T.contiguous() for t in v_tables]).contiguous().to(self.device)
        self.v_bits = v_tables[0].bits
        self.vpb = packed_v_bytes(HD, self.v_bits)
        self.max_tpb = max(t.total_packed_bytes for t in k_tables)
        self.max_ng = max(t.n_groups for t in k_tables)
        self.max_mixed_bytes = max(t.pack_meta["nopack_start"] // 2 + t.pack_meta["nopack_len"] for t in k_tables)
        self.head_perm = torch.stack([t.head_perm for t in k_tables]).long().to(self.device)   # (n_kv, 128)
        self.addrs = (self.desc_dev.data_ptr(), self.rot_k.data_ptr(), self.rot_v.data_ptr())
        self._plans = {}
        self._partition = None
        self._row_strides = {}
        self._early_fresh = 0

    def _make_plan(self, flags):
        p, image = make_decode_plan(self.desc_host, self.n_kv, flags, self.device,
                                    row_strides=self._row_strides.get(bool(flags & _lib.DEC_K_MIXED)))
        if self._partition is not None:
            _lib.check(_lib.lib().bgtq_decode_plan_set_partition(C.byref(p), self._partition.data_ptr()),
                       "bgtq_decode_plan_set_partition")
        if self._early_fresh:
            _lib.check(_lib.lib().bgtq_decode_plan_set_early_fetch(C.byref(p), self._early_fresh),
                       "bgtq_decode_plan_set_early_fetch")
        return p, image

    def set_row_strides(self, kp_st: int, kn_st: int, vp_st: int, vn_st: int, mixed: bool = False) -> None:
        """Row strides (packed-K bytes, K-norm values, packed-V bytes, V-norm values per token) of the cache
        this layer's decode launches will read, for plans made after this call: their specialised kernel is
        compiled for exactly these (see ``bgtq_decode_plan_set_row_strides``)."""
        self._row_strides[bool(mixed)] = (kp_st, kn_st, vp_st, vn_st)

    def set_early_fetch(self, fresh_rows: int) -> None:
        """Let programmatic decode launches of this layer stream the cache before their dependency wait; the
        caller promises what ``bgtq_decode_plan_set_early_fetch`` asks for (0 turns it off again)."""
        self._early_fresh = int(fresh_rows)
        for p in self._plans.values():
            _lib.check(_lib.lib().bgtq_decode_plan_set_early_fetch(C.byref(p[0]), self._early_fresh),
                       "bgtq_decode_plan_set_early_fetch")

    def set_partition(self, table_dev) -> None:
        """Attach (or, with None, detach) a device copy of a ``decode_partition`` table to this layer's decode
        plans; the kernel uses it for launches it was made for and ignores it otherwise."""
        if table_dev is not None and (table_dev.dtype != torch.int32 or not table_dev.is_contiguous()
                                      or table_dev.device != self.device):
            raise ValueError("partition table must be a contiguous int32 tensor on the layer's device")
        self._partition = table_dev
        ptr = table_dev.data_ptr() if table_dev is not None else None
        for p in self._plans.values():
            _lib.check(_lib.lib().bgtq_decode_plan_set_partition(C.byref(p[0]), ptr), "bgtq_decode_plan_set_partition")


def _strides3(t: torch.Tensor):
    """(batch, head, token) element strides of a (B, H, T, X) tensor with unit last stride."""
    st = t.stride()
    if len(st) != 4 or st[3] != 1:
        raise ValueError(f"expected a (B, H, T, X) tensor with contiguous last dim, got {tuple(t.shape)} strides {st}")
    return st[:3]


def encode(layer: LayerTables, k, v, t0, k_packed, k_norms, v_packed, v_norms, *, flags=0,
           k_codes=None, v_codes=None, pos_dev=None, status=None):
    """Encode ``k``/``v`` (B, n_kv, S, 128) fp16 into rows ``t0 .. t0+S`` of the cache tensors
    ``k_packed`` (B, n_kv, T, bytes) u8, ``k_norms`` (B, n_kv, T, groups) f16|f32,
    ``v_packed`` (B, n_kv, T, bytes) u8 and ``v_norms`` (B, n_kv, T) f16.  Either side may be None.
    Bulk row counts (>= 128 rows) run the tcgen05 / tensor-memory encoder; ``_lib.ENC_NO_TCGEN05`` in ``flags``
    (or the environment variable ``BGTQ_ENC_NO_TCGEN05``) keeps them on the warp-MMA one."""
    if k_codes is None and v_codes is None and pos_dev is None and status is None and type(t0) is int:
        r = _lib.host().encode(*layer.addrs, layer.n_kv, layer.vpb, k, v, t0, k_packed, k_norms, v_packed, v_norms, flags | _no_tcgen05())
        if r is not None:
            _lib.done(r, "bgtq_encode")
            return
    ref = k if k is not None else v
    _lib.require_cuda(ref, "k/v")
    B, H, S, D = ref.shape
    if H != layer.n_kv or D != HD:
        raise ValueError("shape does not match the layer tables")
    kps = kns = vps = vns = ks = vs = (0, 0, 0)
    kp_bytes = kn_count = 1
    if k is not None:
        ks = _strides3(k)
        if k.dtype != torch.float16 or k_packed.dtype != torch.uint8:
            raise TypeError("k must be float16 and k_packed uint8")
        if k_norms.dtype == torch.float16:
            flags |= _lib.ENC_K_NORMS_F16
        elif k_norms.dtype != torch.float32:
            raise TypeError("k_norms must be float16 or float32")
        kps, kns = _strides3(k_packed), _strides3(k_norms)
        if t0 + S > k_packed.shape[2]:
            raise ValueError("cache overflow")
        kp_bytes, kn_count = k_packed.shape[3], k_norms.shape[3]
    else:
        flags |= _lib.ENC_SKIP_K
    if v is not None:
        vs = _strides3(v)
        if v.dtype != torch.float16 or v_packed.dtype != torch.uint8 or v_norms.dtype != torch.float16:
            raise TypeError("v must be float16, v_packed uint8, v_norms float16")
        vps = _strides3(v_packed)
        need = HD // 2 if flags & _lib.ENC_V_NIBBLE else layer.vpb
        if v_packed.shape[3] < need:
            raise ValueError("v_packed rows are too short")
        vns = v_norms.stride()[:3]
    else:
        flags |= _lib.ENC_SKIP_V
    _encode_rows(layer, k, ks, v, vs, B, S, int(t0), k_packed, kps, kp_bytes, k_norms, kns, kn_count, v_packed, vps, v_norms, vns,
                 (k_packed if k is not None else v_packed).shape[2], flags, k_codes, v_codes, pos_dev, status)


def _no_tcgen05() -> int:
    return _lib.ENC_NO_TCGEN05 if os.environ.get("BGTQ_ENC_NO_TCGEN05") else 0


def _encode_rows(layer, k, ks, v, vs, B, S, t0, kp, kps, kp_bytes, kn, kns, kn_count, vp, vps, vn, vns, capacity, flags,
                 k_codes=None, v_codes=None, pos_dev=None, status=None):
    """The library call behind :func:`encode`: tensors with their (batch, head, token) strides, nothing checked."""
    ptr = _lib.ptr
    _lib.check(_lib.lib().bgtq_encode(
        ptr(layer.desc_dev), ptr(layer.rot_k), ptr(layer.rot_v), ptr(k), *ks, ptr(v), *vs, B, layer.n_kv, S, t0,
        ptr(kp), *kps, kp_bytes, ptr(kn), *kns, kn_count, ptr(vp), *vps, ptr(vn), *vns,
        ptr(k_codes), ptr(v_codes), flags | _no_tcgen05(), ptr(pos_dev), capacity, ptr(status),
        _lib.stream_ptr((k if k is not None else v).device)), "bgtq_encode")
    _lib.count_launch()


def rotate_q(layer: LayerTables, q: torch.Tensor, out: torch.Tensor = None) -> torch.Tensor:
    """q (B, n_q, 128) or (B, n_q, 1, 128) fp16 -> (B, n_q, 128) fp16 in the packed-K basis."""
    _lib.require_cuda(q, "q")
    if q.dim() == 4:
        q = q[:, :, 0]
    if q.stride(2) != 1 or q.dtype != torch.float16:
        q = q.contiguous().to(torch.float16)
    B, n_q, _ = q.shape
    if out is None:
        out = torch.empty(B, n_q, HD, dtype=torch.float16, device=q.device)
    _lib.check(_lib.lib().bgtq_rotate_q(_lib.ptr(layer.desc_dev), _lib.ptr(layer.rot_k), _lib.ptr(q),
                                        q.stride(0), q.stride(1), _lib.ptr(out), B, n_q, layer.n_kv,
                                        _lib.stream_ptr(q.device)), "bgtq_rotate_q")
    _lib.count_launch()
    return out


def _transformed(t: torch.Tensor) -> bool:
    """A tensor that torch has to see the operations of: gradients (either mode), vmap and the like, tensor subclasses."""
    return (t.requires_grad and torch.is_grad_enabled()) or type(t) is not torch.Tensor or torch.autograd.forward_ad._current_level >= 0 or \
        torch._C._functorch.peek_interpreter_stack() is not None


def rotate_q_bulk(layer: LayerTables, q: torch.Tensor) -> torch.Tensor:
    """Many positions at once: q (B, n_q, S, 128) -> same shape, fp16, in the packed-K basis (the per-row kernel
    behind :func:`rotate_q` is meant for the handful of rows of a decode step).  fp16 queries on the GPU go through the
    tensor cores; queries of another type, on the CPU, or that torch differentiates or maps over, are rotated in fp32 by torch's
    own operators and rounded once."""
    fast = q.dtype == torch.float16 and q.is_cuda and not _transformed(q)
    if fast:
        r = _lib.host().rotate_rows(layer.desc_dev.data_ptr(), layer.rot_k.data_ptr(), layer.n_kv, q)
        if r is not None:
            return _lib.done(r, "bgtq_rotate_q_rows")
    B, n_q, S, D = q.shape
    if fast:
        st = q.stride()
        if st[3] != 1 or (q.data_ptr() | 2 * (st[0] | st[1] | st[2])) & 15:
            q = q.contiguous()
            if q.data_ptr() & 15:
                q = q.clone()
            st = q.stride()
        out = torch.empty(B, n_q, S, D, dtype=torch.float16, device=q.device)
        if out.numel():
            _lib.check(_lib.lib().bgtq_rotate_q_rows(_lib.ptr(layer.desc_dev), _lib.ptr(layer.rot_k), q.data_ptr(), *st[:3],
                                                     out.data_ptr(), B, n_q, layer.n_kv, S, _lib.stream_ptr(q.device)),
                       "bgtq_rotate_q_rows")
            _lib.count_launch()
        return out
    gqa = n_q // layer.n_kv
    qg = q.reshape(B, layer.n_kv, gqa * S, D).float()
    idx = layer.head_perm.view(1, layer.n_kv, 1, D).expand(B, layer.n_kv, gqa * S, D)
    out = torch.matmul(torch.gather(qg, 3, idx), layer.rot_k.view(1, layer.n_kv, D, D))
    return out.to(torch.float16).view(B, n_q, S, D)


def step_prepare(layer: LayerTables, q, k, v, t0, k_packed, k_norms, v_packed, v_norms, *, q_rot=None,
                 flags=0, pos_dev=None, rope=None, ring=None, status=None):
    """``ring=(k_buf, v_buf, n_sink, window)``: three-region mode (``bgtq_step_prepare_ring``), see bgtq.h.
    Rotate q (B, n_q, [1,] 128) into ``q_rot`` and append one token k/v (B, n_kv, 1, 128) at slot
    ``t0`` (or ``*pos_dev``) of the cache tensors, in one launch.  ``q=None`` skips the rotation.
    ``rope=(cos, sin)``, each fp16 (B, 128) (or (B, 1, 128)): q and k are pre-RoPE and the kernel applies
    the rotary embedding of the step's position first (``bgtq_step_prepare_rope``)."""
    _lib.require_cuda(k, "k")
    B, H, S, D = k.shape
    if S != 1 or H != layer.n_kv or D != HD or v.shape != k.shape:
        raise ValueError("step_prepare appends exactly one token per (batch, KV head)")
    if k.dtype != torch.float16 or v.dtype != torch.float16 or k.stride(3) != 1 or v.stride(3) != 1:
        raise TypeError("k and v must be float16 with contiguous last dim")
    if k_norms.dtype == torch.float16:
        flags |= _lib.ENC_K_NORMS_F16
    n_q = 0
    qa = (0, 0, 0)
    if q is not None:
        if q.dim() == 4:
            q = q[:, :, 0]
        if q.dtype != torch.float16 or q.stride(2) != 1:
            q = q.to(torch.float16).contiguous()
        n_q = q.shape[1]
        if q_rot is None:
            q_rot = torch.empty(B, n_q, HD, dtype=torch.float16, device=k.device)
        qa = (_lib.ptr(q), q.stride(0), q.stride(1))
    kps, kns, vps = _strides3(k_packed), _strides3(k_norms), _strides3(v_packed)
    vns = (v_norms.stride(0), v_norms.stride(1), v_norms.stride(2))
    common = (_lib.ptr(layer.desc_dev), _lib.ptr(layer.rot_k), _lib.ptr(layer.rot_v), *qa,
              _lib.ptr(q_rot) if q is not None else 0, n_q,
              _lib.ptr(k), k.stride(0), k.stride(1), _lib.ptr(v), v.stride(0), v.stride(1), B, H, int(t0),
              _lib.ptr(k_packed), *kps, k_packed.shape[3], _lib.ptr(k_norms), *kns, k_norms.shape[3],
              _lib.ptr(v_packed), *vps, _lib.ptr(v_norms), *vns, flags, _lib.ptr(pos_dev),
              int(k_packed.shape[2]), _lib.ptr(status))
    if ring is not None:
        if rope is not None:
            raise NotImplementedError("fused RoPE and the three-region mode cannot be combined")
        k_buf, v_buf, n_sink, window = ring
        if k_buf.stride(2) != HD or k_buf.stride(3) != 1 or v_buf.stride() != k_buf.stride():
            raise ValueError("buffer tensors must be (B, n_kv, cap, 128) with contiguous token rows")
        _lib.check(_lib.lib().bgtq_step_prepare_ring(*common, _lib.ptr(k_buf), _lib.ptr(v_buf), k_buf.stride(0),
                                                     k_buf.stride(1), int(n_sink), int(window),
                                                     _lib.stream_ptr(k.device)), "bgtq_step_prepare_ring")
    elif rope is not None:
        cos, sin = (t.reshape(B, HD) for t in rope)
        if cos.dtype != torch.float16 or sin.dtype != torch.float16 or cos.stride(1) != 1 or sin.stride(1) != 1 \
                or cos.stride(0) != sin.stride(0):
            raise TypeError("rope tables must be float16 (B, 128) with equal row strides")
        _lib.check(_lib.lib().bgtq_step_prepare_rope(*common, _lib.ptr(cos), _lib.ptr(sin), cos.stride(0),
                                                     _lib.stream_ptr(k.device)), "bgtq_step_prepare_rope")
    else:
        _lib.check(_lib.lib().bgtq_step_prepare(*common, _lib.stream_ptr(k.device)), "bgtq_step_prepare")
    _lib.count_launch()
    return q_rot


def default_splits(n_batch: int, n_kv: int, n_tokens: int) -> int:
    return _lib.lib().bgtq_decode_default_splits(n_batch, n_kv, n_tokens)


def decode_grid_size(n_batch: int, n_kv: int, n_splits: int) -> int:
    """CTAs ``decode`` launches for this shape on the current device."""
    n = _lib.lib().bgtq_decode_grid_size(n_batch, n_kv, n_splits)
    if n < 1:
        _lib.check(n, "bgtq_decode_grid_size")
    return n


def decode_partition(n_batch: int, n_kv: int, n_tokens: int, n_splits: int, n_cta: int = None, out=None):
    """Item-range table (host int32 tensor, ``n_cta + 5`` words) that gives CTAs whose range straddles two
    (batch, head) pairs fewer items; copy it to the device and attach it with ``LayerTables.set_partition``."""
    if n_cta is None:
        n_cta = decode_grid_size(n_batch, n_kv, n_splits)
    if out is None:
        out = torch.empty(n_cta + 5, dtype=torch.int32)
    _lib.check(_lib.lib().bgtq_decode_partition(n_batch, n_kv, n_tokens, n_splits, n_cta, out.data_ptr(), out.numel()),
               "bgtq_decode_partition")
    return out


def decode(layer: LayerTables, q_rot, k_packed, k_norms, v_packed, v_norms, t_begin, t_end, *,
           n_splits=None, scale=None, flags=0, part_o=None, part_lse=None, status=None, pos_dev=None, pos_add=0):
    """Split-KV attention partials over cache rows [t_begin, t_end).

    Returns (part_o (B, n_q, n_splits, 128) f32, part_lse (B, n_q, n_splits) f32); slots that hold no
    partial have ``part_lse = -inf`` and an undefined ``part_o`` row (see ``bgtq_decode``)."""
    _lib.require_cuda(q_rot, "q_rot")
    B, n_q, _ = q_rot.shape
    if not q_rot.is_contiguous() or q_rot.dtype != torch.float16:
        raise ValueError("q_rot must be contiguous float16 (B, n_q, 128)")
    if k_norms.dtype != torch.float16 or v_norms.dtype != torch.float16:
        raise TypeError("cache norms must be float16")
    n_tok = t_end - t_begin
    if n_splits is None:
        n_splits = default_splits(B, layer.n_kv, n_tok)
    if scale is None:
        scale = 1.0 / math.sqrt(HD)
    if part_o is None:
        part_o = torch.empty(B, n_q, n_splits, HD, dtype=torch.float32, device=q_rot.device)
        part_lse = torch.empty(B, n_q, n_splits, dtype=torch.float32, device=q_rot.device)
    kps, kns, vps = _strides3(k_packed), _strides3(k_norms), _strides3(v_packed)
    vns = (v_norms.stride(0), v_norms.stride(1), v_norms.stride(2))
    plan = layer.plan(flags)
    _lib.check(_lib.lib().bgtq_decode(
        C.addressof(plan), _lib.ptr(layer.desc_dev), _lib.ptr(q_rot),
        _lib.ptr(k_packed), *kps, _lib.ptr(k_norms), *kns, _lib.ptr(v_packed), *vps, _lib.ptr(v_norms), *vns,
        B, n_q, layer.n_kv, int(t_begin), int(t_end), int(n_splits), float(scale),
        _lib.ptr(part_o), _lib.ptr(part_lse), _lib.ptr(status), _lib.ptr(pos_dev), int(pos_add),
        _lib.stream_ptr(q_rot.device)), "bgtq_decode")
    _lib.count_launch()
    return part_o, part_lse


def attend(layer, q, k_packed, k_norms, v_packed, v_norms, t_begin, t_end, *, rotate, n_splits=None, scale=None, flags=0,
           v_rot=None, buf_o=None, buf_lse=None, want_f32=False, want_lse=False, status=None):
    """Query rotation (``rotate``: q is in the original basis), split-KV decode over rows [t_begin, t_end) and combine
    in one library call.  q (B, n_q, [1,] 128) -> (out fp16 of q's shape, f32 copy (B, n_q, 128) | None, LSE | None)."""
    plan, _image, merged = layer.plan_entry(flags | _lib.DEC_PROGRAMMATIC)
    plan = C.addressof(plan)
    desc, rot_k = (layer.desc_dev.data_ptr(), layer.rot_k.data_ptr()) if rotate else (None, None)      # (of the query rotation)
    n_splits = 0 if n_splits is None else n_splits or -1       # (the library's choice; 0 is refused like -1)
    scale = _SCALE if scale is None else scale
    # (names of their own: the parameters may be the only references to these tensors, and the library takes addresses)
    rot_addr = None if v_rot is None else v_rot.data_ptr()
    status_addr = None if status is None else status.data_ptr()
    native = _lib.host().attend
    try:
        r = native(plan, desc, rot_k, q, k_packed, k_norms, v_packed, v_norms, t_begin, t_end, n_splits, scale, rot_addr, buf_o, buf_lse,
                   want_f32, want_lse, status_addr, layer.n_kv)
    except TypeError:       # (ranges as whole floats, say)
        t_begin, t_end, n_splits = int(t_begin), int(t_end), int(n_splits)
        r = native(plan, desc, rot_k, q, k_packed, k_norms, v_packed, v_norms, t_begin, t_end, n_splits, scale, rot_addr, buf_o, buf_lse,
                   want_f32, want_lse, status_addr, layer.n_kv)
    if r is None:           # another type or layout, or an argument to complain about
        _lib.require_cuda(q, "q")
        if k_norms.dtype != torch.float16 or v_norms.dtype != torch.float16:
            raise TypeError("cache norms must be float16")
        for t in (k_packed, k_norms, v_packed):
            _strides3(t)
        with torch.cuda.device(q.device):
            q = q.to(torch.float16).contiguous()
            r = native(plan, desc, rot_k, q, k_packed, k_norms, v_packed, v_norms, t_begin, t_end, n_splits, scale, rot_addr, buf_o, buf_lse,
                       want_f32, want_lse, status_addr, layer.n_kv)
        if r is None:
            raise ValueError("query, cache and layer do not match")
    return _lib.done(r, "bgtq_attend", (3 if rotate else 2) - merged)


_SCALE = 1.0 / math.sqrt(HD)


@functools.lru_cache(maxsize=None)
def _sm_count(index: int) -> int:
    return torch.cuda.get_device_properties(index).multi_processor_count


def tile_flags(n_batch: int, n_kv: int, n_tokens: int, device) -> int:
    """``DEC_NARROW`` while every SM's share of the tokens fits one narrow tile (16 warps x 16 tokens): twice the warps
    work on half the chain each.  Beyond, the wide tile loads each query fragment for twice the tokens.  A captured layer of
    one sequence with 8 KV heads (K3V3), wide and narrow tile, by tokens per SM: 64: 14.0 and 12.5 us, 192: 14.8 and 13.2, 254: 14.5 and
    14.1, past 256: 14.8 and 15.2, 512: 16.6 and 16.9 (K2V2 alike).  ``n_tokens`` is what the kernel is chosen for: a manager passes its
    capacity, so that one kernel serves the cache's whole life; a short sequence in a large cache runs the wide tile."""
    index = device.index if device.index is not None else torch.cuda.current_device()
    return _lib.DEC_NARROW if n_batch * n_kv * n_tokens <= 256 * _sm_count(index) else 0


def merges(layer, flags: int) -> bool:
    """Whether the layer's decode with these plan flags merges its shares itself in layer steps and attentions."""
    return layer.plan_entry(flags)[2]


def cluster_flags(n_batch: int, n_kv: int, n_tokens: int, device, gqa: int, v_bits: int, grows: bool = False, eager: bool = False) -> int:
    """Plan flags of the form that merges a pair's shares inside the decode launch (``DEC_CLUSTER_SHIFT``; the narrow tile), for
    layer steps and attentions over up to ``n_tokens`` rows, or 0 where the decode over all SMs and its merge launch are faster.
    ``v_bits``: as stored (nibbles: 4).

    A cluster of C CTAs per (batch, KV head) pair saves the second launch and the partials' way through memory, 2 to 4 us (one
    sequence of 8 KV heads, K3V3, 500 tokens: 12.6 -> 10.9 us per layer; 4 sequences at 4000 tokens: 23.1 -> 20.6).  How far that
    carries: see ``_merging_limit``.  C is the largest of 8, 4 and 2 whose clusters all run at once: 14 clusters of 8, 32 of 4 and
    72 of 2 do (16 of 8 and 36 of 4 take two waves); and smaller while a CTA then has at most 8 warps' tokens, or 16 where the CTAs
    would take more than half of the SMs, which the next launch's CTAs start on.  ``grows``: the length goes up from call to call;
    one C for all of them, as each is a kernel of its own.  ``eager``: never captured, so that a launch costs the host's time too."""
    pairs = n_batch * n_kv
    if pairs < 1 or v_bits not in _MOST_SHARE:      # (a call to complain about)
        return 0
    sms = _sm_count(device.index if device.index is not None else torch.cuda.current_device())
    c, most = _merging_limit(pairs, sms, gqa > 4, v_bits, eager)
    if n_tokens > most:
        return 0
    while not grows and c > 2 and 2 * n_tokens <= (256 if 2 * pairs * c > sms else 128) * c:
        c //= 2
    return _lib.DEC_NARROW | c << _lib.DEC_CLUSTER_SHIFT


_MOST_SHARE = {1: 2200, 2: 2200, 3: 2500, 4: 6000}      # tokens of a CTA of a cluster, by V's bits: see _merging_limit


@functools.lru_cache(maxsize=1024)
def _merging_limit(pairs: int, sms: int, wide_groups: bool, v_bits: int, eager: bool):
    """(C, the most tokens its clusters are taken for), from layers of 2 to 72 pairs, 4 and 8 query heads per KV head and V of 2 to 4
    bits timed in both forms at up to eight lengths each, captured and called one by one:
      * a CTA gets tokens / C of them instead of an SM's even share: up to 330 more (3 us) are made up for.  Fewer of a captured
        layer with few pairs, whose split form runs the narrow tile too: 270 with 4-bit values and up to 16 pairs (one sequence of 8 heads,
        4600 tokens: 16.6 -> 17.5 us), 110 less where eight CTAs exchange the rows of more than four query heads (4600 tokens: 16.5 ->
        17.5, K3V3).  Called one by one the second launch costs the host 2.5 us, which carries that far (attention 18.0, 15.6);
      * beside the wide tile clusters fall behind with every token, the more the narrower V is: to 2200, 2500 and 6000 tokens of a
        CTA with 2, 3 and 4 bits (two layers, K3V3, clusters and split form: of 2 CTAs, 72 pairs, 4500 tokens 66.6 and 69.8 us, 5500 75.9
        both, 9000 108.7 and 100.1; of 4, 32 pairs, 8900: 63.9 and 65.6, 9700: 69.0 and 67.0; K2V2, 72 pairs, 4200: 61.5 both,
        7000: 84.3 and 76.4), and to 1050 in clusters of 8 (14 pairs, 7600: 37.7 and 39.0, 8900: 41.0 and 39.4)."""
    for c, most in ((8, 14), (4, 32), (2, 72)):
        if pairs <= most * sms // 148:
            apart = 330
            if not eager:
                wide = c == 8 and wide_groups
                if v_bits == 4 and 4 * (1 if wide else 2) <= pairs <= 16:
                    apart = 270
                if wide and pairs > 4:
                    apart -= 110
            limit = apart * sms * c // (sms - pairs * c) if pairs * c < sms else 1 << 30
            return c, min(limit, c * (1050 if c == 8 else _MOST_SHARE[v_bits]))
    return 0, -1


@functools.lru_cache(maxsize=4096)
def growing_forms(n_batch: int, n_kv: int, n_tokens: int, index, gqa: int, v_bits: int):
    """Plan flags of a call on device ``index`` whose context grows from call to call: of its form, of the split form beside it and of
    the merging form that its shape takes while it is short (0: none).  (A microsecond of arithmetic, asked for per head and layer.)"""
    device = torch.device("cuda" if index is None else f"cuda:{index}")
    split = tile_flags(n_batch, n_kv, n_tokens, device)
    merging, short = (cluster_flags(n_batch, n_kv, n, device, gqa, v_bits, grows=True, eager=True) for n in (n_tokens, 1))
    return merging or split, split, short


_PREFILL_WORKSPACE = 2 << 30        # bytes of dequantised operand tiles per launch


def prefill_attention(layer: LayerTables, q_rot, k_packed, k_norms, v_packed, v_norms, n_tokens, *,
                      q_pos_offset=0, causal=True, scale=None, flags=0, v_rot=None):
    """Attention of q_rot (B, n_q, S_q, 128) fp16 (packed-K basis) over the first ``n_tokens`` cache rows;
    query i has absolute position ``q_pos_offset + i`` and, when ``causal``, sees tokens up to it.
    ``v_rot`` (n_kv, 128, 128) fp32 = R finishes V's rotation.
    Returns (B, n_q, S_q, 128) fp16.  ``_lib.PF_NO_TCGEN05`` in ``flags`` (or the environment variable
    ``BGTQ_PF_NO_TCGEN05``) keeps the products on mma.sync instead of tcgen05 / tensor memory.

    The tcgen05 form dequantises the cache into a workspace from torch's allocator, 768 bytes per token and KV head
    and at most 2 GiB at a time (the batch, then the KV heads, in several launches beyond that).  Where the device
    has no room for it, the call runs on mma.sync, which reads the packed rows themselves."""
    scale = _SCALE if scale is None else scale
    n_tokens, q_pos_offset, causal, flags = int(n_tokens), int(q_pos_offset), bool(causal), int(flags)
    if v_rot is not None:       # the kernels take its address
        if v_rot.dtype != torch.float32 or v_rot.device != q_rot.device:
            raise TypeError("v_rot must be float32 on the queries' device")
        v_rot = v_rot.view(layer.n_kv, HD, HD).contiguous()
    if not (flags & _lib.PF_NO_TCGEN05 or os.environ.get("BGTQ_PF_NO_TCGEN05")):
        try:
            r = _lib.host().prefill(layer.desc_dev.data_ptr(), layer.n_kv, q_rot, k_packed, k_norms, v_packed, v_norms, n_tokens,
                                    q_pos_offset, causal, scale, flags, None if v_rot is None else v_rot.data_ptr(),
                                    _PREFILL_WORKSPACE)
            if r is not None:
                return _lib.done(r, "bgtq_prefill", 2)
            return _prefill_parts(layer, q_rot, k_packed, k_norms, v_packed, v_norms, n_tokens, q_pos_offset, causal, scale, flags, v_rot)
        except torch.OutOfMemoryError:
            pass
    qs, kps, kns, vps, vns = _prefill_strides(q_rot, k_packed, k_norms, v_packed, v_norms)
    B, n_q, S_q, _ = q_rot.shape
    dev = q_rot.device
    out_rot = torch.empty(B, n_q, S_q, HD, dtype=torch.float32, device=dev)
    _lib.check(_lib.lib().bgtq_prefill_attention(
        _lib.ptr(layer.desc_dev), _lib.ptr(q_rot), *qs, _lib.ptr(k_packed), *kps, _lib.ptr(k_norms), *kns,
        _lib.ptr(v_packed), *vps, _lib.ptr(v_norms), *vns, B, n_q, layer.n_kv, S_q, n_tokens, q_pos_offset, causal,
        float(scale), flags | _lib.PF_NO_TCGEN05, _lib.ptr(out_rot), _lib.stream_ptr(dev)), "bgtq_prefill_attention")
    _lib.count_launch()
    if v_rot is None:
        return out_rot.to(torch.float16)
    gqa = n_q // layer.n_kv
    o = torch.matmul(out_rot.view(B, layer.n_kv, gqa * S_q, HD), v_rot.view(1, layer.n_kv, HD, HD))
    return o.view(B, n_q, S_q, HD).to(torch.float16)


def _prefill_strides(q_rot, k_packed, k_norms, v_packed, v_norms):
    _lib.require_cuda(q_rot, "q_rot")
    if q_rot.dim() != 4 or q_rot.shape[3] != HD or q_rot.dtype != torch.float16 or q_rot.stride(3) != 1:
        raise ValueError("q_rot must be float16 (B, n_q, S_q, 128) with contiguous rows")
    if k_norms.dtype != torch.float16 or v_norms.dtype != torch.float16:
        raise TypeError("cache norms must be float16")
    return q_rot.stride()[:3], _strides3(k_packed), _strides3(k_norms), _strides3(v_packed), v_norms.stride()[:3]


def _prefill_parts(layer, q_rot, k_packed, k_norms, v_packed, v_norms, n_tokens, q_pos_offset, causal, scale, flags, v_rot):
    """The tcgen05 form in as many launches as keep the dequantised tiles within their bound: fewer batch entries per
    launch first, then (one entry) fewer KV heads; one of each at least."""
    qs, kps, kns, vps, vns = _prefill_strides(q_rot, k_packed, k_norms, v_packed, v_norms)
    B, n_q, S_q, _ = q_rot.shape
    n_kv, gqa, dev, L = layer.n_kv, n_q // layer.n_kv, q_rot.device, _lib.lib()

    def ws_bytes(n, m):
        return L.bgtq_prefill_workspace_bytes(n, m * gqa, m, S_q, n_tokens, q_pos_offset, causal, v_rot is not None)

    nb, nh = B, n_kv
    while ws_bytes(nb, nh) > _PREFILL_WORKSPACE and nb * nh > 1:
        nb, nh = ((nb + 1) // 2, nh) if nb > 1 else (1, (nh + 1) // 2)
    parts = [(b, min(nb, B - b), h, min(nh, n_kv - h)) for b in range(0, B, nb) for h in range(0, n_kv, nh)]
    ws = torch.empty(max([16] + [ws_bytes(n, m) for _, n, _, m in parts]), dtype=torch.uint8, device=dev)
    out = torch.empty(B, n_q, S_q, HD, dtype=torch.float16, device=dev)
    for b, n, h, m in parts:        # (with fewer heads than all there is one batch entry: its heads' rows are contiguous)
        bs, hs, qh = slice(b, b + n), slice(h, h + m), slice(h * gqa, (h + m) * gqa if m < n_kv else n_q)
        _lib.check(L.bgtq_prefill(
            layer.desc_dev.data_ptr() + h * C.sizeof(_lib.HeadDesc), q_rot[bs, qh].data_ptr(), *qs, k_packed[bs, hs].data_ptr(), *kps,
            k_norms[bs, hs].data_ptr(), *kns, v_packed[bs, hs].data_ptr(), *vps, v_norms[bs, hs].data_ptr(), *vns, n,
            m * gqa if m < n_kv else n_q, m, S_q, n_tokens, q_pos_offset, causal, float(scale), flags,
            None if v_rot is None else v_rot[hs].data_ptr(), ws.data_ptr(), ws.numel(), out[bs, qh].data_ptr(), _lib.stream_ptr(dev)),
            "bgtq_prefill")
        _lib.count_launch(2)
    return out


def combine_ranks(gathered, n_batch, n_q, *, out=None):
    """Merge the all-gathered per-rank messages ``gathered`` (W, n_batch*n_q*129) fp32, each
    [O (B, n_q, 128) | LSE (B, n_q)], into fp16 (B, n_q, 128)."""
    _lib.require_cuda(gathered, "gathered")
    W = gathered.shape[0]
    if out is None:
        out = torch.empty(n_batch, n_q, HD, dtype=torch.float16, device=gathered.device)
    _lib.check(_lib.lib().bgtq_combine_ranks(
        _lib.ptr(gathered), W, gathered.stride(0), n_batch, n_q, _lib.ptr(out), out.stride(0), out.stride(1),
        0, _lib.stream_ptr(gathered.device)), "bgtq_combine_ranks")
    _lib.count_launch()
    return out


def combine(part_o, part_lse, n_kv, *, v_rot=None, buf_o=None, buf_lse=None, out=None,
            want_f32=False, want_lse=False, programmatic=False, o32_out=None, lse_out=None):
    """Merge (B, n_q, S, 128)/(B, n_q, S) partials -> fp16 (B, n_q, 128) [+ f32 copy, total LSE].
    ``programmatic``: launch as a programmatic dependent of the preceding kernel (see bgtq.h)."""
    B, n_q, S, _ = part_o.shape
    dev = part_o.device
    if out is None:
        out = torch.empty(B, n_q, HD, dtype=torch.float16, device=dev)
    o32 = o32_out if o32_out is not None else (
        torch.empty(B, n_q, HD, dtype=torch.float32, device=dev) if want_f32 else None)
    lse = lse_out if lse_out is not None else (
        torch.empty(B, n_q, dtype=torch.float32, device=dev) if want_lse else None)
    _lib.check(_lib.lib().bgtq_combine(
        _lib.ptr(part_o), _lib.ptr(part_lse), S, _lib.ptr(v_rot), _lib.ptr(buf_o), _lib.ptr(buf_lse),
        B, n_q, n_kv, _lib.ptr(out), out.stride(0), out.stride(1), _lib.ptr(o32), _lib.ptr(lse),
        _lib.COMBINE_PROGRAMMATIC if programmatic else 0, _lib.stream_ptr(dev)), "bgtq_combine")
    _lib.count_launch()
    return out, o32, lse


def buffer_attn(q, k_buf, v_buf, n_kv, scale, *, n_sink_tokens=0, n_ring_tokens=0, sink_cap, ring_first=0, ring_size,
                pos_dev=None, out=None):
    """Attention over unquantised fp16 tokens.  q (B, n_q, 128) fp16 (original basis);
    k_buf/v_buf (B, n_kv, cap, 128) fp16 with contiguous token rows: a sink prefix and a ring
    of ``ring_size`` slots starting at slot ``sink_cap`` (see ``bgtq_buffer_attn``)."""
    _lib.require_cuda(q, "q")
    if q.dim() == 4:
        q = q[:, :, 0]
    B, n_q, _ = q.shape
    if out is not None:
        o, lse = out
    else:
        o = torch.empty(B, n_q, HD, dtype=torch.float32, device=q.device)
        lse = torch.empty(B, n_q, dtype=torch.float32, device=q.device)
    if k_buf.stride(2) != HD or k_buf.stride(3) != 1 or v_buf.stride() != k_buf.stride():
        raise ValueError("buffer tensors must be (B, n_kv, cap, 128) with contiguous token rows")
    _lib.check(_lib.lib().bgtq_buffer_attn_pos(
        _lib.ptr(q), q.stride(0), q.stride(1), _lib.ptr(k_buf), _lib.ptr(v_buf), k_buf.stride(0), k_buf.stride(1),
        int(n_sink_tokens), int(n_ring_tokens), int(sink_cap), int(ring_first), int(ring_size),
        B, n_q, n_kv, float(scale), _lib.ptr(o), _lib.ptr(lse), _lib.ptr(pos_dev), _lib.stream_ptr(q.device)),
        "bgtq_buffer_attn_pos")
    _lib.count_launch()
    return o, lse
