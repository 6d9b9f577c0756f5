"""Tensor-level wrappers over the C ABI: they only translate torch tensors
(device memory, strides, the current stream) into the plain structs of
include/sqattn_b200.h.  No arithmetic happens on the Python side."""
from __future__ import annotations

import ctypes as C
import struct
from array import array
from typing import Optional, Sequence

import torch

from . import _lib as L


def _dt(dtype: torch.dtype) -> int:
    if dtype == torch.float16:
        return L.F16
    if dtype == torch.bfloat16:
        return L.BF16
    raise ValueError(f"unsupported dtype {dtype}: float16 or bfloat16 expected")


def _stream() -> int:
    """The current device's current stream, without building a Stream object (a microsecond of every call)."""
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device())


def _require_cuda(*ts):
    for t in ts:
        if t is not None and not t.is_cuda:
            raise RuntimeError("sqattn_b200 runs on CUDA tensors only (there is no CPU path)")


def _desc(t: torch.Tensor, layout: str):
    """(pointer, batch, head and token strides) of the logical [B,H,N,D] view of a 4-D tensor stored HND or NHD."""
    st = t.stride()
    assert len(st) == 4 and st[3] == 1, "Last dim of qkv must be contiguous."
    if layout == "HND":
        return t.data_ptr(), st[0], st[1], st[2]
    if layout == "NHD":
        return t.data_ptr(), st[0], st[2], st[1]
    raise ValueError(f"tensor_layout {layout} not supported")


def _view(t: torch.Tensor, layout: str) -> L.Tensor:
    return L.Tensor(*_desc(t, layout))


_NO_TENSOR = (0, 0, 0, 0)
# The argument structs in the header's order, filled in one call each: setting their fields one by one through ctypes took
# about as long as the launches (a 1000-token call of the operator: 47.3 us field by field, 43.8 like this).
_PREFILL_ARGS = struct.Struct("4q4q4q4q4q4qq11i4x4q2iqQ6i")
_PREP_ARGS = struct.Struct("4q4q4q5q10iqQqii")
assert _PREFILL_ARGS.size == C.sizeof(L.PrefillArgs) and _PREP_ARGS.size == C.sizeof(L.PrepArgs)
_DECODE_ARGS = struct.Struct("4q4q4q4qq5i4xq6iqQqqqqi4xq")
assert _DECODE_ARGS.size == C.sizeof(L.DecodeArgs)


def _decode_args(q, k, v, o, lse, batch, hq, hkv, d, kv_len, dtype, o_dtype, *, kv_lens=0, p_fp8=False, q_is_scaled=False, num_splits=0,
                 reference_tail=False, partial_o=0, partial_lse=0, kv_lens_device=0, peer=0, head_dim_og=0, gather=0) -> L.DecodeArgs:
    """q, k, v, o as _desc gives them; pointers as integers."""
    return L.DecodeArgs.from_buffer(bytearray(_DECODE_ARGS.pack(
        *q, *k, *v, *o, lse, batch, hq, hkv, d, kv_len, kv_lens, dtype, o_dtype, int(p_fp8), int(q_is_scaled), int(num_splits),
        int(reference_tail), 0, 0, partial_o, partial_lse, kv_lens_device, peer, int(head_dim_og), gather)))


def _run_decode(a: L.DecodeArgs, device, workspace_bytes, entry):
    """Workspace and launch.  A rejected plan (0 bytes) goes on to the entry point, which reports why."""
    need = workspace_bytes(C.byref(a))
    if need:
        ws = torch.empty(need, dtype=torch.uint8, device=device)   # the caching allocator's blocks are 512-byte aligned
        a.workspace, a.workspace_bytes = ws.data_ptr(), need
    L.check(entry(C.byref(a), _stream()))
    if not need:
        raise ValueError("sqattn_decode: invalid arguments")


def _shape(t: torch.Tensor, layout: str):
    b, x, y, d = t.shape
    return (b, x, y, d) if layout == "HND" else (b, y, x, d)


_MIRRORS = {}


def poll_device_status(device=None):
    """Cheap, non-synchronising look at the failure word of ``device``: a pinned host int32 that a kernel whose bounded
    wait gave up also writes to (sqattn_set_status_mirror).  Raises SqattnError(ERR_DEVICE_TIMEOUT) once a failure has
    become visible; every operator below calls it on entry, so a caller of the drop-in operator hears about a timed-out
    wait at its next call at the latest (and meanwhile gets NaN, never stale memory).  The device-side word stays set,
    and later launches keep returning NaN, until ``check_device_status`` has cleared it."""
    idx = torch.cuda.current_device() if device is None or device.index is None else device.index
    ent = _MIRRORS.get(idx)
    if ent is None:
        if torch.cuda.is_current_stream_capturing():
            return
        word = torch.zeros(1, dtype=torch.int32).pin_memory()
        with torch.cuda.device(idx):
            L.check(L.lib.sqattn_set_status_mirror(word.data_ptr()))
        ent = _MIRRORS[idx] = (word, C.c_int32.from_address(word.data_ptr()))
    code = ent[1].value
    if code:
        raise L.SqattnError(L.ERR_DEVICE_TIMEOUT, f"a device-side wait gave up on cuda:{idx} (code {code}: 1xx prefill, "
                            "2xx decode, 3xx peer exchange); outputs since then are NaN; call check_device_status() to clear")


def _workspace(nbytes: int, device) -> Optional[torch.Tensor]:
    if nbytes == 0:
        return None
    ws = torch.empty(nbytes + 1024, dtype=torch.uint8, device=device)
    off = (-ws.data_ptr()) % 1024
    return ws[off:off + nbytes] if off else ws


def _floats(values, count: int) -> array:
    """``count`` fp32 numbers in host memory; fewer are followed by zeros, more are refused."""
    x = array("f", map(float, values))
    if len(x) > count:
        raise IndexError("invalid index")
    if len(x) < count:
        x.extend([0.0] * (count - len(x)))
    return x


def _i32(x) -> int:
    """The int32 that a C field would hold."""
    return ((int(x) + 0x80000000) & 0xffffffff) - 0x80000000


def prefill(q8, k8, q4, k4, v, *, mode: int, win8=None, win4=None, sink: int = 0, layout: str = "HND",
            out_dtype=torch.float16, return_lse: bool = False, p_fp8_mode: int = 0, q_is_scaled: bool = False,
            out: Optional[torch.Tensor] = None, out_layout: Optional[str] = None, kv_layout: Optional[str] = None,
            q_row_offset: int = 0, head_dim_og: int = 0, q_split_rows: int = 0, q_row_offset2: int = 0,
            q_fake_quant: Optional[str] = None, round_half_even: bool = False):
    """sqattn_prefill.  win8/win4: per-head sequences (floats for the relative mode, ints for the absolute).
    kv_layout: layout of k/v when it differs from q's; q_row_offset: first row of a query shard; head_dim_og: the
    head_dim before the caller zero-padded the tensors to 64 / 128 (the softmax scale follows it).  q_fake_quant
    ("int" / "e4m3" / "e5m2"): q8 is the raw query and the kernel fake-quantises and scales it tile by tile."""
    _require_cuda(q8, k8, q4, k4, v)
    poll_device_status(q8.device)
    b, hq, n, d = _shape(q8, layout)
    kv_layout = kv_layout or layout
    _, hkv, kv_len, _ = _shape(k8, kv_layout)
    if out is None:
        out = torch.empty(q8.shape, dtype=out_dtype, device=q8.device)
        out_layout = layout
    lse = torch.empty(b, hq, n, dtype=torch.float32, device=q8.device) if return_lse else None
    qd, kd = _desc(q8, layout), _desc(k8, kv_layout)
    if q_fake_quant is not None and q_fake_quant not in L.QTYPE:
        raise ValueError(f"Invalid quantization type: {q_fake_quant}")
    windows = (0, 0, 0, 0)
    if mode == L.MODE_RELATIVE_WINDOW:
        w8, w4 = _floats(win8, hq), _floats(win4, hq)
        windows = (w8.buffer_info()[0], w4.buffer_info()[0], 0, 0)
    elif mode == L.MODE_ABSOLUTE_WINDOW:
        w8, w4 = (C.c_int32 * hq)(*map(int, win8)), (C.c_int32 * hq)(*map(int, win4))
        windows = (0, 0, C.addressof(w8), C.addressof(w4))
    a = L.PrefillArgs.from_buffer(bytearray(_PREFILL_ARGS.pack(
        *qd, *kd, *(qd if q4 is q8 else _desc(q4, layout)), *(kd if k4 is k8 else _desc(k4, kv_layout)), *_desc(v, kv_layout),
        *_desc(out, out_layout), 0 if lse is None else lse.data_ptr(), b, hq, hkv, n, kv_len, d, _dt(q8.dtype), _dt(v.dtype),
        _dt(out.dtype), mode, _i32(sink), *windows, _i32(p_fp8_mode),
        int(q_is_scaled), 0, 0, _i32(q_row_offset), _i32(q_split_rows), _i32(q_row_offset2),   # a shard's second row range, if any
        0 if q_fake_quant is None else L.QTYPE[q_fake_quant] + 1, int(q_fake_quant is not None and round_half_even), _i32(head_dim_og))))
    need = L.lib.sqattn_prefill_workspace_bytes(C.byref(a))
    ws = _workspace(need, q8.device)
    a.workspace, a.workspace_bytes = (ws.data_ptr() if ws is not None else None), need
    L.check(L.lib.sqattn_prefill(C.byref(a), _stream()))
    return (out, lse) if return_lse else out


def prep_qkv(query, key, value, *, qk_qtype: str = "int", v_qtype: str = "int", round_half_even: bool = False,
             skip_bit4: bool = False, k_mean: Optional[torch.Tensor] = None, kv_out_nhd: bool = False,
             out: Optional[dict] = None):
    """sqattn_prep_qkv: NHD inputs -> (q_bit8, q_bit4, k_bit8, k_bit4, v_bit8) contiguous HND; q pre-scaled,
    K/V with their own Hkv heads, v_bit8 in fp16; of longer keys and values the first N rows are prepared.
    k_mean [B,Hkv,D] fp32 overrides the sequence mean of K; kv_out_nhd writes the K/V outputs token-major [B,N,Hkv,D].  Any of query/key/value may be None: only the
    tensors given are prepared (their outputs are returned, the others are None).  ``out`` may hold
    preallocated outputs under the keys q8, q4, k8, k4, v8."""
    given = [t for t in (query, key, value) if t is not None]
    _require_cuda(*given)
    if qk_qtype not in L.QTYPE:
        raise ValueError(f"Invalid quantization type: {qk_qtype}")
    if v_qtype not in L.QTYPE:
        raise ValueError(f"Invalid quantization type: {v_qtype}")
    ref = given[0]
    b, n, _, d = ref.shape
    dev, dt = ref.device, ref.dtype
    out = out or {}
    parts = 0
    q8 = q4 = k8 = k4 = v8 = None
    qd = kd = vd = _NO_TENSOR
    hq = hkv = 1
    if query is not None:
        hq = query.shape[2]
        q8 = out.get("q8")
        if q8 is None:
            q8 = torch.empty((b, hq, n, d), dtype=dt, device=dev)
        if not skip_bit4:
            q4 = out.get("q4") if out.get("q4") is not None else torch.empty_like(q8)
        qd = _desc(query, "NHD")
        parts |= 1
    if key is not None or value is not None:
        kv_in = (key if key is not None else value).shape
        hkv = kv_in[2]
        # one length, one count of KV heads and one set of strides per tensor go down: shorter ones would be read past their end
        if kv_in != (b, n, hkv, d) or (key is not None and value is not None and value.shape != kv_in):
            if any(t.shape[0] != b or t.shape[1] < n or t.shape[2] < hkv or t.shape[3] != d for t in (key, value) if t is not None):
                raise ValueError(f"query, key and value must be [B, N, H, D] of one batch, length and head_dim (keys and values "
                                 f"beyond the first's length are left out), got {[tuple(t.shape) for t in given]}")
    kv_shape = (b, n, hkv, d) if kv_out_nhd else (b, hkv, n, d)
    if key is not None:
        k8 = out.get("k8")
        if k8 is None:
            k8 = torch.empty(kv_shape, dtype=dt, device=dev)
        if not skip_bit4:
            k4 = out.get("k4") if out.get("k4") is not None else torch.empty_like(k8)
        kd = _desc(key, "NHD")
        parts |= 2
    if value is not None:
        v8 = out.get("v8")
        if v8 is None:
            v8 = torch.empty(kv_shape, dtype=torch.float16, device=dev)
        vd = _desc(value, "NHD")
        parts |= 4
    if k_mean is not None:
        assert k_mean.dtype == torch.float32 and k_mean.is_contiguous() and k_mean.shape == (b, hkv, d)
    a = L.PrepArgs.from_buffer(bytearray(_PREP_ARGS.pack(
        *qd, *kd, *vd, *(0 if t is None else t.data_ptr() for t in (q8, q4, k8, k4, v8)), b, hq, hkv, n, d, _dt(dt), L.QTYPE[qk_qtype],
        L.QTYPE[v_qtype], int(round_half_even), int(skip_bit4), 0, 0, 0 if k_mean is None else k_mean.data_ptr(), int(kv_out_nhd), parts)))
    need = L.lib.sqattn_prep_workspace_bytes(C.byref(a))
    ws = torch.empty(need, dtype=torch.uint8, device=dev)
    a.workspace, a.workspace_bytes = ws.data_ptr(), need
    L.check(L.lib.sqattn_prep_qkv(C.byref(a), _stream()))
    return q8, q4, k8, k4, v8


def k_column_sums(key: torch.Tensor) -> torch.Tensor:
    """sqattn_k_column_sums: key [B,N,Hkv,D] -> fp32 [B,Hkv,D] sums over the sequence."""
    _require_cuda(key)
    b, n, hkv, d = key.shape
    sums = torch.empty(b, hkv, d, dtype=torch.float32, device=key.device)
    nbytes = b * hkv * 64 * d * 4
    ws = _workspace(nbytes, key.device)
    view = _view(key, "NHD")
    L.check(L.lib.sqattn_k_column_sums(C.byref(view), b, hkv, n, d, _dt(key.dtype), sums.data_ptr(), ws.data_ptr(),
                                       nbytes, _stream()))
    return sums


def decode(q, k, v, *, layout: str = "HND", out_dtype=torch.float16, return_lse: bool = False, p_fp8: bool = False,
           q_is_scaled: bool = False, kv_lens: Optional[Sequence[int]] = None, kv_len: Optional[int] = None,
           num_splits: int = 0, partial: bool = False, reference_tail: bool = False,
           kv_lens_device: Optional[torch.Tensor] = None, peer=None, head_dim_og: int = 0):
    """sqattn_decode.  q [B,Hq,1,D] (HND) or [B,1,Hq,D] (NHD); k/v caches of capacity >= kv_len.
    partial=True returns (O fp32 [B,Hq,D], LSE fp32 [B,Hq]) of these keys for a later merge.
    reference_tail=True reproduces the reference kernel's zero-score padding of the last 64-key tile.
    kv_lens_device (int32 [B] on the GPU): the lengths are read by the kernel at run time and ``kv_len`` is only the
    capacity the key ranges are planned for, so the call can sit in a CUDA graph that is replayed as the cache grows.
    peer: a filled ``_lib.PeerMergeArgs`` (dist.PeerExchange builds it): the merge of the split-KV partials, the
    exchange with the other GPUs and the merge across GPUs happen in one kernel; returns nothing (the result is
    written to peer.out)."""
    _require_cuda(q, k, v)
    poll_device_status(q.device)
    b, hq, one, d = _shape(q, layout)
    assert one == 1
    _, hkv, cap, _ = _shape(k, layout)
    lens = None
    if kv_lens is not None:
        lens = (C.c_int32 * b)(*[int(x) for x in kv_lens])
    if kv_lens_device is not None:
        if kv_lens is not None:
            raise ValueError("kv_lens and kv_lens_device are exclusive: device lengths are planned for kv_len")
        assert kv_lens_device.is_cuda and kv_lens_device.dtype == torch.int32 and kv_lens_device.numel() == b
    out = lse = po = pl = None
    o_desc, o_dtype = _NO_TENSOR, L.F16
    if peer is None and partial:
        po = torch.empty(b, hq, d, dtype=torch.float32, device=q.device)
        pl = torch.empty(b, hq, dtype=torch.float32, device=q.device)
    elif peer is None:
        out = torch.empty(q.shape, dtype=out_dtype, device=q.device)
        o_desc, o_dtype = _desc(out, layout), _dt(out_dtype)
        if return_lse:
            lse = torch.empty(b, hq, 1, dtype=torch.float32, device=q.device)
    a = _decode_args(_desc(q, layout), _desc(k, layout), _desc(v, layout), o_desc, 0 if lse is None else lse.data_ptr(), b, hq, hkv, d,
                     int(cap if kv_len is None else kv_len), _dt(k.dtype), o_dtype, kv_lens=0 if lens is None else C.addressof(lens),
                     p_fp8=p_fp8, q_is_scaled=q_is_scaled, num_splits=num_splits, reference_tail=reference_tail,
                     partial_o=0 if po is None else po.data_ptr(), partial_lse=0 if pl is None else pl.data_ptr(),
                     kv_lens_device=0 if kv_lens_device is None else kv_lens_device.data_ptr(),
                     peer=0 if peer is None else C.addressof(peer), head_dim_og=head_dim_og)
    _run_decode(a, q.device, L.lib.sqattn_decode_workspace_bytes, L.lib.sqattn_decode)
    if peer is not None:
        return None
    if partial:
        return po, pl
    return (out, lse) if return_lse else out


def tma_ready(t: torch.Tensor) -> bool:
    """The kernels can read ``t`` where it lies: 16-byte aligned rows, no broadcast dimension."""
    st = t.stride()
    return st[3] == 1 and t.data_ptr() % 16 == 0 and all(s % 8 == 0 and (s > 0 or ext == 1) for s, ext in zip(st[:3], t.shape))


def decode_centered(q, k, v, *, layout: str = "HND", out_dtype=torch.float16, return_lse: bool = False,
                    reference_tail: bool = False, head_dim_og: int = 0):
    """sqattn_decode_centered: ``decode`` over K minus its mean over all the keys given, without forming it."""
    _require_cuda(q, k, v)
    poll_device_status(q.device)
    b, hq, one, d = _shape(q, layout)
    assert one == 1
    _, hkv, cap, _ = _shape(k, layout)
    out = torch.empty(q.shape, dtype=out_dtype, device=q.device)
    lse = torch.empty(b, hq, 1, dtype=torch.float32, device=q.device) if return_lse else None
    a = _decode_args(_desc(q, layout), _desc(k, layout), _desc(v, layout), _desc(out, layout), lse.data_ptr() if return_lse else 0,
                     b, hq, hkv, d, cap, _dt(k.dtype), _dt(out_dtype), reference_tail=reference_tail, head_dim_og=head_dim_og)
    _run_decode(a, q.device, L.lib.sqattn_decode_centered_workspace_bytes, L.lib.sqattn_decode_centered)
    return (out, lse) if return_lse else out


def decode_gather(q, idx, counts, k_rows, v_rows, row_stride: int, kv_dtype, *, out_dtype=torch.float16,
                  p_fp8: bool = False, q_is_scaled: bool = False, num_kv_heads: int = 1):
    """sqattn_decode over listed rows (sqattn_decode_args.gather): q [B,Hq,1,D]; key j of (sequence b, KV head h) is row
    idx[b*Hkv+h, j] of the matrix at k_rows[b*Hkv+h] / v_rows[b*Hkv+h] (int64 device tensors of device pointers), rows
    ``row_stride`` elements apart; counts (int32 [B] on the device) are the list lengths, idx.shape[1] the capacity the
    key ranges are planned for.  No host synchronisation."""
    _require_cuda(q, idx, counts, k_rows, v_rows)
    poll_device_status(q.device)
    b, hq, one, d = q.shape
    assert one == 1 and idx.dtype == torch.int32 and idx.is_contiguous() and idx.shape[0] == b * num_kv_heads
    assert counts.dtype == torch.int32 and counts.numel() == b
    assert k_rows.dtype == torch.int64 and v_rows.dtype == torch.int64 and k_rows.numel() == b * num_kv_heads == v_rows.numel()
    g = L.DecodeGather()
    g.idx, g.cap, g.k_rows, g.v_rows, g.row_stride = idx.data_ptr(), idx.shape[1], k_rows.data_ptr(), v_rows.data_ptr(), int(row_stride)
    out = torch.empty(q.shape, dtype=out_dtype, device=q.device)
    a = _decode_args(_desc(q, "HND"), _NO_TENSOR, _NO_TENSOR, _desc(out, "HND"), 0, b, hq, num_kv_heads, d, idx.shape[1], _dt(kv_dtype),
                     _dt(out_dtype), p_fp8=p_fp8, q_is_scaled=q_is_scaled, kv_lens_device=counts.data_ptr(), gather=C.addressof(g))
    _run_decode(a, q.device, L.lib.sqattn_decode_workspace_bytes, L.lib.sqattn_decode)
    return out


def decode_merge(part_o: torch.Tensor, part_lse: torch.Tensor, out_dtype=torch.float16, return_lse: bool = False):
    """sqattn_decode_merge: part_o [P, rows, D] fp32, part_lse [P, rows] fp32 -> O [rows, D]."""
    _require_cuda(part_o, part_lse)
    p, rows, d = part_o.shape
    out = torch.empty(rows, d, dtype=out_dtype, device=part_o.device)
    lse = torch.empty(rows, dtype=torch.float32, device=part_o.device) if return_lse else None
    L.check(L.lib.sqattn_decode_merge(part_o.contiguous().data_ptr(), part_lse.contiguous().data_ptr(), p, rows, d,
                                      out.data_ptr(), _dt(out_dtype), None if lse is None else lse.data_ptr(),
                                      _stream()))
    return (out, lse) if return_lse else out


def check_device_status():
    """Raise if a bounded device-side wait gave up since the last check (synchronises the stream); clears the
    device word and its host mirror, after which launches compute again."""
    ent = _MIRRORS.get(torch.cuda.current_device())
    try:
        L.check(L.lib.sqattn_check_device_status(_stream()))
    finally:
        if ent is not None:
            ent[1].value = 0


def decode_static_scratch(q, k, v, out, *, layout: str = "HND", lse: Optional[torch.Tensor] = None,
                          p_fp8: bool = False, q_is_scaled: bool = False, kv_lens: Optional[Sequence[int]] = None,
                          kv_len: Optional[int] = None, num_splits: int = 0, reference_tail: bool = False):
    """sqattn_decode_static_scratch: decode into the caller's ``out`` (and ``lse``) without any allocation, for
    callers inside a region where device memory may not be allocated.  The split-KV partials use the scratch
    array built into the library (4 MiB + 64 KiB); calls that need more are rejected, and calls must not overlap
    on the GPU.  Make the first call on a device outside stream capture."""
    _require_cuda(q, k, v, out)
    b, hq, one, d = _shape(q, layout)
    assert one == 1
    _, hkv, cap, _ = _shape(k, layout)
    a = L.DecodeArgs()
    a.q, a.k, a.v, a.o = _view(q, layout), _view(k, layout), _view(v, layout), _view(out, layout)
    a.lse = None if lse is None else lse.data_ptr()
    a.batch, a.num_q_heads, a.num_kv_heads, a.head_dim = b, hq, hkv, d
    a.kv_len = int(cap if kv_len is None else kv_len)
    if kv_lens is not None:
        lens = (C.c_int32 * b)(*[int(x) for x in kv_lens])
        a.kv_lens = lens
    a.dtype, a.o_dtype = _dt(k.dtype), _dt(out.dtype)
    a.p_fp8, a.q_is_scaled, a.num_splits, a.reference_tail = int(p_fp8), int(q_is_scaled), int(num_splits), int(reference_tail)
    L.check(L.lib.sqattn_decode_static_scratch(C.byref(a), _stream()))
    return out


def rmsnorm(x: torch.Tensor, weight: torch.Tensor, eps: float, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """sqattn_rmsnorm over the last dimension of x [..., dim] (rows may be strided); out may be x itself."""
    _require_cuda(x, weight)
    dim = x.shape[-1]
    x2 = x.reshape(-1, dim) if x.dim() != 2 else x
    assert x2.stride(1) == 1 and weight.is_contiguous() and weight.numel() == dim
    out = torch.empty(x.shape, dtype=x.dtype, device=x.device) if out is None else out
    o2 = out.reshape(-1, dim) if out.dim() != 2 else out
    assert o2.stride(1) == 1 and o2.shape == x2.shape
    assert o2.data_ptr() == out.data_ptr(), "out must be viewable as [rows, dim] without a copy"
    L.check(L.lib.sqattn_rmsnorm(x2.data_ptr(), weight.data_ptr(), o2.data_ptr(), x2.shape[0], dim, x2.stride(0),
                                 o2.stride(0), float(eps), _dt(x.dtype), _stream()))
    return out


def rope_qk(qkv: torch.Tensor, seq_len: int, num_heads: int, head_dim: int, cos_sin_cache: torch.Tensor, pos0: int,
            pos_device: Optional[torch.Tensor] = None):
    """sqattn_rope_qk: rotate the first num_heads heads of every row of the fused projection qkv [rows, width]
    in place; row r takes position pos0 + r % seq_len of cos_sin_cache [max_len, head_dim] (fp32).  With
    ``pos_device`` (int64 [1] on the GPU) that value is added to pos0 when the kernel runs."""
    _require_cuda(qkv, cos_sin_cache)
    assert qkv.dim() == 2 and qkv.stride(1) == 1
    assert cos_sin_cache.dtype == torch.float32 and cos_sin_cache.is_contiguous() and cos_sin_cache.shape[1] == head_dim
    if pos_device is not None:
        assert pos_device.is_cuda and pos_device.dtype == torch.int64
    L.check(L.lib.sqattn_rope_qk_devpos(qkv.data_ptr(), qkv.stride(0), qkv.shape[0], int(seq_len), int(num_heads),
                                        int(head_dim), cos_sin_cache.data_ptr(), cos_sin_cache.shape[0], int(pos0),
                                        None if pos_device is None else pos_device.data_ptr(), _dt(qkv.dtype), _stream()))
    return qkv


def silu_mul(x: torch.Tensor, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """sqattn_silu_mul: x [..., 2*inter] contiguous -> [..., inter]."""
    _require_cuda(x)
    assert x.is_contiguous() and x.shape[-1] % 2 == 0
    inter = x.shape[-1] // 2
    out = torch.empty(*x.shape[:-1], inter, dtype=x.dtype, device=x.device) if out is None else out
    assert out.is_contiguous()
    L.check(L.lib.sqattn_silu_mul(x.data_ptr(), out.data_ptr(), x.numel() // (2 * inter), inter, _dt(x.dtype), _stream()))
    return out
