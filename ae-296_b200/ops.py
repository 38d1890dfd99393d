"""Python-facing multi-LoRA ops: thin wrappers that pass tensor addresses to the C ABI.

``add_lora_bgmv`` keeps the positional signature the reference's layer code calls
(``punica.ops.add_lora_bgmv(y, x, wa_T_all, wb_T_all, indicies, layer_idx, scale)``,
lightllm/models/lora_gpu.py:138,150,162).  The generalised ops add per-adapter ranks and
scalings, packed pools, adapter-sorted segments and fused q/k/v application.

PyTorch is used for device memory and streams only; all arithmetic runs in the CUDA
library, and there is no fallback path.

The hot calls (``apply``, ``add_lora_bgmv``, ``add_lora_bgmv_static`` and plan building) go through the native
host path first (``csrc/host.cpp``), which reads the tensors in C++ and costs about a microsecond a call; the
Python code that follows each of them raises the error of a call that does not qualify, or prepares what is
missing.
"""
from __future__ import annotations

import ctypes as C
import threading
from typing import List, Optional, Sequence, Tuple

import numpy as np
import torch

from . import _lib
from ._lib import Adapters, LoraError, Proj, check
from .pool import AdapterPool

_DT = {torch.float16: _lib.F16, torch.bfloat16: _lib.BF16, torch.float32: _lib.F32}


def _stream(device) -> int:
    return torch.cuda.current_stream(device).cuda_stream


def _require_cuda(*tensors):
    for t in tensors:
        if not t.is_cuda:
            raise ValueError("LoRA ops need CUDA tensors (no CPU path exists)")


def _adapters_struct(n_adapters, n_layers, r_pool, ranks=None, scalings=None, cum_ranks=None,
                     packed=False, scale=1.0, ranks_pow2=False, total_rank=0) -> Adapters:
    return Adapters(
        ranks.data_ptr() if ranks is not None else None,
        scalings.data_ptr() if scalings is not None else None,
        cum_ranks.data_ptr() if cum_ranks is not None else None,
        n_adapters, n_layers, r_pool, 1 if packed else 0, float(scale), 1 if ranks_pow2 else 0,
        int(total_rank))


def adapters_of(pool: AdapterPool) -> Adapters:
    """The pool's adapter table; promises power-of-two ranks to the library when the host
    copy of the ranks shows it (which selects the TMA kernels)."""
    rh = pool.ranks_host
    if pool.packed:
        pow2 = bool(np.isin(rh, (8, 16, 32, 64)).all())
    else:
        pow2 = bool((rh == pool.r_pool).all()) and pool.r_pool in (8, 16, 32, 64)
    return _adapters_struct(pool.n_adapters, pool.n_layers, pool.r_pool, pool.ranks, pool.scalings,
                            pool.cum_ranks, pool.packed, 1.0, pow2, int(pool.cum_host[-1]))


def _table(adapters) -> Adapters:
    return adapters if isinstance(adapters, Adapters) else adapters_of(adapters)


class LoraPlan:
    """Device-resident segment table of one batch (see ``b200_lora_plan_build``)."""

    def __init__(self, max_tokens: int, n_adapters: int, device="cuda"):
        self.max_tokens, self.n_adapters = int(max_tokens), int(n_adapters)
        nbytes = _lib.lib().b200_lora_plan_bytes(self.max_tokens, self.n_adapters)
        if nbytes == 0:
            raise ValueError("bad plan dimensions")
        self.buf = torch.empty((nbytes + 15) // 16 * 2, dtype=torch.int64, device=device)
        self.buf[:8].zero_()         # the header: a plan that was never built applies nothing
        self.nbytes = self.buf.numel() * 8
        self._keep = None
        self.n_tokens = 0            # rows of the batch the plan was last built for

    def build(self, ids: torch.Tensor, adapters) -> "LoraPlan":
        """``adapters``: the table as an :class:`_lib.Adapters` structure, or the :class:`AdapterPool` it describes."""
        _require_cuda(ids)
        if ids.dtype not in (torch.int32, torch.int64) or not ids.is_contiguous():
            raise ValueError("ids must be a contiguous int32/int64 tensor")
        rc = _lib.host().plan_build(self, ids, adapters)
        if rc > 0:
            rc = _lib.host().plan_build(self, ids, _table(adapters))
        if rc > 0:
            raise ValueError("plan_build: unsupported arguments")
        check(rc, "plan_build")
        return self

    def from_segments(self, seg_starts: torch.Tensor, seg_adapter: torch.Tensor, n_tokens: int,
                      adapters) -> "LoraPlan":
        """``seg_starts`` has one entry per segment and the end of the last one (which may be left out: the
        last segment then ends at ``n_tokens``).  ``adapters`` as for :meth:`build`."""
        _require_cuda(seg_starts, seg_adapter)
        if seg_starts.dtype != torch.int32 or seg_adapter.dtype != torch.int32:
            raise ValueError("segment tables must be int32")
        self._keep = (seg_starts, seg_adapter)
        rc = _lib.host().plan_segments(self, seg_starts, seg_adapter, int(n_tokens), adapters)
        if rc > 0:
            rc = _lib.host().plan_segments(self, seg_starts, seg_adapter, int(n_tokens), _table(adapters))
        if rc > 0:
            raise ValueError("segment tables are contiguous: one start per segment, and optionally the end of the last")
        check(rc, "plan_from_segments")
        return self

    def read(self) -> Tuple[np.ndarray, np.ndarray, np.ndarray]:
        """(perm, seg_starts, seg_adapter) as host arrays; raises on a bad id or segment table."""
        perm = np.zeros(self.max_tokens, np.int32)
        starts = np.zeros(self.max_tokens + 1, np.int32)
        adapter = np.zeros(self.max_tokens, np.int32)
        ns, nt = C.c_int32(0), C.c_int32(0)
        check(_lib.lib().b200_lora_plan_read(
            self.buf.data_ptr(), perm.ctypes.data, starts.ctypes.data, adapter.ctypes.data,
            C.byref(ns), C.byref(nt), _stream(self.buf.device)), "plan_read")
        return perm[:nt.value], starts[:ns.value + 1], adapter[:ns.value]


class LoraWorkspace:
    """Scratch for the ``[T, r]`` intermediate and the split-K partial sums."""

    def check(self) -> None:
        """Synchronises and raises if a kernel recorded a device-side error (expired wait)."""
        check(_lib.lib().b200_lora_workspace_status(self.buf.data_ptr(), _stream(self.buf.device)),
              "workspace_status")

    def __init__(self, max_tokens: int, n_proj: int, max_h_in: int, device="cuda"):
        self.max_tokens, self.n_proj, self.max_h_in = int(max_tokens), int(n_proj), int(max_h_in)
        nbytes = _lib.lib().b200_lora_workspace_bytes(self.max_tokens, self.n_proj, self.max_h_in)
        if nbytes == 0:
            raise ValueError("bad workspace dimensions")
        # 128-byte aligned base: the library's layout aligns v relative to the base address
        raw = torch.empty(nbytes + 128, dtype=torch.uint8, device=device)
        skew = (-raw.data_ptr()) % 128
        self._raw = raw
        self.buf = raw[skew: skew + nbytes]
        self.nbytes = nbytes
        # the control words and v start at zero; the split-K partials behind them (30 times the size) are
        # written before they are read
        off, size = self._v_region()
        self.buf[:off + size].zero_()

    def _v_region(self) -> Tuple[int, int]:
        off, size = C.c_size_t(0), C.c_size_t(0)
        check(_lib.lib().b200_lora_workspace_v_region(self.max_tokens, self.n_proj, C.byref(off), C.byref(size)),
              "workspace_v_region")
        return off.value, size.value

    def v_view(self) -> torch.Tensor:
        """The fp32 shrink result ``v [n_proj, max_tokens, 64]`` inside the workspace
        (what tensor-parallel ranks sum between the shrink and the expand half)."""
        off, size = self._v_region()
        return self.buf[off: off + size].view(torch.float32).view(self.n_proj, self.max_tokens, 64)


def apply(projs: Sequence[Tuple[torch.Tensor, torch.Tensor, AdapterPool]], plan: LoraPlan, layer: int,
          workspace: LoraWorkspace, flags: int = 0, adapters: Optional[Adapters] = None, tp_ctx=None,
          skip_arrival: bool = False) -> None:
    """``y += scale_a * (x @ A_a^T) @ B_a^T`` for up to four projections ``(x, y, pool)`` of one layer.

    All pools must share one adapter table (ranks, scalings, layout).  With ``tp_ctx`` (the library's
    peer-exchange context of a tensor-parallel rank) the call is ``b200_lora_apply_tp``: ``x``, ``y`` and the
    pools are this rank's shards and the shrink result is summed over the ranks inside the call."""
    if tp_ctx is None:
        rc = _lib.host().apply(projs, plan, layer, workspace, flags, adapters)
        if rc <= 0:
            check(rc, "apply")
            return
    if not 1 <= len(projs) <= _lib.MAX_PROJ:
        raise ValueError("1..4 projections per call")
    arr = (Proj * len(projs))()
    io = None
    ydt = None
    for i, (x, y, pool) in enumerate(projs):
        _require_cuda(x, y, pool.wa)
        if x.dim() != 2 or y.dim() != 2 or x.shape[0] != y.shape[0]:
            raise ValueError("x and y must be [T, h] with the same T")
        if x.stride(1) != 1 or y.stride(1) != 1:
            raise ValueError("x and y rows must be contiguous")
        if x.shape[1] != pool.h_in or y.shape[1] != pool.h_out:
            raise ValueError("x/y widths do not match the pool")
        if x.dtype != pool.wa.dtype or x.dtype not in (torch.float16, torch.bfloat16):
            raise ValueError("x and the pool must both be fp16 or both bf16")
        if io is None:
            io, ydt = x.dtype, y.dtype
        if x.dtype != io or y.dtype != ydt or ydt not in (io, torch.float32):
            raise ValueError("all projections share the I/O dtype; y is that dtype or fp32")
        if x.shape[0] != plan.n_tokens:
            raise ValueError(f"the plan was built for {plan.n_tokens} rows, x has {x.shape[0]}")
        arr[i] = Proj(x.data_ptr(), y.data_ptr(), pool.wa.data_ptr(), pool.wb.data_ptr(),
                      x.stride(0), y.stride(0), pool.h_in, pool.h_out)
    ad = adapters if adapters is not None else adapters_of(projs[0][2])
    if tp_ctx is not None:
        check(_lib.lib().b200_lora_apply_tp(
            arr, len(projs), C.byref(ad), plan.buf.data_ptr(), plan.max_tokens, int(projs[0][0].shape[0]), int(layer),
            _DT[io], _DT[ydt], int(flags), workspace.buf.data_ptr(), workspace.nbytes, C.byref(tp_ctx),
            1 if skip_arrival else 0, _stream(projs[0][0].device)), "apply_tp")
        return
    check(_lib.lib().b200_lora_apply(
        arr, len(projs), C.byref(ad), plan.buf.data_ptr(), plan.max_tokens, int(projs[0][0].shape[0]), int(layer),
        _DT[io], _DT[ydt],
        int(flags), workspace.buf.data_ptr(), workspace.nbytes, _stream(projs[0][0].device)), "apply")


# ---- the reference's operator call ---------------------------------------------------------------
_OP_STATE = {}                       # (device, stream, capture) -> (LoraBatch, capacity: tokens, adapters, h_in)
_OP_LOCK = threading.Lock()


def invalidate_plan_cache() -> None:
    """Forget the plans :func:`add_lora_bgmv` keeps.  Needed only after the contents of an index
    tensor were changed behind torch's back (a custom kernel or a raw pointer write, which do not
    bump the tensor's version counter)."""
    _lib.host().bgmv_forget()


def _op_state(ids: torch.Tensor, t: int, n: int, h_in: int) -> None:
    """Makes the plan and workspace behind :func:`add_lora_bgmv` for the current stream large enough.

    The reference's decode loop calls the op 3 x n_layers times per step with the SAME index tensor
    (lightllm/models/lora_gpu.py:138,150,162 with ``select_inds[bsz-1]``).  The plan depends on
    the ids, N, r and the scale only, so it is kept while the very same tensor is passed again
    unmodified (torch's version counter) and rebuilt otherwise.  Every CUDA-graph capture has a plan and
    workspace of its own, allocated inside it (so that the graph's memory pool owns them), and contains the
    build of the plan it applies (its first call): replays rebuild it from the index tensor's contents of the
    moment and touch nothing that eager calls or other graphs use.  The key lives in the native host path;
    the memory is held here, an ended capture's until the stream's next entry is made."""
    dev = ids.device.index
    stream, capture = _lib.host().stream_key(ids)
    with _OP_LOCK:
        for key in [k for k in _OP_STATE if k[:2] == (dev, stream) and k[2] not in (0, capture)]:
            del _OP_STATE[key]
        _, old = _OP_STATE.get((dev, stream, capture), (None, (0, 0, 0)))
        dims = (max(t, old[0]), max(n, old[1]), max(h_in, old[2]))
        if dims == old:                  # another thread has made it meanwhile
            return
        batch = LoraBatch(*dims, 1, ids.device)
        # registered before the old memory goes: no call can still be enqueueing with that then
        _lib.host().bgmv_register(stream, dev, capture, batch.plan.buf.data_ptr(), batch.plan.nbytes,
                                  batch.workspace.buf.data_ptr(), batch.workspace.nbytes, *dims)
        _OP_STATE[dev, stream, capture] = (batch, dims)


def add_lora_bgmv(y: torch.Tensor, x: torch.Tensor, wa_T_all: torch.Tensor, wb_T_all: torch.Tensor,
                  indicies: torch.Tensor, layer_idx: int, scale: float) -> None:
    """In place ``y[t] += scale * (x[t] @ wa_T_all[i_t, layer]^T) @ wb_T_all[i_t, layer]^T``.

    Same arguments as the reference's decode op: ``y [T, h_out]``, ``x [T, h_in]``,
    ``wa_T_all [N, L, r, h_in]``, ``wb_T_all [N, L, h_out, r]`` contiguous fp16/bf16 CUDA
    tensors, ``indicies [T]`` int64 (or int32) CUDA tensor.  Returns ``None``.

    One launch for a few tokens (a cluster per token, as many as run at once), else two (shrink, expand), when
    the index tensor is the one of the previous call on this stream, unmodified; one more (the plan kernel) when it is new.
    """
    rc = _lib.host().bgmv(y, x, wa_T_all, wb_T_all, indicies, layer_idx, scale)
    if rc <= 0:
        check(rc, "add_lora_bgmv")
        return
    _require_cuda(y, x, wa_T_all, wb_T_all, indicies)
    if wa_T_all.dim() != 4 or wb_T_all.dim() != 4:
        raise ValueError("weight pools must be [N, L, r, h_in] and [N, L, h_out, r]")
    n, l, r, h_in = wa_T_all.shape
    h_out = wb_T_all.shape[2]
    if tuple(wb_T_all.shape) != (n, l, h_out, r):
        raise ValueError("wa_T_all / wb_T_all shapes disagree")
    t = x.shape[0]
    if tuple(x.shape) != (t, h_in) or tuple(y.shape) != (t, h_out) or indicies.numel() != t:
        raise ValueError("x, y, indicies shapes disagree with the pools")
    for ten in (y, x, wa_T_all, wb_T_all, indicies):
        if not ten.is_contiguous():
            raise ValueError("add_lora_bgmv needs contiguous tensors")
    if not (y.dtype == x.dtype == wa_T_all.dtype == wb_T_all.dtype) or x.dtype not in (torch.float16, torch.bfloat16):
        raise ValueError("fp16 or bf16 tensors of one dtype expected")
    if indicies.dtype not in (torch.int32, torch.int64):
        raise ValueError("indicies must be int32 or int64")
    _op_state(indicies, t, n, h_in)
    rc = _lib.host().bgmv(y, x, wa_T_all, wb_T_all, indicies, int(layer_idx), float(scale))
    if rc > 0:
        raise ValueError("add_lora_bgmv: unsupported arguments")
    check(rc, "add_lora_bgmv")


def add_lora_bgmv_once(y: torch.Tensor, x: torch.Tensor, wa_T_all: torch.Tensor, wb_T_all: torch.Tensor,
                       indicies: torch.Tensor, layer_idx: int, scale: float, workspace: torch.Tensor) -> None:
    """The same op as ONE C-ABI call (``b200_add_lora_bgmv``): plan and scratch live in the
    caller's ``workspace`` (any dtype, ``b200_add_lora_bgmv_workspace_bytes`` bytes or more, no
    preparation needed) and the plan is rebuilt by every call.  For bindings that cannot keep
    state between calls; tensors as for :func:`add_lora_bgmv`, shapes are not re-validated."""
    _require_cuda(y, x, wa_T_all, wb_T_all, indicies, workspace)
    n, l, r, h_in = wa_T_all.shape
    h_out = wb_T_all.shape[2]
    t = x.shape[0]
    check(_lib.lib().b200_add_lora_bgmv(
        y.data_ptr(), x.data_ptr(), wa_T_all.data_ptr(), wb_T_all.data_ptr(), indicies.data_ptr(),
        1 if indicies.dtype == torch.int64 else 0, t, h_in, h_out, n, l, r, int(layer_idx), float(scale),
        _DT[x.dtype], workspace.data_ptr(), workspace.numel() * workspace.element_size(), _stream(x.device)),
        "add_lora_bgmv")


def add_lora_bgmv_workspace_bytes(n_tokens: int, n_adapters: int, h_in: int) -> int:
    return int(_lib.lib().b200_add_lora_bgmv_workspace_bytes(n_tokens, n_adapters, h_in))


def add_lora_bgmv_static(y: torch.Tensor, x: torch.Tensor, wa_T_all: torch.Tensor, wb_T_all: torch.Tensor,
                         indicies: torch.Tensor, layer_idx: int, scale: float) -> None:
    """``add_lora_bgmv`` for callers that must not allocate device memory.

    Same arguments and result as :func:`add_lora_bgmv`, but the library's built-in scratch
    array is used instead of a workspace tensor, so nothing is allocated - not by this wrapper
    either.  Meant for processes that have given all of HBM to their KV cache or that may not
    call ``cudaMalloc`` after start-up.  Accepts at most 64 tokens, 1024 adapters and
    ``h_in <= 8192`` (larger calls raise).  All calls on a GPU share that one array: issue them
    on one stream, or order the streams, because overlapping calls race.  Make the first call
    on a device outside stream capture (it performs a one-time address lookup)."""
    rc = _lib.host().bgmv_static(y, x, wa_T_all, wb_T_all, indicies, layer_idx, scale)
    if rc <= 0:
        check(rc, "add_lora_bgmv_static")
        return
    _require_cuda(y, x, wa_T_all, wb_T_all, indicies)
    n, l, r, h_in = wa_T_all.shape
    h_out = wb_T_all.shape[2]
    t = x.shape[0]
    if tuple(wb_T_all.shape) != (n, l, h_out, r) or tuple(x.shape) != (t, h_in) or tuple(y.shape) != (t, h_out) \
            or indicies.numel() != t:
        raise ValueError("x, y, indicies shapes disagree with the pools")
    for ten in (y, x, wa_T_all, wb_T_all, indicies):
        if not ten.is_contiguous():
            raise ValueError("add_lora_bgmv_static needs contiguous tensors")
    if not (y.dtype == x.dtype == wa_T_all.dtype == wb_T_all.dtype) or x.dtype not in (torch.float16, torch.bfloat16):
        raise ValueError("fp16 or bf16 tensors of one dtype expected")
    if indicies.dtype not in (torch.int32, torch.int64):
        raise ValueError("indicies must be int32 or int64")
    rc = _lib.host().bgmv_static(y, x, wa_T_all, wb_T_all, indicies, int(layer_idx), float(scale))
    if rc > 0:
        raise ValueError("add_lora_bgmv_static: unsupported arguments")
    check(rc, "add_lora_bgmv_static")


def add_lora_bgmv_static_status(device=None) -> None:
    """Synchronises and raises if the last :func:`add_lora_bgmv_static` call on ``device`` saw an
    adapter id out of range (that call left ``y`` unchanged) or an expired device-side wait."""
    dev = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    with torch.cuda.device(dev):
        check(_lib.lib().b200_add_lora_bgmv_static_status(_stream(dev)), "add_lora_bgmv_static_status")


class LoraBatch:
    """Plan + workspace of one batch, reused across layers and projections."""

    def __init__(self, max_tokens: int, n_adapters: int, max_h_in: int, n_proj: int = 4, device="cuda"):
        self.plan = LoraPlan(max_tokens, n_adapters, device)
        self.workspace = LoraWorkspace(max_tokens, n_proj, max_h_in, device)
        self.tiles = False

    def set_ids(self, ids: torch.Tensor, pool: AdapterPool, tiles: bool = False) -> "LoraBatch":
        """Per-token adapter ids.  ``tiles=True`` also launches the tcgen05 tile kernel for
        tall contiguous runs (mixed prefill + decode batches); decode batches leave it off."""
        self.plan.build(ids, pool)
        self.tiles = tiles
        return self

    def set_segments(self, seg_starts, seg_adapter, n_tokens, pool: AdapterPool, tiles: bool = True) -> "LoraBatch":
        self.plan.from_segments(seg_starts, seg_adapter, n_tokens, pool)
        self.tiles = tiles
        return self

    def apply(self, projs, layer: int, flags: int = 0, tp_ctx=None, skip_arrival: bool = False) -> None:
        if not self.tiles:
            flags |= _lib.NO_TENSOR
        apply(projs, self.plan, layer, self.workspace, flags, tp_ctx=tp_ctx, skip_arrival=skip_arrival)


def add_lora_bgmv_v2(y, x, pool: AdapterPool, indicies, layer_idx: int, flags: int = 0) -> None:
    """BGMV with per-adapter ranks and scalings taken from ``pool`` (dense or packed)."""
    b = LoraBatch(x.shape[0], pool.n_adapters, pool.h_in, 1, x.device).set_ids(indicies, pool)
    b.apply([(x, y, pool)], layer_idx, flags)


def add_lora_sgmv(y, x, pool: AdapterPool, seg_starts, seg_adapter, layer_idx: int, flags: int = 0) -> None:
    """SGMV on adapter-sorted rows: segment ``s`` = rows ``[seg_starts[s], seg_starts[s+1])``."""
    b = LoraBatch(x.shape[0], pool.n_adapters, pool.h_in, 1, x.device)
    b.set_segments(seg_starts, seg_adapter, x.shape[0], pool)
    b.apply([(x, y, pool)], layer_idx, flags)
