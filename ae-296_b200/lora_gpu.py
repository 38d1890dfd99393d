"""Host-side mirror of the reference's GPU LoRA layer object.

``Lora_GPU`` keeps the constructor keys, attribute names and the three
``invoke_one_layer_{q,k,v}(x, layer_id, prefill=False)`` methods of
lightllm/models/lora_gpu.py:16-163, so the layer-infer code
(lightllm/models/llama/layer_infer/transformer_layer_infer.py:101-111) can call it
unchanged.  Differences, all on purpose:

* the decode op is this package's CUDA BGMV instead of ``punica.ops.add_lora_bgmv``, with one
  plan per batch size and stream (built once per ``set_indices``, not per call) and q/k/v of a layer computed in one fused pass;
* prefill uses the same kernels on request-aligned segments (slot ``b`` <-> request ``b``)
  instead of two ``torch.bmm`` calls and two transposed copies; ``prefill_mid_round``
  reproduces that op's fp16 rounding of the ``[B, L, r]`` intermediate;
* adapter ids come from ``set_indices`` (the reference draws random ids once,
  lora_gpu.py:120, reading past its pool when ``batch_size < 32``);
* no sockets, no swapper, no process exit on error: errors raise.
"""
from __future__ import annotations

from typing import Optional

import torch

import numpy as np

from . import _lib
from .ops import LoraBatch, _adapters_struct, apply
from .pool import AdapterPool


class _Kept:
    """A plan + workspace that calls of one kind keep, and what the plan was built from."""

    def __init__(self, batch: LoraBatch, rows: int):
        self.batch, self.rows = batch, rows
        self.built = None


class Lora_GPU:
    def __init__(self, configJson, shared: bool = False, dtype=torch.float16, prefill_mid_round: bool = True):
        self.device = torch.cuda.current_device()
        self.n_layers = configJson["n_layers"]
        self.batch_size = configJson["batch_size"]
        self.lora_rank = configJson["lora_rank"]
        self.in_size = configJson["hidden_dim"]
        self.tp_degree = configJson["tp_degree"]
        self.output_size = configJson["hidden_dim"] // self.tp_degree
        self.max_prefill_batch_size = configJson["max_prefill_batch_size"]
        self.prefill_mid_round = prefill_mid_round
        dev = f"cuda:{self.device}"

        def pool(n, scale):
            down = (torch.randn(n, self.n_layers, self.lora_rank, self.in_size, device=dev) * scale).to(dtype)
            up = (torch.randn(n, self.n_layers, self.output_size, self.lora_rank, device=dev) * scale).to(dtype)
            return down, up

        # decode pools: [N, L, r, H] and [N, L, H/tp, r]   (lora_gpu.py:33-40)
        self.q_down, self.q_up = pool(self.batch_size, 0.001)
        self.k_down, self.k_up = pool(self.batch_size, 0.001)
        self.v_down, self.v_up = pool(self.batch_size, 0.001)
        # prefill slots (lora_gpu.py:54-72)
        self.q_down_prefill, self.q_up_prefill = pool(self.max_prefill_batch_size, 0.001)
        self.k_down_prefill, self.k_up_prefill = pool(self.max_prefill_batch_size, 0.001)
        self.v_down_prefill, self.v_up_prefill = pool(self.max_prefill_batch_size, 0.001)
        g = torch.Generator(device=dev).manual_seed(0)
        self.select_inds = [torch.randint(0, self.batch_size, (i + 1,), device=dev, generator=g)
                            for i in range(self.batch_size)]

        def view(down, up, n):       # the reference's tensors described as a dense pool of uniform rank
            return AdapterPool(down, up, None, None, None, n, self.n_layers, self.in_size, self.output_size,
                               self.lora_rank, False, np.full(n, self.lora_rank, np.int32),
                               np.arange(n + 1, dtype=np.int64) * self.lora_rank)

        self._decode_pools = [view(d, u, self.batch_size) for d, u in
                              ((self.q_down, self.q_up), (self.k_down, self.k_up), (self.v_down, self.v_up))]
        self._prefill_pools = [view(d, u, self.max_prefill_batch_size) for d, u in
                               ((self.q_down_prefill, self.q_up_prefill), (self.k_down_prefill, self.k_up_prefill),
                                (self.v_down_prefill, self.v_up_prefill))]
        self._ad_decode = _adapters_struct(self.batch_size, self.n_layers, self.lora_rank, scale=1.0)
        self._ad_prefill = _adapters_struct(self.max_prefill_batch_size, self.n_layers, self.lora_rank, scale=1.0)
        # Plan + workspace per (decode batch size, or None for prefill; stream; graph capture or 0), so that a
        # step on another stream, and every replay of a graph, which builds its plan again, leaves this one's alone.
        self._kept = {}
        self._use_key = _lib.host().use_key
        self._indices_version = {}       # decode batch size -> how often set_indices has set it
        self._fused = None               # (use of x, layer, prefill) -> the k and v deltas computed with q

    def set_indices(self, indices: torch.Tensor) -> None:
        """Adapter slot of each decode token for batches of ``len(indices)`` tokens.  A captured graph goes on
        with the index tensor that it was captured with (its contents at each replay), which the caller keeps."""
        bsz = indices.numel()
        self.select_inds[bsz - 1] = indices.to(device=f"cuda:{self.device}")
        self._indices_version[bsz] = self._indices_version.get(bsz, 0) + 1
        self._fused = None

    def _keep(self, x, where, kind, rows, n_adapters) -> _Kept:
        """What is kept for calls of ``kind`` on the stream and in the capture ``where``, with room for ``rows``.  A capture's is allocated inside it, so its memory belongs to the graph's pool; the
        reference here goes when the stream, which is in one capture at a time, makes its next."""
        kept = self._kept.get((kind, where))
        if kept is None or kept.rows < rows:
            for key in [k for k in self._kept if k[1][0] == where[0] and k[1][1] not in (0, where[1])]:
                del self._kept[key]
            kept = self._kept[kind, where] = _Kept(LoraBatch(rows, n_adapters, self.in_size, 3, x.device), rows)
        return kept

    # ---- the three calls the layer code makes ------------------------------------------
    # The layer code asks for q, k and v of one layer in that order with the same input
    # (lightllm/models/llama/layer_infer/transformer_layer_infer.py:108-111).  The q call computes
    # all three deltas in one fused pass (x is read once, one shrink and one expand launch instead
    # of three each) and the k and v calls hand out their parts; a k or v call that does not follow
    # such a q call, on the same stream and in the same graph capture, computes its own.
    def _invoke(self, which, x, layer_id, prefill):
        use = self._use_key(x)
        key = (use, int(layer_id), bool(prefill))
        if which > 0 and self._fused is not None and self._fused[0] == key:
            out = self._fused[1][which]
            if which == 2:
                self._fused = None
            return out
        projs = (0, 1, 2) if which == 0 else (which,)
        ys = (self._prefill if prefill else self._decode)(x, use[0], layer_id, projs)
        if which == 0:
            self._fused = (key, ys)
        return ys[which]

    def invoke_one_layer_q(self, x, layer_id, prefill=False):
        return self._invoke(0, x, layer_id, prefill)

    def invoke_one_layer_k(self, x, layer_id, prefill=False):
        return self._invoke(1, x, layer_id, prefill)

    def invoke_one_layer_v(self, x, layer_id, prefill=False):
        return self._invoke(2, x, layer_id, prefill)

    def _decode(self, x, where, layer_id, projs):
        """x ``[bsz, H]``; token ``t`` uses slot ``select_inds[bsz-1][t]`` (lora_gpu.py:137-138)."""
        bsz = x.shape[0]
        kept = self._keep(x, where, bsz, bsz, self.batch_size)
        batch = kept.batch
        version = self._indices_version.get(bsz, 0)
        if kept.built != version:
            batch.plan.build(self.select_inds[bsz - 1], self._ad_decode)
            kept.built = version
        y = x.new_empty((3, bsz, self.output_size)).unbind(0)
        apply([(x, y[i], self._decode_pools[i]) for i in projs], batch.plan, layer_id, batch.workspace,
              _lib.NO_TENSOR | _lib.OVERWRITE, self._ad_decode)
        return y                         # only those of `projs` hold anything

    def _prefill(self, x, where, layer_id, projs):
        """x ``[B, L, H]``: request ``b`` uses prefill slot ``b`` (lora_gpu.py:125-128).  One plan +
        workspace (per stream) serves every shape: it grows to the largest batch seen and the segment table is
        rebuilt (one small kernel) when ``(B, L)`` changes, so nothing accumulates per shape."""
        bsz, seqlen, hidden = x.shape
        rows = bsz * seqlen
        kept = self._keep(x, where, None, rows, self.max_prefill_batch_size)
        batch = kept.batch
        if kept.built != (bsz, seqlen):
            starts = torch.arange(0, (bsz + 1) * seqlen, seqlen, dtype=torch.int32, device=x.device)
            slots = torch.arange(bsz, dtype=torch.int32, device=x.device)
            batch.plan.from_segments(starts, slots, rows, self._ad_prefill)
            kept.built = (bsz, seqlen)
        y = x.new_empty((3, rows, self.output_size)).unbind(0)
        flags = _lib.OVERWRITE | (_lib.MID_ROUND if self.prefill_mid_round else 0)
        x2 = x.reshape(rows, hidden)
        apply([(x2, y[i], self._prefill_pools[i]) for i in projs], batch.plan, layer_id, batch.workspace, flags,
              self._ad_prefill)
        return {i: y[i].view(bsz, seqlen, self.output_size) for i in projs}
