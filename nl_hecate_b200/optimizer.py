"""Flat-arena AdamW for the outer parameters.

Host-side mirror of the per-tensor loop in
core/src/gpu_stacked_optimizer.rs:522-683 (``gpu_stacked_adamw_update``) and of
``FrequencyAwareAdamW::step`` (core/src/adamw.rs:195-395): all parameters, their
gradients and both moments live in four flat fp32 arenas with one layout, so
that the step is ONE global-norm reduction and ONE multi-tensor kernel (and,
data-parallel, ONE all-reduce over ``g``). Per-tensor state that the reference
keeps in separate launches travels in a descriptor table: the tensor's own
bias corrections (shared tensors use the global step, CMS level tensors their
level's fire count), whether it is active this step (pulse gating), and the
post-update clamp (``b_theta`` in [-10, 2]).
"""
from __future__ import annotations

import numpy as np
import torch

from . import ffi
from .dispatch import call

CHUNK = 8192  # elements per CTA work item
RING = 4      # steps of descriptors that may be in flight
_DESC = np.dtype(ffi.AdamWTensorDesc)


class FlatAdamW:
    def __init__(self, sizes, device="cuda", beta1=0.9, beta2=0.999, eps=1e-8, weight_decay=0.1,
                 clamp=None, no_decay=()):
        self.sizes = [int(s) for s in sizes]
        self.beta1, self.beta2, self.eps, self.weight_decay = beta1, beta2, eps, weight_decay
        self.clamp = dict(clamp or {})
        self.no_decay = set(no_decay)
        self.slices = []
        off = 0
        for n in self.sizes:
            self.slices.append((off, n))
            off += (n + 7) // 8 * 8          # 32-byte aligned in fp32, 16-byte aligned in a bf16 shadow of the arena
        self.arena_len = max(off, 4)
        dev = torch.device(device)
        z = lambda: torch.zeros(self.arena_len, dtype=torch.float32, device=dev)
        self.w, self.g, self.m, self.v = z(), z(), z(), z()
        ct, cs, cl = [], [], []
        for ti, (o, n) in enumerate(self.slices):
            for c0 in range(0, n, CHUNK):
                ct.append(ti); cs.append(o + c0); cl.append(min(CHUNK, n - c0))
        self.n_chunks = len(ct)
        self.chunk_tensor = torch.tensor(ct, dtype=torch.int32, device=dev)
        self.chunk_start = torch.tensor(cs, dtype=torch.int64, device=dev)
        self.chunk_len = torch.tensor(cl, dtype=torch.int32, device=dev)
        # Per-tensor descriptors of one step. The table travels through a small ring of pinned host rows:
        # prepare() fills the next one while the GPU may still have to read the previous ones, so the
        # host runs ahead of the device.
        nt = len(self.sizes)
        pinned = torch.zeros(RING, nt * _DESC.itemsize, dtype=torch.uint8)
        if dev.type == "cuda":
            pinned = pinned.pin_memory()
        self._desc_ring = pinned
        self._desc_rows = pinned.numpy().view(_DESC)
        self._row_options = [None] * RING      # the (weight_decay, no_decay, clamp) that a row was filled with
        self._desc_dev = torch.empty(nt * _DESC.itemsize, dtype=torch.uint8, device=dev)
        self._partial = torch.empty(148 * 8, dtype=torch.float32, device=dev)
        self.norm = torch.zeros(1, dtype=torch.float32, device=dev)
        self.scale = torch.ones(1, dtype=torch.float32, device=dev)
        # one event per ring row, recorded after the stream-ordered upload of that row; prepare()
        # waits on it before it rewrites the row, so a host that runs ahead of the GPU cannot
        # replace step t's descriptors before step t's copy has read them
        self._uploaded = [torch.cuda.Event() for _ in range(RING)] if dev.type == "cuda" else None
        self._row_busy = [False] * RING
        self._row = 0
        self._captured_row = None      # set when a graph captured the upload of a row: that row is then reused
        self._on_device = False        # the caller uploaded the prepared row itself

    def view(self, arena: torch.Tensor, i: int) -> torch.Tensor:
        o, n = self.slices[i]
        return arena[o:o + n]

    def prepare(self, steps, active=None, lr_scale=1.0):
        """Host part of a step: fill the next row of the descriptor ring (bias corrections from each
        tensor's own 1-based step count, activity, learning-rate scale). The device reads it after
        launch() or upload(); a row is rewritten only when the upload that last used it has completed. A
        graph that captured launch() without an upload() before it reads the same row at every replay:
        its caller waits for a replay before it prepares the next one."""
        nt = len(self.sizes)
        if nt and type(steps) is list and len(steps) >= nt and steps[:nt].count(steps[0]) == nt:   # one count for all
            t = [max(int(steps[0]), 1)]
        else:
            t = [max(int(steps[i]), 1) for i in range(nt)]
        bc = {x: (1.0 / (1.0 - self.beta1 ** x), 1.0 / (1.0 - self.beta2 ** x)) for x in set(t)}
        act = [1] if active is None else [bool(active[i]) for i in range(nt)]
        r = (self._row + 1) % RING if self._captured_row is None else self._captured_row
        if self._row_busy[r]:
            self._uploaded[r].synchronize()
            self._row_busy[r] = False
        row = self._desc_rows[r]
        row["bc1_inv"] = [bc[x][0] for x in t]
        row["bc2_inv"] = [bc[x][1] for x in t]
        row["lr_scale"] = lr_scale
        row["active"] = act
        options = (self.weight_decay, self.no_decay, self.clamp)
        if options != self._row_options[r]:     # these rarely change: compared, not rewritten, each step
            row["weight_decay"] = [0.0 if i in self.no_decay else self.weight_decay for i in range(nt)]
            row["clamp_lo"] = [self.clamp[i][0] if i in self.clamp else 0.0 for i in range(nt)]
            row["clamp_hi"] = [self.clamp[i][1] if i in self.clamp else 0.0 for i in range(nt)]
            row["has_clamp"] = [i in self.clamp for i in range(nt)]
            self._row_options[r] = (self.weight_decay, set(self.no_decay), dict(self.clamp))
        self._row = r
        self._on_device = False

    def upload(self):
        """Stream-ordered copy of the prepared descriptors to the device, for a caller that replays a
        captured launch(): with an upload() before the capture and before every replay the graph holds no
        copy from a fixed host row. launch() uploads by itself what the caller has not."""
        self._upload()
        self._on_device = True

    def _upload(self):
        r = self._row
        self._desc_dev.copy_(self._desc_ring[r], non_blocking=True)
        if self._uploaded is None:
            pass
        elif torch.cuda.is_current_stream_capturing():
            self._captured_row = r
        else:
            self._uploaded[r].record()
            self._row_busy[r] = True

    def launch(self, lr, max_grad_norm=0.0):
        """Device part of a step (stream-ordered, capturable in a CUDA graph): descriptor upload,
        global-norm clip scale, multi-tensor AdamW. Returns the device scalar with the pre-clip
        gradient norm (valid only when max_grad_norm > 0)."""
        if not self._on_device:
            self._upload()
        scale_ptr = None
        if max_grad_norm > 0.0:
            call("nlh_arena_grad_norm_clip", g=self.g, n=self.arena_len,
                 max_grad_norm=max_grad_norm, partial=self._partial,
                 partial_capacity=self._partial.numel(), out_norm=self.norm, out_scale=self.scale)
            scale_ptr = self.scale
        call("nlh_adamw_multi_tensor", w=self.w, g=self.g, m=self.m, v=self.v,
             descs_dev=self._desc_dev, chunk_tensor_dev=self.chunk_tensor,
             chunk_start_dev=self.chunk_start, chunk_len_dev=self.chunk_len,
             n_chunks=self.n_chunks, grad_scale_ptr=scale_ptr, lr=lr, beta1=self.beta1,
             beta2=self.beta2, eps=self.eps)
        return self.norm

    def step(self, lr, steps, active=None, max_grad_norm=0.0):
        """One optimizer step. ``steps[i]`` is tensor i's own 1-based step count (bias
        correction), ``active[i]`` False skips it."""
        self.prepare(steps, active)
        return self.launch(lr, max_grad_norm)
