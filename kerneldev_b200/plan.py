"""Attention plans: the per-batch product of the tile classifier.

A plan holds the packed token descriptors, the class (EMPTY / FULL / PARTIAL) of every
128x128 tile of the mask and the work lists the kernels walk. It depends only on the
metadata (``in_span``, ``span_id``, ``is_prefix``, ``lens``, ``causal``), not on the head, so one
plan serves all heads and -- because ``model.GPTModel`` passes the same three metadata tensors
to every layer (model.py:243-244) -- all layers of a step. Plans are cached on the identity and
version of the metadata tensors (the cache keeps their memory alive, so an address cannot be
reused while its plan is cached; a plan whose metadata nobody else holds any more leaves the cache with the next new plan). A CUDA
graph keeps the plans that its launches read, whatever becomes of the cache. Metadata rewritten in place through raw pointers -- by
kd_metadata_from_tokens into preallocated buffers, or through ``.data`` -- does not change a tensor's
version: call ``clear_plan_cache()`` after such a write.

The plans and their cache live in the host extension (csrc/host.cpp); ``AttentionPlan`` is the view of one
of them from Python.

Device status. Kernels report problems (a bounded wait that ran out, a span id out of range) in the
plan's status word and, in the same breath, in a pinned host mirror whose address the plan carries; the
next call that uses the plan (or ``poll()``) looks at the mirror without synchronising and raises, so a
failed launch surfaces one call later at the latest -- normally at the backward of the same step. The
words of the last 64 plans that left the cache for newer ones are looked at whenever a plan is made for it: what the
last launch of a step reports surfaces with a later step's new metadata. A
launch that succeeds costs no copy. ``KD_CHECK_STATUS=1`` makes every call synchronise and check at once.
"""
from __future__ import annotations

import ctypes
import weakref

import torch

from . import _capi, _host

_ext = _host.load()


class AttentionPlan:
    """Device-resident plan for B sequences of T tokens (layout: kd_plan_layout in kd_attention.h)."""

    def __init__(self, B, T, device, in_span=None, span_id=None, is_prefix=None, lens=None,
                 causal=True, rules=False):
        device = torch.device(device)
        if device.index is None:
            device = torch.device(device.type, torch.cuda.current_device())
        self._bind(_ext.Plan(B, T, device, in_span, span_id, is_prefix, lens, bool(causal), bool(rules)))

    def _bind(self, core):
        self._core = core
        self.B, self.T, self.device, self.buf = core.B, core.T, core.device, core.buf
        self.layout = _capi.plan_layout(self.B, self.T)
        self.NT, self.NP = self.layout.NT, self.layout.NP
        self._status_dev, self._status_host = core.status_dev, core.status_host

    @classmethod
    def _of(cls, core):
        """The one Python view of a plan of the extension (while somebody holds it)."""
        plan = _VIEWS.get(core)
        if plan is None:
            plan = object.__new__(cls)
            plan._bind(core)
            _VIEWS[core] = plan
        return plan

    # ---- views into the plan buffer -------------------------------------------------------------
    def _view(self, off, nbytes, dtype, shape):
        return self.buf[off:off + nbytes].view(dtype).view(shape)

    @property
    def ptr(self) -> int:
        return self.buf.data_ptr()

    @property
    def desc(self) -> torch.Tensor:
        n = self.B * self.NT * _capi.KD_TILE
        return self._view(self.layout.off_desc, n * 4, torch.int32, (self.B, self.NT * _capi.KD_TILE))

    @property
    def tile_classes(self) -> torch.Tensor:
        """uint8 (B, NT, NT): class of tile [b][q_tile][k_tile]."""
        n = self.B * self.NT * self.NT
        return self._view(self.layout.off_cls, n, torch.uint8, (self.B, self.NT, self.NT))

    @property
    def stats(self) -> torch.Tensor:
        """int32 (B, 2): number of FULL and PARTIAL tiles per sequence."""
        return self._view(self.layout.off_stats, self.B * 8, torch.int32, (self.B, 2))

    @property
    def fwd_counts(self) -> torch.Tensor:
        return self._view(self.layout.off_fwd_cnt, self.B * self.NP * 4, torch.int32, (self.B, self.NP))

    @property
    def bwd_counts(self) -> torch.Tensor:
        return self._view(self.layout.off_bwd_cnt, self.B * self.NT * 4, torch.int32, (self.B, self.NT))

    def use_on_current_stream(self) -> None:
        """Orders the current stream after the classifier when the plan was built on another one."""
        self._core.use_on_current_stream()

    def status(self) -> int:
        """Reads the device status word (synchronises the current stream)."""
        return int(self._status_dev.item()) & 0xFFFFFFFF

    def mirror_status(self) -> None:
        """Enqueues a copy of the status word to the pinned host mirror (kernels write the mirror themselves)."""
        self._status_host.copy_(self._status_dev, non_blocking=True)

    def poll(self) -> None:
        """Raises if the host mirror holds a status a finished launch reported. Never synchronises."""
        s = int(self._status_host[0]) & 0xFFFFFFFF
        if s:
            self._report(s)

    def check_status(self) -> None:
        """Synchronises the current stream, reads the device status word and raises if it is set."""
        s = self.status()
        if s:
            self._report(s)

    def _report(self, s: int) -> None:
        # the word is cleared so that one event is reported once and later launches start clean
        self._status_dev.zero_()
        self._status_host.zero_()
        if s & _capi.KD_STATUS_SPAN_RANGE:
            raise ValueError("span_id values must fit in 24 signed bits (|span_id| < 2**23)")
        if s & _capi.KD_STATUS_TIMEOUT:
            raise RuntimeError(f"a device-side wait timed out (status 0x{s:08x}, wait site 0x{s & 0xFFFF:x}); "
                               "the results of that launch are invalid")
        raise RuntimeError(f"device status 0x{s:08x}")

    def dense_mask(self) -> torch.Tensor:
        """bool (B, T, T) mask materialised on the device from the descriptors."""
        out = torch.empty((self.B, self.T, self.T), dtype=torch.uint8, device=self.device)
        stream = torch.cuda.current_stream(self.device).cuda_stream
        with torch.cuda.device(self.device):
            _capi.check(_capi.load().kd_mask_dense(self.ptr, self.B, self.T, out.data_ptr(), stream))
        return out.view(torch.bool)

    def nonempty_tiles(self) -> int:
        """Total number of non-EMPTY 128x128 tiles over the batch (one head)."""
        return int(self.stats.sum().item())


# the core is alive as long as its view is (the view holds it), so its hash cannot be reused while it is a key
_VIEWS: "weakref.WeakValueDictionary" = weakref.WeakValueDictionary()


class _PlanCacheView:
    """The extension's plan cache seen from Python: the cached plans, least recently used first."""

    def values(self):
        return [AttentionPlan._of(core) for core in _ext.cached_plans()]

    def clear(self):
        _ext.clear_plans()

    def __len__(self):
        return len(_ext.cached_plans())


_CACHE = _PlanCacheView()


def get_plan(B, T, device, in_span=None, span_id=None, is_prefix=None, lens=None, causal=True,
             rules=False) -> AttentionPlan:
    """Returns a cached plan for this metadata, classifying on the device if it is new."""
    return AttentionPlan._of(_ext.get_plan(B, T, torch.device(device), in_span, span_id, is_prefix, lens, bool(causal), bool(rules)))


def clear_plan_cache() -> None:
    _CACHE.clear()
