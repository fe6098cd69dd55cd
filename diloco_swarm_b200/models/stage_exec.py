"""Host side of the native stage executor (csrc/stage.cu): its handle and the work areas that its passes run in.

A work area is one tensor per microbatch in flight (``saved``, what the backward needs) or per stream (``scratch``,
what lives within a call).  They are kept between calls: a pass then allocates nothing, and the caching allocator
never has to wait for the side stream before it can give a block out again.
"""
from __future__ import annotations

import ctypes
import threading
import weakref
from collections import OrderedDict
from typing import Dict, List, Optional, Tuple

import torch

from ..ops import kernels as K
from ..ops._lib import check, cuda_lib, ptr

KEEP_AREA_BYTES = 8 << 30        # finished `saved` areas are kept up to this much in all, one of any size
MAX_STREAMS = 4                  # scratch areas kept (one per calling stream)


class SavedArea:
    """``saved`` area of one microbatch, with the point on the streams after which it may be written again.
    ``home``: the stream that it was allocated on."""
    __slots__ = ("buf", "free", "stream", "home")

    def __init__(self, buf: torch.Tensor, home: torch.cuda.Stream):
        self.buf, self.free, self.stream, self.home = buf, None, None, home

    def used_on(self, stream: torch.cuda.Stream) -> None:
        """Once dropped, the memory goes back to ``home``'s pool: the allocator has to know of everybody else."""
        if stream != self.home:
            self.buf.record_stream(stream)


class StageExec:
    def __init__(self, n: int, d: int, heads: int, vocab: int, status, side: Optional[torch.cuda.Stream],
                 ends: List[Optional[torch.Tensor]], blocks: List[List[torch.Tensor]], device: torch.device):
        """``ends``: wte, wpe, dwte, dwpe, lnf_w, lnf_b, dlnf_w, dlnf_b, head_w, dhead_w, count (None where the stage
        has no such part); ``blocks``: the 24 tensors of each block in the order of dsw_stage_create."""
        desc = [n, d, heads, vocab, status.ptr, side.cuda_stream if side is not None else 0]
        desc += [ptr(t) or 0 for t in ends]
        for b in blocks:
            desc += [t.data_ptr() for t in b]
        lib = cuda_lib()
        h = ctypes.c_void_p()
        with torch.cuda.device(device):
            check(lib.dsw_stage_create((ctypes.c_longlong * len(desc))(*desc), len(desc), ctypes.byref(h)),
                  "dsw_stage_create", 0)
        self.handle, self.lib, self.side, self.device, self.d = h.value, lib, side, device, d
        self._keep = (status, ends, blocks)
        weakref.finalize(self, lib.dsw_stage_destroy, self.handle)
        # A pass is several calls of the library on work areas that the passes of a stream share, so a thread holds this
        # from the first to the last of them.
        self.lock = threading.RLock()
        self.capturing = False
        self._sizes: Dict[tuple, Tuple[int, int]] = {}
        self._scratch: "OrderedDict[Tuple[str, int], torch.Tensor]" = OrderedDict()
        self._idle: List[SavedArea] = []

    def enter(self) -> torch.cuda.Stream:
        """The calling stream of a pass that begins (the lock is held), looked at for a capture by the caller."""
        self.capturing = torch.cuda.is_current_stream_capturing()
        return torch.cuda.current_stream()

    # ------------------------------------------------------------------ work areas
    def sizes(self, B: int, T: int, keep: bool, grad: bool, chunks: int) -> Tuple[int, int]:
        key = (B, T, keep, grad, chunks)
        got = self._sizes.get(key)
        if got is None:
            a, b = ctypes.c_size_t(), ctypes.c_size_t()
            check(self.lib.dsw_stage_sizes(self.handle, B, T, int(keep), int(grad), chunks, ctypes.byref(a),
                                           ctypes.byref(b)), "dsw_stage_sizes", 0)
            if len(self._sizes) > 1024:
                self._sizes.clear()
            got = self._sizes[key] = (a.value, b.value)
        return got

    def _alloc(self, nbytes: int) -> torch.Tensor:
        buf = torch.empty(max(nbytes, 256), dtype=torch.uint8, device=self.device)
        if self.side is not None:
            buf.record_stream(self.side)          # should it be dropped while side work still reads it
        return buf

    def area(self, kind: str, nbytes: int, stream: torch.cuda.Stream) -> torch.Tensor:
        """Scratch of this calling stream, at least ``nbytes``: its contents live within one pass.  Under a capture of
        the caller's it is the capture's own, and so are the areas of ``take``: replays must not meet other passes there,
        and a capture cannot wait for work from outside of it."""
        if self.capturing:
            return self._alloc(nbytes)
        key = (kind, stream.cuda_stream)
        buf = self._scratch.get(key)
        if buf is None or buf.numel() < nbytes:
            self._scratch.pop(key, None)
            buf = None                            # the old block may serve the new request
            buf = self._scratch[key] = self._alloc(nbytes)
            while len(self._scratch) > 2 * MAX_STREAMS:
                self._scratch.popitem(last=False)
        return buf

    def take(self, nbytes: int, stream: torch.cuda.Stream) -> SavedArea:
        if self.capturing:
            return SavedArea(self._alloc(nbytes), stream)
        for i, a in enumerate(self._idle):
            if a.buf.numel() == nbytes:
                del self._idle[i]
                stream.wait_event(a.free)
                if a.stream != stream:
                    stream.wait_stream(a.stream)
                a.used_on(stream)
                return a
        while self._idle and self._idle_bytes() + nbytes > KEEP_AREA_BYTES:
            self._idle.pop(0)                     # areas of another size go back to the allocator
        return SavedArea(self._alloc(nbytes), stream)

    def give(self, area: SavedArea, stream: torch.cuda.Stream) -> None:
        """The backward that read ``area`` has been queued on ``stream`` (and the side stream)."""
        if self.capturing:
            return
        if area.free is None:
            area.free = torch.cuda.Event()
        area.free.record(self.side if self.side is not None else stream)
        area.stream = stream
        area.used_on(stream)
        if not self._idle or self._idle_bytes() + area.buf.numel() <= KEEP_AREA_BYTES:
            self._idle.append(area)

    def _idle_bytes(self) -> int:
        return sum(a.buf.numel() for a in self._idle)

    def graphs(self) -> Tuple[int, int]:
        """(runs replayed so far, captures that failed)"""
        a, b = ctypes.c_int(), ctypes.c_int()
        check(self.lib.dsw_stage_graphs(self.handle, ctypes.byref(a), ctypes.byref(b)), "dsw_stage_graphs", 0)
        return a.value, b.value

    @staticmethod
    def keeps(nbytes: int) -> int:
        """How many finished areas of a size wait for the next microbatches."""
        return max(1, KEEP_AREA_BYTES // nbytes)

    def seal(self) -> None:
        """Passes that have no CUDA graph yet get none any more."""
        check(self.lib.dsw_stage_seal(self.handle), "dsw_stage_seal", 0)

    # ------------------------------------------------------------------ passes
    def forward(self, ids, x, saved: torch.Tensor, y, logits, B: int, T: int, keep: bool, stream) -> None:
        check(self.lib.dsw_stage_forward(self.handle, ptr(ids), ptr(x), saved.data_ptr(), ptr(y), ptr(logits), B, T,
                                         int(keep), stream.cuda_stream), "dsw_stage_forward", 0)

    def head(self, saved: torch.Tensor, scratch: torch.Tensor, targets, mask, scale: float, loss, B: int, T: int,
             keep: bool, grad: bool, chunks: int, stream) -> None:
        check(self.lib.dsw_stage_head(self.handle, saved.data_ptr(), scratch.data_ptr(), targets.data_ptr(), ptr(mask),
                                      scale, loss.data_ptr(), B, T, int(keep), int(grad), chunks,
                                      int(K.deterministic()), stream.cuda_stream), "dsw_stage_head", 0)

    def backward(self, hi: int, lo: int, dy, x, ids, saved: torch.Tensor, scratch: torch.Tensor, dx0, B: int, T: int,
                 chunks: int, stream) -> None:
        check(self.lib.dsw_stage_backward(self.handle, hi, lo, ptr(dy), ptr(x), ptr(ids), saved.data_ptr(),
                                          scratch.data_ptr(), ptr(dx0), B, T, chunks, int(K.deterministic()),
                                          stream.cuda_stream), "dsw_stage_backward", 0)
