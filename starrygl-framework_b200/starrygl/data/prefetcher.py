"""Mini-batch prefetcher on the GPU: sampling + feature gather of the next batches run while the model consumes the
current one.

The reference's training scripts import a ``HostToDevicePrefetcher`` (``starrygl.data.prefetcher``, used at
test/test_offline.py:137-140 as ``HostToDevicePrefetcher(loader=..., device=..., ...)``) that is not part of the
reference tree; its job -- hide the data path behind the model -- is done here with ``depth`` pre-bound
:class:`~starrygl.graph.pipeline.SampleGatherPipeline` objects, each on its own stream.  ``loader`` yields the roots
of one mini-batch as ``(roots, query_times)`` int64 tensors (CUDA, or pinned host memory) of at most ``max_roots``
entries.  Iterating yields :class:`PrefetchedBatch` objects in loader order, already ordered into the consumer's
current stream; a batch's tensors alias the buffers of its pipeline object and may be read by kernels enqueued on that
stream until the next batch is requested, which hands the pipeline object to the batch ``depth`` places on.
"""
import ctypes as C
from collections import deque
from typing import Iterable, Optional

import torch

from .. import _C, ops
from ..graph.pipeline import SampleGatherPipeline


class PrefetchedBatch:
    """Block structure and gathered edge-feature rows of one mini-batch (device tensors, capacity-sized; the valid
    prefix has ``offsets[n_roots]`` edges -- :meth:`num_edges` reads it, one synchronisation)."""

    def __init__(self, pipe: SampleGatherPipeline, n_roots: int, ready: torch.cuda.Event, total=None):
        self.pipe, self.n_roots, self.ready = pipe, n_roots, ready
        self._total = total               # (address, ctypes words, sequence number, their buffer) of the pinned edge count
        self.offsets, self.nbr, self.dst, self.ts, self.eid, self.dt = (pipe.offsets[:n_roots + 1], pipe.nbr, pipe.dst,
                                                                        pipe.ts, pipe.eid, pipe.dt)
        self.edge_feats = pipe.out_feats

    def wait(self, stream: Optional[torch.cuda.Stream] = None):
        """Make ``stream`` (default: the current one) wait for this batch -- no host blocking."""
        (stream or _C.current_stream()).wait_event(self.ready)
        return self

    def num_edges(self) -> int:
        if self.n_roots == 0:             # (its count would race with that of the slot's batch before)
            return 0
        if self._total is not None:
            addr, words, seq, _ = self._total
            if words[1] < seq:
                _C.check(_C.lib().sgl_wait_word(addr + 8, seq, self.pipe.stream.cuda_stream))
            if words[1] == seq:           # (a later batch of the slot may have overwritten it)
                return words[0]
        self.ready.synchronize()
        return int(self.offsets[self.n_roots].item())


# places among the arguments of sgl_prefetch_batch
_HOST, _DEVICE, _COUNT, _SEQ = slice(0, 2), slice(8, 10), 10, slice(34, 36)


class HostToDevicePrefetcher:
    def __init__(self, loader: Iterable, g: ops.TCSR, edge_feats: Optional[torch.Tensor], fanout: int,
                 policy: str = "recent", max_roots: int = 4096, depth: int = 4, device=None, **sampler_options):
        self.loader, self.depth = loader, max(1, int(depth))
        self.streams = [torch.cuda.Stream(g.device) for _ in range(self.depth)]
        self.pipes = [SampleGatherPipeline(g, edge_feats, fanout, policy, max_roots, stream=s, **sampler_options)
                      for s in self.streams]
        self._held = [deque() for _ in range(self.depth)]      # per slot: (event behind a batch, its inputs), oldest first
        self._spare = [[] for _ in range(self.depth)]          # events of batches that are done
        self._totals = torch.zeros(2 * self.depth, dtype=torch.int64).pin_memory()   # per slot: edges, sequence number
        self._seq, self._fn = 0, _C.host().sgl_prefetch_batch
        self._bound = [None] * self.depth

    def _bind(self, slot):
        """The arguments of a slot's foreign call, those that change from batch to batch at their places (_HOST, _DEVICE, _COUNT, _SEQ)."""
        p, g = self.pipes[slot], self.pipes[slot].g
        a, table = p.args, p.feats
        addr = self._totals.data_ptr() + 16 * slot
        words = (C.c_int64 * 2).from_address(addr)
        args = [0, 0, g.indptr.data_ptr(), g.nbr.data_ptr(), g.ts.data_ptr(), g.eid.data_ptr(), g.fence.data_ptr() if g.fence is not None else 0,
                g.num_nodes, 0, 0, 0, p.k, a["pol"], a["eq"], a["off"], a["keep"], a["seed"], 0, p.nbr.data_ptr(), p.dst.data_ptr(),
                p.ts.data_ptr(), p.dt.data_ptr(), p.eid.data_ptr(), p.offsets.data_ptr(), 0 if table is None else table.data_ptr(),
                0 if table is None else table.shape[0], 0 if table is None else p.row_bytes, 0 if table is None else p.src_pitch,
                0 if table is None else p.out_feats.data_ptr(), p.mode, p.status.ptr(), p.ws.data_ptr(), p.ws.numel(), addr, 0, 0,
                p.stream.cuda_stream]
        return args, addr, words

    def _submit(self, slot, roots, root_ts):
        pipe, st = self.pipes[slot], self.streams[slot]
        n = roots.numel()
        if n > pipe.max_roots:
            raise _C.SglError(f"batch of {n} roots exceeds max_roots={pipe.max_roots}")
        as_is = roots.dtype == torch.int64 and root_ts.dtype == torch.int64 and root_ts.numel() == n
        if roots.is_cuda and not as_is:
            raise _C.SglError("prefetcher: roots on the GPU are int64 and come with as many int64 query times")
        if self._bound[slot] is None:
            self._bound[slot] = self._bind(slot)
        args, addr, words = self._bound[slot]
        on_host, on_device = (0, 0), (pipe.roots.data_ptr(), pipe.root_ts.data_ptr())
        roots, root_ts = roots.contiguous(), root_ts.contiguous()
        if as_is and roots.is_cuda and root_ts.is_cuda:
            on_device = roots.data_ptr(), root_ts.data_ptr()
        elif as_is and roots.is_pinned() and root_ts.is_pinned():
            on_host = roots.data_ptr(), root_ts.data_ptr()
        else:                             # pageable, of another type, or one time for all: staged by a copy, behind what the consumer still does with the slot
            st.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(st):
                pipe.roots[:n].copy_(roots, non_blocking=True)
                pipe.root_ts[:n].copy_(root_ts, non_blocking=True)
        # The kernels read the inputs where they are, which no allocator knows: they are held until their batch is done,
        # whatever becomes of the batch object.
        held, spare = self._held[slot], self._spare[slot]
        if len(held) >= 8:               # (not for every batch: asking costs as much as recording)
            if held[-1][0].query():
                spare.extend(e for e, _ in held)
                held.clear()
            while held and held[0][0].query():
                spare.append(held.popleft()[0])
        ready = spare.pop() if spare else torch.cuda.Event()
        self._seq += 1
        args[_HOST], args[_DEVICE], args[_COUNT], args[_SEQ] = on_host, on_device, n, (self._seq, _C.stream_ptr())
        # The call orders the slot's reuse behind everything the consumer has enqueued so far on its stream: the work on the
        # batch that occupied this slot (handed out just before) and the kernels that produced ``roots``.  The batch submitted
        # now is only needed ``depth`` requests later, so this does not stall the consumer.
        self._fn(*args)
        ready.record(st)
        held.append((ready, (roots, root_ts)))
        return PrefetchedBatch(pipe, n, ready, (addr, words, self._seq, self._totals))

    def __iter__(self):
        it = iter(self.loader)
        queue = deque()
        slot = 0
        for roots, root_ts in it:
            if len(queue) == self.depth:
                yield queue.popleft().wait()
            queue.append(self._submit(slot, roots, root_ts))
            slot = (slot + 1) % self.depth
        while queue:
            yield queue.popleft().wait()

    def __del__(self):
        try:                              # the inputs and counts of batches that are still under way go with the object
            for held in self._held:
                if held:
                    held[-1][0].synchronize()
        except Exception:
            pass

    def check(self):
        for p in self.pipes:
            p.status.check("prefetcher")
