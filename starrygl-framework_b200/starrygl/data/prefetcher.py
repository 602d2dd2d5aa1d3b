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
        self._seq, self._fn = 0, _C.lib().sgl_prefetch_batch
        self._bound = [None] * self.depth

    def _bind(self, slot):
        """Everything of a slot's foreign call that does not change from batch to batch."""
        v, p, g = C.c_void_p, self.pipes[slot], self.pipes[slot].g
        a = p.args
        addr = self._totals.data_ptr() + 16 * slot
        words = (C.c_int64 * 2).from_address(addr)
        var = v(0), v(0), v(0), v(0), C.c_int64(0), C.c_int64(0), v(0)       # host roots / times, targets / times, n, seq, consumer
        table = p.feats
        args = [var[0], var[1], v(g.indptr.data_ptr()), v(g.nbr.data_ptr()), v(g.ts.data_ptr()), v(g.eid.data_ptr()),
                v(g.fence.data_ptr() if g.fence is not None else 0), C.c_int64(g.num_nodes), var[2], var[3], var[4], C.c_int(p.k),
                C.c_int(a["pol"]), C.c_int(a["eq"]), C.c_int64(a["off"]), C.c_int(a["keep"]), C.c_uint64(a["seed"]), C.c_uint32(0),
                v(p.nbr.data_ptr()), v(p.dst.data_ptr()), v(p.ts.data_ptr()), v(p.dt.data_ptr()), v(p.eid.data_ptr()),
                v(p.offsets.data_ptr()), v(0 if table is None else table.data_ptr()), C.c_int64(0 if table is None else table.shape[0]),
                C.c_int64(0 if table is None else p.row_bytes), C.c_int64(0 if table is None else p.src_pitch),
                v(0 if table is None else p.out_feats.data_ptr()), C.c_int(p.mode), v(p.status.ptr()), v(p.ws.data_ptr()),
                C.c_size_t(p.ws.numel()), v(addr), var[5], var[6], v(p.stream.cuda_stream)]
        return args, var, addr, words

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
        args, (h_r, h_t, d_r, d_t, c_n, c_seq, c_cons), addr, words = self._bound[slot]
        h_r.value = h_t.value = None
        d_r.value, d_t.value = pipe.roots.data_ptr(), pipe.root_ts.data_ptr()
        roots, root_ts = roots.contiguous(), root_ts.contiguous()
        if as_is and roots.is_cuda and root_ts.is_cuda:
            d_r.value, d_t.value = roots.data_ptr(), root_ts.data_ptr()
        elif as_is and roots.is_pinned() and root_ts.is_pinned():
            h_r.value, h_t.value = roots.data_ptr(), root_ts.data_ptr()
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
        c_n.value, c_seq.value, c_cons.value = n, self._seq, _C.stream_ptr()
        # The call orders the slot's reuse behind everything the consumer has enqueued so far on its stream: the work on the
        # batch that occupied this slot (handed out just before) and the kernels that produced ``roots``.  The batch submitted
        # now is only needed ``depth`` requests later, so this does not stall the consumer.
        _C.check(self._fn(*args))
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
