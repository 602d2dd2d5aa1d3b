"""Python-visible surface of the native sampler module.

Same names and call signatures as the reference's pybind module ``libstarrygl_comm``
(csrc/srcs/starrygl/export.cu:20-254): ``from_edge_index``, ``CUDAGraph`` with ``submit_query`` / ``get`` /
``get_seeds_in_chunks`` / ``get_negative_root`` / ``sample_src_in_chunks_khop``, and the result types
``TemporalRoot``, ``NegativeRoot``, ``TemporalNeighbor``, ``TemporalResult``; plus the communicator and the sharded
feature table the same module exports (``create_nccl_id``, ``DistContext``,
csrc/include/starrygl/commContext.cu.hpp:259-268; ``init_p2p``, ``ShardTensorItem``, ``ShardTensor``,
csrc/include/starrygl/feature.cu.hpp:713-750).  The work is done by libsgl_b200.so
through its C ABI; result attributes are the tensors the kernels wrote (no second device copy per attribute
read, unlike export.cu:28-185).

Semantics (where the reference's CUDA code is ill-defined, the CPU sampler's rule is used):
candidates of a query (node, t) are the node's out-edges with ts < t (ts <= t with ``equal_root_time``; and
ts >= t - allowed_offset when ``allowed_offset`` >= 0); "recent" keeps the last k in ascending time, "uniform"
k distinct ones in ascending position; ``neighbors_dt`` = ts - t as int64; hop l+1 queries every neighbour of
hop l at the time of the edge that reached it (or at the root's time with ``keep_root_time``).
"""
import ctypes as C
import queue
import threading
from bisect import bisect_left
from collections import deque
from typing import List, Optional

import torch

from .. import ops
from .. import _C


def _empty(dev):
    return torch.empty(0, dtype=torch.int64, device=dev)


class TemporalRoot:
    """Roots of a batch: ``roots[r]`` has query times ``ts[ts_ptr[r]:ts_ptr[r+1]]``; query q is backed by the events
    ``q_eid[q_ptr[q]:q_ptr[q+1]]``."""

    def __init__(self, roots, ts_ptr, ts, q_ptr=None, q_eid=None):
        dev = roots.device
        self.roots, self.ts_ptr, self.ts = roots, ts_ptr, ts
        self.q_ptr = q_ptr if q_ptr is not None else _empty(dev)
        self.q_eid = q_eid if q_eid is not None else _empty(dev)

    @property
    def root_num(self):
        return self.roots.numel()

    @property
    def root_ts_num(self):
        return self.ts.numel()

    def __repr__(self):
        return f"<TemporalRoot with {self.root_num} roots>"


class NegativeRoot:
    def __init__(self, roots, ts):
        self.roots, self.ts = roots, ts

    @property
    def root_num(self):
        return self.roots.numel()

    def __repr__(self):
        return f"<NegativeRoot with {self.root_num} roots>"


class _Sizes:
    """What a result and its hops share: where the sizes (of the hops, of the pieces of the id map) are on the device, and not the arrays --
    a result holds its hops, and a hop that held the result would keep both, and the arrays of every other hop, until a garbage collection."""

    def __init__(self):
        self.status = None               # device status word of the graph that produced the result
        self.counts, self.known = [], []           # device counts (until they are read), and sizes (None: not read yet)

    def add(self, d_total) -> int:
        self.counts.append(d_total)
        self.known.append(None)
        return len(self.known) - 1

    def read(self):
        """One read-back of all sizes that are not known yet."""
        counts = [d for d in self.counts if d is not None]
        if not counts:
            return
        if self.status is not None:      # the kernels' error bits ride along in the same copy
            counts.append(self.status.t.to(torch.int64))
        host = torch.cat(counts).tolist()
        if self.status is not None:
            bits = int(host.pop())
            if bits:
                self.status.t.zero_()
                raise _C.SglError(f"sampling: device status {bits} ({_C.decode_status(bits)})")
        for i, d in enumerate(self.counts):
            if d is not None:
                self.known[i], self.counts[i] = host.pop(0), None


class TemporalNeighbor:
    """One hop: query q owns ``neighbors[root_start_ptr[q]:root_end_ptr[q]]`` (``root_start_ptr`` is the full
    exclusive prefix with one extra entry, ``root_end_ptr`` its shift by one).

    The hop's arrays are produced at capacity with their length on the device, so building the object costs no
    synchronisation.  Consumers that stay on the GPU use the capacity views (``hop``: ``nbr`` / ``ts`` / ``eid`` /
    ``dt_i64`` / ``offsets`` and the device count ``hop.d_total``).  The attributes of the reference's type (trimmed
    tensors, ``neighbor_num``) are cut to size on first use; all hops of a result are cut with ONE read-back of their
    counts (``TemporalResult.materialize``)."""

    def __init__(self, hop: ops.Hop, owner: "TemporalResult" = None, n_queries: Optional[int] = None):
        self.hop = hop
        self._sizes = None if owner is None else owner._sizes
        self._at = None if owner is None else owner._sizes.add(hop.d_total)
        last = owner.neighbors_list[-1] if owner is not None and owner.neighbors_list else None
        self._at_before = last._at if last is not None and last._sizes is self._sizes else None
        self._n = None                  # number of sampled neighbours, once known on the host
        self._nq = n_queries            # number of queries (None: known only once the previous hop has been cut)
        self._neighbors_override = None

    def _cut(self) -> int:
        if self._n is None:
            if self._sizes is None:
                self._n = self.hop.total()
            else:
                self._sizes.read()
                self._n = self._sizes.known[self._at]
                if self._nq is None and self._at_before is not None:      # queries of hop l = neighbours of hop l - 1
                    self._nq = self._sizes.known[self._at_before]
        return self._n

    @classmethod
    def from_arrays(cls, start_ptr, neighbors, neighbors_ts, neighbors_eid):
        """Layer given directly by its CSR arrays (``start_ptr`` with one extra entry)."""
        hop = ops.Hop(neighbors, None, neighbors_ts, None, neighbors_eid, start_ptr, neighbors.numel(), torch.zeros_like(neighbors_ts))
        self = cls(hop, None, start_ptr.numel() - 1)
        self._n = neighbors.numel()
        return self

    @property
    def neighbor_num(self) -> int:
        return self._cut()

    @property
    def root_start_ptr(self):
        self._cut()
        return self.hop.offsets if self._nq is None else self.hop.offsets[:self._nq + 1]

    @property
    def root_end_ptr(self):
        o = self.root_start_ptr
        return torch.cat([o[1:], o[-1:]])

    @property
    def neighbors(self):
        if self._neighbors_override is not None:
            return self._neighbors_override[:self._cut()]
        return self.hop.nbr[:self._cut()]

    @neighbors.setter
    def neighbors(self, value):
        self._neighbors_override = value

    @property
    def neighbors_ts(self):
        return self.hop.ts[:self._cut()]

    @property
    def neighbors_eid(self):
        return self.hop.eid[:self._cut()]

    @property
    def neighbors_dt(self):
        return self.hop.dt_i64[:self._cut()]

    @property
    def start_ptr(self):   # name used by the reference's block builder (starrygl/graph/graph.py:174)
        return self.root_start_ptr

    def __repr__(self):
        return f"<TemporalNeighbor with {self.neighbor_num} neighbors>"


class TemporalResult:
    def __init__(self, roots: TemporalRoot, neg_roots: Optional[NegativeRoot] = None):
        self.roots = roots
        self.neg_roots = neg_roots
        self.neighbors_list: List[TemporalNeighbor] = []
        self._remap_pieces = []          # (new global ids at capacity, where among the sizes their number is) per relabelled list
        self._remapper = None
        self._sizes = _Sizes()

    @property
    def _status(self):
        return self._sizes.status

    @_status.setter
    def _status(self, word):
        self._sizes.status = word

    @property
    def neighbors(self):
        return self.neighbors_list

    def materialize(self):
        """The one read-back of a result: the sizes of every hop (and of every piece of the id map) in a single copy."""
        self._sizes.read()
        prev = None
        for nb in self.neighbors_list:      # queries of hop l+1 = neighbours of hop l
            nb._cut()
            if nb._nq is None and prev is not None:
                nb._nq = prev._n
            prev = nb
        if self._remap_pieces:
            self._remapper = torch.cat([ids[:self._sizes.known[i]] for ids, i in self._remap_pieces])
            self._remap_pieces = []

    @property
    def nodes_remapper_id(self):
        if self._remapper is None:
            if self._remap_pieces:
                self.materialize()
            else:
                self._remapper = _empty(self.roots.roots.device)
        return self._remapper

    def __repr__(self):
        return f"<TemporalResult with {len(self.neighbors_list)} neighbor layers>"


# Arrays of a query up to this size share one allocation (what keeps one keeps the others' memory); larger ones have one each.
_SHARED_MOST = 32 << 20


class _QueryPlan:
    """Layout of the arrays of a query of one shape (events at most, negatives, fan-out, hops)."""

    def __init__(self, cap, n_neg, fanout, hops):
        L = _C.lib()
        self.places = C.c_int64 * (8 + 8 * hops)
        sec = self.places()
        self.words = int(L.sgl_query_layout(cap, n_neg, fanout, hops, sec))
        if self.words < 0:
            raise _C.SglError("query: bad shape")
        self.ws_bytes = int(L.sgl_query_ws_bytes(cap, n_neg, fanout, hops))
        self.size = [int(w) for w in sec]
        self.at, at = self.places(), 0
        for s, w in enumerate(self.size):
            self.at[s] = at
            at += w
        self.shared = 8 * self.words <= _SHARED_MOST


class _Arena:
    """All arrays of one query (see ``sgl_query``) with their sizes known on the host: ``cut(section, n)`` is a view.  ``buf``: one
    tensor, or a list of one per section."""

    def __init__(self, buf, plan, hops, meta):
        self.buf, self.hops = buf, hops
        self.device = buf.device if plan.shared else buf[0].device
        self._at = plan.at if plan.shared else None
        self.n_roots, self.n_pairs, self.n_events, self.n_queries = meta[:4]
        self.edges = meta[9:9 + hops]
        self.n_new = sum(meta[9 + hops:10 + 2 * hops])

    def cut(self, section, n, floats=False):
        t, s = (self.buf, self._at[section]) if self._at is not None else (self.buf[section], 0)
        return _C.host().cut(t, s, n, floats)

    def ptr(self, section):
        return self.buf.data_ptr() + 8 * self._at[section] if self._at is not None else self.buf[section].data_ptr()

    def holds(self, t, name):
        """Is ``t`` the root array ``name`` as the query left it?"""
        section, count, extra = _ArenaRoot._SECTIONS[name]
        return t.is_cuda and t.dtype == torch.int64 and t.is_contiguous() and t.data_ptr() == self.ptr(section) and \
            t.numel() == getattr(self, count) + extra


class _ArenaRoot(TemporalRoot):
    """Roots of a query under their local ids; the tensors are cut out of the query's arena on first use."""

    _SECTIONS = {"roots": (1, "n_roots", 0), "ts_ptr": (2, "n_roots", 1), "ts": (6, "n_pairs", 0), "q_ptr": (3, "n_pairs", 1),
                 "q_eid": (4, "n_events", 0)}

    def __init__(self, arena):
        self._a = arena

    def __getattr__(self, name):
        spec = _ArenaRoot._SECTIONS.get(name)
        if spec is None:
            raise AttributeError(name)
        a = self.__dict__["_a"]
        t = self.__dict__[name] = a.cut(spec[0], getattr(a, spec[1]) + spec[2])
        return t

    @property
    def root_num(self):
        t = self.__dict__.get("roots")
        return self._a.n_roots if t is None else t.numel()

    @property
    def root_ts_num(self):
        t = self.__dict__.get("ts")
        return self._a.n_pairs if t is None else t.numel()


class _ArenaNeighbor(TemporalNeighbor):
    """One hop of a query, cut out of the query's arena."""

    def __init__(self, arena, level):
        self._a, self._l, self._b = arena, level, 7 + 8 * level
        self._n = arena.edges[level]
        self._nq = arena.n_queries if level == 0 else arena.edges[level - 1]
        self._neighbors_override = None

    def _cut(self):
        return self._n

    @property
    def hop(self):
        a, b, n = self._a, self._b, self._n
        return ops.Hop(a.cut(b, n), a.cut(b + 1, n), a.cut(b + 2, n), a.cut(b + 3, n, True), a.cut(b + 5, n),
                       a.cut(b + 7, self._nq + 1), n, a.cut(b + 4, n))

    @property
    def neighbors(self):
        return self._neighbors_override if self._neighbors_override is not None else self._a.cut(self._b + 6, self._n)

    @neighbors.setter
    def neighbors(self, value):
        self._neighbors_override = value

    @property
    def root_start_ptr(self):
        return self._a.cut(self._b + 7, self._nq + 1)

    @property
    def neighbors_ts(self):
        return self._a.cut(self._b + 2, self._n)

    @property
    def neighbors_eid(self):
        return self._a.cut(self._b + 5, self._n)

    @property
    def neighbors_dt(self):
        return self._a.cut(self._b + 4, self._n)


class _QueryFuture:
    """A query whose kernels are enqueued; ``wait()`` reads its sizes and builds the result."""

    def __init__(self, stream, slot, buf, plan, hops, neg):
        self.stream, self.slot, self.buf, self.plan, self.hops, self.neg = stream, slot, buf, plan, hops, neg

    def wait(self):
        hops = self.hops
        addr, words = self.slot
        n = 10 + 2 * hops
        try:
            _C.host().sgl_wait_word(addr + 8 * n, 1, self.stream.cuda_stream)
            meta = words[:n]
        finally:                          # (the stream has come to its end either way)
            _FREE_SLOTS.append(self.slot)
        bits = meta[5] & 0xFFFFFFFF
        if bits:
            raise _C.SglError(f"submit_query: device status {bits} ({_C.decode_status(bits)})")
        arena = _Arena(self.buf, self.plan, hops, meta)
        out = TemporalResult(_ArenaRoot(arena), self.neg)
        out.neighbors_list = [_ArenaNeighbor(arena, l) for l in range(hops)]
        out._remapper = arena.cut(7 + 8 * hops, arena.n_new)
        return out


def query_blocks(root, neg_roots, neighbors):
    """Source nodes, source times and column indices of the blocks of a query's hops (self loops included) in one launch;
    None when the parts are not those of one query as ``CUDAGraph.get`` returned it.  Yields (dst count, nid, ts, indices)."""
    if not neighbors or not isinstance(root, _ArenaRoot):
        return None
    a = root._a
    if len(neighbors) != a.hops or any(not isinstance(nb, _ArenaNeighbor) or nb._a is not a or nb._l != l
                                       or nb._neighbors_override is not None for l, nb in enumerate(neighbors)):
        return None
    n_neg = 0 if neg_roots is None else neg_roots.root_num
    # parts that were replaced since take the general path, which uses what they hold now
    if n_neg != a.n_queries - a.n_pairs or any(k in root.__dict__ and not a.holds(root.__dict__[k], k) for k in ("roots", "ts", "ts_ptr")):
        return None
    neg = neg_ts = None
    if n_neg:
        neg, neg_ts = neg_roots.roots.contiguous(), neg_roots.ts.contiguous()          # (a column of a table, say)
        if any(not t.is_cuda or t.dtype != torch.int64 or t.numel() != n_neg for t in (neg, neg_ts)):
            return None
    parts = []
    for l, n in enumerate(a.edges):
        parts += (a.ptr(7 + 8 * l + 6), a.ptr(7 + 8 * l + 2), n)
    blocks = _C.host().query_blocks(a.device.index, a.ptr(6), a.ptr(2), a.ptr(1), neg, neg_ts, a.n_roots, a.n_pairs, a.n_queries, *parts)
    return [(d, *arrays) for d, arrays in blocks]


# Free pinned result words of queries, (address, ctypes array); as many as queries were ever in flight together, kept for the next
# graph (pinning memory takes a millisecond).
_FREE_SLOTS: list = []
_SLOT_BLOCKS: list = []


class CUDAGraph:
    """Temporal graph on one GPU + an asynchronous sampling queue (FIFO results)."""

    def __init__(self, g: ops.TCSR, ev, chunk_size, mapper, stream, rank):
        self.g = g
        self.ev = ev                      # events in time order: (src, ts, eid)
        self.chunk_size, self.mapper, self.rank = chunk_size, mapper, rank
        self.stream = stream
        self.status = ops.StatusWord(g.device)
        self.relabel = ops.NodeRelabeler(g.num_nodes, g.device)
        self._tasks = queue.Queue()
        self._results = deque()
        self._closed = False
        self._worker = None               # started by the first task that has to wait for the GPU on the way
        self._pending = 0                 # tasks that the worker has not finished
        self._lock = threading.Lock()
        self._ev_index = None
        self._plans = {}

    # ---- synchronous entry points -----------------------------------------------------------------------
    def get_negative_root(self, negative_root: torch.Tensor, negative_time: torch.Tensor) -> NegativeRoot:
        return NegativeRoot(negative_root.to(self.g.device, torch.int64), negative_time.to(self.g.device, torch.int64))

    def get_seeds_in_chunks(self, chunks: torch.Tensor, time_begin: int, time_end: int,
                            using_full_timestamp: bool = False) -> TemporalRoot:
        with torch.cuda.stream(self.stream):
            roots, ts_ptr, ts, q_ptr, q_eid = ops.seeds_in_window(self.ev, self.g, chunks, self.mapper, int(time_begin),
                                                                  int(time_end), status=self.status)
            if using_full_timestamp:
                # every root gets all time steps of the window (snapshot graphs): time steps without an event own no event
                ts_ptr, ts, q_ptr = ops.densify_time_groups(ts_ptr, ts, q_ptr, int(time_begin), int(time_end))
        return TemporalRoot(roots, ts_ptr, ts, q_ptr, q_eid)

    def sample_src_in_chunks_khop(self, postive_root: TemporalRoot, negative_root: Optional[NegativeRoot], k: int,
                                  layers: int, allowed_offset: int, equal_root_time: bool, keep_root_time: bool,
                                  sample_type: str) -> TemporalResult:
        if sample_type not in ("recent", "uniform"):
            raise RuntimeError("undefined sampling strategy")
        dev = self.g.device
        with torch.cuda.stream(self.stream):
            # one query per (root, timestamp) of the positive roots, then one per negative root
            reps = postive_root.ts_ptr[1:] - postive_root.ts_ptr[:-1] if postive_root.root_num else _empty(dev)
            q_nodes = torch.repeat_interleave(postive_root.roots, reps) if postive_root.root_num else _empty(dev)
            q_ts = postive_root.ts
            if negative_root is not None and negative_root.root_num:
                q_nodes = torch.cat([q_nodes, negative_root.roots])
                q_ts = torch.cat([q_ts, negative_root.ts])
            out = TemporalResult(postive_root, negative_root)
            out._status = self.status
            tgt, tgt_ts, d_n, n_q = q_nodes.contiguous(), q_ts.contiguous(), None, q_nodes.numel()
            for l in range(int(layers)):
                hop = ops.sample_layer(self.g, tgt, tgt_ts, int(k), sample_type, d_n=d_n,
                                       equal_root_time=bool(equal_root_time), allowed_offset=int(allowed_offset),
                                       keep_root_time=bool(keep_root_time), rng_stream=l, want_dt_i64=True,
                                       status=self.status)
                out.neighbors_list.append(TemporalNeighbor(hop, out, n_q))
                # the next hop queries this hop's neighbours: arrays at capacity, their number stays on the device
                tgt, tgt_ts, d_n, n_q = hop.nbr, hop.ts, hop.d_total, None
        return out

    def slice_by_chunk_ts(self, chunks, time_begin, time_end, using_full_timestamp=False, stream=0) -> "TemporalResult":
        """Sub-graph of the chunks' nodes inside ``[time_begin, time_end)``: ``roots`` = the nodes that keep an edge with
        their distinct timestamps (``ts_ptr`` / ``ts``), one neighbour layer whose ``root_start_ptr`` has one entry per
        (node, timestamp) group (reference: csrc/include/starrygl/sample.cu.hpp:1189-1291)."""
        ev_ts = self.ev[1]
        with torch.cuda.stream(self.stream):
            lo, hi = ops.lower_bound(ev_ts, torch.tensor([int(time_begin), int(time_end)], dtype=torch.int64,
                                                         device=ev_ts.device)).tolist()
            nodes, node_ptr, group_ts, group_ptr, nbr, ts, eid = ops.slice_window(
                self.g, chunks, self.mapper, int(time_begin), int(time_end), max(hi - lo, 0), status=self.status)
            if using_full_timestamp:
                node_ptr, group_ts, group_ptr = ops.densify_time_groups(node_ptr, group_ts, group_ptr, int(time_begin),
                                                                        int(time_end))
        out = TemporalResult(TemporalRoot(nodes, node_ptr, group_ts))
        out.neighbors_list.append(TemporalNeighbor.from_arrays(group_ptr, nbr, ts, eid))
        return out

    def _remap(self, result: TemporalResult, reset: bool):
        """Node-level relabel: roots first, then every hop; local ids in ascending global id among the new ids."""
        if reset:
            self.relabel.reset()
        pieces = result._remap_pieces
        loc, new_ids, d_new = self.relabel.insert(result.roots.roots, status=self.status)
        result.roots = TemporalRoot(loc, result.roots.ts_ptr, result.roots.ts, result.roots.q_ptr, result.roots.q_eid)
        pieces.append((new_ids, result._sizes.add(d_new)))
        for nb in result.neighbors_list:      # capacity arrays + device counts: no read-back between the hops
            loc, new_ids, d_new = self.relabel.insert(nb.hop.nbr, d_n=nb.hop.d_total, status=self.status)
            nb.neighbors = loc
            pieces.append((new_ids, result._sizes.add(d_new)))

    # ---- asynchronous queue ----------------------------------------------------------------------------------
    def submit_query(self, time_start, time_end, chunk_list, test_generate_samples, test_generate_samples_ts,
                     sample_type, layers, fanout, allowed_offset, equal_root_time, keep_root_time, op) -> None:
        """Queue one task; results come back from :meth:`get` in the order of submission.  Sampling tasks are enqueued on
        the graph's stream at once -- one foreign call, nothing waits for the GPU; tasks whose sizes the host has to learn on
        the way (the chunk slice, windows above the mini-batch limit) run on a worker thread, and while it has work
        everything behind goes through it, so that the relabel's numbering keeps the order."""
        if self._closed:
            raise RuntimeError("graph is closed")
        neg = self.get_negative_root(test_generate_samples, test_generate_samples_ts)
        task = (int(time_start), int(time_end), chunk_list, neg, sample_type, int(layers), int(fanout), int(allowed_offset),
                bool(equal_root_time), bool(keep_root_time), op)
        with self._lock:
            if self._pending == 0:
                try:
                    fut = self._enqueue(*task)
                except BaseException as e:       # delivered to the caller of get()
                    fut = {"event": None, "value": None, "error": e}
                if fut is not None:
                    self._results.append(fut)
                    return
            made = torch.cuda.Event()            # the caller's tensors are ready behind it
            made.record(torch.cuda.current_stream(self.g.device))
            fut = {"event": threading.Event(), "value": None, "error": None, "made": made}
            self._pending += 1
            if self._worker is None:
                self._worker = threading.Thread(target=_serve, args=(self._tasks, self.g.device), daemon=True)
                self._worker.start()
            self._tasks.put((self, fut, task))
            self._results.append(fut)

    def _window(self, t0, t1):
        """Host-known bounds of the window's events: (first, at most) from every 256th timestamp of the stream."""
        if self._ev_index is None:
            with torch.cuda.stream(self.stream):      # (events out of order are still being sorted there)
                # (a view of the copy: a look-up costs 0.3 us, in an array 1.0; a list is made in 0.14 ms for 2 M events, in 5 for 50 M)
                self._ev_index = memoryview(self.ev[1][::256].cpu().numpy())
        idx, m = self._ev_index, self.ev[1].numel()
        first = max(bisect_left(idx, t0) - 1, 0) * 256
        last = min(bisect_left(idx, t1) * 256, m)
        if last <= first:
            first, last = min(first, m - 1), min(first, m - 1) + 1
        return first, last - first

    @staticmethod
    def _slot():
        try:
            return _FREE_SLOTS.pop()
        except IndexError:
            block = torch.zeros(64 * 32, dtype=torch.int64, pin_memory=True)
            _SLOT_BLOCKS.append(block)
            new = [(block.data_ptr() + 256 * i, (C.c_int64 * 32).from_address(block.data_ptr() + 256 * i)) for i in range(64)]
            _FREE_SLOTS.extend(new[1:])
            return new[0]

    def _enqueue(self, t0, t1, chunks, neg, stype, layers, fanout, off, eq, keep, op) -> Optional[_QueryFuture]:
        g = self.g
        m = self.ev[1].numel()
        if stype not in ("recent", "uniform") or m == 0 or not 0 <= layers <= 8 or fanout < 1:
            return None
        if not (-2 ** 63 <= t0 < 2 ** 63 and -2 ** 63 <= t1 < 2 ** 63):
            return None                     # (refused there; the foreign call would take the low 64 bits)
        first, cap = self._window(t0, t1)
        if cap > 1_200_000:                 # above the mini-batch sort's limit
            return None
        dev = g.device
        sp = self.stream.cuda_stream
        n_neg = neg.root_num
        key = (cap, n_neg, fanout, layers)
        plan = self._plans.get(key)
        if plan is None:
            if len(self._plans) > 64:
                self._plans.clear()
            plan = self._plans[key] = _QueryPlan(*key)
        producer = _C.stream_ptr() if torch._C._cuda_getDevice() == dev.index else torch.cuda.current_stream(dev).cuda_stream
        neg_ids, neg_ts = neg.roots.contiguous(), neg.ts.contiguous()
        if self.mapper is not None and chunks is not None and self.mapper.numel():
            self.stream.wait_stream(torch.cuda.current_stream(dev))
        rl, st, extra = self.relabel, self.stream, 10 + 2 * layers
        mask, node_chunk, n_chunks, buf = None, None, 0, None
        at, words, meta = C.addressof(plan.at), plan.words, extra
        if self.mapper is not None or not plan.shared:
            with _C.on_stream(st):
                mask, node_chunk, n_chunks = ops.chunk_mask(g, chunks, self.mapper)
                if not plan.shared:
                    buf = [torch.empty(w, dtype=torch.int64, device=dev) for w in (*plan.size, extra)]
                    places = plan.places(*[t.data_ptr() // 8 for t in buf[:-1]])
                    at, words, meta = C.addressof(places), 0, buf[-1].data_ptr()
        epoch = rl.epoch + (1 if op == "f" else 0)       # the reference restarts the numbering on "f"
        slot = self._slot()
        slot[1][extra] = 0
        try:
            own, = _C.host().query(
                g.indptr, g.nbr, g.ts, g.eid, g.fence, g.num_nodes, *self.ev, first, cap, t0, t1, node_chunk, mask, n_chunks, neg_ids, neg_ts,
                fanout, layers, _C.POLICY[stype], eq, off, keep, ops.bits_for(g.num_nodes - 1), ops.bits_for(g.ts_max - g.ts_min), g.ts_min,
                rl.mapper, rl.mask, epoch, op == "f", rl.next_local, at, words, meta, slot[0], plan.ws_bytes, producer, st.stream_id,
                st.device_index, st.device_type, sp)
        except BaseException:             # refused before anything ran: the numbering goes on as it was
            _FREE_SLOTS.append(slot)
            raise
        buf = own if buf is None else buf
        rl.epoch = epoch
        fut = _QueryFuture(self.stream, slot, buf, plan, layers, neg)
        fut._keep = (neg_ids, neg_ts, mask)   # inputs of kernels that may still be queued
        return fut

    def get(self) -> Optional[TemporalResult]:
        try:
            fut = self._results.popleft()
        except IndexError:
            return None
        if isinstance(fut, _QueryFuture):
            return fut.wait()
        if fut["event"] is not None:
            fut["event"].wait()
        if fut["error"] is not None:
            raise fut["error"]
        return fut["value"]

    def _do(self, fut, task):
        """One task on the worker thread."""
        t0, t1, chunks, neg, stype, layers, fanout, off, eq, keep, op = task
        try:
            self.stream.wait_event(fut["made"])
            nat = self._enqueue(*task)
            if nat is not None:
                fut["value"] = nat.wait()
            else:
                if stype in ("recent", "uniform"):
                    roots = self.get_seeds_in_chunks(chunks, t0, t1, False)
                    res = self.sample_src_in_chunks_khop(roots, neg, fanout, layers, off, eq, keep, stype)
                else:
                    # any other policy name is the "cluster" slice: the chunks' whole sub-graph inside the window, dense
                    # time steps (csrc/include/starrygl/sample.cu.hpp:1953-1961)
                    res = self.slice_by_chunk_ts(chunks, t0, t1, True)
                    res._status = self.status
                with torch.cuda.stream(self.stream):
                    self._remap(res, op == "f")
                    self.status.check("submit_query")
                self.stream.synchronize()
                fut["value"] = res
        except BaseException as e:   # delivered to the caller of get()
            fut["error"] = e
        with self._lock:
            self._pending -= 1
        fut["event"].set()

    def close(self):
        if not self._closed:
            self._closed = True
            self._tasks.put(None)

    def __del__(self):
        try:
            self.close()
            # queries that nobody fetched: their kernels still use the graph's arrays, their negatives and result words
            left = [f for f in self._results if isinstance(f, _QueryFuture)]
            if left:
                self.stream.synchronize()
                _FREE_SLOTS.extend(f.slot for f in left)
        except Exception:
            pass


def _serve(tasks, device):
    """Worker of one graph; holds the graph only while it has a task of it."""
    torch.cuda.set_device(device)
    while True:
        item = tasks.get()
        if item is None:
            return
        graph, fut, task = item
        graph._do(fut, task)
        del item, graph, fut, task


def from_edge_index(n: int, chunk_size: int, src: torch.Tensor, dst: torch.Tensor, ts: torch.Tensor, eid: torch.Tensor,
                    mapper: Optional[torch.Tensor] = None, stream=0, rank: int = 0) -> CUDAGraph:
    """Build the time-sorted CSR (rows = source nodes, neighbours = destinations) on GPU ``rank``.

    ``stream`` is a ``torch.cuda.Stream``, a raw ``cudaStream_t`` value, or 0/None for a stream owned by the graph.
    Raises ``RuntimeError`` for non-CUDA / non-int64 inputs and for node ids outside [0, n).
    """
    for name, t in (("src", src), ("dst", dst), ("ts", ts), ("eid", eid)):
        if not isinstance(t, torch.Tensor) or not t.is_cuda:
            raise RuntimeError(f"Graph construction failed: {name} must be a CUDA tensor")
        if t.dtype != torch.int64:
            raise RuntimeError(f"Graph construction failed: {name} must be int64")
    dev = src.device
    if isinstance(stream, torch.cuda.Stream):
        s = stream
    elif stream:
        s = torch.cuda.ExternalStream(int(stream), device=dev)
    else:
        s = torch.cuda.Stream(device=dev)
    if mapper is not None and mapper.numel():
        m = mapper.to(torch.int64).cpu()
        if bool((m[1:] < m[:-1]).any()):
            raise RuntimeError("Graph construction failed: chunk mapper must be non-decreasing in node id")
    s.wait_stream(torch.cuda.current_stream(dev))
    try:
        with torch.cuda.stream(s):
            g = ops.tcsr_build(src, dst, ts, eid, int(n))
            ev = ops.time_ordered_events(src, ts, eid)
    except _C.SglError as e:
        raise RuntimeError(f"Graph construction failed: {e}") from e
    return CUDAGraph(g, ev, chunk_size, mapper, s, rank)


# ---------------------------------------------------------------------------------------------------------------------
# communicator + sharded feature table
# ---------------------------------------------------------------------------------------------------------------------

def create_nccl_id() -> bytes:
    """Unique id of a new communicator, to be handed to every rank out of band (the reference puts it into the
    process group's store, starrygl/utils/context.py:111-117)."""
    import ctypes as C
    buf = C.create_string_buffer(128)
    _C.check(_C.lib().sgl_comm_unique_id(buf, 128))
    return buf.raw


class DistContext:
    """One rank of the library's own NCCL communicator: ``DistContext(rank, world_size, local_size, id)`` with
    ``rank()``, ``size()``, ``device()`` (csrc/include/starrygl/commContext.cu.hpp:11-60, :259-268).  The device of the
    rank is ``rank % local_size`` and is made current, as the reference's constructor does."""

    def __init__(self, rank: int, world_size: int, local_size: int, id: bytes):
        import ctypes as C
        if not (isinstance(id, (bytes, bytearray)) and len(id) >= 128):
            raise RuntimeError("DistContext: id must be the bytes create_nccl_id() returned")
        if local_size < 1 or not (0 <= rank < world_size):
            raise RuntimeError("DistContext: bad rank / size")
        self._rank, self._world, self._local = int(rank), int(world_size), int(local_size)
        self._device = self._rank % self._local
        torch.cuda.set_device(self._device)
        self.handle = C.c_void_p()
        _C.check(_C.lib().sgl_comm_init(C.byref(self.handle), self._rank, self._world, bytes(id)))
        from ..route.exchange import NativeComm
        NativeComm.adopt(self.handle, self._rank, self._world)     # the routes of this process use this communicator

    def rank(self) -> int:
        return self._rank

    def size(self) -> int:
        return self._world

    def device(self) -> int:
        return self._device


def init_p2p(devices: List[int]) -> int:
    """Enable peer access from the current GPU to the listed ones where the hardware allows it; returns how many of
    them are reachable.  With one process per GPU the mappings of other ranks' memory enable it when they are opened,
    so this matters only for a process that drives several GPUs."""
    import ctypes as C
    arr = (C.c_int * max(len(devices), 1))(*[int(d) for d in devices])
    ok = C.c_int(0)
    _C.check(_C.lib().sgl_init_p2p(arr, len(devices), C.byref(ok)))
    return ok.value


class ShardTensorItem:
    """Description of one shard that can travel between processes: owner rank and device, an inter-process handle of
    its memory, its shape and element size (csrc/include/starrygl/feature.cu.hpp:94-140)."""

    def __init__(self):
        self.rank, self.group, self.device = 0, 0, -1
        self.mem_handle, self.shape, self.element_size, self.dtype = b"", [], 4, "float32"

    def share_ipc(self):
        return (self.device, self.element_size, self.mem_handle, list(self.shape), self.rank, self.dtype)

    def from_ipc(self, ipc_data):
        self.device, self.element_size, self.mem_handle, shape = ipc_data[:4]
        self.shape = list(shape)
        if len(ipc_data) > 4:
            self.rank = int(ipc_data[4])
        if len(ipc_data) > 5:
            self.dtype = ipc_data[5]
        return self


class ShardTensor:
    """Row table sharded over the GPUs of one node; ``tensor[ids]`` with packed ids ``(partition << 48) | local row``
    returns the rows in the order of the ids (csrc/include/starrygl/feature.cu.hpp:142-422).

    Shard p belongs to rank p.  The owner appends its own CUDA tensor, every other rank appends the
    ``ShardTensorItem`` the owner published (``share_ipc``) and thereby maps the owner's memory.  The gather is ONE
    kernel that reads every row from its owner's memory over NVLink; the reference's plan -- split the ids by owner,
    send the ids, gather at the owner, send the rows back, scatter to the original order -- is what
    :meth:`gather_by_exchange` does for ranks without a mapping of each other's memory."""

    def __init__(self, device: int, context: Optional[DistContext] = None):
        self._device = int(device)
        self.context = context
        self._local = {}          # partition -> tensor owned here (kept alive)
        self._bases, self._rows = [], []
        self._opened = []
        self._row_shape, self._dtype = None, None
        self._tables = None

    # ---- building ------------------------------------------------------------------------------------------------
    def _check_layout(self, shape, dtype):
        if self._row_shape is None:
            self._row_shape, self._dtype = tuple(shape[1:]), dtype
        elif tuple(shape[1:]) != self._row_shape or dtype != self._dtype:
            raise RuntimeError("ShardTensor: all shards must have the same row shape and dtype")

    def append(self, item, target_device: Optional[int] = None):
        """Append the next partition's shard: a CUDA tensor of this process, or a ``ShardTensorItem`` of another."""
        import ctypes as C
        self._tables = None
        if isinstance(item, torch.Tensor):
            if not item.is_cuda or not item.is_contiguous():
                raise RuntimeError("ShardTensor.append: a local shard must be a contiguous CUDA tensor")
            self._check_layout(item.shape, item.dtype)
            self._local[len(self._bases)] = item
            self._bases.append(item.data_ptr())
            self._rows.append(int(item.shape[0]))
            return
        dtype = getattr(torch, item.dtype)
        self._check_layout(item.shape, dtype)
        ptr = C.c_void_p()
        _C.check(_C.lib().sgl_p2p_open(item.mem_handle, C.byref(ptr)))
        self._opened.append(ptr)
        self._bases.append(ptr.value)
        self._rows.append(int(item.shape[0]))

    def share_ipc(self) -> List[ShardTensorItem]:
        """Items for the shards this process owns (the memory must come from ``cudaMalloc``, i.e. be a whole torch
        allocation or one made with ``ShardTensor.alloc_shared``)."""
        out = []
        for part, t in self._local.items():
            it = ShardTensorItem()
            it.rank, it.device, it.shape, it.element_size = part, t.device.index, list(t.shape), t.element_size()
            it.dtype = str(t.dtype).replace("torch.", "")
            it.mem_handle = _ipc_handle(t)
            out.append(it)
        return out

    @classmethod
    def from_local(cls, local: torch.Tensor, context: Optional[DistContext] = None) -> "ShardTensor":
        """Collective convenience: every rank of the default process group passes its own shard (allocated with
        :func:`shared_empty`); the handles are exchanged through the group and every rank maps all shards."""
        import torch.distributed as dist
        rank, world = dist.get_rank(), dist.get_world_size()
        me = cls(local.device.index, context)
        mine = ShardTensorItem()
        mine.rank, mine.device, mine.shape, mine.element_size = rank, local.device.index, list(local.shape), local.element_size()
        mine.dtype = str(local.dtype).replace("torch.", "")
        mine.mem_handle = _ipc_handle(local)
        box = [None] * world
        dist.all_gather_object(box, mine.share_ipc())
        for p in range(world):
            me.append(local if p == rank else ShardTensorItem().from_ipc(box[p]))
        dist.barrier()
        return me

    # ---- queries ---------------------------------------------------------------------------------------------------
    def shape(self):
        return [sum(self._rows)] + list(self._row_shape or [])

    def size(self, dim: int) -> int:
        return self.shape()[dim]

    def numel(self) -> int:
        n = 1
        for d in self.shape():
            n *= d
        return n

    def stride(self, dim: int) -> int:
        s = 1
        for d in self.shape()[dim + 1:]:
            s *= d
        return s

    def device(self) -> int:
        return self._device

    def device_count(self) -> int:
        return len(self._bases)

    # ---- gather ------------------------------------------------------------------------------------------------------
    def _device_tables(self, dev):
        if self._tables is None:
            self._tables = (torch.tensor(self._bases, dtype=torch.int64, device=dev),
                            torch.tensor(self._rows, dtype=torch.int64, device=dev), ops.StatusWord(dev))
        return self._tables

    def __getitem__(self, indices: torch.Tensor) -> torch.Tensor:
        if not indices.is_cuda:
            raise RuntimeError("ShardTensor: the ids must be on the GPU")
        bases, rows, st = self._device_tables(indices.device)
        return ops.shard_gather(bases, rows, len(self._bases), self._row_shape, self._dtype, indices, status=st)

    def check(self):
        """Raise if a gather since the last check met an id outside its shard (one synchronisation)."""
        if self._tables is not None:
            self._tables[2].check("ShardTensor gather")

    def unregister(self):
        for p in self._opened:
            _C.lib().sgl_p2p_close(p)
        self._opened, self._bases, self._rows, self._local, self._tables = [], [], [], {}, None

    @staticmethod
    def gather_by_exchange(local: torch.Tensor, indices: torch.Tensor, group=None) -> torch.Tensor:
        """The same result without peer mappings, in the reference's five steps: ids ordered by owner, id exchange,
        gather at the owner, row exchange, rows put back in the order of ``indices``.  Collective over ``group``."""
        from ..route.exchange import exchange_rows
        from ..route.route import Route
        route, asked_rows, order = Route.all_to_all_ind2ptr(indices, group)
        mine = ops.gather_rows(local, asked_rows)                                   # what the others asked me for
        got = torch.empty((indices.numel(),) + tuple(local.shape[1:]), dtype=local.dtype, device=indices.device)
        exchange_rows(mine, route.recv_sizes, got, route.send_sizes, group).wait()  # rows arrive in owner order
        out = torch.empty_like(got)
        ops.scatter_rows(out, order, got)                                           # back to the order of the ids
        return out


def shared_empty(rows: int, row_shape, dtype=torch.float32):
    """A zero-filled CUDA tensor in memory of its own allocation, as inter-process handles need (a slice of torch's caching
    allocator cannot be exported on its own).  Returns the tensor; its memory is released with the tensor."""
    import ctypes as C
    n = int(rows)
    per = torch.empty(0, dtype=dtype).element_size()
    for d in row_shape:
        per *= int(d)
    nbytes = max(n * per, 256)
    base, handle = C.c_void_p(), C.create_string_buffer(64)
    _C.check(_C.lib().sgl_p2p_alloc(nbytes, C.byref(base), handle, 64))
    dev = torch.device("cuda", torch.cuda.current_device())
    t = _tensor_over(base.value, nbytes, dev).view(dtype)[: n * per // torch.empty(0, dtype=dtype).element_size()]
    t = t.view((n,) + tuple(int(d) for d in row_shape))
    _SHARED[t.data_ptr()] = (handle.raw, base)
    return t


_SHARED = {}   # data_ptr -> (ipc handle, base pointer) of tensors made by shared_empty


def _ipc_handle(t: torch.Tensor) -> bytes:
    hit = _SHARED.get(t.data_ptr())
    if hit is None:
        raise RuntimeError("ShardTensor: a shard that other processes map must be allocated with shared_empty()")
    return hit[0]


def _tensor_over(ptr: int, nbytes: int, dev) -> torch.Tensor:
    """uint8 tensor viewing foreign device memory through the CUDA array interface."""
    class _Mem:
        __cuda_array_interface__ = {"shape": (nbytes,), "typestr": "|u1", "data": (ptr, False), "version": 3}
    return torch.as_tensor(_Mem(), device=dev)
