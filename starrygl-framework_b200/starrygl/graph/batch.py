"""Multi-hop mini-batch builder on the GPU: sampling, (node, ts)-pair dedup/relabel and per-hop CSC.

Produces the per-layer dictionaries of the reference's offline builder
(``MaterializedMultiLayerBuilder.build_aligned_batch``, prepare_sample.py:313-377) without its route
planning: layer 0 = sorted unique (id, ts) pairs of the roots + ``inv_map``; layer l+1 = CSC over the
previous list (``indptr``, ``indices``, ``eid``, ``edge_ts``, ``edge_dt``) + the merged sorted pair list
(``gids``, ``ts``).  All hops are enqueued on the current stream without an intermediate host
synchronisation: the number of edges a hop produced is handed to the next kernels as a device count.
``finish()`` performs the single synchronisation that is needed to give the tensors their final shapes.
"""
import ctypes as C
from collections import OrderedDict
from typing import List, Optional, Sequence

import torch

from .. import _C, ops


# Results up to this size share one allocation (a tensor that is kept keeps the others' memory), together with the raw arrays when
# they are small; larger ones have an allocation each.
_SHARED_MOST, _WHOLE_MOST = 32 << 20, 2 << 20


class _Plan:
    """What a batch of one shape (number of roots, fan-outs) needs: the size of every section and where it goes, the scratch
    size and the fan-outs as the library reads them.  Sections that :meth:`DeviceBatch.finish` returns are kept apart from the
    raw arrays of the hops, which go with the :class:`DeviceBatch`."""

    def __init__(self, n: int, fanouts: Sequence[int]):
        L = _C.lib()
        hops = len(fanouts)
        self.fan = (C.c_int32 * max(hops, 1))(*[int(k) for k in fanouts])
        self.places = C.c_int64 * (3 + 14 * hops)
        sec = self.places()
        if int(L.sgl_build_batch_layout(n, self.fan, hops, sec)) < 0:
            raise _C.SglError("build_batch: bad batch shape")
        self.ws_bytes = int(L.sgl_build_batch_ws_bytes(n, self.fan, hops))
        self.size = [int(w) for w in sec]
        kept = [0, 1, 2]
        for l in range(hops):
            kept += [3 + 14 * l + i for i in ((2, 3, 4, 5, 6, 7, 8) if l == 0 else (6, 7, 9, 10, 11, 12, 13))]
        self.kept = kept
        self.whole = 8 * sum(self.size) <= _WHOLE_MOST
        start, words, raw = [0] * len(self.size), 0, 0       # place in the results, or -1 - place in the raw arrays
        for s in kept:
            start[s] = words
            words += self.size[s]
        for s in sorted(set(range(len(self.size))) - set(kept)):
            if self.whole:
                start[s] = words
                words += self.size[s]
            else:
                start[s] = -1 - raw
                raw += self.size[s]
        self.start, self.at, self.words, self.raw_words = start, self.places(*start), words, raw
        self.fan_at, self.at_at = C.addressof(self.fan), C.addressof(self.at)
        self.shared = 8 * words <= _SHARED_MOST


_PLANS: "OrderedDict" = OrderedDict()


def _plan(n, fanouts) -> _Plan:
    key = (n, *fanouts)
    p = _PLANS.get(key)
    if p is None:
        p = _PLANS[key] = _Plan(n, fanouts)
        if len(_PLANS) > 64:
            _PLANS.popitem(last=False)
    return p


_HOP = ("indptr", "indices", "eid", "edge_ts", "edge_dt", "gids", "ts")     # of a layer behind the roots


class _MetaStatus(ops.StatusWord):
    """The status word of a batch that came without one: the last word of its meta block."""

    def __init__(self, meta):
        self.t = meta[-1:].view(torch.int32)[:1]


class DeviceBatch:
    """Un-trimmed result of :func:`build_batch_async`: every array at capacity, the counts on the device.  ``results``: one tensor
    for all sections that a caller gets to keep, or a dictionary of one each; ``raw``: the others."""

    def __init__(self, g, n, fanouts, plan, results, raw, meta, status):
        self.g, self.n, self.fanouts = g, n, list(fanouts)
        self._plan, self._results, self._raw, self._own_meta, self._status = plan, results, raw, meta, status
        self._shared = not isinstance(results, dict)
        self._layers = None

    @property
    def _meta(self):
        """Counts and status word: the block that was given, or the end of the raw arrays."""
        if self._own_meta is None:
            self._own_meta = self._raw[self._raw.numel() - (2 + 2 * len(self.fanouts)):]
        return self._own_meta

    @property
    def status(self):
        if self._status is None:
            self._status = _MetaStatus(self._meta)
        return self._status

    @property
    def counts(self):
        """Device int64 scalars (1-element tensors): root list, then per hop sampled edges and merged list."""
        return [self._meta[i:i + 1] for i in range(1 + 2 * len(self.fanouts))]

    def _place(self, section):
        """(tensor, offset) of a section."""
        s = self._plan.start[section]
        if s < 0:
            return self._raw, -1 - s
        return (self._results, s) if self._shared else (self._results[section], 0)

    def _view(self, section, count, floats=False):
        t, s = self._place(section)
        if floats:
            return t[s:s + (count + 1) // 2].view(torch.float32)[:count]
        return t[s:s + count]

    def addresses(self):
        """Address of every section (0: a raw array)."""
        start = self._plan.start
        if not self._shared:
            return [0 if s < 0 else self._results[i].data_ptr() for i, s in enumerate(start)]
        base = self._results.data_ptr()
        return [0 if s < 0 else base + 8 * s for s in start]

    @property
    def layers(self):
        """Capacity-sized tensors per layer."""
        if self._layers is None:
            v, n = self._view, self.n
            out = [{"gids": v(0, n), "ts": v(1, n), "inv_map": v(2, n)}]
            t = c = n
            counts = self.counts
            for l, k in enumerate(self.fanouts):
                b, e = 3 + 14 * l, t * k
                hop = ops.Hop(v(b, e), v(b + 1, e), v(b + 2, e), v(b + 3, e, True), v(b + 4, e), v(b + 5, t + 1), e)
                d = {"raw_nbr": hop.nbr, "raw_ts": hop.ts, "inv": v(b + 8, e), "hop": hop, "gids": v(b + 6, c + e), "ts": v(b + 7, c + e)}
                if l == 0:
                    d.update(indptr=hop.offsets, indices=d["inv"], eid=hop.eid, edge_ts=hop.ts, edge_dt=hop.dt)
                else:
                    d.update(indptr=v(b + 9, c + 1), indices=v(b + 10, e), edge_ts=v(b + 11, e), edge_dt=v(b + 12, e, True), eid=v(b + 13, e))
                out.append(d)
                t, c = e, c + e
            self._layers = out
        return self._layers

    def _read(self):
        """The one read-back: every count and, when the batch owns it, the status word."""
        n = 2 + 2 * len(self.fanouts)
        host = _C.read_words(self._meta, n) if n < 512 else self._meta.tolist()
        return host[:-1], host[-1] & 0xFFFFFFFF

    def finish(self) -> List[dict]:
        """One host synchronisation: read every count, check the device status word, trim the arrays."""
        host, bits = self._read()
        if isinstance(self._status, ops.StatusWord) and not isinstance(self._status, _MetaStatus):
            self._status.check("build_batch")
        elif bits:
            raise _C.SglError(f"build_batch: device status {bits} ({_C.decode_status(bits)})")
        return self._trim(host)

    def _cuts(self, pieces):
        """Views of the first ``count`` values of sections, (section, count, fp32?) thrice each."""
        if not self._shared:
            return [self._view(*pieces[i:i + 3]) for i in range(0, len(pieces), 3)]
        at = self._plan.start
        return _C.host().cuts(self._results, *[at[x] if i % 3 == 0 else x for i, x in enumerate(pieces)])

    def _trim(self, host):
        self._host = host
        hops = len(self.fanouts)
        if 0 not in host[1:2 * hops + 1:2]:
            out, last = self._trim_but_last(host)
            if hops:
                out[-1]["gids"], out[-1]["ts"] = last(host[-1])
            return out
        first = self._cuts((0, host[0], 0, 1, host[0], 0, 2, self.n, 0))
        out, prev_n = [dict(zip(("gids", "ts", "inv_map"), first))], host[0]
        for l in range(hops):
            n_edges, n_next = host[1 + 2 * l], host[2 + 2 * l]
            if n_edges == 0 and not self._any_target_has_edges(l, out):
                # the reference emits an empty layer and stops when no target has any edge at all
                # (prepare_sample.py:352-361)
                z = torch.zeros(0, dtype=torch.int64, device=self.g.device)
                out.append({"indptr": torch.zeros(1, dtype=torch.int64, device=self.g.device), "indices": z,
                            "eid": z, "edge_ts": z, "edge_dt": torch.zeros(0, dtype=torch.float32, device=self.g.device),
                            "gids": z, "ts": z})
                break
            out.append(dict(zip(_HOP, self._cuts(self._hop(l, prev_n, n_edges) + (3 + 14 * l + 6, n_next, 0, 3 + 14 * l + 7, n_next, 0)))))
            prev_n = n_next
        return out

    @staticmethod
    def _hop(l, prev_n, n_edges):
        b = 3 + 14 * l
        # (the first hop's edges are in CSC order as they were sampled, see sgl_build_batch)
        ip, ix, ts, dt, ei = (b + 5, b + 8, b + 2, b + 3, b + 4) if l == 0 else (b + 9, b + 10, b + 11, b + 12, b + 13)
        return ip, prev_n + 1, 0, ix, n_edges, 0, ei, n_edges, 0, ts, n_edges, 0, dt, n_edges, 1

    def _trim_but_last(self, host):
        """The layers as :meth:`_trim` returns them without the last list, whose length ``host`` does not say yet, and a function of
        that length for its two arrays; None where a hop has no edges."""
        hops = len(self.fanouts)
        if 0 in host[1:2 * hops:2]:
            return None
        pieces, prev_n = (0, host[0], 0, 1, host[0], 0, 2, self.n, 0), host[0]
        for l in range(hops):
            pieces += self._hop(l, prev_n, host[1 + 2 * l])
            if l + 1 < hops:
                prev_n = host[2 + 2 * l]
                pieces += (3 + 14 * l + 6, prev_n, 0, 3 + 14 * l + 7, prev_n, 0)
        got = self._cuts(pieces)
        out = [dict(zip(("gids", "ts", "inv_map"), got))]
        for l in range(hops):
            out.append(dict(zip(_HOP if l + 1 < hops else _HOP[:5], got[3 + 7 * l:10 + 7 * l])))
        b = 3 + 14 * (hops - 1)
        return out, lambda n: self._cuts((b + 6, n, 0, b + 7, n, 0))

    def _any_target_has_edges(self, l, out):
        tgt = out[0]["gids"] if l == 0 else self._view(3 + 14 * (l - 1), self._host[1 + 2 * (l - 1)])
        if tgt.numel() == 0:
            return False
        deg = self.g.indptr[tgt + 1] - self.g.indptr[tgt]
        return bool((deg > 0).any().item())


def _enqueue(g, roots, root_ts, fanouts, policy, lo, hi, equal_root_time, allowed_offset, seed, status, side, host=None,
             meta=None, together=False, early=None, ready=None) -> DeviceBatch:
    """``lo`` / ``hi``: lowest and highest timestamp that can occur; ``host``: pinned address that receives the counts, ``early`` one
    that receives all but the last while the last list is merged, ``ready`` that of a word that becomes 1 when everything else is there;
    ``meta``: block of 2 + 2 * hops device words for the counts and the status (default: behind the raw arrays);
    ``together``: one allocation for the results whatever their size (for callers that keep none of them)."""
    n, hops = roots.numel(), len(fanouts)
    plan = _plan(n, fanouts)
    at, words, kept = plan.at_at, plan.words, None
    if not (plan.whole or plan.shared or together):
        kept = {s: torch.empty(plan.size[s], dtype=torch.int64, device=g.device) for s in plan.kept}
        places, words = plan.places(*plan.at), 0
        for s, t in kept.items():
            places[s] = t.data_ptr() // 8
        at = C.addressof(places)
    results, raw = _C.host().build_batch(
        g.indptr, g.nbr, g.ts, g.eid, g.fence, g.num_nodes, roots, root_ts, plan.fan_at, hops,
        _C.POLICY[policy] if isinstance(policy, str) else int(policy), bool(equal_root_time), int(allowed_offset), int(seed),
        ops.bits_for(g.num_nodes - 1), ops.bits_for(hi - lo), lo, at, words, -1 if plan.whole else plan.raw_words,
        2 + 2 * hops if meta is None else 0, meta, plan.ws_bytes, None if status is None else status.ptr(), host, early, ready,
        None if side is None else side.cuda_stream)
    return DeviceBatch(g, n, fanouts, plan, results if kept is None else kept, raw, meta, status)


def _graph_range(g, lo, hi):
    """Timestamps of the batch's lists: the queries' and the graph's."""
    return min(g.ts_min, lo), max(g.ts_max, hi)


def build_batch_async(g: ops.TCSR, roots: torch.Tensor, root_ts: torch.Tensor, fanouts: Sequence[int],
                      policy: str = "recent", *, ts_range: Optional[Sequence[int]] = None, equal_root_time=False,
                      allowed_offset=-1, seed=0, status: Optional[ops.StatusWord] = None,
                      side_streams: Optional[Sequence[torch.cuda.Stream]] = None) -> DeviceBatch:
    """Enqueue the whole batch construction on the current stream, in one foreign call.

    ``ts_range`` = (lowest, highest) timestamp that can occur among the roots' query times; together with the
    graph's own timestamp range it fixes the width of the (id, ts) sort key.  When omitted it is read from
    ``root_ts`` (one extra synchronisation).

    Hop l+1 samples the raw output of hop l, and a hop's CSC needs the relabel before it but not its own: with several hops
    both run next to the relabels and are joined into the current stream.  ``side_streams`` (the first is used) is needed
    for that only while a CUDA graph is being captured.
    """
    if ts_range is None:
        ts_range = _root_range(g, root_ts)
    lo, hi = _graph_range(g, int(ts_range[0]), int(ts_range[1]))
    fanouts = list(fanouts)
    return _enqueue(g, roots, root_ts, fanouts, policy, lo, hi, equal_root_time, allowed_offset, seed, status,
                    side_streams[0] if side_streams else None)


def _root_range(g, root_ts):
    if not root_ts.numel():
        return g.ts_min, g.ts_max
    lo, hi = torch.stack(root_ts.aminmax()).tolist()
    return lo, hi


_EARLY = 256                 # place of the early counts among the thread's result words
_SYNC_OPTIONS = {"ts_range", "equal_root_time", "allowed_offset", "seed"}


def build_batch(g, roots, root_ts, fanouts, policy="recent", **kw) -> List[dict]:
    """Synchronous form of :func:`build_batch_async`."""
    if kw.get("ts_range") is not None or not _SYNC_OPTIONS.issuperset(kw):
        return build_batch_async(g, roots, root_ts, fanouts, policy, **kw).finish()
    # Query times nearly always lie in the graph's own time range (events of the stream): the batch is enqueued with that range
    # instead of waiting for the smallest and largest query time.  The kernels flag a time outside of it; then the range is read
    # and the batch built again, and while a graph's queries stay outside they are read first.  Only that is remembered: the
    # width of the sort keys is always that of the batch at hand.
    fanouts = list(fanouts)
    if g.__dict__.get("_queried_outside", False):
        a, b = _root_range(g, root_ts)
        g.__dict__["_queried_outside"] = a < g.ts_min or b > g.ts_max
        return build_batch_async(g, roots, root_ts, fanouts, policy, **{**kw, "ts_range": (a, b)}).finish()
    addr, words = _C.host_words()
    last = 1 + 2 * len(fanouts)
    if last + 2 > len(words):
        return build_batch_async(g, roots, root_ts, fanouts, policy, **kw).finish()
    staged = bool(fanouts) and roots.numel() > 0 and last + 2 <= _EARLY
    try:
        db = _enqueue(g, roots, root_ts, fanouts, policy, g.ts_min, g.ts_max, kw.get("equal_root_time", False), kw.get("allowed_offset", -1),
                      kw.get("seed", 0), None, None, addr, early=addr + 8 * _EARLY if staged else None)
        wait, sp, laid = _C.host().sgl_wait_word, _C.stream_ptr(), None     # (not in front of it: the device waits for nothing else)
        if staged:
            # laid out while the device merges the last list: a fifth of a small batch's time is the making of tensors
            wait(addr + 8 * (_EARLY + last), 1, sp)
            laid = db._trim_but_last(words[_EARLY:_EARLY + last])
        wait(addr + 8 * (last + 1), 1, sp)
    except BaseException:
        _C.abandon()
        raise
    host, bits = words[:last], words[last] & 0xFFFFFFFF
    if bits & 2:
        g.__dict__["_queried_outside"] = True
        return build_batch(g, roots, root_ts, fanouts, policy, **kw)
    if bits:
        raise _C.SglError(f"build_batch: device status {bits} ({_C.decode_status(bits)})")
    if laid is None:
        return db._trim(host)
    out, last_list = laid
    out[-1]["gids"], out[-1]["ts"] = last_list(host[-1])
    return out


def batch_kernel_launches(num_nodes: int, num_roots: int, fanouts: Sequence[int], ts_span: int) -> int:
    """Kernels of this library that one mini-batch of :func:`build_batch_async` launches at the given capacities: count and
    fill of every hop, the sort of every relabel (above the mini-batch sort's limit with a delivery
    kernel more), and for every hop after the first the two CSC kernels, the sort behind them and the column map."""
    L = _C.lib()
    id_bits, ts_bits = ops.bits_for(num_nodes - 1), ops.bits_for(ts_span)

    def sort(n, bits):
        k = L.sgl_radix_sort_launches(n, bits)
        return k if k <= 2 else k + 1
    total = sort(num_roots, id_bits + ts_bits)
    cur, targets = num_roots, num_roots
    for l, k in enumerate(fanouts):
        edges = targets * k
        total += 2 + sort(cur + edges, id_bits + ts_bits)
        total += 0 if l == 0 else 1 + (2 if edges > 2048 else 0) + sort(edges, ops.bits_for(cur) + ts_bits)
        cur, targets = cur + edges, edges
    return int(total)


class BatchGraph:
    """The whole multi-hop batch construction of :func:`build_batch_async` captured once as a CUDA graph for a fixed
    number of roots, and replayed per mini-batch.  The plain call is submitted as one graph launch too and on a stream of its
    own is the faster of the two (4,096 roots uniform [10, 10]: 0.103 ms a batch, 0.111 as a replay); a replay costs the host one
    launch and two copies and is for callers that drive several batches side by side (four in flight: 0.068 ms a batch).

    The result tensors are the same objects for every batch: consume (or copy) a result before the next ``run``.
    """

    def __init__(self, g: ops.TCSR, num_roots: int, fanouts: Sequence[int], policy: str = "recent", *,
                 ts_range: Sequence[int], equal_root_time=False, allowed_offset=-1, seed=0,
                 stream: Optional[torch.cuda.Stream] = None):
        dev = g.device
        self.g, self.num_roots = g, int(num_roots)
        self.stream = stream or torch.cuda.Stream(dev)
        self.roots = torch.zeros(self.num_roots, dtype=torch.int64, device=dev)
        self.root_ts = torch.full((self.num_roots,), int(ts_range[0]), dtype=torch.int64, device=dev)
        self.status = ops.StatusWord(dev)
        self._side = [torch.cuda.Stream(dev)]
        kw = dict(ts_range=ts_range, equal_root_time=equal_root_time, allowed_offset=allowed_offset, seed=seed,
                  status=self.status, side_streams=self._side)
        # scratch used inside the graph must not be shared with eager calls: the capture gets its own workspace
        saved = _C.WORKSPACE
        _C.WORKSPACE = self._workspace = _C.Workspace()
        try:
            torch.cuda.synchronize(dev)
            with torch.cuda.stream(self.stream):
                build_batch_async(g, self.roots, self.root_ts, fanouts, policy, **kw)     # warm-up: sizes the scratch
            self.stream.synchronize()
            self.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(self.graph, stream=self.stream):
                self.batch = build_batch_async(g, self.roots, self.root_ts, fanouts, policy, **kw)
        finally:
            _C.WORKSPACE = saved
        self.stream.synchronize()
        self.kernel_launches = batch_kernel_launches(g.num_nodes, self.num_roots, fanouts, int(ts_range[1]) - min(g.ts_min, int(ts_range[0])))

    def run(self, roots: torch.Tensor, root_ts: torch.Tensor) -> DeviceBatch:
        """Enqueue one batch (exactly ``num_roots`` roots, already on the GPU); returns the un-trimmed device batch,
        whose ``finish()`` synchronises and trims."""
        if roots.numel() != self.num_roots:
            raise ValueError(f"this graph was captured for {self.num_roots} roots, got {roots.numel()}")
        with torch.cuda.stream(self.stream):
            self.roots.copy_(roots, non_blocking=True)
            self.root_ts.copy_(root_ts, non_blocking=True)
            self.graph.replay()
        return self.batch
