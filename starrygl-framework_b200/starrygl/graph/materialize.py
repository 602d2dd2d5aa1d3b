"""Materialised mini-batches: the per-slot files of the reference's offline pipeline, built on the GPU.

``MaterializedMultiLayerBuilder`` has the constructor and the ``build_aligned_batch`` signature of the reference's
class (prepare_sample.py:179-406).  One call builds, for one task slice of one partition, the list of per-layer
dictionaries -- layer 0: ``gids``, ``ts``, ``inv_map``, ``num_neg`` + the task tensors + ``comm_plan``; layer l+1:
``indptr``, ``indices``, ``eid``, ``edge_ts``, ``edge_dt``, ``gids``, ``ts`` -- and writes it with ``torch.save`` in the
layout the reference's loader reads (all tensors on the CPU, ``comm_plan`` = one ``CommPlan`` or ``None`` per layer
list).  Sampling, (node, ts) relabel, CSC and the route plans run through the library
(``sgl_build_batch``, ``sgl_plan_routes``); the T-CSR is built once per partition.

Supported policy space = what the GPU sampler implements: continuous graphs (``graph_type == 'c'``), ``recent`` and
``uniform`` layers, ``end_offset`` 0 (strictly earlier edges) or 1 (edges at the query time included; integer
timestamps).  ``cluster`` / ``full`` layers and discrete graphs raise ``NotImplementedError``.  Negative destinations
of a ``'neg'`` task are drawn from a seeded torch generator (the reference draws from the unseeded global numpy state).
"""
import ctypes as C
import threading
from typing import List, Optional

import numpy as np
import torch

from .. import _C, ops
from ..cache.cache_route import CommPlan
from .batch import _EARLY, _HOP, _enqueue, _graph_range, _root_range


_PINNED_MOST, _PINNED_TOTAL = 256 << 20, 2 << 30
_SHARED_MOST = 32 << 20
_STAGE = threading.local()                # of a thread: pinned buffer for the roots of its tasks, a stream per device for early copies
_READY = 511                              # place of the word that says so among the thread's result words


def _pinned_now() -> int:
    """Bytes of pinned memory in use through torch's host allocator."""
    try:
        return int(torch._C._cuda_hostMemoryStats()["allocated_bytes"]["current"])      # (a tenth of the cost of the flat form)
    except (AttributeError, KeyError, TypeError):
        return int(torch.cuda.host_memory_stats().get("allocated_bytes.current", 0))


def _dev_i64(x, dev):
    if isinstance(x, np.ndarray):
        x = torch.from_numpy(np.ascontiguousarray(x))
    return x.to(dev, torch.int64).contiguous()


def prepare_distributed_metadata(node_parts, edge_index, num_parts: int, output_dir=None):
    """Partition book and replica table of a partitioned graph, in the reference's file layout
    (``prepare_distributed_metadata``, prepare_nparts_louvain.py:457-484).

    An event belongs to the partition of its destination.  ``partition_book[p]`` = the nodes partition p stores: the ones
    it owns (ascending id) followed by its halo -- sources of its events that another partition owns (ascending id).
    ``partition_book.pt`` holds ``(partition_book, node_parts, edge_parts)``, ``replica_table.pt`` the CSR over node id of
    every ``(rank, local slot)`` copy.  One-time set-up on whatever device the inputs live on; the files hold CPU tensors.
    Returns ``(partition_book, replica_table)``."""
    import os

    from ..cache.replica_table import build_replica_table
    node_parts = torch.as_tensor(node_parts, dtype=torch.int64)
    src, dst = (torch.as_tensor(x, dtype=torch.int64).to(node_parts.device) for x in edge_index)
    edge_parts = node_parts[dst]
    src_parts = node_parts[src]
    book = []
    for pid in range(int(num_parts)):
        owned = torch.nonzero(node_parts == pid, as_tuple=True)[0]
        halo = torch.unique(src[(edge_parts == pid) & (src_parts != pid)])
        book.append(torch.cat([owned, halo]).cpu())
    table = build_replica_table(node_parts.numel(), book, int(num_parts))
    if output_dir is not None:
        os.makedirs(output_dir, exist_ok=True)
        torch.save((book, node_parts.cpu(), edge_parts.cpu()), os.path.join(output_dir, "partition_book.pt"))
        torch.save(table, os.path.join(output_dir, "replica_table.pt"))
    return book, table


class MaterializedMultiLayerBuilder:
    def __init__(self, partition_data, num_nodes, node_parts, rep_table, pid, num_parts, device=None):
        dev = torch.device(device) if device is not None else torch.device("cuda", torch.cuda.current_device())
        if dev.type != "cuda":
            raise _C.SglError("MaterializedMultiLayerBuilder: the data path has no CPU implementation")
        self.device = dev
        src, dst, ts = (_dev_i64(partition_data[k], dev) for k in ("src", "dst", "ts"))
        eid = _dev_i64(partition_data["eid"], dev) if "eid" in partition_data else None
        if "cid" in partition_data and np.any(np.asarray(partition_data["cid"]) != 0):
            raise NotImplementedError("cluster ids: 'cluster' layers are not implemented on the GPU path")
        self.num_nodes = int(num_nodes)
        # rows keyed by the destination of an event, neighbour = its source, ascending time (prepare_sample.py:192-203)
        self.g = ops.tcsr_build(dst, src, ts, eid, self.num_nodes)
        self.node_parts = None if node_parts is None else _dev_i64(node_parts, dev)
        self.rep_table = None if rep_table is None else rep_table.to(dev)
        self.pid, self.num_parts = int(pid), int(num_parts)
        self.gen = torch.Generator(device="cpu")
        self.gen.manual_seed(0)

    def _roots(self, node_parts, ts_parts):
        """(nodes, times, (lowest, highest time)) of a task on the GPU: host arrays go through one pinned buffer and one copy,
        and their time range is read where they are."""
        parts = [x.numpy() if torch.is_tensor(x) and not x.is_cuda else x for x in (*node_parts, *ts_parts)]
        if not all(isinstance(x, np.ndarray) for x in parts):
            f = lambda xs: torch.cat([_dev_i64(x, self.device) for x in xs])
            return f(node_parts), f(ts_parts), None
        n, total = sum(len(x) for x in parts[:len(node_parts)]), sum(len(x) for x in parts)
        # (a buffer of this thread's own: several may build slots with one builder)
        if getattr(_STAGE, "buf", None) is None or _STAGE.buf.numel() < total:
            _STAGE.buf = torch.empty(max(2 * total, 1024), dtype=torch.int64, pin_memory=True)
        st, at = _STAGE.buf.numpy(), 0
        for x in parts:
            st[at:at + len(x)] = x
            at += len(x)
        d = _STAGE.buf[:total].to(self.device, non_blocking=True)     # (the slot's end waits for the stream)
        t = parts[len(node_parts)]
        return d[:n], d[n:], (int(t.min()), int(t.max())) if len(t) else None

    # ---- layers and route plans of one slot on the host (prepare_sample.py:266-310) -------------------------------
    def _build(self, roots, root_ts, ts_range, fanouts, policy, inclusive, seed) -> List[dict]:
        """Batch, then the plan of every layer list, all enqueued without a host round trip; the arrays that are there before the last list
        is merged cross PCIe next to that merge and the plans (8,000 roots, two hops, 8 MB: 437 us, so 390 - 407), the others after one
        read-back of every size."""
        g, P, hops = self.g, self.num_parts, len(fanouts)
        if ts_range is None:
            ts_range = _root_range(g, root_ts)
        planned = self.rep_table is not None and self.node_parts is not None and P > 1
        nb = 2 + 2 * hops
        meta = torch.empty(nb + ((hops + 1) * (P + 1) if planned else 0), dtype=torch.int64, device=self.device)
        lo, hi = _graph_range(g, *ts_range)
        addr, result = _C.host_words()
        staged = hops > 0 and roots.numel() > 0 and meta.numel() < _EARLY and _EARLY + nb < _READY
        early = copies = None
        try:
            db = _enqueue(g, roots, root_ts, fanouts, policy, lo, hi, inclusive, -1, seed, None, None, None, meta[:nb], True,
                          addr + 8 * _EARLY if staged else None, addr + 8 * _READY if staged else None)
            n, place = roots.numel(), db.addresses()
            plans, room = self._plan(place, n, fanouts, meta) if planned else ([], None)
            if staged:
                sp, wait = _C.stream_ptr(), _C.host().sgl_wait_word
                wait(addr + 8 * (_EARLY + nb - 1), 1, sp)
                counts = result[_EARLY:_EARLY + nb - 1]
                if 0 not in counts[1::2]:
                    picks = self._picks(place, counts, n, hops, "early")
                    copies = self._copies()
                    with _C.on_stream(copies):
                        early = list(zip(picks, self._export([p[2:] for p in picks], lambda: wait(addr + 8 * _READY, 1, sp))))
            return self._finish(db, meta, place, n, hops, plans, early)
        except BaseException:
            _C.abandon()
            raise
        finally:
            if copies is not None:                  # (whatever becomes of the slot: they write to memory of its own)
                copies.synchronize()

    def _plan(self, place, n, fanouts, meta):
        """Enqueues the route plan of every layer list; sizes go behind the batch's counts in ``meta``.  Returns (address, capacity) of
        every plan's arrays and the tensor that holds them."""
        P, nb = self.num_parts, 2 + 2 * len(fanouts)
        lists, c, t = [(place[0], n)], n, n         # (address of the ids, capacity) of every layer list
        for l, k in enumerate(fanouts):
            t *= k
            c += t
            lists.append((place[3 + 14 * l + 6], c))
        caps = [max(c * max(P - 1, 1), 1) for _, c in lists]
        room = torch.empty(3 * sum(caps), dtype=torch.int64, device=self.device)
        rt, sp, mp, at, plans = self.rep_table, _C.stream_ptr(), meta.data_ptr(), room.data_ptr(), []
        for cap in caps:
            plans.append((at, cap))
            at += 24 * cap
        k = len(lists)
        words = C.c_int64 * k
        ids, ns, cp = words(*[a for a, _ in lists]), words(*[c for _, c in lists]), words(*caps)
        d_ns, outs = words(*[mp + 16 * i for i in range(k)]), words(*[a for a, _ in plans])
        cnts = words(*[mp + 8 * (nb + i * (P + 1)) for i in range(k)])
        ref = C.addressof
        ws = _C.WORKSPACE.get(_C.host().sgl_plan_routes_ws_bytes(k, ref(ns), ref(cp)), self.device, sp)
        _C.host().sgl_plan_routes(k, ref(ids), ref(ns), ref(d_ns), self.node_parts.data_ptr(), self.node_parts.numel(), self.pid,
                                  rt.indptr.data_ptr(), rt.indices.data_ptr(), rt.locs.data_ptr(), P, ref(cp), ref(outs), ref(cnts),
                                  mp + 8 * (nb - 1), ws.data_ptr(), ws.numel(), sp)
        return plans, room

    def _copies(self):
        """The calling thread's stream for copies next to what its current stream does."""
        streams = _STAGE.__dict__.setdefault("streams", {})
        s = streams.get(self.device.index)
        if s is None:
            s = streams[self.device.index] = torch.cuda.Stream(self.device)
        return s

    @staticmethod
    def _picks(place, host, n, hops, part):
        """(layer, name, address, count, bytes per value) of the layers' arrays: those that are there before the last list is merged
        ("early"; the last of the counts is not looked at), the others ("late"), or all."""
        out = []

        def sec(layer, name, section, count, size=8, late=False):
            if part == "all" or late == (part == "late"):
                out.append((layer, name, place[section], count, size))
        sec(0, "gids", 0, host[0]); sec(0, "ts", 1, host[0]); sec(0, "inv_map", 2, n)
        for l in range(hops):
            e, b, last = host[1 + 2 * l], 3 + 14 * l, l + 1 == hops
            ip, ix, ts, dt, ei = (5, 8, 2, 3, 4) if l == 0 else (9, 10, 11, 12, 13)
            sec(l + 1, "indptr", b + ip, host[2 * l] + 1); sec(l + 1, "indices", b + ix, e, 8, last); sec(l + 1, "eid", b + ei, e)
            sec(l + 1, "edge_ts", b + ts, e); sec(l + 1, "edge_dt", b + dt, e, 4)
            sec(l + 1, "gids", b + 6, host[2 + 2 * l], 8, last); sec(l + 1, "ts", b + 7, host[2 + 2 * l], 8, last)
        return out

    def _finish(self, db, meta, place, n, hops, plans, early) -> List[dict]:
        """``early``: the early arrays of the layers on the host, on their way; None: nothing is."""
        P, nb = self.num_parts, 2 + 2 * hops
        host = _C.read_words(meta, meta.numel()) if meta.numel() < 512 else meta.tolist()    # the one synchronisation before the copy
        bits = host[nb - 1] & 0xFFFFFFFF
        if bits:
            raise _C.SglError(f"build_batch: device status {bits} ({_C.decode_status(bits)})")
        stopped = next((l for l in range(hops) if host[1 + 2 * l] == 0), None)
        layers = None
        if stopped is not None:                     # perhaps a hop without any edge, where the builder stops
            layers = db._trim(host[:nb - 1])
            if len(layers) == hops + 1 and layers[-1]["indptr"].numel() > 1:
                layers = None
        picks = self._picks(place, host, n, hops, "all" if early is None else "late") if layers is None else []
        sizes = [host[nb + i * (P + 1):nb + (i + 1) * (P + 1)] for i in range(len(plans))]
        routed = [(at + 8 * j * cap, s[P], 8) for (at, cap), s in zip(plans, sizes) for j in range(3)]
        got = self._export([p[2:] for p in picks] + routed)
        if layers is None:
            arrays = {p[:2]: t for p, t in [*(early or ()), *zip(picks, got)]}
            final = [{k: arrays[0, k] for k in ("gids", "ts", "inv_map")}]
            final += [{k: arrays[l, k] for k in _HOP} for l in range(1, hops + 1)]
            got = got[len(picks):]
        else:
            final = [{k: v.cpu() for k, v in d.items()} for d in layers]
        routes = []
        for i in range(len(final)):
            if not plans or sizes[i][P] == 0:
                routes.append(None)
            else:
                routes.append(CommPlan(send_ranks=got[3 * i], send_sizes=torch.tensor(sizes[i][:P], dtype=torch.int64),
                                       send_indices=got[3 * i + 1], send_remote_indices=got[3 * i + 2]))
        if len(final) >= 2 and final[-1]["indptr"].numel() == 1:
            routes[-1] = None                       # the reference stops at an empty layer with no plan for it
        final[0]["comm_plan"] = routes
        _C.current_stream(self.device).synchronize()               # the copies of _export
        return final

    def _export(self, picks, ready=None):
        """Host tensors of device arrays (address, count, bytes per value), on their way: the caller waits for the copies.  ``ready``
        returns once the arrays may be read.  Up to 32 MiB in all they are pieces of one buffer, packed by a kernel and filled by one
        copy, above that (and above the kernel's 96 arrays, nine hops) each has its own.
        The memory is pinned (a copy to fresh pageable memory takes several times as long) as long as not too much is."""
        n, at, offs = len(picks), 0, []
        for _, count, size in picks:
            offs.append(at)
            at += (count * size + 15) & ~15
        pin = at <= _PINNED_MOST and _pinned_now() + at <= _PINNED_TOTAL
        src, size = (C.c_void_p * max(n, 1))(*[p[0] for p in picks]), (C.c_int64 * max(n, 1))(*[p[1] * p[2] for p in picks])
        types = {8: torch.int64, 4: torch.float32}
        if at > _SHARED_MOST or n > 96:
            out = [torch.empty(count, dtype=types[s], pin_memory=pin) for _, count, s in picks]
            if ready is not None:
                ready()
            _C.check(_C.lib().sgl_copy_arrays(n, src, size, (C.c_void_p * n)(*[t.data_ptr() for t in out]), _C.stream_ptr()))
            return out
        h = torch.empty(at // 8, dtype=torch.int64, pin_memory=pin)
        d = torch.empty(max(at, 16) // 8, dtype=torch.int64, device=self.device)
        places, ref = (C.c_int64 * max(n, 1))(*offs), C.addressof
        if ready is not None:
            ready()
        _C.host().sgl_export_arrays(n, ref(src), ref(size), ref(places), d.data_ptr(), h.data_ptr(), at, None, at, _C.stream_ptr())
        # (pieces with a storage of their own size: what saves or shares one does not take the others along)
        buf = h.numpy()
        return [torch.frombuffer(buf, dtype=types[s], count=count, offset=o) if count else torch.empty(0, dtype=types[s])
                for o, (_, count, s) in zip(offs, picks)]

    # ---- one slot ------------------------------------------------------------------------------------------------
    def build_aligned_batch(self, task_param, save_path, layer_configs, num_neg=1, global_dst_pool=None, cluster_ids=None,
                            seed: Optional[int] = None) -> List[dict]:
        task_type, task_nodes = task_param
        dev = self.device
        extra = {}
        if task_type == 'link':
            task_src, task_dst, task_ts, task_label, task_eid = task_nodes
            l0_nodes, l0_ts, ts_range = self._roots((task_src, task_dst), (task_ts, task_ts))
            extra = {"task_ts": task_ts, "task_src": task_src, "task_dst": task_dst, "task_label": task_label,
                     "task_eid": task_eid}
        elif task_type == 'node':
            task_node, task_ts, task_label = task_nodes
            l0_nodes, l0_ts, ts_range = self._roots((task_node,), (task_ts,))
            extra = {"task_node": task_node, "task_ts": task_ts, "task_label": task_label}
        elif task_type == 'neg':
            if num_neg <= 0 or global_dst_pool is None:
                raise ValueError("a 'neg' task needs num_neg > 0 and a destination pool")
            task_ts = task_nodes
            pool = torch.as_tensor(np.asarray(global_dst_pool), dtype=torch.int64)
            if seed is not None:
                self.gen.manual_seed(int(seed))
            pick = torch.randint(0, pool.numel(), (len(task_ts) * num_neg,), generator=self.gen)
            neg = pool[pick]
            l0_nodes = neg.to(dev)
            l0_ts, ts_range = _dev_i64(task_ts, dev).repeat_interleave(num_neg), None
            extra = {"task_nodes": neg, "task_ts": task_ts, "task_label": 'neg_set'}
        else:
            raise ValueError(f"Unsupported task type: {task_type}")

        meta = layer_configs.get('meta', {})
        if meta.get('graph_type', 'c') != 'c':
            raise NotImplementedError("discrete graphs (graph_type != 'c') are not implemented on the GPU path")
        end_offset = int(meta.get('end_offset', 0))
        if end_offset not in (0, 1):
            raise NotImplementedError("end_offset must be 0 (edges strictly before the query time) or 1 (inclusive)")
        kinds = {c['type'] for c in layer_configs['layer']}
        if not kinds <= {'recent', 'uniform'}:
            raise NotImplementedError(f"layer types {sorted(kinds - {'recent', 'uniform'})} are not implemented on the GPU path")
        if len(kinds) > 1:
            raise NotImplementedError("all layers of a batch use one policy")
        policy = kinds.pop() if kinds else 'recent'
        fanouts = [int(c['fanout']) for c in layer_configs['layer']]

        seed = 0 if seed is None else int(seed)
        final = self._build(l0_nodes, l0_ts, ts_range, fanouts, policy, bool(end_offset), seed)

        def host(x):
            if isinstance(x, np.ndarray):
                return torch.from_numpy(x)
            return x.cpu() if torch.is_tensor(x) else x
        final[0]["num_neg"] = num_neg
        final[0].update({k: host(v) for k, v in extra.items()})
        if save_path is not None:
            torch.save(final, save_path)
        return final
