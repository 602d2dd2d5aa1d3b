"""Performance cases of the mini-batch data path: what a temporal-GNN training program asks of this framework per
batch, slot or partition, through the public entry points.

Nine kinds of work (``kind`` of a case):

  tcsr      build the time-sorted adjacency (and its search index) of a partition's event list
  sample    one hop of temporal neighbour sampling, cut to size
  batch     whole mini-batch: (node, time) relabel, every hop, per-hop CSC
  prefetch  mini-batches from pinned host roots through the prefetcher: sampling + edge-feature rows
  cache     node-feature rows through the device cache, with the list of misses
  state     node memory: read rows and times of a batch's nodes, write the updated ones back
  mail      mailbox step: read messages, newest message per node of a batch, write it to the mailbox
  query     the asynchronous graph API: time windows queued, sampled, relabelled and assembled to blocks
  slot      one slot of the offline builder: layers plus the route plan of every layer, on the host

Sizes are those of the repository's configurations (160 k to 50 M events; 200-event to 32 x 4,000-event batches with
three roots per event; recent-10 / recent-20 / uniform [10,10]; rows of 100, 128, 172 and 186 values, fp32 and bf16;
10 M-row node table behind a 10 % cache; 312,500-node partitions).  Graphs have power-law out-degrees and events in
time order unless a case says otherwise.  Every result is integer or copied bytes: all cases compare exactly.
"""
import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "starrygl-framework_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from starrygl import ops  # noqa: E402
from starrygl.cache.NodeState import DistNodeState  # noqa: E402
from starrygl.cache.replica_table import CSRReplicaTable  # noqa: E402
from starrygl.data.prefetcher import HostToDevicePrefetcher  # noqa: E402
from starrygl.graph.batch import build_batch  # noqa: E402
from starrygl.graph.graph import AsyncBlock, pyGraph  # noqa: E402
from starrygl.graph.materialize import MaterializedMultiLayerBuilder  # noqa: E402
from starrygl.nn.memory.mailbox import mailbox  # noqa: E402
from starrygl.utils.partition_book import PartitionState  # noqa: E402

I64 = torch.int64
TS_MAX = 10_000_000


# ------------------------------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------------------------------

def listed():
    return [
        # the small configuration's whole training set becomes an adjacency: 160 k events in time order
        dict(name="tcsr_160k", kind="tcsr", nodes=10_000, edges=160_000, ordered=True),
        # the sampler benchmark's graph, events in no particular order: the largest single build of the repository's
        # configurations that runs on one partition
        dict(name="tcsr_50m", kind="tcsr", nodes=1_000_000, edges=50_000_000, ordered=False),
        # one hop for a 32 x 4,000-event mega-batch (source, destination, negative of every event)
        dict(name="sample_recent20_384k", kind="sample", nodes=1_000_000, edges=50_000_000, roots=384_000, fanout=20,
             policy="recent", offset=-1, inclusive=False),
        # a training batch of the small configuration: 200 events, one negative each, one layer of 10 most recent
        dict(name="batch_recent10_600", kind="batch", nodes=10_000, edges=160_000, roots=600, fanouts="10", policy="recent"),
        # the sampler benchmark's two-hop batch
        dict(name="batch_uniform10x10_4096", kind="batch", nodes=1_000_000, edges=50_000_000, roots=4096, fanouts="10,10",
             policy="uniform"),
        # the two-layer model's mega-batch: 32 x 4,000 events
        dict(name="batch_uniform10x10_384k", kind="batch", nodes=1_000_000, edges=50_000_000, roots=384_000, fanouts="10,10",
             policy="uniform"),
        # the single-GPU training loop's input side: four batches of 4,096 roots in flight, 172-value edge features
        dict(name="prefetch_recent20_4x4096", kind="prefetch", nodes=200_000, edges=8_000_000, roots=4096, batches=4, fanout=20,
             policy="recent", dim=172, dtype="float32"),
        # node features of one batch's 200,000 ids through a 10 % cache, stored in bf16
        dict(name="cache_bf16_200k", kind="cache", rows=10_000_000, dim=128, dtype="bfloat16", ids=200_000, share=0.1),
        # memory of the distributed configuration's partition: 4,000 events, recent-10
        dict(name="state_132k_of_312k", kind="state", nodes=312_500, all_nodes=2_500_000, dim=100, reads=132_000, writes=12_000),
        # messages of the same batch: 4,000 events, memory 100 + 100, edge features 172
        dict(name="mail_4000", kind="mail", nodes=312_500, slots=1, dim=100, edge_dim=172, events=4000),
        # the graph API's two-layer query for a window of about 1,000 events plus as many negatives
        dict(name="query_1000_events", kind="query", nodes=50_000, edges=2_000_000, events=1000, windows=2, layers=2, fanout=10,
             policy="recent"),
        # one slot of the offline pipeline on one of four partitions
        dict(name="slot_4000_events", kind="slot", nodes=200_000, edges=2_000_000, events=4000, fanouts="10,10", policy="recent",
             parts=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _graph_size(rng, hi=50_000_000):
    m = _log_int(rng, 160_000, hi)
    return dict(nodes=max(1000, int(m / rng.uniform(10, 60))), edges=m)


def draw(rng):
    kind = rng.choice(["tcsr", "sample", "batch", "prefetch", "cache", "state", "mail", "query", "slot"])
    policy = rng.choice(["recent", "uniform"])
    if kind == "tcsr":
        return dict(kind=kind, ordered=rng.random() < 0.5, **_graph_size(rng))
    if kind == "sample":
        return dict(kind=kind, roots=_log_int(rng, 200, 384_000), fanout=rng.choice([5, 10, 15, 20]), policy=policy,
                    offset=rng.choice([-1, -1, TS_MAX // 20]), inclusive=rng.random() < 0.25, **_graph_size(rng))
    if kind == "batch":
        return dict(kind=kind, roots=_log_int(rng, 200, 384_000), fanouts=rng.choice(["10", "20", "5,5", "10,5", "10,10"]),
                    policy=policy, **_graph_size(rng))
    if kind == "prefetch":
        return dict(kind=kind, roots=_log_int(rng, 200, 8192), batches=rng.randint(2, 6), fanout=rng.choice([10, 20]),
                    policy=policy, dim=rng.choice([100, 128, 172, 186]), dtype=rng.choice(["float32", "float32", "bfloat16"]),
                    **_graph_size(rng, 8_000_000))
    if kind == "cache":
        return dict(kind=kind, rows=_log_int(rng, 200_000, 10_000_000), dim=rng.choice([64, 100, 128, 172, 256]),
                    dtype=rng.choice(["float32", "bfloat16"]), ids=_log_int(rng, 2000, 400_000), share=rng.choice([0.05, 0.1, 0.3]))
    if kind == "state":
        n = _log_int(rng, 10_000, 2_000_000)
        w = _log_int(rng, 200, min(n // 2, 100_000))
        return dict(kind=kind, nodes=n, all_nodes=n * rng.randint(1, 8), dim=rng.choice([64, 100, 128, 172, 372]),
                    reads=w * rng.randint(1, 11), writes=w)
    if kind == "mail":
        slots = rng.choice([1, 1, 10])
        return dict(kind=kind, nodes=_log_int(rng, 10_000, 1_000_000 // slots), slots=slots, dim=rng.choice([64, 100, 128]),
                    edge_dim=rng.choice([16, 172, 186]), events=_log_int(rng, 200, 32_000))
    if kind == "query":
        return dict(kind=kind, events=_log_int(rng, 100, 10_000), windows=rng.randint(1, 3), layers=rng.randint(1, 2),
                    fanout=rng.choice([5, 10, 20]), policy=policy, **_graph_size(rng, 4_000_000))
    return dict(kind=kind, events=_log_int(rng, 200, 16_000), fanouts=rng.choice(["10", "5,5", "10,10"]), policy=policy,
                parts=rng.randint(2, 8), **_graph_size(rng, 4_000_000))


# ------------------------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------------------------

def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _events(nodes, edges, gen, ordered=True):
    """Sources with a power-law out-degree (exponent 2.1), uniform destinations, times uniform in [0, 1e7)."""
    dev = _dev()
    w = torch.rand(nodes, device=dev, generator=gen).clamp_min_(1e-9).pow_(-1.0 / 1.1).double()
    cdf = torch.cumsum(w, 0)
    cdf /= cdf[-1].clone()
    src = torch.searchsorted(cdf, torch.rand(edges, device=dev, dtype=torch.double, generator=gen)).clamp_max_(nodes - 1)
    dst = torch.randint(0, nodes, (edges,), device=dev, generator=gen)
    ts = (torch.rand(edges, device=dev, dtype=torch.double, generator=gen) * TS_MAX).long()
    if ordered:
        ts = ts.sort().values
    return src, dst, ts, torch.arange(edges, device=dev)


class _Names:
    """The number of sampled edges and of distinct pairs is a property of a graph's shape.  So that a case has one amount
    of work, its shape comes from its sizes alone (``shape``); the seed renames it: ids move to other places of the id
    space in the same order, times by a constant (``node`` and ``time``).  A fifth of the ids stays without events."""

    def __init__(self, case, gen):
        dev = _dev()
        self.shape = torch.Generator(device=dev).manual_seed(1 + case["nodes"])
        self.active = int(case["nodes"] * 0.8)
        gaps = torch.rand(self.active, device=dev, generator=gen) < 0.15
        self._id = ((1 + gaps.long()).cumsum(0) - 1).clamp_max_(case["nodes"] - 1)
        self._shift = int(torch.randint(0, TS_MAX, (1,), device=dev, generator=gen))

    def node(self, v):
        return self._id[v]

    def time(self, t):
        return t + self._shift


def _roots(src, ts, n, gen):
    """Roots as link prediction asks for them: an event's source at the event's own time."""
    pick = torch.randint(0, src.numel(), (n,), device=src.device, generator=gen)
    return src[pick], ts[pick]


def _zipf(n, size, gen, s=1.1):
    """Bounded Zipf(s) ranks in [0, n) by the inverse of the continuous distribution."""
    u = torch.rand(size, device=_dev(), dtype=torch.double, generator=gen)
    x = ((n ** (1.0 - s) - 1.0) * u + 1.0).pow_(1.0 / (1.0 - s))
    return (x.long() - 1).clamp_(0, n - 1)


def _fanouts(case):
    return [int(k) for k in case["fanouts"].split(",")]


def prepare(case, seed):
    dev = _dev()
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("sample", "batch", "prefetch", "query", "slot"):
        names = _Names(case, gen)
        shape = names.shape
        src, dst, ts, eid = _events(names.active, case["edges"], shape)
        src, dst, ts = names.node(src), names.node(dst), names.time(ts)
    if kind == "tcsr":
        src, dst, ts, eid = _events(case["nodes"], case["edges"], gen, case["ordered"])
        s.update(src=src, dst=dst, ts=ts, eid=eid)
    elif kind in ("sample", "batch"):
        s["g"] = ops.tcsr_build(src, dst, ts, eid, case["nodes"])
        s["roots"], s["times"] = _roots(src, ts, case["roots"], shape)
        s["status"] = ops.StatusWord(dev)
    elif kind == "prefetch":
        g = ops.tcsr_build(src, dst, ts, eid, case["nodes"])
        feats = torch.empty(case["edges"], case["dim"], dtype=getattr(torch, case["dtype"]), device=dev).normal_(generator=gen)
        loader = []
        for _ in range(case["batches"]):
            q, qt = _roots(src, ts, case["roots"], shape)
            loader.append((q.cpu().pin_memory(), qt.cpu().pin_memory()))
        s["loader"] = HostToDevicePrefetcher(loader, g, feats, case["fanout"], case["policy"], max_roots=case["roots"],
                                             depth=case["batches"])
    elif kind == "cache":
        n = case["rows"]
        s["table"] = torch.empty(n, case["dim"], dtype=getattr(torch, case["dtype"]), device=dev).normal_(generator=gen)
        perm = torch.randperm(n, device=dev, generator=gen)
        hot = perm[:int(n * case["share"])]
        s["hitmap"] = torch.full((n,), -1, dtype=torch.int32, device=dev)
        s["hitmap"][hot] = torch.arange(hot.numel(), dtype=torch.int32, device=dev)
        s["cache"] = s["table"][hot].contiguous()
        # the ranks of the batch, and with them the hits, come from the sizes; which ids they are from the seed
        s["ids"] = perm[_zipf(n, case["ids"], torch.Generator(device=dev).manual_seed(n))].contiguous()
    elif kind == "state":
        loc = torch.randperm(case["all_nodes"], device=dev, generator=gen)[:case["nodes"]].contiguous()
        s["state"] = DistNodeState(PartitionState(loc, case["nodes"], node_mode="map", num_nodes=case["all_nodes"]), case["dim"],
                                   device=dev)
        s["state"].data.normal_(generator=gen)
        s["state"].ts.uniform_(0, 1e6, generator=gen)
        s["read"] = loc[_zipf(case["nodes"], case["reads"], gen)].contiguous()
        s["write"] = loc[torch.randperm(case["nodes"], device=dev, generator=gen)[:case["writes"]]].contiguous()
        s["rows"] = torch.empty(case["writes"], case["dim"], device=dev).normal_(generator=gen)
        s["row_ts"] = torch.empty(case["writes"], device=dev).uniform_(0, 1e6, generator=gen)
    elif kind == "mail":
        n, b, d = case["nodes"], case["events"], case["dim"]
        s["box"] = mailbox(n, case["slots"], d, case["edge_dim"], device=dev)
        s["box"].mailbox.normal_(generator=gen)
        perm = torch.randperm(n, device=dev, generator=gen)
        shape = torch.Generator(device=dev).manual_seed(n)     # which events share a node; the seed says which nodes
        s["src"] = perm[_zipf(n, b, shape)].contiguous()
        s["dst"] = perm[torch.randint(0, n, (b,), device=dev, generator=shape)].contiguous()
        s["nodes"] = torch.cat([s["src"], s["dst"], torch.randint(0, n, (b,), device=dev, generator=gen)])
        s["ts"] = torch.randint(0, TS_MAX, (b,), device=dev, generator=gen).sort().values
        s["mem_src"], s["mem_dst"] = (torch.empty(b, d, device=dev).normal_(generator=gen) for _ in range(2))
        s["edge"] = torch.empty(b, case["edge_dim"], device=dev).normal_(generator=gen)
    elif kind == "query":
        s["g"] = pyGraph(src, dst, ts, case["nodes"], 1, eid=eid)
        s["chunks"] = torch.zeros(1, dtype=I64, device=dev)
        # consecutive windows of about ``events`` events each, from the middle of the stream on
        first = case["edges"] // 2
        cuts = [first + i * case["events"] for i in range(case["windows"] + 1)]
        s["cuts"] = ts[torch.tensor(cuts, device=dev)].tolist()
        s["neg"] = [(names.node(torch.randint(0, names.active, (case["events"],), device=dev, generator=shape)),
                     ts[cuts[i]:cuts[i + 1]].contiguous()) for i in range(case["windows"])]
        s["policy"] = {"sample_type": case["policy"], "layers": case["layers"], "fanout": case["fanout"]}
    elif kind == "slot":
        n, parts = case["nodes"], case["parts"]
        every = names.node(torch.arange(names.active, device=dev))
        node_parts = torch.zeros(n, dtype=I64, device=dev)
        node_parts[every] = torch.randint(0, parts, (names.active,), device=dev, generator=shape)
        # a copy on the owner and on about a quarter of the other partitions
        held = torch.zeros(n, parts, dtype=torch.bool, device=dev)
        held[every] = torch.rand(names.active, parts, device=dev, generator=shape) < 0.25
        held[torch.arange(n, device=dev), node_parts] = True
        slot = held.long().cumsum(0) - 1
        indptr = torch.zeros(n + 1, dtype=I64, device=dev)
        indptr[1:] = held.sum(1).cumsum(0)
        rank = torch.arange(parts, device=dev).expand(n, parts)
        table = CSRReplicaTable(indptr, rank[held].contiguous(), slot[held].contiguous())
        data = {k: v.cpu().numpy() for k, v in (("src", src), ("dst", dst), ("ts", ts), ("eid", eid))}
        s["builder"] = MaterializedMultiLayerBuilder(data, n, node_parts, table, 0, parts)
        a = case["edges"] // 2
        b = a + case["events"]
        label = (torch.arange(case["events"]) % 2).numpy()
        s["task"] = ("link", (data["src"][a:b], data["dst"][a:b], data["ts"][a:b], label, data["eid"][a:b]))
        s["layers"] = {"meta": {"graph_type": "c", "end_offset": 0},
                       "layer": [{"type": case["policy"], "fanout": k} for k in _fanouts(case)]}
    return s


# ------------------------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------------------------

def run(s):
    return _RUN[s["case"]["kind"]](s)


def _run_tcsr(s):
    g = ops.tcsr_build(s["src"], s["dst"], s["ts"], s["eid"], s["case"]["nodes"])
    return [g.indptr, g.nbr, g.ts, g.eid, g.ts_min, g.ts_max]


def _run_sample(s):
    c = s["case"]
    h = ops.sample_layer(s["g"], s["roots"], s["times"], c["fanout"], c["policy"], equal_root_time=c["inclusive"],
                         allowed_offset=c["offset"], status=s["status"]).trimmed()
    return [h.nbr, h.dst, h.ts, h.dt, h.eid, h.offsets]


def _run_batch(s):
    return build_batch(s["g"], s["roots"], s["times"], _fanouts(s["case"]), s["case"]["policy"])


def _run_prefetch(s):
    out = []
    for b in s["loader"]:
        n = b.num_edges()
        out.append([b.offsets, b.nbr[:n], b.dst[:n], b.ts[:n], b.eid[:n], b.dt[:n], b.edge_feats[:n]])
    return out


def _run_cache(s):
    rows, miss_pos, miss_ids, counts = ops.cache_gather(s["cache"], s["hitmap"], s["table"], s["ids"])
    hits, misses = counts.tolist()
    return [rows, miss_pos[:misses], miss_ids[:misses], hits, misses]


def _run_state(s):
    st = s["state"]
    rows, ts = st[s["read"]]
    st.update(s["write"], s["rows"], s["row_ts"])
    return [rows, ts, st.data, st.ts]


def _run_mail(s):
    box = s["box"]
    msg, msg_ts = box.get_message(s["nodes"])
    index, mail, mail_ts = box.get_update_mail(s["src"], s["dst"], s["ts"], s["edge"], s["mem_src"], s["mem_dst"])
    box.set_mailbox_local(index, mail, mail_ts)
    return [msg, msg_ts, index, mail, mail_ts, box.mailbox, box.mailbox_ts, box.next_mail_pos]


def _run_query(s):
    g, cuts = s["g"], s["cuts"]
    for i, (neg, neg_ts) in enumerate(s["neg"]):
        g.async_sample(cuts[i], cuts[i + 1], s["chunks"], s["policy"],
                       {"test_generate_samples": neg, "test_generate_samples_ts": neg_ts}, op="f")
    out = []
    for _ in s["neg"]:
        r = g.get_last_sample()
        root, _, blocks, mapper = AsyncBlock.to_block(r.roots, r.neg_roots, r.neighbors, r.nodes_remapper_id)
        out.append([root.roots, root.ts_ptr, root.ts, root.q_eid, mapper] +
                   [[b.indptr, b.indices, b.srcdata["nid"], b.srcdata["ts"], b.edata["eid"], b.edata["dt"]] for b in blocks])
    return out


def _run_slot(s):
    layers = s["builder"].build_aligned_batch(s["task"], None, s["layers"], seed=1)
    plans = [None if p is None else [p.send_ranks, p.send_sizes, p.send_indices, p.send_remote_indices]
             for p in layers[0]["comm_plan"]]
    keys = ("gids", "ts", "inv_map", "indptr", "indices", "eid", "edge_ts", "edge_dt")
    return [{k: d[k] for k in keys if k in d} for d in layers], plans


_RUN = dict(tcsr=_run_tcsr, sample=_run_sample, batch=_run_batch, prefetch=_run_prefetch, cache=_run_cache, state=_run_state,
            mail=_run_mail, query=_run_query, slot=_run_slot)


# ------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------------------------
# Share of the fan-out that the synthetic graphs fill: an event's source at the event's time nearly always has enough
# earlier edges, a neighbour reached from it (a uniform node) often has few.
_FILL = (0.9, 0.28)


def _hop_edges(roots, fanouts):
    out, n = [], roots
    for l, k in enumerate(fanouts):
        n = n * k * _FILL[min(l, 1)]
        out.append(n)
    return out


def _batch_bytes(roots, fanouts):
    total, targets, pairs = 16.0 * roots, roots, roots
    total += 24.0 * roots                                   # first list and its inverse map
    for e in _hop_edges(roots, fanouts):
        total += 16.0 * targets + 24.0 * e                  # row bounds, sampled edges
        total += 8.0 * pairs + 28.0 * e                     # row pointer; indices, edge id, time, time difference
        targets, pairs = e, pairs + e
        total += 16.0 * pairs                               # merged list
    return total


def work(case):
    kind = case["kind"]
    size = 2 if case.get("dtype") == "bfloat16" else 4
    if kind == "tcsr":
        b = 56.0 * case["edges"] + 8.0 * case["nodes"]
    elif kind == "sample":
        b = 40.0 * case["roots"] + 60.0 * _hop_edges(case["roots"], [case["fanout"]])[0]
    elif kind == "batch":
        b = _batch_bytes(case["roots"], _fanouts(case))
    elif kind == "prefetch":
        e = _hop_edges(case["roots"], [case["fanout"]])[0]
        b = case["batches"] * (40.0 * case["roots"] + e * (60.0 + 2.0 * size * case["dim"]))
    elif kind == "cache":
        b = case["ids"] * (2.0 * size * case["dim"] + 12.0) + 16.0 * 0.25 * case["ids"]
    elif kind == "state":
        b = (case["reads"] + case["writes"]) * (8.0 * case["dim"] + 24.0)
    elif kind == "mail":
        width = 2 * case["dim"] + case["edge_dim"]
        b = case["events"] * (3 * (8.0 * width * case["slots"] + 16.0) + 2 * 16.0 + 4.0 * width + 2 * 1.8 * (8.0 * width + 12.0))
    elif kind == "query":
        b = case["windows"] * (1.5 * _batch_bytes(2 * case["events"], [case["fanout"]] * case["layers"]) + 24.0 * case["events"])
    else:
        b = 2.0 * _batch_bytes(2 * case["events"], _fanouts(case))
    return {"bytes": b, "flops": 0}


def tolerance(case):
    return "exact"
