"""The workloads whose speed this framework is measured by, through the entry
points that a timing flow calls.

A case is a dict of plain values; its "kind" says which calls one pass makes:

  rc        RcBatch.run: BFS order and Elmore load / delay / ldelay / impulse
            (and sink slews) of a forest of RC nets resident on the device
  rc_host   rc_timing_host: the same on host arrays, copies included (what a
            caller of rct_bfs_and_compute_cuda pays)
  relevel   fanin_csr + LevelizeBatch: levels of a gate-level design's timing
            graph from its arc list, as after a netlist change
  levelize  LevelizeBatch.run: levels of a resident pin graph
  update    RcBatch.run + TimingGraph.propagate: a full timing update of a
            gate-level design (arrival, slew, required time, slack)
  sizing    SizingDesign.run_prepared: one batch of gate resizes, their nets
            re-timed, the design propagated, the worst slack

All sizes are those of the repository's benchmark and tests or lie between
them: RC nets of 2..4096 nodes (log-uniform) and of 2..16 nodes (the nets of
the generated designs), huge nets of 5k..20k nodes, pin graphs of up to 5M
pins / 12M arcs, designs of 2k..240k gates.
"""
import math
import tempfile

import numpy as np
import torch

import opentimer_b200 as otg
from opentimer_b200 import designgen
from opentimer_b200.prop import TimingGraph
from opentimer_b200.sizing import SizingDesign, resize_trace

DEV = "cuda"
NC = 4


def listed():
    return [
        # the smallest call: the dirty nets of one engineering change
        {"name": "rc_eco", "kind": "rc", "nets": 64, "lo": 2, "hi": 16, "log": False,
         "sinks": True},
        # the nets of a placed design: few nodes each, many of them
        {"name": "rc_design", "kind": "rc", "nets": 250_000, "lo": 2, "hi": 16, "log": False,
         "sinks": True},
        # one sizing iteration's dirty nets in a design with long wires
        {"name": "rc_dirty", "kind": "rc", "nets": 2_500, "lo": 2, "hi": 512, "log": True,
         "sinks": False},
        # the headline mix, heavy-tailed net sizes
        {"name": "rc_mixed", "kind": "rc", "nets": 100_000, "lo": 2, "hi": 4096, "log": True,
         "sinks": True},
        # clock and reset trees: a few nets of many thousand nodes
        {"name": "rc_trees", "kind": "rc", "nets": 24, "lo": 5_000, "hi": 20_000, "log": True,
         "sinks": False},
        # the drop-in call on a design's nets in host memory
        {"name": "rc_host", "kind": "rc_host", "nets": 60_000, "lo": 2, "hi": 16, "log": False,
         "sinks": True},
        # levels of a 60k-gate design after a netlist change
        {"name": "relevel_60k", "kind": "relevel", "gates": 60_000, "back": 600},
        # levels of a flat multi-million-pin graph
        {"name": "levelize_5m", "kind": "levelize", "pins": 5_000_000, "arcs": 12_000_000,
         "levels": 200},
        # a block: a full update where latency is everything
        {"name": "update_2k", "kind": "update", "gates": 2_000, "back": 50},
        # a design of the usual size and depth
        {"name": "update_60k", "kind": "update", "gates": 60_000, "back": 600},
        # a large design with the logic depth of pipelined logic
        {"name": "update_240k", "kind": "update", "gates": 240_001, "back": 10_000},
        # one iteration of gate sizing on a block
        {"name": "sizing_6k", "kind": "sizing", "gates": 6_000, "resizes": 60},
    ]


def _between(rng, lo, hi):
    """An integer between lo and hi, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rc", "rc", "rc", "rc_trees", "rc_host", "relevel", "levelize", "update",
                       "update", "sizing"])
    if kind == "rc":
        hi = rng.choice([16, 24, 33, 64, 128, 512, 1500, 4096])
        log = hi > 32
        mean = (hi - 2) / math.log(hi / 2) if log else (hi + 2) / 2
        most = min(250_000, int(50_000_000 / mean))
        return {"kind": "rc", "nets": _between(rng, 50, most), "lo": 2, "hi": hi, "log": log,
                "sinks": rng.random() < 0.5}
    if kind == "rc_trees":
        return {"kind": "rc", "nets": _between(rng, 1, 40), "lo": 5_000,
                "hi": _between(rng, 6_000, 20_000), "log": True, "sinks": rng.random() < 0.5}
    if kind == "rc_host":
        return {"kind": "rc_host", "nets": _between(rng, 100, 60_000), "lo": 2,
                "hi": rng.choice([8, 16, 24]), "log": False, "sinks": rng.random() < 0.5}
    if kind == "relevel":
        gates = _between(rng, 2_000, 120_000)
        return {"kind": "relevel", "gates": gates, "back": max(50, gates // rng.choice([25, 100]))}
    if kind == "levelize":
        pins = _between(rng, 20_000, 5_000_000)
        return {"kind": "levelize", "pins": pins, "arcs": int(pins * rng.uniform(1.8, 2.4)),
                "levels": _between(rng, 20, 200)}
    if kind == "update":
        gates = _between(rng, 2_000, 240_000)
        return {"kind": "update", "gates": gates,
                "back": max(50, gates // rng.choice([25, 50, 100]))}
    return {"kind": "sizing", "gates": _between(rng, 1_000, 6_000),
            "resizes": _between(rng, 1, 60)}


# ------------------------------------------------------------------ inputs

def _sizes(case, seed):
    """nodes_start of the case's nets: the same sizes for every seed, in
    another order."""
    r = np.random.default_rng(case["nets"])
    lo, hi, k = case["lo"], case["hi"], case["nets"]
    if case["log"]:
        n = np.floor(np.exp(r.uniform(math.log(lo), math.log(hi + 1), k))).astype(np.int64)
        n = np.clip(n, lo, hi)
    else:
        n = r.integers(lo, hi + 1, k)
    ns = np.zeros(k + 1, np.int64)
    np.cumsum(np.random.default_rng(seed).permutation(n), out=ns[1:])
    return ns.astype(np.int32)


def _rc_forest(case, seed):
    """The repository's synthetic RC forest on the device: 70% random trees,
    30% chains with side branches, ids by first appearance over the shuffled
    resistors, per-corner pin caps on the leaves.  With sinks, two nodes in
    five of a net (never its root, at least one) are pins with a slew."""
    ns = torch.from_numpy(_sizes(case, seed)).to(DEV)
    f = otg.synth_forest(seed, ns, with_sinks=False)
    if not case["sinks"]:
        f.pop("driver_slew")
        return f
    start = ns.long()
    n = start[1:] - start[:-1]
    net = torch.repeat_interleave(torch.arange(n.numel(), device=DEV), n)
    key = net.double() + 0.99 * _rand(_generator(seed), net.numel()).double()
    key[start[:-1] + f["roots"].long()] = torch.arange(n.numel(), device=DEV).double() + 0.995
    rank = torch.empty_like(net)
    rank[torch.argsort(key)] = torch.arange(net.numel(), device=DEV)
    want = torch.clamp((2 * n) // 5, min=1)
    pins = (rank - start[net] < want[net]).nonzero()[:, 0]
    f["sinks_start"] = _excl(want).to(torch.int32)
    f["sink_nodes"] = (pins - start[net[pins]]).to(torch.int32)
    return f


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV)


def _excl(x):
    """Exclusive prefix sum with the total at the end."""
    out = torch.zeros(x.numel() + 1, dtype=torch.int64, device=x.device)
    out[1:] = torch.cumsum(x, 0)
    return out


CELLS = ("INV_X1", "INV_X2", "INV_X4", "NAND2_X1", "NAND2_X2", "NAND2_X4", "NOR2_X1", "NOR2_X2",
         "NOR2_X4", "DFF_X1")


def _library(seed):
    """The generated cell library's tables and timing records, and each
    cell's pin caps."""
    libs = {"early": {}, "late": {}}
    designgen.liberty(seed, 1.0, "late", libs["late"])
    designgen.liberty(seed, 0.9, "early", libs["early"])
    arrays, _, _ = designgen.timing_graph({
        "libs": libs, "gates": [], "ports_in": ["clk"], "ports_out": [], "nets": {},
        "at": {}, "slew": {}, "rat": {}, "period": 1.0})
    rec = arrays["records"]
    ins = {"INV": ("A",), "NAND2": ("A1", "A2"), "NOR2": ("A1", "A2"), "DFF": ("D", "CK")}
    caps = np.zeros((len(CELLS), 2), np.float32)
    out_rec = np.full((2, len(CELLS), 2), -1, np.int64)  # [split][cell][input] -> record
    for c, cell in enumerate(CELLS):
        for k, cp in enumerate(ins[cell.split("_")[0]]):
            caps[c, k] = libs["late"][cell]["caps"][cp]
            for el in (0, 1):
                if cell.startswith("DFF"):  # input 1 drives Q; D is checked (setup k=0, hold k=1)
                    out_rec[el, c, k] = (rec[(cell, el, "Q", 0)] if k == 1 else
                                         rec[(cell, el, "D", 1 if el == 0 else 0)])
                else:
                    out_rec[el, c, k] = rec[(cell, el, "ZN", k)]
    return arrays, caps, out_rec


def _design(gates, back, seed):
    """A gate-level design by the rules of the repository's generator (INV /
    NAND2 / NOR2 in three drives, 5% flops on one clock, sources at a mean
    look-back of `back` signals, RC trees of a net's pins and up to
    13 inner nodes), built with tensors: (graph arrays for TimingGraph, RC
    forest).  The signals that the first inputs leave over, `back` of them,
    drive the primary outputs.  Every seed gives another design with the
    same numbers of pins, arcs and nodes."""
    g = _generator(seed)
    lib, caps, out_rec = _library(seed % 1000 + 1)
    n_pi = 64
    G, S = gates, n_pi + gates
    ar = lambda n: torch.arange(n, device=DEV)  # noqa: E731
    r = torch.argsort(_rand(g, G)).double() / G
    drive = (_rand(g, G) * 3).long()
    nand = _rand(g, G) < 0.5
    dff, inv = r < 0.05, (r >= 0.05) & (r < 0.35)
    cell = torch.where(dff, 9, torch.where(inv, drive, torch.where(nand, 3 + drive, 6 + drive)))
    two = ~dff & ~inv  # two data inputs
    width = torch.where(inv, 2, 3)
    clk = n_pi
    base = n_pi + 1 + _excl(width)  # first pin of every gate
    out_pin = base[:G] + width - 1
    # data inputs: the first takes the signals in a locally shuffled order,
    # the second looks back a geometric number of signals
    key = ar(S) + _rand(g, S) * back
    order = torch.argsort(key)
    first = torch.where(ar(G) + n_pi >= back, order[(ar(G) + n_pi - back).clamp(min=0)],
                        (_rand(g, G) * n_pi).long())
    first = torch.minimum(first, ar(G) + n_pi - 1)
    look = (torch.log1p(-_rand(g, G).double()) / math.log1p(-1.0 / back)).ceil().clamp(min=1).long()
    second = (ar(G) + n_pi - look).clamp(min=0)
    # sinks: (net, pin, cap); net i is signal i's, net S the clock's
    i2, ff = two.nonzero()[:, 0], dff.nonzero()[:, 0]
    tcaps = torch.from_numpy(caps).to(DEV)
    s_net = torch.cat([first, second[i2], torch.full_like(ff, S)])
    s_pin = torch.cat([base[:G], base[:G][i2] + 1, base[:G][ff] + 1])
    s_cap = torch.cat([tcaps[cell, 0], tcaps[cell[i2], 1], tcaps[cell[ff], 1]])
    P = int(base[G]) + back
    s_net = torch.cat([s_net, order[S - back:]])
    s_pin = torch.cat([s_pin, int(base[G]) + ar(back)])
    s_cap = torch.cat([s_cap, torch.full((back,), 4.0, device=DEV)])
    by = torch.argsort(s_net, stable=True)
    s_net, s_pin, s_cap = s_net[by], s_pin[by], s_cap[by]
    N = S + 1
    fan = torch.bincount(s_net, minlength=N)
    driver = torch.cat([ar(n_pi), out_pin, torch.tensor([clk], device=DEV)])
    # RC trees: position 0 is the driver, 1.. the sinks, then inner nodes
    n = fan + 1 + (torch.argsort(_rand(g, N)) * 14) // N
    ns = _excl(n)
    V = int(ns[-1])
    net = torch.repeat_interleave(ar(N), n)
    pos = ar(V) - ns[net]
    nd = _rand(g, V).double()
    local = torch.empty(V, dtype=torch.int64, device=DEV)
    local[torch.argsort(net.double() + nd * 0.999)] = pos  # a random id per node
    child = (pos > 0).nonzero()[:, 0]
    enet, p = net[child], pos[child]
    # parents in a random order of the positions that starts at the driver
    ndq = torch.where(pos == 0, 0.0, nd * 0.5 + 0.25)
    rank = torch.empty(V, dtype=torch.int64, device=DEV)
    rank[torch.argsort(net.double() + ndq)] = ar(V)
    at_rank = torch.argsort(rank)
    par = at_rank[ns[enet] + ((rank[child] - ns[enet]).double() *
                              _rand(g, p.numel()).double()).long()]
    e = torch.stack([local[par], local[child]], 1)
    e = torch.where((_rand(g, p.numel()) < 0.5)[:, None], e, e.flip(1))
    e = e[torch.argsort(enet.double() + _rand(g, p.numel()).double() * 0.999)]
    ground = (0.1 + 2.9 * _rand(g, V)) * (16.0 / n.float()).clamp(max=1.0)[net]
    row = ns[:-1]
    s_idx = ar(s_net.numel()) - _excl(fan)[s_net] + 1  # position of the sink in its net
    s_row = ns[s_net] + s_idx
    ground[s_row] += s_cap
    cap = torch.empty(V, NC, device=DEV)
    cap[ns[net] + local] = ground[:, None].expand(V, NC)
    i32 = lambda x: x.to(torch.int32).contiguous()  # noqa: E731
    rc = {"nodes_start": i32(ns), "edges": i32(e), "roots": i32(local[row]),
          "res": ((0.5 + 19.5 * _rand(g, p.numel())) * 1e-3).contiguous(), "cap": cap}
    # arcs: net arcs by net, then per split the cells' arcs
    frm, to = [driver[s_net]], [s_pin]
    anet, node = [s_net], [local[s_row]]
    rec = [torch.full((s_net.numel(), 2), -1, dtype=torch.int64, device=DEV)]
    trec = torch.from_numpy(out_rec).to(DEV)
    tests, count = [], s_net.numel()
    pin_net = torch.full((P,), -1, dtype=torch.int64, device=DEV)
    pin_net[s_pin] = s_net
    pin_net[driver] = ar(N)
    comb = (~dff).nonzero()[:, 0]
    for el in (0, 1):
        for src, dst, k, who in ((base[:G][comb], out_pin[comb], 0, comb),
                                 (base[:G][i2] + 1, out_pin[i2], 1, i2),
                                 (base[:G][ff] + 1, out_pin[ff], 1, ff),
                                 (base[:G][ff] + 1, base[:G][ff], 0, ff)):
            t = torch.full((who.numel(), 2), -1, dtype=torch.int64, device=DEV)
            t[:, el] = trec[el, cell[who], k]
            if k == 0 and who is ff:
                tests.append(count + ar(who.numel()))
            count += who.numel()
            frm.append(src)
            to.append(dst)
            rec.append(t)
            anet.append(pin_net[dst])
            node.append(torch.full_like(src, -1))
    A = count
    kind = torch.ones(A, dtype=torch.int64, device=DEV)
    kind[:s_net.numel()] = 0
    nan4 = lambda: torch.full((P, NC), math.nan, device=DEV)  # noqa: E731
    pi_at, pi_slew, po_rat = nan4(), nan4(), nan4()
    pi_at[:n_pi] = (0.05 * _rand(g, n_pi))[:, None]
    pi_slew[:n_pi] = (0.01 + 0.09 * _rand(g, n_pi))[:, None]
    pi_at[clk] = torch.tensor([0.0, 0.5, 0.0, 0.5], device=DEV)
    pi_slew[clk] = 0.02
    po_rat[int(base[G]):] = torch.tensor([0.0, 0.0, 1.0, 1.0], device=DEV)
    host = lambda x: i32(x).cpu().numpy()  # noqa: E731
    arrays = {"num_pins": P, "arc_from": host(torch.cat(frm)), "arc_to": host(torch.cat(to)),
              "arc_kind": host(kind), "arc_timing": host(torch.cat(rec)),
              "arc_net": host(torch.cat(anet)), "arc_node": host(torch.cat(node)),
              "test_arc": host(torch.cat(tests)), "pi_at": pi_at.cpu().numpy(),
              "pi_slew": pi_slew.cpu().numpy(), "po_rat": po_rat.cpu().numpy(),
              "timing": lib["timing"], "lut_meta": lib["lut_meta"], "lut_data": lib["lut_data"],
              "period": 1.0}
    return arrays, rc


def _pin_graph(case, seed):
    """A levelled pin graph (fanin CSR, fanout counts, seed): every pin above
    level 0 has a fanin one level down, the other arcs come from any earlier
    level, and one pin in 5000 drives 500..5000 others."""
    g = _generator(seed)
    n, levels = case["pins"], case["levels"]
    ar = lambda k: torch.arange(k, device=DEV)  # noqa: E731
    lvl = (_rand(g, n) * levels).long()
    lvl[:levels] = ar(levels)
    lvl = torch.sort(lvl)[0]
    pin_at = torch.argsort(_rand(g, n))  # sorted position -> pin
    starts = torch.searchsorted(lvl, ar(levels + 1))
    rest = ar(n)[int(starts[1]):]
    k = lvl[rest]
    a, b = starts[k - 1], starts[k]
    src = [a + (_rand(g, rest.numel()).double() * (b - a)).long()]
    dst = [rest]
    hubs = int(0.0002 * n)
    if hubs:
        p = (_rand(g, hubs).double() * int(starts[levels // 2])).long()
        lo = starts[lvl[p] + 1]
        cnt = 500 + (_rand(g, hubs) * 4501).long()
        cnt = torch.minimum(cnt, torch.full_like(cnt, max(1, n // 20)))
        src.append(torch.repeat_interleave(p, cnt))
        lo = torch.repeat_interleave(lo, cnt)
        dst.append(lo + (_rand(g, lo.numel()).double() * (n - lo)).long())
    extra = max(0, case["arcs"] - sum(x.numel() for x in dst))
    d = int(starts[1]) + (_rand(g, extra).double() * (n - int(starts[1]))).long()
    src.append((_rand(g, extra).double() * starts[lvl[d]]).long())
    dst.append(d)
    s, d = pin_at[torch.cat(src)], pin_at[torch.cat(dst)]
    arcs = torch.unique(d * n + s)
    d, s = arcs // n, arcs % n
    out_deg = torch.bincount(s, minlength=n)
    i32 = lambda x: x.to(torch.int32).contiguous()  # noqa: E731
    return (i32(_excl(torch.bincount(d, minlength=n))), i32(s), i32(out_deg),
            i32((out_deg == 0).nonzero()[:, 0]))


# ------------------------------------------------------------------ passes

def prepare(case, seed):
    kind = case["kind"]
    if kind == "rc":
        return {"kind": kind, "batch": otg.RcBatch(**_rc_forest(case, seed))}
    if kind == "rc_host":
        f = {k: np.ascontiguousarray(v.cpu().numpy()) for k, v in _rc_forest(case, seed).items()}
        return {"kind": kind, "forest": f}
    if kind == "relevel":
        arrays, _ = _design(case["gates"], case["back"], seed)
        return {"kind": kind, "pins": arrays["num_pins"],
                "from": torch.from_numpy(arrays["arc_from"]).to(DEV),
                "to": torch.from_numpy(arrays["arc_to"]).to(DEV)}
    if kind == "levelize":
        return {"kind": kind, "batch": _defined(otg.LevelizeBatch(*_pin_graph(case, seed)))}
    if kind == "update":
        arrays, rc = _design(case["gates"], case["back"], seed)
        return {"kind": kind, "batch": otg.RcBatch(**rc), "graph": TimingGraph(arrays)}
    with tempfile.TemporaryDirectory() as d:
        keep = {}
        designgen.write_design(d, seed=case["gates"], gates=case["gates"], keep=keep,
                               rc_nodes=(2, 512), rc_log=True, lib_seed=seed % 100_000)
        design = SizingDesign(d, keep)
    steps = resize_trace(keep, seed + 1, 1, case["resizes"])
    return {"kind": "sizing", "design": design, "prep": design.prepare(steps)}


def _defined(lb):
    """The entries of level_ends past the last level are nobody's output."""
    lb.level_ends.zero_()
    return lb


def _rc_out(b):
    out = {k: getattr(b, k) for k in ("node2bfs", "pid", "edges", "load", "delay", "ldelay",
                                      "impulse")}
    if b.sink_slew is not None:
        out["sink_slew"] = b.sink_slew
    return out


def run(state):
    kind = state["kind"]
    if kind == "rc":
        return _rc_out(state["batch"].run())
    if kind == "rc_host":
        f = state["forest"]
        out = otg.rc_timing_host(**f)
        out["edges"] = f["edges"]
        return out
    if kind == "relevel":
        start, fanin, out_deg, front = otg.fanin_csr(state["pins"], state["from"], state["to"])
        lb = otg.LevelizeBatch(start, fanin, out_deg, front).run()
        return [start, fanin, out_deg, front, lb.order, lb.level, lb.counts]
    if kind == "levelize":
        lb = state["batch"].run()
        return [lb.order, lb.level, lb.level_ends, lb.counts]
    if kind == "update":
        b = state["batch"].run()
        g = state["graph"].propagate(b)
        return {**_rc_out(b), **g.out}
    d = state["design"]
    d.run_prepared(state["prep"], 0, 1)
    return {"worst_slack": state["prep"]["wns"], "load": d.batch.load, "delay": d.batch.delay,
            "impulse": d.batch.impulse, **d.graph.out}


def work(case):
    kind = case["kind"]
    if kind in ("rc", "rc_host"):
        ns = _sizes(case, 1)
        V, N = int(ns[-1]), case["nets"]
        sinks = 0.4 * V if case["sinks"] else 0
        return {"bytes": 108.0 * V - 20.0 * N + 28.0 * N + 20.0 * sinks, "flops": 40.0 * V}
    if kind == "levelize":
        return {"bytes": 4.0 * case["arcs"] + 16.0 * case["pins"], "flops": 0.0}
    G = case["gates"]
    pins, arcs = 2.75 * G, 5.2 * G
    if kind == "relevel":
        return {"bytes": 12.0 * arcs + 20.0 * pins, "flops": 0.0}
    nodes = 9.3 * G
    graph = {"bytes": 36.0 * arcs + 128.0 * pins, "flops": 8 * 40.0 * arcs}
    if kind == "update":
        return {"bytes": graph["bytes"] + 108.0 * nodes + 8.0 * G,
                "flops": graph["flops"] + 40.0 * nodes}
    dirty = 2.0 * case["resizes"]  # nets of 2..512 nodes
    return {"bytes": graph["bytes"] + 92.0 * 108.0 * dirty,
            "flops": graph["flops"] + 40.0 * 92.0 * dirty}


# ---------------------------------------------------------- 64-bit results

def _grouped(keys, size):
    """CSR of item indices grouped by key."""
    return _excl(torch.bincount(keys, minlength=size)), torch.argsort(keys, stable=True)


def _take(start, items, rows):
    """The items of the given CSR rows, and for each the index into rows."""
    cnt = start[rows + 1] - start[rows]
    which = torch.repeat_interleave(torch.arange(rows.numel(), device=DEV), cnt)
    off = torch.arange(which.numel(), device=DEV) - _excl(cnt)[which]
    return items[start[rows][which] + off], which


def _rc_exact(f):
    """The Elmore quantities of a forest in 64 bits, in BFS order (distance
    ascending, local id descending)."""
    ns, roots = f["nodes_start"].long(), f["roots"].long()
    N, V = roots.numel(), f["cap"].shape[0]
    n = ns[1:] - ns[:-1]
    net = torch.repeat_interleave(torch.arange(N, device=DEV), n)
    enet = torch.repeat_interleave(torch.arange(N, device=DEV), n - 1)
    x, y = f["edges"][:, 0].long() + ns[enet], f["edges"][:, 1].long() + ns[enet]
    E = x.numel()
    start, arcs = _grouped(torch.cat([x, y]), V)
    ends = torch.cat([y, x])
    dist = torch.full((V,), -1, dtype=torch.int64, device=DEV)
    parent = torch.arange(V, device=DEV)
    pres = torch.zeros(V, dtype=torch.float64, device=DEV)
    res = f["res"].double()
    front = ns[:-1] + roots
    dist[front] = 0
    levels = [front]
    while True:
        a, which = _take(start, arcs, front)
        v = ends[a]
        new = dist[v] < 0
        v, a, u = v[new], a[new], front[which[new]]
        if v.numel() == 0:
            break
        dist[v] = len(levels)
        parent[v] = u
        pres[v] = res[torch.where(a >= E, a - E, a)]
        levels.append(v)
        front = v
    cap = f["cap"].double()

    def up(q):
        q = q.clone()
        for v in reversed(levels[1:]):
            q.index_add_(0, parent[v], q[v])
        return q

    def down(w):
        q = torch.zeros_like(w)
        for v in levels[1:]:
            q[v] = q[parent[v]] + w[v]
        return q

    load = up(cap)
    delay = down(pres[:, None] * load)
    ldelay = up(cap * delay)
    impulse = 2.0 * down(pres[:, None] * ldelay) - delay * delay
    local = torch.arange(V, device=DEV) - ns[net]
    big = 1 << 20
    order = torch.argsort((net * big + dist) * big + (big - 1 - local))
    out = {k: None for k in ("node2bfs", "pid", "edges")}
    out.update({"load": load[order], "delay": delay[order], "ldelay": ldelay[order],
                "impulse": impulse[order]})
    if "sinks_start" in f:
        ss = f["sinks_start"].long()
        snet = torch.repeat_interleave(torch.arange(N, device=DEV), ss[1:] - ss[:-1])
        si = f["driver_slew"].double()[snet]
        out["sink_slew"] = torch.sqrt(si * si + impulse[ns[snet] + f["sink_nodes"].long()])
    by_node = {"load": load, "delay": delay, "impulse": impulse}
    return out, by_node


def _seg(idx, q):
    """Index of the upper end of q's segment (the outer ones extrapolate)."""
    return torch.searchsorted(idx, q.contiguous()).clamp(1, idx.numel() - 1)


def _table(vals, i1, i2, x, y):
    """Bilinear interpolation of tables vals[..., 7, 7] at (x, y)."""
    a, b = _seg(i1, x), _seg(i2, y)
    at = lambda p, q: vals.gather(-1, (p * i2.numel() + q)[..., None])[..., 0]  # noqa: E731
    fx = (x - i1[a - 1]) / (i1[a] - i1[a - 1])
    fy = (y - i2[b - 1]) / (i2[b] - i2[b - 1])
    lo = at(a - 1, b - 1) + fx * (at(a, b - 1) - at(a - 1, b - 1))
    hi = at(a - 1, b) + fx * (at(a, b) - at(a - 1, b))
    return lo + fy * (hi - lo)


def _update_exact(case, seed):
    """The update in 64 bits: every arc by the level of the pin it ends at."""
    ar, rc = _design(case["gates"], case["back"], seed)
    out, node = _rc_exact(rc)
    t = lambda k: torch.from_numpy(np.asarray(ar[k])).to(DEV)  # noqa: E731
    P = ar["num_pins"]
    frm, to, kind = t("arc_from").long(), t("arc_to").long(), t("arc_kind").long()
    tm, anet, anode = t("arc_timing").long(), t("arc_net").long(), t("arc_node").long()
    timing, meta = t("timing").long(), t("lut_meta").long()
    data = t("lut_data").double()
    ns = rc["nodes_start"].long()
    A = frm.numel()
    inf = math.inf
    # tables by (record, which = delay | slew | constraint, output transition)
    lut = timing[:, 3:9].reshape(-1, 3, 2)
    off = meta[lut.clamp(min=0), 2]
    vals = data[off[..., None] + 14 + torch.arange(49, device=DEV)]
    slew_ax, load_ax = data[off[lut[:, 0, 0] >= 0][0, 0, 0] + torch.arange(14, device=DEV)].split(7)
    root = ns[anet.clamp(min=0)] + rc["roots"].long()[anet.clamp(min=0)]
    load = node["load"][root].reshape(A, 2, 2)  # [arc][split][out transition]
    sink = ns[anet.clamp(min=0)] + anode.clamp(min=0)
    nd, ni = (node[k][sink].reshape(A, 2, 2) for k in ("delay", "impulse"))
    # [arc][split][from][to] combinations that a cell arc propagates or checks
    rec = tm[:, :, None, None].expand(A, 2, 2, 2)
    r0 = rec.clamp(min=0)
    fr = torch.arange(2, device=DEV).reshape(1, 1, 2, 1).expand(A, 2, 2, 2)
    tr = torch.arange(2, device=DEV).reshape(1, 1, 1, 2).expand(A, 2, 2, 2)
    sense, edge = timing[r0, 0], timing[r0, 1]
    ok = (rec >= 0) & ((edge != 1) | (fr == 0)) & ((edge != 2) | (fr == 1))
    ok &= ((sense != 0) | (fr == tr)) & ((sense != 1) | (fr != tr))
    cons = timing[r0, 2] > 0
    is_net = (kind == 0)[:, None, None, None]
    go = torch.where(is_net, fr == tr, ok & ~cons)
    sign = torch.tensor([1.0, -1.0], dtype=torch.float64, device=DEV)[:, None]  # MIN, MAX
    # forward: worst = the largest of sign-flipped values; -inf is empty
    W = lambda x: torch.where(torch.isnan(x), torch.full_like(x, -inf), x)  # noqa: E731
    flip = lambda x: x.reshape(-1, 2, 2) * -sign  # noqa: E731
    at, sl = W(flip(t("pi_at").double())), W(flip(t("pi_slew").double()))
    delay = torch.full((A, 2, 2, 2), math.nan, dtype=torch.float64, device=DEV)
    fstart, farcs = _grouped(frm, P)
    indeg = torch.bincount(to, minlength=P)
    front = (indeg == 0).nonzero()[:, 0]
    waves = []
    while front.numel():
        a, _ = _take(fstart, farcs, front)
        if a.numel() == 0:
            break
        indeg.index_add_(0, to[a], torch.full_like(a, -1))
        front = torch.unique(to[a])
        front = front[indeg[front] == 0]
        waves.append(front)
    instart, inarcs = _grouped(to, P)
    for pins in waves:
        a, _ = _take(instart, inarcs, pins)
        s_in = (sl[frm[a]] * -sign)[:, :, :, None].expand(-1, 2, 2, 2)
        a_in = (at[frm[a]] * -sign)[:, :, :, None].expand(-1, 2, 2, 2)
        live = go[a] & torch.isfinite(s_in)
        q = torch.where(live, s_in, torch.ones_like(s_in))
        ld = load[a][:, :, None, :].expand(-1, 2, 2, 2)
        d_cell = _table(vals[r0[a], 0, tr[a]], slew_ax, load_ax, q, ld)
        s_cell = _table(vals[r0[a], 1, tr[a]], slew_ax, load_ax, q, ld)
        s_net = torch.copysign(torch.sqrt(q * q + ni[a][:, :, None, :]), q)
        d_net = nd[a][:, :, None, :].expand(-1, 2, 2, 2)
        s_out = torch.where(is_net[a], s_net, s_cell)
        d = torch.where(is_net[a], d_net, d_cell)
        d = torch.where(live | (is_net[a] & go[a]), d, torch.full_like(d, math.nan))
        delay[a] = d
        m = -sign.reshape(1, 2, 1, 1)
        cand_s = torch.where(live, s_out * m, torch.full_like(d, -inf)).amax(2)
        arr = go[a] & torch.isfinite(a_in) & ~torch.isnan(d)
        cand_a = torch.where(arr, (a_in + d) * m, torch.full_like(d, -inf)).amax(2)
        idx = to[a][:, None, None].expand(-1, 2, 2)
        sl.scatter_reduce_(0, idx, cand_s, "amax")
        at.scatter_reduce_(0, idx, cand_a, "amax")
    un = lambda x: torch.where(torch.isfinite(x), x * -sign, torch.full_like(x, math.nan))  # noqa: E731
    at, sl = un(at), un(sl)
    # tests: required times at the checked pins
    rat = W(flip(t("po_rat").double()) * -1.0)
    ta = t("test_arc").long()
    u, v = frm[ta], to[ta]
    el = (tm[ta, 1] >= 0).long()
    r = tm[ta].max(1)[0]
    fel = 1 - el
    rel_at, rel_sl = at[u, fel, 0], sl[u, fel, 0]
    for rf in (0, 1):
        c = _table(vals[r, 2, rf], slew_ax, slew_ax, rel_sl, sl[v, el, rf])
        val = torch.where(el == 0, c + rel_at, rel_at + ar["period"] - c)
        sgn = torch.where(el == 0, 1.0, -1.0)
        w = torch.where(torch.isnan(val), torch.full_like(val, -inf), val * sgn)
        flat = rat.view(-1)
        flat.scatter_reduce_(0, (v * 2 + el) * 2 + rf, w, "amax")
    # backward, last wave first; required times relax the other way round
    srt = lambda x: torch.where(torch.isfinite(x), x * sign, torch.full_like(x, math.nan))  # noqa: E731
    checks = ok & cons
    for pins in [*reversed(waves), None]:
        if pins is None:
            pins = (torch.bincount(to, minlength=P) == 0).nonzero()[:, 0]
        a, _ = _take(fstart, farcs, pins)
        if a.numel() == 0:
            continue
        wr = srt(rat[to[a]])
        cand = wr[:, :, None, :] - delay[a]
        cand = torch.where(go[a] & ~torch.isnan(cand), cand * sign.reshape(1, 2, 1, 1),
                           torch.full_like(cand, -inf)).amax(3)
        idx = frm[a][:, None, None].expand(-1, 2, 2)
        rat.scatter_reduce_(0, idx, cand, "amax")
        # a check's slack moves the required time of the other split's clock
        av, wa = at[frm[a]], at[to[a]]
        c = av.flip(1)[:, :, :, None] + (wa - wr)[:, :, None, :]
        c = torch.where(checks[a] & ~torch.isnan(c), c * -sign.reshape(1, 2, 1, 1),
                        torch.full_like(c, -inf)).amax(3).flip(1)
        rat.scatter_reduce_(0, idx, c, "amax")
    rat = srt(rat)
    slack = (at - rat) * sign
    flat4 = lambda x: x.reshape(P, NC)  # noqa: E731
    out.update({"at": flat4(at), "slew": flat4(sl), "rat": flat4(rat), "slack": flat4(slack)})
    return out


def exact(case, seed):
    """What run() returns in 64 bits (None: whole numbers)."""
    if case["kind"] == "rc":
        return _rc_exact(_rc_forest(case, seed))[0]
    if case["kind"] == "rc_host":
        out = _rc_exact(_rc_forest(case, seed))[0]
        return {k: None if v is None else v.cpu().numpy() for k, v in out.items()}
    if case["kind"] == "update":
        return _update_exact(case, seed)
    return None  # whole numbers, or a design whose files have to be read first
