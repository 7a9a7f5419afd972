"""The workloads that the speed of this library is judged by: what a serving host has the MoE expert path do, through the
public entry points, from one EXL3 linear to an 8192-row prefill chunk.

A case is a dict of plain values:
  kind    "linear"  one EXL3 linear (exl3_linear)
          "layers"  MoE layers after routing (Moe.run), each with weights of its own; with `graph` the walk over the layers is
                    replayed through GraphCache, as a host's decode loop does; with `routed` the router runs in front of every
                    layer (route); with `host` the host-buffer call is used (Moe.run_host)
          "tables"  the owners that hosts with a combine of their own call: Grouping.run + ExpertGpu.run_rows (<= 16 rows) or
                    FastExperts.run
          "route"   router logits + sigmoid top-k of a chunk (route)
  hidden, inter, experts, slots, rows: sizes of the bank and of the window (slots = top-k + 1)
  layers  distinct weight banks walked by one pass
  lo, hi, shared, shared_lo, shared_hi: the expert-parallel window of a rank (routed experts [lo, hi), the shared expert
          computed here or not, and for chunks of more than 16 rows the rows it is computed for)
  bias    the rows of a window share one routing bias (speculative verify: about half of their experts overlap)
  shared_x  gate and up have one input scale vector, so one rotated copy of the input serves both
Weights are random trellis words; the output scales put the pre-activations of SwiGLU at unit variance, as trained weights do.
"""
import math

import numpy as np
import torch

import __graft_entry__ as entry

LINEAR_K = (256, 512, 768, 1024, 1536, 2048, 2304, 3072, 4096)
MAX_FLOPS = 8192 * 8 * 6 * 4096 * 512                       # the largest listed case
MAX_STACK_BYTES = 15e9                                      # a 47-layer stack of the benchmark's layer


def _layers(name, rows, **kw):
    c = dict(name=name, kind="layers", hidden=2048, inter=1536, experts=64, slots=5, rows=rows, layers=1, graph=False, routed=False,
             host=False, bias=False, shared_x=False, lo=0, hi=kw.get("experts", 64), shared=1, shared_lo=0, shared_hi=0)
    c.update(kw)
    return c


def _tables(name, rows, **kw):
    return _layers(name, rows, kind="tables", **kw)


UPSTREAM = dict(hidden=4096, inter=512, experts=288, slots=9, hi=288, shared=0)   # one of four tensor-parallel shards


def listed():
    return [
        # one quantised linear (a projection outside the expert path), the smallest call there is
        dict(name="linear-1", kind="linear", K=2048, N=1536, rows=1),
        # one token of one request through the whole stack, the decode loop's captured graph
        _layers("decode-1", 1, layers=47, graph=True),
        # the same without a graph and with the router in front of every layer: launches and host calls count
        _layers("decode-1-routed", 1, layers=8, routed=True),
        # eight requests' tokens handed over in host memory, layer by layer, the result read back
        _layers("decode-8-host", 8, layers=4, host=True),
        # speculative verify window, sixteen rows of overlapping experts, captured graph
        _layers("verify-16", 16, layers=8, graph=True, bias=True),
        # an odd verify window on a tensor-parallel shard of the larger model, table-driven owners
        _tables("verify-11-tables", 11, layers=4, bias=True, **UPSTREAM),
        # the ragged tail of a prompt
        _layers("chunk-40", 40),
        # an ordinary short prompt
        _layers("prefill-500", 500),
        # the benchmark's prefill chunk
        _layers("prefill-4096", 4096),
        # the share of one of eight expert-parallel ranks of that chunk
        _layers("prefill-4096-ep", 4096, lo=8, hi=16, shared_lo=512, shared_hi=1024),
        # the largest chunk, on the tensor-parallel shard, table-driven owners
        _tables("prefill-8192-tables", 8192, shared_x=True, **UPSTREAM),
        # the router of the benchmark's prefill chunk
        dict(name="route-4096", kind="route", hidden=2048, experts=64, slots=5, rows=4096),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(("linear", "decode", "decode", "routed", "host", "verify", "verify", "tables", "chunk", "chunk", "prefill", "prefill",
                       "prefill-tables", "prefill-ep", "route"))
    if what == "linear":
        return dict(kind="linear", K=rng.choice(LINEAR_K), N=128 * rng.randint(1, 32), rows=rng.randint(1, 16))
    size = rng.choice((dict(hidden=2048, inter=1536, experts=64, slots=5),) * 3 + (
        dict(hidden=4096, inter=512, experts=288, slots=9), dict(hidden=rng.choice((1024, 1536, 2304, 3072)), inter=rng.choice((256, 512, 768, 1024, 2048)),
                                                                 experts=rng.randint(8, 128), slots=rng.randint(3, 9))))
    if size["slots"] > size["experts"]:
        size["slots"] = size["experts"]
    if what == "route":
        return dict(kind="route", hidden=size["hidden"], experts=size["experts"], slots=size["slots"], rows=_log(rng, 1, 8192))
    bank = _expert_bytes(size) * (size["experts"] + 1)
    pair = 6 * size["hidden"] * size["inter"]
    c = _layers(None, 0, **size)
    del c["name"]
    c["hi"] = size["experts"]
    if what in ("decode", "routed", "host", "verify") or (what == "tables"):
        c["rows"] = rng.randint(1, 4) if what in ("decode", "routed") else rng.randint(1, 16)
        c["bias"] = what in ("verify", "tables")
        c["layers"] = max(1, min(rng.randint(2, 24), int(MAX_STACK_BYTES / bank)))
        c["graph"] = what in ("decode", "verify") and rng.random() < 0.8
        c["routed"], c["host"] = what == "routed", what == "host"
        if what == "routed" or what == "host":
            c["layers"] = min(c["layers"], 8)
        if what == "tables":
            c["kind"], c["shared"] = "tables", rng.randint(0, 1)
        return c
    c["shared_x"] = rng.random() < 0.3
    most = min(8192, MAX_FLOPS // (pair * size["slots"]))
    c["rows"] = rng.randint(17, 256) if what == "chunk" else min(_log(rng, 257, 8192), most)
    if what == "prefill-tables":
        c["kind"], c["shared"] = "tables", rng.randint(0, 1)
    if what == "prefill-ep":
        world = rng.choice((2, 4, 8))
        w, rank = -(-size["experts"] // world), rng.randrange(world)
        c["lo"], c["hi"] = min(rank * w, size["experts"]), min((rank + 1) * w, size["experts"])
        per = -(-c["rows"] // world)
        c["shared_lo"], c["shared_hi"] = min(rank * per, c["rows"]), min((rank + 1) * per, c["rows"])
        if c["shared_lo"] == c["shared_hi"]:
            c["shared_lo"] = c["shared_hi"] = 0
            c["shared"] = 0
    return c


# ---- what a host has in hand before the call -----------------------------------------------------------------------

_stream = None


def stream():
    """The one stream of the host's decode loop (graphs cannot be captured on the default stream)."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def _scales(g, e, n, s=1.0):
    sign = torch.where(torch.rand((e, n), device="cuda", generator=g) < 0.5, -s, s)
    return (sign * (0.5 + torch.rand((e, n), device="cuda", generator=g))).to(torch.float16)


def _words(g, e, K, N):
    return torch.randint(-(1 << 31), (1 << 31) - 1, (e, K // 16, N // 16, 32), dtype=torch.int32, device="cuda", generator=g)


def _bank(g, c):
    H, I, E1 = c["hidden"], c["inter"], c["experts"] + 1
    sg, sd = 1.0 / (1.244 * math.sqrt(H)), 1.0 / (1.244 * math.sqrt(I))
    b = {"gt": _words(g, E1, H, I), "ut": _words(g, E1, H, I), "dt": _words(g, E1, I, H), "suh_g": _scales(g, E1, H), "suh_u": _scales(g, E1, H),
         "suh_d": _scales(g, E1, I), "svh_g": _scales(g, E1, I, sg), "svh_u": _scales(g, E1, I, sg), "svh_d": _scales(g, E1, H, sd)}
    if c["shared_x"]:
        b["suh_u"] = b["suh_g"]
    return b


def _routing(g, c):
    """Sigmoid top-k of N(0, 1) logits: picks int32 [rows][slots], weights fp32 [rows][slots], the shared expert last."""
    logits = torch.randn((c["rows"], c["experts"]), device="cuda", generator=g)
    if c["bias"]:
        logits = logits + torch.randn((1, c["experts"]), device="cuda", generator=g)
    top, ids = torch.sigmoid(logits).topk(c["slots"] - 1, dim=1)
    picks = torch.cat([ids.to(torch.int32), torch.full((c["rows"], 1), c["experts"], dtype=torch.int32, device="cuda")], 1)
    weights = torch.cat([top / top.sum(1, keepdim=True), torch.ones((c["rows"], 1), device="cuda")], 1)
    return picks.contiguous(), weights.contiguous()


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h


def _kept(view, owner):
    """A view of an owner's buffer is valid while the owner lives: the view keeps it."""
    view.owner = owner
    return view


class State:
    pass


def prepare(case, seed):
    pkg = entry.load_package()
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    s, c = State(), case
    s.case, s.pkg, s.rows = c, pkg, c["rows"]
    if c["kind"] == "linear":
        K, N = c["K"], c["N"]
        s.x = torch.randn((s.rows, K), device="cuda", generator=g).to(torch.float16)
        s.words, s.suh, s.svh = _words(g, 1, K, N), _scales(g, 1, K), _scales(g, 1, N)
        return s
    E, S, H, rows = c["experts"], c["slots"], c["hidden"], c["rows"]
    if c["kind"] == "route" or c.get("routed"):
        n = c.get("layers", 1)
        s.wr = [(torch.randn((E, H), device="cuda", generator=g) / math.sqrt(H)).to(torch.bfloat16) for _ in range(n)]
        s.logits = [torch.empty((rows, E), device="cuda") for _ in range(n)]
        s.picks = [torch.empty((rows, S), dtype=torch.int32, device="cuda") for _ in range(n)]
        s.weights = [torch.empty((rows, S), device="cuda") for _ in range(n)]
        s.x = [torch.randn((rows, H), device="cuda", generator=g).to(torch.bfloat16) for _ in range(n)]
        if c["kind"] == "route":
            return s
    else:
        s.x = [torch.randn((rows, H), device="cuda", generator=g).to(torch.bfloat16) for _ in range(c["layers"])]
        s.picks, s.weights = map(list, zip(*[_routing(g, c) for _ in range(c["layers"])]))
    s.banks = [_bank(g, c) for _ in range(c["layers"])]
    s.w = [pkg.weights_struct(b) for b in s.banks]
    cfg = pkg.make_config(H, c["inter"], E, S, max_rows=rows, shared_exl3=c["shared"], expert_lo=c["lo"], expert_hi=c["hi"],
                          shared_rows=(c["shared_lo"], c["shared_hi"]))
    if c["kind"] == "tables":
        s.grouping = [pkg.Grouping(cfg) for _ in range(c["layers"])]
        s.tables = [(q.ids, q.count, q.members) for q in s.grouping]
        s.owner = [(pkg.ExpertGpu if rows <= 16 else pkg.FastExperts)(cfg) for _ in range(c["layers"])]
        s.out = [_kept(o.y if rows <= 16 else o.output, o) for o in s.owner]
        return s
    s.owner = [pkg.Moe(cfg) for _ in range(c["layers"])]
    s.out = [_kept(o.output, o) for o in s.owner]
    if c["host"]:
        s.x, s.picks, s.weights = ([_pinned(t) for t in v] for v in (s.x, s.picks, s.weights))
        s.out = [torch.empty((rows, H), dtype=torch.float32, pin_memory=True) for _ in s.owner]
    if c["graph"]:
        s.cache = pkg.GraphCache(bounded=False)
    return s


def _step(s):
    for l, owner in enumerate(s.owner):
        owner.run(s.w[l], s.x[l], s.picks[l], s.weights[l], s.rows)


def run(s):
    c, pkg = s.case, s.pkg
    if c["kind"] == "linear":
        return pkg.exl3_linear(s.x, s.words, s.suh, s.svh, c["K"], c["N"])
    if c["kind"] == "route":
        pkg.route(s.x[0], s.wr[0], s.logits[0], s.picks[0], s.weights[0])
        return [s.logits[0], s.picks[0], s.weights[0]]
    if c["kind"] == "tables":
        for l, owner in enumerate(s.owner):
            s.grouping[l].run(s.picks[l], s.rows)
            ids, count, members = s.tables[l]
            if s.rows <= 16:
                owner.run_rows(s.w[l], s.x[l], s.picks[l], ids, count, members, s.rows, s.rows)
            else:
                owner.run(s.w[l], s.x[l], s.picks[l], ids, count, members, s.rows, s.rows, shared_x=c["shared_x"])
        return s.out
    if c["graph"]:
        s.cache.run(s.rows, lambda: _step(s), stream=stream())
        return s.out
    for l, owner in enumerate(s.owner):
        if c["host"]:
            owner.run_host(s.w[l], s.x[l], s.picks[l], s.weights[l], s.rows, s.out[l])
            continue
        if c["routed"]:
            pkg.route(s.x[l], s.wr[l], s.logits[l], s.picks[l], s.weights[l])
        owner.run(s.w[l], s.x[l], s.picks[l], s.weights[l], s.rows)
    return s.out


# ---- what a pass cannot do without ------------------------------------------------------------------------------------

def _expert_bytes(c):
    """Packed words (4 bits a weight) and the six fp16 scale vectors of one expert."""
    H, I = c["hidden"], c["inter"]
    return 3 * H * I // 2 + 2 * (3 * H + 3 * I)


def _distinct(c):
    """Routed experts of [lo, hi) that a window of this case touches, on average."""
    g = np.random.Generator(np.random.PCG64(1))
    n, rows, E, k = 0.0, min(c["rows"], 2048), c["experts"], c["slots"] - 1
    times = 20 if rows <= 16 else 2
    for _ in range(times):
        logits = g.standard_normal((rows, E)) + (g.standard_normal((1, E)) if c["bias"] else 0.0)
        ids = np.unique(np.argpartition(-logits, k - 1, axis=1)[:, :k])
        n += ((ids >= c["lo"]) & (ids < c["hi"])).sum() / times
    return float(n)


def work(case):
    c, rows = case, case["rows"]
    if c["kind"] == "linear":
        K, N = c["K"], c["N"]
        return {"bytes": K * N / 2 + 2 * (K + N) + 2 * rows * (K + N), "flops": 2 * rows * K * N}
    H, E, S = c["hidden"], c["experts"], c["slots"]
    route = {"bytes": 2 * rows * H + 2 * E * H + 4 * rows * E + 8 * rows * S, "flops": 2 * rows * E * H}
    if c["kind"] == "route":
        return route
    routed = rows * (S - 1) * (c["hi"] - c["lo"]) / E
    shared = 0 if not c["shared"] else c["shared_hi"] - c["shared_lo"] if c["shared_hi"] else rows
    out = 4 * H * (routed + shared if c["kind"] == "tables" else rows)
    b = (_distinct(c) + (shared > 0)) * _expert_bytes(c) + 2 * rows * H + rows * S * (4 if c["kind"] == "tables" else 8) + out
    f = 6 * H * c["inter"] * (routed + shared)
    if c["routed"]:
        b, f = b + route["bytes"], f + route["flops"]
    return {"bytes": c["layers"] * b, "flops": c["layers"] * f}


def tolerance(case):
    if case["kind"] == "route":
        return {"rel": 1e-5, "differ": 1e-3}              # fp32 sums of bf16 products; near ties may fall the other way
    return {"rel": 1e-3}                                  # fp16 and bf16 intermediates, fp32 accumulation
