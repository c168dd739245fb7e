"""The performance cases: what a user of the framework has it do, through its public calls.

Batch runs of the Alpha101 and Alpha158 factor graphs (``runGraph`` on torch or numpy data, fp32,
fp64 and the sliding-moment form; many universes in one ``runGraphBatch``), one tick of a stream
(``StreamContext``) and of a serving pool, and the two utilities behind a factor run (``corrWith``
as rank IC, ``aggregrate``).  Every case is a dict of plain values; ``prepare`` makes its inputs and
output buffers from a seed, ``run`` is one pass, ``exact`` the same results in 64 bits from plain
torch: an interpreter of the factor graphs' definitions (``kunquant_gb300/graphs``).
"""
import functools
import gzip
import json
import math
import os
import random
import re

import numpy as np
import torch

from kunquant_gb300 import runner as kr
from kunquant_gb300 import serve

GRAPHS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kunquant_gb300", "graphs")
FIELDS = ("open", "high", "low", "close", "volume", "amount")

# ------------------------------------------------------------------ the cases
# "kind" names the public call; for batch runs "graph" is the shipped library and "module" its module.


def listed():
    return [
        # the reference's own benchmark: 64 stocks x 260 days, numpy in and out; a research notebook's
        # smallest call, where latency counts
        dict(name="alpha101_notebook", kind="numpy", graph="alpha101_f32", stocks=64, days=260, nan=0.0),
        # one index (300 stocks), two years, data already on the GPU
        dict(name="alpha158_index", kind="batch", graph="alpha158_f32", stocks=300, days=500, nan=0.005),
        # the benchmark's default workload: a whole market over ten years
        dict(name="alpha158_market", kind="batch", graph="alpha158_f32", stocks=5000, days=2500, nan=0.005),
        # Alpha101 on a wide market: rows longer than a block's registers hold at 8 keys a thread
        dict(name="alpha101_market", kind="batch", graph="alpha101_f32", stocks=8192, days=2500, nan=0.005),
        # an odd mid-size universe: rows of under 1024 stocks, unaligned rows
        dict(name="alpha101_midcap", kind="batch", graph="alpha101_f32", stocks=997, days=1251, nan=0.005),
        # double precision
        dict(name="alpha158_double", kind="batch", graph="alpha158_f64", stocks=801, days=1000, nan=0.005),
        # the sliding-moment form, an odd stock count
        dict(name="alpha158_slide", kind="batch", graph="alpha158_slide_f32", stocks=3111, days=1777, nan=0.005),
        # uneven universes in one call
        dict(name="alpha101_universes", kind="universes", graph="alpha101_f32", count=12, stocks=3000, days=1500,
             sizes=4242, nan=0.005),
        # live trading, one universe: push a bar of every input, run, read every factor
        dict(name="stream_tick", kind="tick", graph="alpha101_stream_f32", stocks=4096, history=260),
        # live serving: the sessions of a pool advance together, tables on the GPU
        dict(name="serve_step", kind="serve", graph="alpha101_stream_f32", sessions=48, stocks=5000, sizes=7,
             history=64),
        # rank IC of a set of factors against the next return
        dict(name="rank_ic", kind="ic", factors=32, stocks=5000, days=1250, rank=True),
        # daily bars to monthly ones
        dict(name="monthly_bars", kind="aggregate", inputs=6, stocks=5000, days=2500, group=21),
    ]


def _between(rng, lo, hi):
    """Log-uniform whole number in [lo, hi]; now and then a round one."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, n // 8 * 8) if rng.random() < 0.25 else n


def draw(rng):
    pick = rng.choice(["numpy", "batch158", "batch101", "batch158", "batch101", "double", "slide", "universes",
                       "tick", "serve", "ic", "aggregate"])
    nan = rng.choice([0.0, 0.005, 0.02])
    if pick == "numpy":
        return dict(kind="numpy", graph=rng.choice(["alpha101_f32", "alpha158_f32"]), stocks=_between(rng, 16, 300),
                    days=_between(rng, 60, 500), nan=nan)
    if pick == "batch158":
        return dict(kind="batch", graph="alpha158_f32", stocks=_between(rng, 32, 5000), days=_between(rng, 60, 2500),
                    nan=nan)
    if pick == "batch101":
        return dict(kind="batch", graph="alpha101_f32", stocks=_between(rng, 32, 8192), days=_between(rng, 60, 2500),
                    nan=nan)
    if pick == "double":
        return dict(kind="batch", graph=rng.choice(["alpha101_f64", "alpha158_f64"]), stocks=_between(rng, 32, 1500),
                    days=_between(rng, 60, 1000), nan=nan)
    if pick == "slide":
        return dict(kind="batch", graph="alpha158_slide_f32", stocks=_between(rng, 32, 5000),
                    days=_between(rng, 120, 2500), nan=nan)
    if pick == "universes":
        return dict(kind="universes", graph=rng.choice(["alpha101_f32", "alpha158_f32"]), count=rng.randint(4, 16),
                    stocks=_between(rng, 300, 3000), days=_between(rng, 250, 1500), sizes=rng.randint(1, 10 ** 6),
                    nan=nan)
    if pick == "tick":
        return dict(kind="tick", graph=rng.choice(["alpha101_stream_f32", "alpha158_stream_f32"]),
                    stocks=_between(rng, 4, 768) * 8, history=_between(rng, 64, 260))
    if pick == "serve":
        return dict(kind="serve", graph="alpha101_stream_f32", sessions=_between(rng, 1, 64),
                    stocks=_between(rng, 300, 5000), sizes=rng.randint(1, 10 ** 6), history=_between(rng, 16, 64))
    if pick == "ic":
        return dict(kind="ic", factors=_between(rng, 1, 48), stocks=_between(rng, 50, 6000),
                    days=_between(rng, 60, 1250), rank=rng.random() < 0.5)
    return dict(kind="aggregate", inputs=_between(rng, 1, 6), stocks=_between(rng, 50, 6000),
                days=_between(rng, 120, 2500), group=rng.choice([5, 21, 63]))


# Alphas that rank or compare values which are equal but for rounding (correlations of ranks over a few
# days): their value at a tie hangs on the order of the additions, so 64 bits say nothing about them.
TIES = {"alpha%03d" % n for n in (13, 15, 16, 27, 29, 31, 45, 50, 71, 74, 75, 78, 81, 85, 88, 92, 94, 96, 98)}


# ------------------------------------------------------------------ inputs
def _ohlcv(stocks, days, seed, nan=0.0):
    """Synthetic daily bars [days][stocks] on the GPU, fp32: the distribution of
    kunquant_gb300/synth.py."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal():
        return torch.randn((days, stocks), generator=g, device="cuda")

    first = torch.rand((1, stocks), generator=g, device="cuda") * 90 + 10
    close = first * torch.exp(torch.cumsum(normal() * 0.02, 0))
    before = torch.cat([first, close[:-1]])
    opened = before * torch.exp(normal() * 0.005)
    out = {"open": opened,
           "high": torch.maximum(opened, close) * (1 + (normal() * 0.01).abs()),
           "low": torch.minimum(opened, close) * (1 - (normal() * 0.01).abs()),
           "close": close,
           "volume": torch.exp(13 + normal())}
    out["amount"] = out["volume"] * (opened + close) * 0.5
    if nan:
        for k in FIELDS:
            out[k][torch.rand((days, stocks), generator=g, device="cuda") < nan] = float("nan")
    return out


def _bars(case, seed):
    d = _ohlcv(case["stocks"], case["days"], seed, case["nan"])
    if _type(case) == torch.float64:
        d = {k: v.double() for k, v in d.items()}
    return d


def _type(case):
    return torch.float64 if case["graph"].endswith("_f64") else torch.float32


def _sizes(case):
    """(stocks, days) of each universe."""
    r = random.Random(case["sizes"])
    return [(int(math.exp(r.uniform(math.log(37), math.log(case["stocks"])))), r.randint(120, case["days"]))
            for _ in range(case["count"])]


def _session_sizes(case):
    r = random.Random(case["sizes"])
    return [int(math.exp(r.uniform(math.log(100), math.log(case["stocks"])))) for _ in range(case["sessions"])]


def _families(names):
    """Output names grouped by factor family (RESI5, RESI10, ... -> RESI), or alpha numbers by tens:
    the buffers that a program lays out for the results, one [n][days][stocks] block a family."""
    fam = {}
    for n in names:
        key = ("ties" if n in TIES else n[:-1]) if n.startswith("alpha") else re.sub(r"\d+$", "", n)
        fam.setdefault(key, []).append(n)
    return fam


def _parts(n):
    """Rows in each of the parts that a table of n factor rows is returned in."""
    return -(-n // 60)


def _module(graph):
    return graph[:-4] if graph != "alpha101_f64" and graph != "alpha158_f64" else graph


@functools.lru_cache(None)
def _load(graph):
    return kr.Library.predefined(graph).getModule(_module(graph))


@functools.lru_cache(None)
def _executor():
    """One executor for the whole program, as the reference's users keep one thread pool."""
    return kr.createMultiThreadExecutor(8)


def _blocks(names, shape, make):
    """{family: [n][shape] block} and {name: its slice}."""
    blocks, outputs = {}, {}
    for fam, members in _families(names).items():
        blocks[fam] = make((len(members),) + shape)
        for i, n in enumerate(members):
            outputs[n] = blocks[fam][i]
    return blocks, outputs


# ------------------------------------------------------------------ prepare / run
def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "ex": _executor()}
    if kind in ("batch", "numpy"):
        s["mod"], s["days"] = _load(case["graph"]), case["days"]
        names, shape = s["mod"].getOutputNames(), (case["days"], case["stocks"])
        s["inputs"] = _bars(case, seed)
        if kind == "numpy":
            s["inputs"] = {k: v.cpu().numpy() for k, v in s["inputs"].items()}
            s["blocks"], s["outputs"] = _blocks(names, shape, lambda n: np.empty(n, np.float32))
        else:
            s["blocks"], s["outputs"] = _blocks(names, shape, lambda n: torch.empty(n, dtype=_type(case),
                                                                                    device="cuda"))
    elif kind == "universes":
        s["mod"] = _load(case["graph"])
        names = s["mod"].getOutputNames()
        s["inputs"] = [_ohlcv(n, t, seed * 64 + i, case["nan"]) for i, (n, t) in enumerate(_sizes(case))]
        s["blocks"] = [torch.empty((len(names), t, n), device="cuda") for n, t in _sizes(case)]
        s["outputs"] = [{k: b[i] for i, k in enumerate(names)} for b in s["blocks"]]
    elif kind == "tick":
        s["mod"] = _load(case["graph"])
        s["ctx"] = kr.StreamContext(s["ex"], s["mod"], case["stocks"])
        names, fields = s["mod"].getOutputNames(), s["mod"].getInputNames()
        bars = {k: v.cpu().numpy() for k, v in _ohlcv(case["stocks"], case["history"] + 8, seed).items()}
        s["put"] = {k: s["ctx"].queryBufferHandle(k) for k in fields}
        s["get"] = [s["ctx"].queryBufferHandle(k) for k in names]
        for t in range(case["history"]):
            for k, h in s["put"].items():
                s["ctx"].pushData(h, bars[k][t])
            s["ctx"].run()
        s["bars"] = [{k: bars[k][case["history"] + j].copy() for k in fields} for j in range(8)]
        s["rows"], s["at"] = np.empty((len(names), case["stocks"]), np.float32), 0
        s["part"] = _parts(len(names))
    elif kind == "serve":
        s["mod"] = _load(case["graph"])
        sizes = _session_sizes(case)
        cap, fields = sum(sizes), s["mod"].getInputNames()
        s["pool"] = serve.ServePool(s["ex"], s["mod"], capacity_stocks=cap, max_sessions=64,
                                    max_session_stocks=5000, start=False)
        s["sessions"] = [s["pool"].open(n) for n in sizes]
        bars = _ohlcv(cap, case["history"] + 8, seed)
        tables = [torch.stack([bars[k][t] for k in fields]) for t in range(case["history"] + 8)]
        s["table"] = torch.empty((len(s["mod"].getOutputNames()), cap), device="cuda")
        for t in range(case["history"]):
            s["pool"].step(s["sessions"], device_inputs=tables[t], device_outputs=s["table"])
        s["tables"], s["at"], s["part"] = tables[case["history"]:], 0, _parts(len(s["table"]))
    elif kind == "ic":
        g = torch.Generator(device="cuda").manual_seed(seed)
        shape = (case["days"], case["stocks"])
        s["y"] = torch.randn(shape, generator=g, device="cuda") * 0.02
        s["factors"] = [torch.randn(shape, generator=g, device="cuda") * (k + 1) + s["y"] * 5
                        for k in range(case["factors"])]
        s["ics"] = torch.empty((case["factors"], case["days"]), device="cuda")
        s["rank"] = case["rank"]
    else:
        bars = _ohlcv(case["stocks"], case["days"], seed)
        s["inputs"] = [bars[k] for k in FIELDS[:case["inputs"]]]
        s["labels"] = [torch.arange(case["days"], device="cuda").div(case["group"], rounding_mode="floor").float()
                       for _ in s["inputs"]]
        groups = -(-case["days"] // case["group"])
        s["outs"] = [{k: torch.empty((groups, case["stocks"]), device="cuda") for k in AGGREGATES}
                     for _ in s["inputs"]]
    return s


AGGREGATES = ("sum", "min", "max", "first", "last", "count", "mean")


def run(s):
    kind = s["kind"]
    if kind in ("batch", "numpy"):
        kr.runGraph(s["ex"], s["mod"], s["inputs"], 0, s["days"], outputs=s["outputs"])
        return s["blocks"]
    if kind == "universes":
        kr.runGraphBatch(s["ex"], s["mod"], s["inputs"], outputs_list=s["outputs"])
        return s["blocks"]
    if kind == "tick":
        ctx, bar = s["ctx"], s["bars"][s["at"] % 8]
        s["at"] += 1
        for k, h in s["put"].items():
            ctx.pushData(h, bar[k])
        ctx.run()
        for i, h in enumerate(s["get"]):
            s["rows"][i] = ctx.getCurrentBuffer(h)
        return [s["rows"][i:i + s["part"]] for i in range(0, len(s["rows"]), s["part"])]
    if kind == "serve":
        table = s["tables"][s["at"] % 8]
        s["at"] += 1
        s["pool"].step(s["sessions"], device_inputs=table, device_outputs=s["table"])
        return list(s["table"].split(s["part"]))
    if kind == "ic":
        kr.corrWith(s["ex"], s["factors"], s["y"], list(s["ics"]), rank_inputs=s["rank"])
        return s["ics"]
    kr.aggregrate(s["ex"], s["inputs"], s["labels"], s["outs"])
    return s["outs"]


# ------------------------------------------------------------------ work
def _io(graph):
    return (6, 158) if "158" in graph else (6, 82)


@functools.lru_cache(None)
def _flops_per_cell(graph):
    """Operations at one stock and day that no way of computing the graph's definition saves: one a
    pointwise op or window reduction, two a running sum, the logarithm of the row or window an order."""
    cost = {"FastWindowedSum": 2, "Rank": 13, "SkipListState": 6, "Input": 0, "Output": 0, "ConstantOp": 0,
            "WindowedTempOutput": 0, "IterValue": 0, "BackRef": 0, "ForeachBackWindow": 0, "WindowLoopIndex": 0}
    g = _graph(graph.replace("_slide", "").replace("_stream", ""))
    return sum(cost.get(o["k"], 1) for st in g["stages"] for o in st["ops"])


def work(case):
    kind = case["kind"]
    if kind in ("batch", "numpy"):
        cells, size = case["stocks"] * case["days"], 8 if case["graph"].endswith("_f64") else 4
        return {"bytes": sum(_io(case["graph"])) * size * cells, "flops": _flops_per_cell(case["graph"]) * cells}
    if kind == "universes":
        cells = sum(n * t for n, t in _sizes(case))
        return {"bytes": sum(_io(case["graph"])) * 4 * cells, "flops": _flops_per_cell(case["graph"]) * cells}
    if kind in ("tick", "serve"):
        # the bars and the factors, and the state that a tick has to read at least once: one row of
        # every input that its longest windows hold is replaced, so the windows themselves are not counted
        cells = case["stocks"] if kind == "tick" else sum(_session_sizes(case))
        return {"bytes": sum(_io(case["graph"])) * 4 * cells, "flops": _flops_per_cell(case["graph"]) * cells}
    cells = case["stocks"] * case["days"]
    if kind == "ic":
        return {"bytes": 4 * (case["factors"] + 1) * cells + 4 * case["factors"] * case["days"],
                "flops": (10 + (13 if case["rank"] else 0)) * case["factors"] * cells}
    groups = -(-case["days"] // case["group"])
    return {"bytes": 4 * case["inputs"] * (cells + case["days"] + 7 * groups * case["stocks"]),
            "flops": 7 * case["inputs"] * cells}


# ------------------------------------------------------------------ 64-bit results
def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "numpy"):
        got = _evaluate(case["graph"], _bars(case, seed))
        return {f: None if f == "ties" else torch.stack([got[n] for n in members])
                for f, members in _families(list(got)).items()}
    if kind == "universes":
        if "101" in case["graph"]:  # each block holds alphas of TIES
            return None
        return [torch.stack(list(_evaluate(case["graph"], _ohlcv(n, t, seed * 64 + i, case["nan"])).values()))
                for i, (n, t) in enumerate(_sizes(case))]
    if kind == "tick":
        bars = _ohlcv(case["stocks"], case["history"] + 8, seed)
        got = _evaluate(case["graph"], {k: v[:case["history"] + 1] for k, v in bars.items()})
        return _rows({k: v[-1] for k, v in got.items()})
    if kind == "serve":
        sizes = _session_sizes(case)
        bars, cols, at = _ohlcv(sum(sizes), case["history"] + 8, seed), [], 0
        for n in sizes:
            got = _evaluate(case["graph"], {k: v[:case["history"] + 1, at:at + n] for k, v in bars.items()})
            cols.append({k: v[-1] for k, v in got.items()})
            at += n
        return _rows({k: torch.cat([c[k] for c in cols]) for k in cols[0]})
    s = prepare(case, seed)
    if kind == "ic":
        y, rows = s["y"].double(), []
        for f in s["factors"]:
            x = _rank(f.double()) if case["rank"] else f.double()
            a, b = x - x.mean(1, keepdim=True), y - y.mean(1, keepdim=True)
            rows.append((a * b).sum(1) / ((a * a).sum(1) * (b * b).sum(1)).sqrt())
        return torch.stack(rows)
    res = []
    for x in s["inputs"]:
        parts = [p.double() for p in x.split(case["group"])]
        res.append({"sum": torch.stack([p.sum(0) for p in parts]), "min": torch.stack([p.amin(0) for p in parts]),
                    "max": torch.stack([p.amax(0) for p in parts]), "first": torch.stack([p[0] for p in parts]),
                    "last": torch.stack([p[-1] for p in parts]),
                    "count": torch.stack([torch.full_like(p[0], len(p)) for p in parts]),
                    "mean": torch.stack([p.mean(0) for p in parts])})
    return res


def _rows(got):
    """The last rows of the factors, in run()'s parts; no value for a part that holds one of TIES."""
    names, part = list(got), _parts(len(got))
    return [None if TIES & set(names[i:i + part]) else torch.stack([got[n] for n in names[i:i + part]])
            for i in range(0, len(names), part)]


@functools.lru_cache(None)
def _graph(graph):
    with gzip.open(os.path.join(GRAPHS, graph + ".json.gz")) as f:
        return json.loads(f.read())


def _rank(x):
    """Average rank in the row over the number of non-NaN values, in (0, 1]."""
    bad = x.isnan()
    full = torch.where(bad, torch.full_like(x, math.inf), x)
    order = full.sort(1).values
    n = (~bad).sum(1, keepdim=True).double()
    lo = torch.searchsorted(order, full.contiguous()).double()
    hi = torch.minimum(torch.searchsorted(order, full.contiguous(), right=True).double(), n)
    return torch.where(bad, math.nan, (lo + hi + 1) * 0.5 / n)


def _back(x, n):
    """The value n rows ago, NaN before the first row."""
    if n == 0:
        return x
    out = torch.full_like(x, math.nan)
    if n < x.shape[0]:
        out[n:] = x[:-n]
    return out


def _quantile(x, w, q):
    out = torch.full_like(x, math.nan)
    at = q * (w - 1)
    i = int(at)
    for t in range(w - 1, x.shape[0], 128):
        win = x[t - w + 1:t + 128].unfold(0, w, 1).sort(-1).values  # NaN sorts last
        v = win[..., i] if at == i else win[..., i] + (win[..., i + 1] - win[..., i]) * (at - i)
        out[t:t + 128] = torch.where(win[..., w - 1].isnan(), math.nan, v)
    return out


class _Regression:
    """Window regression of the value on its place in the window, 1 .. w, over its non-NaN rows."""

    def __init__(self, x, w):
        self.w = w
        n, sx, sxx, sy = (torch.zeros_like(x) for _ in range(4))
        for back in range(w):
            y = _back(x, back)
            ok = (~y.isnan()).double()
            n, sx, sxx, sy = n + ok, sx + ok * (w - back), sxx + ok * (w - back) ** 2, sy + y.nan_to_num(0.0)
        self.mx, self.my = sx / n, sy / n
        self.vx, self.vy, self.c = (torch.zeros_like(x) for _ in range(3))
        for back in range(w):
            y = _back(x, back)
            ok = ~y.isnan()
            dx, dy = torch.where(ok, w - back - self.mx, 0.0), torch.where(ok, y - self.my, 0.0)
            self.vx, self.vy, self.c = self.vx + dx * dx, self.vy + dy * dy, self.c + dx * dy

    def slope(self):
        return self.c / self.vx

    def rsq(self):
        return self.c * self.c / (self.vx * self.vy)

    def resi(self, x):
        return x - (self.my + self.slope() * (self.w - self.mx))


_POINTWISE = {
    "Add": torch.add, "Sub": torch.sub, "Mul": torch.mul, "Div": torch.div,
    "Max": lambda a, b: torch.where(a > b, a, b), "Min": lambda a, b: torch.where(a < b, a, b),
    "GreaterThan": torch.gt, "GreaterEqual": torch.ge, "LessThan": torch.lt, "LessEqual": torch.le,
    "Equals": torch.eq, "Or": torch.logical_or, "And": torch.logical_and, "Not": torch.logical_not,
    "Sqrt": torch.sqrt, "Abs": torch.abs, "Log": torch.log, "Exp": torch.exp,
    "Sign": lambda a: torch.where(a.isnan(), a, torch.sign(a)),
    "Select": lambda c, a, b: torch.where(c, a, b), "ReturnFirstValue": lambda a, *_: a,
}
_CONSTANT = {"AddConst": torch.add, "SubConst": torch.sub, "MulConst": torch.mul, "DivConst": torch.div,
             "GreaterThanConst": torch.gt, "LessThanConst": torch.lt}


def _pointwise(op, args, like):
    k = op["k"]
    if k == "ConstantOp":
        return torch.full_like(like, float(op["value"]))
    if k == "SetInfOrNanToValue":
        return torch.where(args[0].isfinite(), args[0], float(op["value"]))
    if k in _CONSTANT:
        c = torch.full((), float(op["value"]), dtype=torch.float64, device=like.device)
        return _CONSTANT[k](c, args[0]) if op.get("swap") else _CONSTANT[k](args[0], c)
    return _POINTWISE[k](*args)


class _Reduction:
    def __init__(self, op, like, current):
        self.k, self.current = op["k"], current
        w = op.get("window", 1)
        self.weight = self.step = 2.0 / ((1.0 + w) * w)
        start = {"ReduceMul": 1.0, "ReduceMin": math.inf, "ReduceArgMin": math.inf, "ReduceMax": -math.inf,
                 "ReduceArgMax": -math.inf}.get(self.k, 0.0)
        self.v, self.bad = torch.full_like(like, start), torch.zeros_like(like, dtype=torch.bool)
        self.more = torch.zeros_like(like) if self.k in ("ReduceRank", "ReduceArgMin", "ReduceArgMax") else None

    def add(self, x, back):
        if self.k == "ReduceAdd":
            self.v = self.v + x
        elif self.k == "ReduceMul":
            self.v = self.v * x
        elif self.k == "ReduceDecayLinear":
            self.v, self.weight = self.v + x * self.weight, self.weight + self.step
        elif self.k == "ReduceRank":
            self.v, self.more = self.v + (x < self.current), self.more + (x == self.current)
            self.bad |= x.isnan()
        else:
            better = x > self.v if self.k.endswith("Max") else x < self.v
            if self.more is not None:
                self.more = torch.where(better, float(back), self.more)
            self.v = torch.where(better, x, self.v)
            self.bad |= x.isnan()

    def value(self):
        if self.k == "ReduceRank":
            return torch.where(self.bad | self.current.isnan(), math.nan, self.v + (self.more + 1) / 2)
        got = self.more if self.more is not None else self.v
        return torch.where(self.bad, math.nan, got)


class _Values(dict):
    def __getitem__(self, i):
        v = dict.__getitem__(self, i)
        return v.value() if isinstance(v, _Reduction) else v


def _stage(stage, buffers):
    """The series that one stage makes of the ones it reads: {buffer: [days][stocks]}."""
    ops, val, made, loops, before = stage["ops"], _Values(), {}, {}, None
    like = buffers[stage["in"][0]]
    reduction = {}

    def loop_of(i):
        first = ops[ops[i]["in"][0]]
        return ops[i]["in"][0] if first["k"] == "ForeachBackWindow" else first.get("p", -1)

    for i, o in enumerate(ops):
        k, a = o["k"], o["in"]
        if o.get("p", -1) >= 0:
            continue
        if k == "Input":
            val[i] = buffers[o["buf"]]
        elif k in ("Output", "WindowedTempOutput"):
            val[i] = val[a[0]]
            if k == "Output":
                made[o["buf"]] = val[i]
        elif k == "ForeachBackWindow":
            own = [j for j, r in enumerate(ops) if r["k"].startswith("Reduce") and loop_of(j) == i]
            body, reds = ([], []) if not o.get("copy_prev_body") else (list(loops[before][0]), list(loops[before][1]))
            body += [j for j, b in enumerate(ops) if b.get("p", -1) == i]
            for j in own:
                val[j] = reduction[j] = _Reduction(ops[j], like, val[ops[j]["in"][1]] if ops[j]["k"] == "ReduceRank" else None)
            reds += own
            loops[i], before = (body, reds), i
            for back in range(o["window"] - 1, o.get("segment_end", 0) - 1, -1):
                for j in body:
                    b = ops[j]
                    val[j] = (_back(val[b["in"][1]], back) if b["k"] == "IterValue" else
                              _pointwise(b, [val[x] for x in b["in"]], like))
                for j in reds:
                    reduction[j].add(val[ops[j]["in"][0]], back)
        elif k.startswith("Reduce"):
            pass
        elif k == "BackRef":
            val[i] = _back(val[a[0]], o["window"])
        elif k == "FastWindowedSum":
            val[i] = sum(_back(val[a[0]], b) for b in range(o["window"]))
        elif k == "WindowedLinearRegression":
            val[i] = _Regression(val[a[0]], o["window"])
        elif k.startswith("WindowedLinearRegression"):
            val[i] = (val[a[0]].rsq() if "RSq" in k else val[a[0]].slope() if "Slope" in k else
                      val[a[0]].resi(val[a[1]]))
        elif k == "SkipListState":
            val[i] = (val[a[1]], o["window"])
        elif k == "SkipListQuantile":
            val[i] = _quantile(*val[a[0]], float(o["q"]))
        elif k == "Rank":
            val[i] = _rank(val[a[0]])
        elif k == "Scale":
            val[i] = val[a[0]] / val[a[0]].abs().nan_to_num(0.0, math.inf).sum(1, keepdim=True)
        else:
            val[i] = _pointwise(o, [val[x] for x in a], like)
    return made


def _evaluate(graph, bars):
    """{output: [days][stocks]} of a graph in 64 bits."""
    g = _graph(graph.replace("_slide", "").replace("_stream", ""))
    buffers = {b["id"]: bars[b["name"]].double() for b in g["buffers"] if b["kind"] == "INPUT"}
    users, todo = {b["id"]: 0 for b in g["buffers"]}, list(g["stages"])
    for st in todo:
        for b in st["in"]:
            users[b] += 1
    kind = {b["id"]: b["kind"] for b in g["buffers"]}
    while todo:
        st = next(s for s in todo if all(b in buffers for b in s["in"]))
        todo.remove(st)
        buffers.update(_stage(st, buffers))
        for b in st["in"]:
            users[b] -= 1
            if not users[b] and kind[b] == "TEMP":
                del buffers[b]
    return {b["name"]: buffers[b["id"]] for b in g["buffers"] if b["kind"] == "OUTPUT"}
