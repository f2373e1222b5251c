"""The work a user of this framework has it do, as cases that can be timed and checked.

Every case goes through the public Python entry points (nt2_gb300.lib, nt2_gb300.expr).  The kinds:

  price     Black-Scholes call and put of one option book (sigma one number or a table; both arithmetic policies)
  greeks    prices and gradients of a book in one pass (the fused reverse-mode kernel)
  functors  a user's own expressions of NT2's functors, one tie of several outputs (run-time compiled)
  gradient  reverse mode of a user's own program (run-time compiled)
  reduce    sum, dot, a fold of an expression, and globalmax with its position over whole tables
  stats     mean, stdev and maximum (with position) of a table along both dimensions
  scan      running sums and maxima of a table along both dimensions, and over all of it
  median    medians of a table along both dimensions, and of all of it
  video     NT2's image demos: sigma-delta motion detection frame by frame, then rgb2yuv
  batch     many uneven tables, each with its own expression, in one run
"""
import ctypes
import math

import torch

from nt2_gb300 import expr as E
from nt2_gb300 import lib

DEVICE = "cuda"
R, SIGMA = 0.02, 0.30
POLICY = {"fast": lib.PREC_FAST, "nt2": lib.PREC_NT2}


def f32(v):
    """The value a float argument has once it crosses the C ABI."""
    return float(torch.tensor(v, dtype=torch.float32))


# ------------------------------------------------------------------- the cases
def listed():
    return [
        # one quote request's strip of options: what a call costs when there is almost nothing to compute
        {"name": "price_4k", "kind": "price", "n": 4099, "policy": "fast", "sigma": "scalar"},
        # the framework's headline: NT2's Black-Scholes over 2^20 options
        {"name": "price_1m", "kind": "price", "n": 1 << 20, "policy": "fast", "sigma": "scalar"},
        # a volatility surface priced bit-identically to NT2 (a user validating against the CPU library)
        {"name": "price_nt2_3m", "kind": "price", "n": 3000017, "policy": "nt2", "sigma": "table"},
        # a whole book's risk run, larger than L2
        {"name": "greeks_32m", "kind": "greeks", "n": 1 << 25},
        # an elementwise formula of transcendental functors, three results from two tables
        {"name": "functors_16m", "kind": "functors", "n": 1 << 24, "which": "all", "policy": "fast"},
        # calibration: gradients of the pricing program written by the user, the rate's summed
        {"name": "gradient_16m", "kind": "gradient", "n": 16777213, "form": "textbook"},
        # norms and projections of long vectors
        {"name": "reduce_100m", "kind": "reduce", "n": 100000000},
        # summary statistics of a matrix of observations
        {"name": "stats_table", "kind": "stats", "rows": 6000, "cols": 8192},
        # cumulative returns and drawdown levels of many series, of ragged lengths
        {"name": "scan_table", "kind": "scan", "rows": 4099, "cols": 8190},
        # robust location of the same kind of matrix
        {"name": "median_table", "kind": "median", "rows": 4000, "cols": 3001},
        # a second of full-HD video through both image demos
        {"name": "video_1080p", "kind": "video", "height": 1080, "width": 1920, "frames": 16},
        # a nightly batch: tables from a thousand to a million elements, four expressions
        {"name": "batch_1024", "kind": "batch", "tables": 1024, "most": 1 << 20, "policy": "fast"},
    ]


def _log_int(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def _side(rng, lo, hi):
    """A table's extent: as often a round number as any other."""
    n = _log_int(rng, lo, hi)
    return max(8, n // 8 * 8) if rng.random() < 0.5 else n


def draw(rng):
    kind = rng.choice(["price", "price", "greeks", "functors", "gradient", "reduce", "stats", "scan", "median", "video",
                       "batch"])
    if kind == "price":
        return {"kind": kind, "n": _log_int(rng, 1000, 1 << 24), "policy": rng.choice(["fast", "fast", "nt2"]),
                "sigma": rng.choice(["scalar", "table"])}
    if kind == "greeks":
        return {"kind": kind, "n": _log_int(rng, 1000, 1 << 25)}
    if kind == "functors":
        return {"kind": kind, "n": _log_int(rng, 10000, 1 << 24), "which": rng.choice(["all", "trig", "pow", "special"]),
                "policy": rng.choice(["fast", "fast", "nt2"])}
    if kind == "gradient":
        return {"kind": kind, "n": _log_int(rng, 10000, 1 << 24), "form": rng.choice(["textbook", "demo"])}
    if kind == "reduce":
        return {"kind": kind, "n": _log_int(rng, 10000, 100000000)}
    if kind in ("stats", "scan", "median"):
        rows = _side(rng, 40, 40000)
        most = {"stats": 48000000, "scan": 32000000, "median": 12000000}[kind] // rows
        return {"kind": kind, "rows": rows, "cols": _side(rng, 40, max(48, min(40000, most)))}
    if kind == "video":
        w = rng.choice([320, 641, 1280, 1920, 2048])
        return {"kind": kind, "height": w * 9 // 16, "width": w, "frames": rng.randint(1, 16)}
    return {"kind": kind, "tables": _log_int(rng, 16, 1024), "most": _log_int(rng, 1 << 13, 1 << 20),
            "policy": rng.choice(["fast", "fast", "nt2"])}


# ------------------------------------------------------------------ the inputs
def _uniform(g, n, lo, hi):
    return torch.rand(n, device=DEVICE, generator=g) * (hi - lo) + lo


def _book(g, n):
    """Spot, strike, expiry as NT2's demo draws them."""
    return _uniform(g, n, 5, 30), _uniform(g, n, 1, 100), _uniform(g, n, 0.25, 10)


def _price(case, g):
    n = case["n"]
    s = {"S_K_T": _book(g, n), "call": torch.empty(n, device=DEVICE), "put": torch.empty(n, device=DEVICE)}
    s["sigma"] = _uniform(g, n, 0.05, 0.8) if case["sigma"] == "table" else None
    return s


def _greeks(case, g):
    n = case["n"]
    return {"S_K_T": _book(g, n), "sigma": _uniform(g, n, 0.05, 0.8), "gc": _uniform(g, n, -1, 1),
            "gp": _uniform(g, n, -1, 1), "outs": [torch.empty(n, device=DEVICE) for _ in range(7)]}


def _functors(case, g):
    n = case["n"]
    names = ["trig", "pow", "special"] if case["which"] == "all" else [case["which"]]
    return {"x": _uniform(g, n, 0.25, 4.25), "y": _uniform(g, n, -2, 2), "names": names,
            "outs": [torch.empty(n, device=DEVICE) for _ in names]}


def _gradient(case, g):
    n = case["n"]
    S, K, T = _book(g, n)
    ins = [S, K, T, _uniform(g, n, 0.05, 0.8)]
    if case["form"] == "demo":  # the rate a table too, one result
        ins.append(_uniform(g, n, 0.01, 0.05))
        return {"ins": ins, "outs": [torch.empty(n, device=DEVICE)], "cts": [_uniform(g, n, -1, 1)]}
    return {"ins": ins, "outs": [torch.empty(n, device=DEVICE), torch.empty(n, device=DEVICE)],
            "cts": [_uniform(g, n, -1, 1), _uniform(g, n, -1, 1)]}


def _reduce(case, g):
    n = case["n"]
    return {"x": torch.randn(n, device=DEVICE, generator=g) * 0.5 + 0.05, "y": _uniform(g, n, 0, 2),
            "sum": lib.Reducer(DEVICE), "dot": lib.Reducer(DEVICE)}


def _table(case, g):
    """A rows x cols table, column-major (NT2's layout): x[i + rows * j]."""
    return {"x": torch.randn(case["rows"] * case["cols"], device=DEVICE, generator=g) + 0.1}


def _video(case, g):
    h, w, f = case["height"], case["width"], case["frames"]
    scene = torch.randint(20, 230, (h // 8 + 1, w // 8 + 1), device=DEVICE, generator=g)
    scene = scene.repeat_interleave(8, 0).repeat_interleave(8, 1)[:h, :w].to(torch.float32)
    frames = (scene + torch.randn(f, h, w, device=DEVICE, generator=g) * 3).clamp_(0, 255)
    for k in range(f):  # something bright that moves
        at = (k * w // max(f, 1)) // 2
        frames[k, h // 3: h // 2, at: at + w // 10] = 250
    frames = frames.to(torch.uint8).reshape(f, h * w).contiguous()
    rgb = [_uniform(g, h * w, 0, 1) for _ in range(3)]
    return {"frames": frames, "bkg": scene.to(torch.uint8).reshape(-1).contiguous(),
            "var": torch.ones(h * w, dtype=torch.uint8, device=DEVICE),
            "labels": torch.empty_like(frames), "rgb": rgb, "yuv": [torch.empty_like(rgb[0]) for _ in range(3)]}


BATCH_INPUTS = 3  # every table has three input tables' room; expressions use what they need


class _Batch:
    """A batch handle that goes when its state goes."""

    def __init__(self, items, precision):
        self.h = ctypes.c_void_p()
        tune = lib.BatchTune(0, 0, 0, precision, 0)
        lib.check(lib.load().nt2g_batch_create(items, len(items), ctypes.byref(tune), ctypes.byref(self.h)))

    def __del__(self):
        try:
            lib.load().nt2g_batch_destroy(self.h)
        except Exception:
            pass


def _batch_sizes(case):
    """Table sizes, log-uniform, and each table's expression (0..3): the same for every seed."""
    import random
    rng = random.Random(case["tables"] * 1000003 + case["most"])
    return [_log_int(rng, 1000, case["most"]) for _ in range(case["tables"])], \
           [rng.randrange(4) for _ in range(case["tables"])]


def _batch(case, g):
    sizes, kinds = _batch_sizes(case)
    at, total = [], 0
    for n in sizes:  # tables start at multiples of 64 elements, as an allocator places them
        at.append(total)
        total += (n + 63) // 64 * 64
    book = _book(g, total)
    plain = [torch.randn(total, device=DEVICE, generator=g) for _ in range(BATCH_INPUTS)]
    out = [torch.zeros(total, device=DEVICE), torch.zeros(total, device=DEVICE)]
    items, keep = (lib.BatchItem * len(sizes))(), []
    for i, (n, k, a) in enumerate(zip(sizes, kinds, at)):
        src = book if k in (0, 3) else plain
        if k == 3:  # the user's own program: NT2's demo form, the volatility a scalar of each table
            T = [E.Table(t[a:a + n]) for t in src]
            it, prog, args = E.batch_item([out[0][a:a + n]], [_demo_call(*T, E.Scalar(0.2 + 0.01 * (i % 40)),
                                                                         E.Scalar(R))])
            keep.append((prog, args))
            items[i] = it
            continue
        items[i].expr, items[i].n = k, n
        used = [0, 1, 2] if k != lib.BATCH_SAXPY else [0]
        for j in used:
            items[i].inp[j] = src[j].data_ptr() + 4 * a
        for j in range(2 if k == lib.BATCH_BLACKSCHOLES else 1):
            items[i].out[j] = out[j].data_ptr() + 4 * a
        items[i].s[0], items[i].s[1] = (SIGMA, R) if k == lib.BATCH_BLACKSCHOLES else (0.5 + 0.01 * (i % 100), 0.0)
    return {"book": book, "plain": plain, "out": out, "keep": keep, "batch": _Batch(items, POLICY[case["policy"]])}


def prepare(case, seed):
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    make = {"price": _price, "greeks": _greeks, "functors": _functors, "gradient": _gradient, "reduce": _reduce,
            "stats": _table, "scan": _table, "median": _table, "video": _video, "batch": _batch}[case["kind"]]
    return {"case": case, **make(case, g)}


# ------------------------------------------------------------------- the passes
def _textbook(S, K, T, sig, r):
    """Call and put as NT2's user writes them."""
    sq = E.sqrt(T)
    d1 = (E.log(S / K) + E.fma(E.sqr(sig), 0.5, r) * T) / (sig * sq)
    d2 = E.fnms(sig, sq, d1)
    e = K * E.exp(-r * T)
    return [E.fnms(e, E.normcdf(d2), S * E.normcdf(d1)), E.fnms(S, E.normcdf(-d1), e * E.normcdf(-d2))]


def _demo_call(S, X, T, v, r):
    """NT2's demo Black-Scholes: the call alone, through fastnormcdf."""
    da = E.sqrt(T)
    d1 = E.log(S / X) + (E.fma(E.sqr(v), 0.5, r) * T) / (v * da)
    d2 = E.fnms(v, da, d1)
    return E.fnms(X * E.exp(-r * T), E.fastnormcdf(d2), S * E.fastnormcdf(d1))


FUNCTORS = {"trig": lambda x, y: E.sin(x) * E.cos(y), "pow": E.pow, "special": lambda x, y: E.erf(y) + E.gammaln(x)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "price":
        lib.blackscholes(*state["S_K_T"], state["call"], state["put"], R, sigma=state["sigma"], sigma_s=SIGMA,
                         precision=POLICY[case["policy"]])
        return {"call": state["call"], "put": state["put"]}
    if kind == "greeks":
        lib.blackscholes_vjp(*state["S_K_T"], state["sigma"], R, state["gc"], state["gp"], state["outs"])
        return list(state["outs"])
    if kind == "functors":
        x, y = E.Table(state["x"]), E.Table(state["y"])
        E.assign(state["outs"], [FUNCTORS[k](x, y) for k in state["names"]], precision=POLICY[case["policy"]])
        return dict(zip(state["names"], state["outs"]))
    if kind == "gradient":
        tables = [E.Table(t) for t in state["ins"]]
        if case["form"] == "demo":
            return E.vjp(state["outs"], [_demo_call(*tables)], state["cts"], state["ins"])
        r = E.Scalar(R)
        return E.vjp(state["outs"], _textbook(*tables, r), state["cts"], state["ins"] + [r])
    if kind == "reduce":
        x, y = state["x"], state["y"]
        total, projection = state["sum"](x)[0], state["dot"](x, y)[0]
        _, weighted = E.fold(E.exp(E.Table(x)) * E.Table(y), "sum", out64=True)
        largest, where = lib.fold(x, 1, x.numel(), 1, "max", index=True)
        return {"sum": total, "dot": projection, "fold": weighted, "max": largest, "where": where}
    if kind in ("stats", "scan", "median"):
        x, m, n = state["x"], case["rows"], case["cols"]
        down, across, whole = (1, m, n), (m, n, 1), (1, m * n, 1)
        if kind == "stats":
            out = {}
            for name, view in (("cols", down), ("rows", across)):
                out[name] = [lib.fold(x, *view, "mean"), lib.fold(x, *view, "stdev"),
                             *lib.fold(x, *view, "max", index=True)]
            return out
        if kind == "scan":
            return {"sum_cols": lib.scan(x, *down, "sum"), "max_rows": lib.scan(x, *across, "max"),
                    "sum_all": lib.scan(x, *whole, "sum")}
        return {"cols": lib.median(x, *down), "rows": lib.median(x, *across), "all": lib.median(x, *whole)}
    if kind == "video":
        for frame, label in zip(state["frames"], state["labels"]):
            lib.sigmadelta(frame, state["bkg"], state["var"], label)
        lib.rgb2yuv(*state["rgb"], *state["yuv"])
        return {"labels": state["labels"], "bkg": state["bkg"], "var": state["var"], "yuv": list(state["yuv"])}
    lib.check(lib.load().nt2g_batch_run(state["batch"].h, lib._stream()))
    return list(state["out"])


# ------------------------------------------------------- what a pass has to move
BS_FLOPS, FUNCTOR_FLOPS = 120, {"trig": 60, "pow": 80, "special": 140}


def work(case):
    kind = case["kind"]
    if kind in ("price", "greeks", "functors", "gradient", "reduce"):
        n = case["n"]
        if kind == "price":
            return {"bytes": (24 if case["sigma"] == "table" else 20) * n, "flops": BS_FLOPS * n}
        if kind == "greeks":
            return {"bytes": 52 * n, "flops": 2 * BS_FLOPS * n}
        if kind == "functors":
            names = list(FUNCTORS) if case["which"] == "all" else [case["which"]]
            return {"bytes": (8 + 4 * len(names)) * n, "flops": sum(FUNCTOR_FLOPS[k] for k in names) * n}
        if kind == "gradient":
            return {"bytes": (44 if case["form"] == "demo" else 40) * n, "flops": 3 * BS_FLOPS * n}
        return {"bytes": 24 * n, "flops": 60 * n}  # x; x and y; x and y; x
    if kind in ("stats", "scan", "median"):
        m, n = case["rows"], case["cols"]
        if kind == "stats":  # six calls, each reading the table
            return {"bytes": 24 * m * n + 20 * (m + n), "flops": 6 * 8 * m * n}
        if kind == "scan":
            return {"bytes": 24 * m * n, "flops": 3 * 8 * m * n}
        return {"bytes": 12 * m * n + 4 * (m + n + 1), "flops": 3 * 4 * m * n}
    if kind == "video":
        p = case["height"] * case["width"]
        return {"bytes": 6 * p * case["frames"] + 24 * p, "flops": 20 * p * case["frames"] + 10 * p}
    sizes, kinds = _batch_sizes(case)
    per = {0: 20, 1: 12, 2: 16, 3: 16}
    return {"bytes": sum(per[k] * n for n, k in zip(sizes, kinds)),
            "flops": sum({0: BS_FLOPS, 1: 2, 2: 60, 3: 80}[k] * n for n, k in zip(sizes, kinds))}


# ------------------------------------------------------------- the same in 64 bits
def _ncdf(x):
    return 0.5 * torch.erfc(-x * math.sqrt(0.5))


def _fast_ncdf(x):
    """NT2's fastnormcdf (Abramowitz and Stegun 26.2.17)."""
    c = [0.31938153, -0.356563782, 1.781477937, -1.821255978, 1.330274429]
    l = x.abs()
    k = 1 / (1 + 0.2316419 * l)
    w = k * (c[0] + k * (c[1] + k * (c[2] + k * (c[3] + k * c[4])))) * torch.exp(-l * l / 2) / math.sqrt(2 * math.pi)
    return torch.where(x < 0, w, 1 - w)


def _bs64(S, K, T, sig, r):
    sq = torch.sqrt(T)
    d1 = (torch.log(S / K) + (r + sig * sig / 2) * T) / (sig * sq)
    d2 = d1 - sig * sq
    e = K * torch.exp(-r * T)
    return S * _ncdf(d1) - e * _ncdf(d2), e * _ncdf(-d2) - S * _ncdf(-d1)


def _demo64(S, X, T, v, r):
    da = torch.sqrt(T)
    d1 = torch.log(S / X) + ((r + v * v / 2) * T) / (v * da)
    return S * _fast_ncdf(d1) - X * torch.exp(-r * T) * _fast_ncdf(d1 - v * da)


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    d = lambda ts: [t.double() for t in ts]  # noqa: E731
    r, sigma = f32(R), f32(SIGMA)
    if kind == "price":
        call, put = _bs64(*d(s["S_K_T"]), s["sigma"].double() if s["sigma"] is not None else sigma, r)
        return {"call": call, "put": put}
    if kind == "greeks":
        parts = []
        n = case["n"]
        for a in range(0, n, 1 << 22):  # in slices: the tape of all of it at once is large
            cut = lambda t: t[a:a + (1 << 22)]  # noqa: E731
            ins = [t.requires_grad_() for t in d([cut(t) for t in (*s["S_K_T"], s["sigma"])])]
            rate = torch.full_like(ins[0], r).requires_grad_()
            call, put = _bs64(*ins, rate)
            grads = torch.autograd.grad((cut(s["gc"]).double() * call + cut(s["gp"]).double() * put).sum(), ins + [rate])
            parts.append([call.detach(), put.detach(), *grads])
        return [torch.cat(p) for p in zip(*parts)]
    if kind == "functors":
        x, y = d([s["x"], s["y"]])
        f = {"trig": lambda: torch.sin(x) * torch.cos(y), "pow": lambda: torch.pow(x, y),
             "special": lambda: torch.erf(y) + torch.lgamma(x)}
        return {k: f[k]() for k in s["names"]}
    if kind == "gradient":
        ins = [t.requires_grad_() for t in d(s["ins"])]
        cts = d(s["cts"])
        if case["form"] == "demo":
            return list(torch.autograd.grad((_demo64(*ins) * cts[0]).sum(), ins))
        rate = torch.tensor(r, dtype=torch.float64, device=DEVICE, requires_grad=True)
        call, put = _bs64(*ins, rate)
        return list(torch.autograd.grad((call * cts[0] + put * cts[1]).sum(), ins + [rate]))
    if kind == "reduce":
        x, y = d([s["x"], s["y"]])
        return {"sum": x.sum().reshape(1), "dot": (x * y).sum().reshape(1), "fold": (x.exp() * y).sum().reshape(1),
                "max": x.max().reshape(1), "where": None}
    if kind in ("stats", "scan", "median"):
        x = s["x"].double().reshape(case["cols"], case["rows"])  # a column of NT2's is a row of torch's
        if kind == "stats":
            return {name: [x.mean(dim), x.std(dim), x.amax(dim), None] for name, dim in (("cols", 1), ("rows", 0))}
        if kind == "scan":
            return {"sum_cols": x.cumsum(1).reshape(-1), "max_rows": x.cummax(0).values.reshape(-1),
                    "sum_all": x.reshape(-1).cumsum(0)}

        def middle(v):
            v, n = v.sort(-1).values, v.shape[-1]
            return (v[..., (n - 1) // 2] + v[..., n // 2]) / 2
        return {"cols": middle(x), "rows": middle(x.t().contiguous()), "all": middle(x.reshape(1, -1))}
    if kind == "video":
        r_, g_, b_ = d(s["rgb"])
        y = f32(0.299) * r_ + f32(0.587) * g_ + f32(0.114) * b_
        return {"labels": None, "bkg": None, "var": None, "yuv": [y, f32(0.492) * (b_ - y), f32(0.877) * (r_ - y)]}
    sizes, kinds = _batch_sizes(case)
    out, at = [t.double() for t in s["out"]], 0
    for i, (n, k) in enumerate(zip(sizes, kinds)):
        cut = lambda ts: [t[at:at + n].double() for t in ts]  # noqa: E731
        if k == lib.BATCH_BLACKSCHOLES:
            out[0][at:at + n], out[1][at:at + n] = _bs64(*cut(s["book"]), sigma, r)
        elif k == lib.BATCH_SAXPY:
            out[0][at:at + n] += f32(0.5 + 0.01 * (i % 100)) * s["plain"][0][at:at + n].double()
        elif k == lib.BATCH_EXPR3:
            x, y, z = cut(s["plain"])
            out[0][at:at + n] = torch.exp(-x * x) * y.abs().sqrt() + torch.log1p(z.abs())
        else:
            out[0][at:at + n] = _demo64(*cut(s["book"]), f32(0.2 + 0.01 * (i % 40)), r)
        at += (n + 63) // 64 * 64
    return out
