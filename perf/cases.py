"""The calls whose speed is measured: what a program that uses the skeleton library has it do.

A case is one call of a skeleton (or one launch of a batch plan) through the public entry points, on arrays that are
already on the device, as they are between the operations of an array program.  Sizes and distributions are those of
the library's benchmark and tests: uniform integers, N(0,1) floats, lognormal segments, Zipf(1.1) and uniform bins.
Scalars such as seeds and stencil weights are passed with every call, as a program does.
"""
import importlib
import math

import numpy as np
import torch

acc = importlib.import_module("accelerate-llvm_gb300")

DTYPES = {"i32": torch.int32, "i64": torch.int64, "f32": torch.float32, "f64": torch.float64}
SIZE = {"i32": 4, "i64": 8, "f32": 4, "f64": 8}
FLAVOURS = ("scanl1", "scanl", "scanl_", "scanr1", "scanr", "scanr_")
SEEDED = ("scanl", "scanl_", "scanr", "scanr_")

# Stencil patterns in use: the box filter, the 5-point Laplacian of the serving mix, a 5 x 5 smoothing kernel; in
# three dimensions the box and the 7-point heat step.
BOX = [[1.0 / 9] * 3] * 3
LAPLACE = [[0.0, 0.25, 0.0], [0.25, -1.0, 0.25], [0.0, 0.25, 0.0]]
SMOOTH = [[a * b / 256.0 for b in (1, 4, 6, 4, 1)] for a in (1, 4, 6, 4, 1)]
BOX3 = [[[1.0 / 27] * 3] * 3] * 3
STAR3 = [[[0.0, 0.0, 0.0], [0.0, 0.1, 0.0], [0.0, 0.0, 0.0]],
         [[0.0, 0.1, 0.0], [0.1, 0.4, 0.1], [0.0, 0.1, 0.0]],
         [[0.0, 0.0, 0.0], [0.0, 0.1, 0.0], [0.0, 0.0, 0.0]]]
PATTERNS = {"box": BOX, "laplace": LAPLACE, "smooth": SMOOTH, "box3": BOX3, "star3": STAR3}


def listed():
    return [
        # Row sums of a matrix: the everyday reduction, a few microseconds of device time.
        {"name": "fold_rows_i32", "kind": "fold", "type": "i32", "op": "+", "prec": "default", "zip": False,
         "outer": 4096, "inner": 1024},
        # The sum of an array far larger than L2, with the default (compensated) accumulation.
        {"name": "fold_f32_2e28", "kind": "fold", "type": "f32", "op": "+", "prec": "default", "zip": False,
         "outer": 1, "inner": 1 << 28},
        # Offsets from a short array of counts: the smallest call, bound by its latency.
        {"name": "scan_small_i32", "kind": "scan", "type": "i32", "op": "+", "prec": "default", "zip": False,
         "flavour": "scanl", "outer": 1, "inner": 10_007},
        # Running sums along the rows of a matrix of odd extents.
        {"name": "scan_rows_f32", "kind": "scan", "type": "f32", "op": "+", "prec": "default", "zip": False,
         "flavour": "scanl1", "outer": 1001, "inner": 4099},
        # The prefix sum of an array far larger than L2.
        {"name": "scan_i64_2e28", "kind": "scan", "type": "i64", "op": "+", "prec": "default", "zip": False,
         "flavour": "scanl1", "outer": 1, "inner": 1 << 28},
        # Segment maxima of a short ragged array, from segment lengths.
        {"name": "foldseg_small_i32", "kind": "foldseg", "type": "i32", "op": "max", "prec": "default", "zip": False,
         "n": 100_003, "nseg": 1_563, "lengths": True},
        # Segment sums of a large ragged array (sparse rows, groups), compensated.
        {"name": "foldseg_f32_2e26", "kind": "foldseg", "type": "f32", "op": "+", "prec": "default", "zip": False,
         "n": 1 << 26, "nseg": 1 << 20, "lengths": False},
        # A histogram of skewed indices, the counts of many events over a vocabulary.
        {"name": "histogram_2e28", "kind": "permute", "type": "i32", "op": "+", "index": "i32", "source": False,
         "n": 1 << 28, "m": 1 << 16, "zipf": True},
        # Values summed by key (scatter-add), every key about equally frequent.
        {"name": "keyed_sum_f32", "kind": "permute", "type": "f32", "op": "+", "index": "i32", "source": True,
         "n": 20_000_003, "m": 50_021, "zipf": False},
        # A 3 x 3 box filter over a large image.
        {"name": "stencil_f32_8192", "kind": "stencil", "type": "f32", "pattern": "box", "boundary": "clamp",
         "h": 8192, "w": 8192},
        # A 3 x 3 x 3 filter over a volume.
        {"name": "stencil3d_f32_512", "kind": "stencil3d", "type": "f32", "pattern": "box3", "boundary": "clamp",
         "d": 512, "h": 512, "w": 512},
        # Many independent folds and scans of uneven sizes in one launch of a captured plan.
        {"name": "batch_1000", "kind": "batch", "count": 1000, "low": 8, "high": 22},
    ]


def _log(rng, low, high):
    """A whole number, spread evenly over the logarithm of its range."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _rows(rng, n):
    """n elements as (outer, inner): one row, or rows of an even or odd length."""
    if rng.random() < 0.5:
        return 1, n
    inner = _log(rng, 16, max(17, n // 2))
    return max(1, n // inner), inner


def draw(rng):
    kind = rng.choice(("fold", "scan", "foldseg", "permute", "stencil", "stencil3d", "fold", "scan", "foldseg",
                       "permute", "batch"))
    if kind in ("fold", "scan"):
        t = rng.choice(("i32", "i64", "f32", "f64"))
        zipped = rng.random() < 0.25
        n = _log(rng, 1 << 12, (1 << (28 if kind == "fold" else 27)) * 4 // SIZE[t] // (2 if zipped else 1))
        outer, inner = _rows(rng, n)
        case = {"kind": kind, "type": t, "op": rng.choice(("+", "+", "max", "min")),
                "prec": rng.choice(("default", "default", "plain")), "zip": zipped, "outer": outer, "inner": inner}
        if kind == "scan":
            case["flavour"] = rng.choice(FLAVOURS)
        return case
    if kind == "foldseg":
        t = rng.choice(("i32", "f32", "f32", "f64"))
        n = _log(rng, 1 << 12, (1 << 26) * 4 // SIZE[t])
        return {"kind": kind, "type": t, "op": rng.choice(("+", "+", "max")),
                "prec": rng.choice(("default", "default", "plain", "fp64")), "zip": rng.random() < 0.2, "n": n,
                "nseg": max(1, n // _log(rng, 16, 512)), "lengths": rng.random() < 0.3}
    if kind == "permute":
        t = rng.choice(("i32", "i32", "f32", "i64"))
        source = t != "i32" or rng.random() < 0.4
        n = _log(rng, 1 << 12, 1 << (26 if source else 28))
        return {"kind": kind, "type": t, "op": rng.choice(("+", "+", "max")) if t != "f32" else "+",
                "index": rng.choice(("i32", "i32", "i64")), "source": source, "n": n,
                "m": _log(rng, 1 << 8, 1 << 20), "zipf": rng.random() < 0.3}
    if kind == "stencil":
        return {"kind": kind, "type": rng.choice(("f32", "f32", "f64", "i32")),
                "pattern": rng.choice(("box", "laplace", "smooth")),
                "boundary": rng.choice(("clamp", "mirror", "wrap", "constant")),
                "h": _log(rng, 64, 8192), "w": _log(rng, 64, 8192)}
    if kind == "stencil3d":
        return {"kind": kind, "type": rng.choice(("f32", "f32", "f64")), "pattern": rng.choice(("box3", "star3")),
                "boundary": rng.choice(("clamp", "mirror", "wrap", "constant")),
                "d": _log(rng, 32, 512), "h": _log(rng, 32, 512), "w": _log(rng, 32, 512)}
    return {"kind": kind, "count": _log(rng, 32, 1000), "low": rng.choice((8, 9, 10)), "high": rng.choice((18, 20, 22))}


# ----------------------------------------------------------------- inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _values(t, n, g, op="+"):
    if t[0] == "i" and op != "+":  # minima and maxima of keys from the whole range
        high = (1 << (31 if t == "i32" else 62)) - 1
        return torch.randint(-high, high, (n,), dtype=DTYPES[t], device="cuda", generator=g)
    if t == "i32":
        return torch.randint(-1024, 1025, (n,), dtype=torch.int32, device="cuda", generator=g)
    if t == "i64":
        return torch.randint(-(1 << 20), (1 << 20) + 1, (n,), dtype=torch.int64, device="cuda", generator=g)
    return torch.randn(n, dtype=DTYPES[t], device="cuda", generator=g)


def _lengths(n, nseg, g):
    """nseg lognormal lengths (sigma 1.5, 2 % empty, none above 2^16 before scaling) that sum to n."""
    lens = torch.empty(nseg, dtype=torch.float64, device="cuda").log_normal_(math.log(48.0), 1.5, generator=g)
    lens.clamp_(max=float(1 << 16))
    lens[torch.rand(nseg, device="cuda", generator=g) < 0.02] = 0.0
    ends = torch.cumsum(lens, 0)
    ends = torch.round(ends * (n / ends[-1].clamp(min=1.0))).to(torch.int64)
    ends[-1] = n
    return torch.diff(ends, prepend=ends.new_zeros(1))


def _indices(case, g):
    n, m, dt = case["n"], case["m"], DTYPES[case["index"]]
    if not case["zipf"]:
        return torch.randint(0, m, (n,), dtype=dt, device="cuda", generator=g)
    p = torch.arange(1, m + 1, dtype=torch.float64, device="cuda").pow(-1.1)
    cdf = torch.cumsum(p / p.sum(), 0)
    where = torch.randperm(m, device="cuda", generator=g).to(dt)
    idx = torch.empty(n, dtype=dt, device="cuda")
    for s in range(0, n, 1 << 26):
        u = torch.rand(min(1 << 26, n - s), dtype=torch.float64, device="cuda", generator=g)
        idx[s:s + u.numel()] = where[torch.searchsorted(cdf, u).clamp_(max=m - 1)]
    return idx


def _seed(case):
    """The seed of a fold or a seeded scan: the neutral value of its operation over these inputs."""
    if case["op"] == "+":
        return 0
    low = {"i32": -(1 << 31), "i64": -(1 << 63)}.get(case["type"], -1e30)
    return low if case["op"] == "max" else -low - (case["type"][0] == "i")


def _requests(case):
    """(kind, type, first element, elements) of each request of a batch; the plan is the program's, the data the seed's."""
    rng = np.random.default_rng(case["count"])
    sizes = np.exp(rng.uniform(math.log(2 ** case["low"]), math.log(2 ** case["high"]), size=case["count"]))
    at, reqs = {"i32": 0, "f32": 0}, []
    for i, n in enumerate(sizes.astype(np.int64).tolist()):
        kind, t = ("fold", "scan")[i % 2], ("i32", "f32")[i // 2 % 2]
        reqs.append((kind, t, at[t], n))
        at[t] += n
    return reqs, at


def prepare(case, seed):
    kind, g, st = case["kind"], _generator(seed), {"case": case}
    if kind in ("fold", "scan"):
        shape = (case["outer"], case["inner"]) if case["outer"] > 1 else (case["inner"],)
        n = case["outer"] * case["inner"]
        st["xs"] = _values(case["type"], n, g, case["op"]).view(shape)
        if case["zip"]:
            st["ys"] = _values(case["type"], n, g, case["op"]).view(shape)
    elif kind == "foldseg":
        st["xs"] = _values(case["type"], case["n"], g, case["op"])
        if case["zip"]:
            st["ys"] = _values(case["type"], case["n"], g, case["op"])
        lens = _lengths(case["n"], case["nseg"], g)
        if not case["lengths"] or case["zip"]:
            lens = torch.nn.functional.pad(torch.cumsum(lens, 0), (1, 0))
        st["seg"] = lens.to(torch.int32)
    elif kind == "permute":
        t = case["type"]
        st["idx"] = _indices(case, g)
        st["xs"] = _values(t, case["n"], g, case["op"]) if case["source"] else 1
        st["defaults"] = torch.full((case["m"],), _seed(case), dtype=DTYPES[t], device="cuda")
    elif kind in ("stencil", "stencil3d"):
        t = case["type"]
        shape = (case["d"], case["h"], case["w"]) if kind == "stencil3d" else (case["h"], case["w"])
        if t == "i32":
            st["xs"] = torch.randint(-1000, 1000, shape, dtype=torch.int32, device="cuda", generator=g)
        else:
            st["xs"] = torch.rand(shape, dtype=DTYPES[t], device="cuda", generator=g)
        st["weights"] = _weights(case)
        st["cval"] = 0.5 if t[0] == "f" else 7
    else:
        reqs, total = _requests(case)
        pool = {t: _values(t, n, g) for t, n in total.items()}
        scans = {t: torch.zeros(sum(n for k, u, _, n in reqs if k == "scan" and u == t), dtype=DTYPES[t],
                                device="cuda") for t in total}
        folds = {t: torch.zeros(sum(k == "fold" and u == t for k, u, _, _ in reqs), dtype=DTYPES[t], device="cuda")
                 for t in total}
        at, plan = {("scan", t): 0 for t in total} | {("fold", t): 0 for t in total}, []
        for k, t, first, n in reqs:
            o, size = at[k, t], n if k == "scan" else 1
            plan.append((k, pool[t][first:first + n], (scans if k == "scan" else folds)[t][o:o + size],
                         0 if k == "fold" else None))
            at[k, t] = o + size
        st["batch"] = acc.Batch("+", plan)
        st["batch"].capture()
        st["out"] = [folds["i32"], folds["f32"], scans["i32"], scans["f32"]]
    return st


def _weights(case):
    w = PATTERNS[case["pattern"]]
    if case["type"] != "i32":
        return w
    # Integer filters are the small whole numbers that the real ones are scaled from.
    scale = {"box": 9, "laplace": 4, "smooth": 256}[case["pattern"]]
    return [[int(round(v * scale)) for v in row] for row in w]


# ----------------------------------------------------------------- the calls
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "fold":
        if case["zip"]:
            return acc.fold_zipwith(case["op"], "*", _seed(case), st["xs"], st["ys"], prec=case["prec"])
        return acc.fold(case["op"], _seed(case), st["xs"], prec=case["prec"])
    if kind == "scan":
        z = _seed(case) if case["flavour"] in SEEDED else None
        if case["zip"]:
            return acc.scan_zipwith(case["flavour"], case["op"], "*", z, st["xs"], st["ys"], prec=case["prec"])
        if z is None:
            return getattr(acc, case["flavour"])(case["op"], st["xs"], prec=case["prec"])
        return getattr(acc, case["flavour"])(case["op"], z, st["xs"], prec=case["prec"])
    if kind == "foldseg":
        if case["zip"]:
            return acc.fold_seg_zipwith(case["op"], "*", _seed(case), st["xs"], st["ys"], st["seg"], prec=case["prec"])
        return acc.fold_seg(case["op"], _seed(case), st["xs"], st["seg"], prec=case["prec"],
                            offsets=not case["lengths"])
    if kind == "permute":
        return acc.permute(case["op"], st["defaults"], st["idx"], st["xs"])
    if kind == "stencil":
        return acc.stencil(st["weights"], st["xs"], case["boundary"], cval=st["cval"])
    if kind == "stencil3d":
        return acc.stencil3d(st["weights"], st["xs"], case["boundary"], cval=st["cval"])
    st["batch"].launch()
    return st["out"]


# ----------------------------------------------------------------- what a call cannot do without
def work(case):
    kind = case["kind"]
    if kind in ("fold", "scan"):
        n, outer, e = case["outer"] * case["inner"], case["outer"], SIZE[case["type"]]
        reads = n * (2 if case["zip"] else 1)
        writes = outer
        if kind == "scan":
            writes = n + (outer if case["flavour"] in SEEDED else 0)
        return {"bytes": e * (reads + writes), "flops": n * (2 if case["zip"] else 1)}
    if kind == "foldseg":
        e, n = SIZE[case["type"]], case["n"]
        reads = n * (2 if case["zip"] else 1)
        return {"bytes": e * (reads + case["nseg"]) + 4 * (case["nseg"] + 1), "flops": reads}
    if kind == "permute":
        e, n = SIZE[case["type"]], case["n"]
        return {"bytes": n * (SIZE[case["index"]] + (e if case["source"] else 0)) + 2 * e * case["m"], "flops": n}
    if kind in ("stencil", "stencil3d"):
        n = case["h"] * case["w"] * case.get("d", 1)
        taps = int(np.count_nonzero(np.array(PATTERNS[case["pattern"]])))
        return {"bytes": 2 * SIZE[case["type"]] * n, "flops": 2 * taps * n}
    reqs, _ = _requests(case)
    return {"bytes": sum(4 * n + 4 if k == "fold" else 8 * n for k, _, _, n in reqs), "flops": sum(r[3] for r in reqs)}


# ----------------------------------------------------------------- the same in 64 bits, by plain torch
def _exact_scan(case, x):
    back = case["flavour"].startswith("scanr")
    if back:
        x = x.flip(-1)
    if case["flavour"] in SEEDED:
        x = torch.cat([torch.full(x.shape[:-1] + (1,), float(_seed(case)), dtype=x.dtype, device=x.device), x], -1)
    if case["op"] == "+":
        y = torch.cumsum(x, -1)
    else:
        y = (torch.cummax if case["op"] == "max" else torch.cummin)(x, -1).values
    totals = None
    if case["flavour"] in ("scanl_", "scanr_"):
        y, totals = y[..., :-1], y[..., -1].contiguous()
    if back:
        y = y.flip(-1)
    return y.contiguous() if totals is None else (y.contiguous(), totals)


def _ends(i, size, boundary):
    """Indices outside of the array brought back into it; -1 where the boundary's constant stands."""
    if boundary == "constant":
        return torch.where((i < 0) | (i >= size), torch.full_like(i, -1), i)
    if boundary == "clamp":
        return i.clamp(0, size - 1)
    if boundary == "wrap":
        return i % size
    return torch.where(i < 0, -i, torch.where(i >= size, 2 * (size - 1) - i, i))


def _exact_stencil(case, st):
    x, dt = st["xs"].double(), DTYPES[case["type"]]
    w = np.array(st["weights"], dtype=np.float64)
    w = torch.from_numpy(w).to(dt).double().numpy()
    y = torch.zeros_like(x)
    for at in np.ndindex(*w.shape):
        if w[at] == 0.0:
            continue
        part = x
        for dim, k in enumerate(at):
            shift = k - w.shape[dim] // 2
            if shift == 0:
                continue
            i = _ends(torch.arange(x.shape[dim], device="cuda") + shift, x.shape[dim], case["boundary"])
            outside = i < 0
            part = part.index_select(dim, i.clamp(min=0))
            if case["boundary"] == "constant":
                part.movedim(dim, 0)[outside] = st["cval"]
        y += float(w[at]) * part
    return y


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        st = prepare(case, seed)
        reqs, total = _requests(case)
        x = _values("i32", total["i32"], g := _generator(seed))
        x = _values("f32", total["f32"], g).double()
        folds, scans = [], []
        for k, t, first, n in reqs:
            if t == "f32":
                part = x[first:first + n]
                (folds if k == "fold" else scans).append(part.sum().view(1) if k == "fold" else torch.cumsum(part, 0))
        st["batch"].close()
        return [None, torch.cat(folds), None, torch.cat(scans)]
    if case["type"][0] == "i":
        return None
    st = prepare(case, seed)
    if kind in ("fold", "scan", "foldseg"):
        x = st["xs"]
        if case["zip"]:
            x = x * st["ys"]  # a zipped element is a value of the array's type
        x = x.double()
        if kind == "scan":
            return _exact_scan(case, x)
        if kind == "fold":
            return x.sum(-1) if case["op"] == "+" else (x.amax(-1) if case["op"] == "max" else x.amin(-1))
        seg = st["seg"].long()
        lens = seg if case["lengths"] and not case["zip"] else torch.diff(seg)
        where = torch.repeat_interleave(torch.arange(case["nseg"], device="cuda"), lens)
        y = torch.full((case["nseg"],), float(_seed(case)), dtype=torch.float64, device="cuda")
        return y.index_add_(0, where, x) if case["op"] == "+" else y.scatter_reduce_(0, where, x, "amax")
    if kind == "permute":
        return torch.zeros(case["m"], dtype=torch.float64, device="cuda").index_add_(0, st["idx"].long(),
                                                                                     st["xs"].double())
    return _exact_stencil(case, st)
