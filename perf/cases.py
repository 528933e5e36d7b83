"""The work whose speed counts: what programs built on this library have it
do, through its public entry points.

A case is a dict of plain values.  Its "kind" is one of
  hierarchize  nodal values on the device -> surpluses on the device;
  refine       one iteration of limits-adaptive refinement: sample, hierarchize,
               surpluses and max |surplus| per subspace back;
  evaluate     a hierarchized grid and query points on the device -> values;
  host         the reference's calling style: host values and host points in,
               host results out (sg_set_values, sg_hierarchize, sg_evaluate);
  batch        many grids of mixed shape hierarchized and evaluated together;
  serve        requests of uneven size against a pool of resident grids.
The handles run with the options a program gets without asking for others;
FP64 hierarchization is the one option that programs choose (for accuracy).

Functions are products over the dims, f(x) = prod_k g_k(x_k), with g_k drawn
from the seed: smooth (exp(-w (x - c)^2) with w about 1) or localized (w = 50
near 0.3).  The surpluses of a product are products of 1-D surpluses, which
gives every exact result in closed form: exact() builds them in 64 bits, and
evaluates by a convolution over level sums instead of a sum over subspaces.
"""
import functools
import math

import numpy as np
import torch

import adaptive_sparse_grid_bench_b200 as sg

FN_BUMP = 3  # SG_FN_BUMP: exp(-p[1] sum_k (x_k - p[0])^2)


# ---- the cases -------------------------------------------------------------

def listed():
    full14 = "9,9,9,9,9,9"
    return [
        # one call on a small low-dimensional grid inside a larger program
        # (the shape of the reference's CPU case): launches and latency
        {"name": "hier_d4_n8", "kind": "hierarchize", "d": 4, "n": 8, "limits": "", "fp64": False, "local": False},
        # the reference's large grid, N = 33.0 M: memory traffic
        {"name": "hier_d10_n10", "kind": "hierarchize", "d": 10, "n": 10, "limits": "", "fp64": False, "local": False},
        # the accurate option at a middling size, N = 1.07 M
        {"name": "hier_fp64_d7_n9", "kind": "hierarchize", "d": 7, "n": 9, "limits": "", "fp64": True, "local": False},
        # one step of the refinement driver on a grid near its end (d = 6,
        # limits below n - 1): N = 13.3 M
        {"name": "refine_d6_n12", "kind": "refine", "d": 6, "n": 12, "limits": "9,8,9,8,9,8", "local": True},
        # a single request of a few points on a small grid: the smallest call
        {"name": "eval_d3_n6_7pts", "kind": "evaluate", "d": 3, "n": 6, "limits": "", "points": 7, "local": False},
        # an odd, small number of points on the large grid, as an optimizer
        # or a sampler asks for per step
        {"name": "eval_d10_n10_1000pts", "kind": "evaluate", "d": 10, "n": 10, "limits": "", "points": 1000, "local": False},
        # the reference's CPU case: d = 4, n = 8, 65,536 points
        {"name": "eval_d4_n8_64k", "kind": "evaluate", "d": 4, "n": 8, "limits": "", "points": 65536, "local": False},
        # a refined low-dimensional grid, half the points around its feature
        {"name": "eval_d6_n14_300k", "kind": "evaluate", "d": 6, "n": 14, "limits": full14, "points": 300007, "local": True},
        # the headline evaluation: the large grid, a long array of points
        {"name": "eval_d10_n10_4m", "kind": "evaluate", "d": 10, "n": 10, "limits": "", "points": 1 << 22, "local": False},
        # host arrays in, host results out, a middling grid and point count
        {"name": "host_d5_n9_20k", "kind": "host", "d": 5, "n": 9, "limits": "", "points": 20011, "local": False},
        # a batch of independent grids, d in 2..12 and n in 3..9, with
        # log-uniform 256..65,536 points each
        {"name": "batch_96", "kind": "batch", "grids": 96, "shapes": 3, "max_points": 2_000_000},
        # a burst of requests (log-uniform 1..65,536 points) on resident grids
        {"name": "serve_48", "kind": "serve", "grids": 24, "requests": 48, "shapes": 4, "max_points": 2_000_000},
    ]


MAX_N, MAX_S = 1 << 25, 120_000  # largest drawn grid: points, subspaces
MAX_PAIRS = 1 << 38               # largest drawn evaluation: points x subspaces


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_grid(rng, max_n=MAX_N, max_s=MAX_S):
    d = rng.randint(1, 14)
    top = 1
    while top < 16 and _sizes(d, top + 1)[0] <= max_n and _sizes(d, top + 1)[1] <= max_s:
        top += 1
    n = rng.randint(min(3, top), top)
    limits = ""
    if rng.random() < 0.33 and n > 2:
        limits = ",".join(str(rng.randint(n // 2, n - 1)) for _ in range(d))
    return d, n, limits


def draw(rng):
    kind = rng.choice(["hierarchize"] * 3 + ["evaluate"] * 5 + ["refine", "host", "batch", "serve"])
    if kind == "batch":
        return {"kind": kind, "grids": rng.randint(8, 96), "shapes": rng.randint(10, 1 << 20),
                "max_points": rng.choice([100_000, 500_000, 2_000_000])}
    if kind == "serve":
        return {"kind": kind, "grids": rng.randint(4, 24), "requests": rng.randint(4, 60),
                "shapes": rng.randint(10, 1 << 20), "max_points": rng.choice([100_000, 500_000, 2_000_000])}
    if kind == "host":
        d, n, limits = _draw_grid(rng, 1 << 21)
    else:
        d, n, limits = _draw_grid(rng)
    case = {"kind": kind, "d": d, "n": n, "limits": limits, "local": kind == "refine" or rng.random() < 0.3}
    if kind == "hierarchize":
        case["fp64"] = rng.random() < 0.25
    if kind in ("evaluate", "host"):
        s = _sizes(d, n, limits)[1]
        case["points"] = _log_int(rng, 1, min(1 << 18 if kind == "host" else 1 << 22, max(1, MAX_PAIRS // s)))
    return case


# ---- grid shapes (the compact layout, restated) ------------------------------

def _limits(d, n, limits=""):
    return [min(int(v), n - 1) for v in limits.split(",")] if limits else [n - 1] * d


@functools.lru_cache(maxsize=None)
def _counts(d, n, limits=""):
    """Level vectors per level sum 0..n-1."""
    c = [1] + [0] * (n - 1)
    for lim in _limits(d, n, limits):
        c = [sum(c[s - l] for l in range(min(s, lim) + 1)) for s in range(n)]
    return c


def _sizes(d, n, limits=""):
    """(points, subspaces)"""
    c = _counts(d, n, limits)
    return sum(v << s for s, v in enumerate(c)), sum(c)


@functools.lru_cache(maxsize=64)
def _level_vectors(d, n, limits=""):
    """Per level sum, the level vectors in memory order, (count, d) int64."""
    rows = [np.zeros((1, 0), np.int64)] + [np.zeros((0, 0), np.int64)] * (n - 1)
    for lim in _limits(d, n, limits):
        rows = [np.concatenate([np.pad(rows[s - l], ((0, 0), (0, 1)), constant_values=l)
                                for l in range(min(s, lim) + 1) if rows[s - l].shape[0]]
                               or [np.zeros((0, rows[0].shape[1] + 1), np.int64)]) for s in range(n)]
    return rows


def _product_values(d, n, limits, tables):
    """prod_k tables[k][2^l_k - 1 + i_k] at every grid point in compact order,
    float64; tables: (d, 2^n - 1) float64 on the target device."""
    dev = tables.device
    out = torch.empty(_sizes(d, n, limits)[0], dtype=torch.float64, device=dev)
    at = 0
    for s, lv in enumerate(_level_vectors(d, n, limits)):
        if not lv.shape[0]:
            continue
        lv = torch.from_numpy(lv).to(dev)
        p = torch.arange(1 << s, device=dev).unsqueeze(0)
        shift = torch.zeros((lv.shape[0], 1), dtype=torch.int64, device=dev)
        v = None
        for k in range(d - 1, -1, -1):
            size = torch.ones_like(shift) << lv[:, k:k + 1]
            f = tables[k][(size - 1) + ((p >> shift) & (size - 1))]
            v = f if v is None else v * f
            shift = shift + lv[:, k:k + 1]
        out[at:at + v.numel()] = v.reshape(-1)
        at += v.numel()
    return out


# ---- functions and points ----------------------------------------------------

def _function(seed, d, local):
    """(w, c) per dim of g_k(x) = exp(-w_k (x - c_k)^2)."""
    r = np.random.RandomState((seed * 7919 + 17) % (1 << 31))
    if local:
        return np.full(d, 50.0), np.full(d, 0.25 + 0.1 * r.rand())  # the form of SG_FN_BUMP
    return 0.3 + r.rand(d), r.rand(d)


def _nodal_tables(w, c, n):
    """g_k at the points of levels 0..n-1, (d, 2^n - 1)."""
    x = np.concatenate([(2 * np.arange(1 << l) + 1) / float(2 << l) for l in range(n)])
    return np.exp(-np.asarray(w)[:, None] * (x[None] - np.asarray(c)[:, None]) ** 2)


def _surplus_tables(w, c, n):
    """1-D surpluses of g_k: value minus the mean of its two neighbours on
    the next coarser grid (0 outside)."""
    g = lambda x: np.exp(-np.asarray(w)[:, None] * (x[None] - np.asarray(c)[:, None]) ** 2) * ((x > 0) & (x < 1))  # noqa: E731
    cols = []
    for l in range(n):
        h = 1.0 / (2 << l)
        x = (2 * np.arange(1 << l) + 1) * h
        cols.append(g(x) - 0.5 * (g(x - h) + g(x + h)))
    return np.concatenate(cols, axis=1)


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _points(seed, m, d, local):
    """m x d float32 in [0, 1): uniform; with `local`, the second half around
    0.3 with sigma 0.1, clipped into [0, 1)."""
    gen = torch.Generator(device=_device()).manual_seed(seed * 31 + 5)
    x = torch.rand((m, d), generator=gen, device=_device())
    if local:
        h = m - m // 2
        x[h:] = torch.clamp(0.3 + 0.1 * torch.randn((m - h, d), generator=gen, device=_device()), 0.0, 1.0 - 2.0 ** -24)
    return x


def _nodal(case, seed):
    w, c = _function(seed, case["d"], case["local"])
    t = torch.from_numpy(_nodal_tables(w, c, case["n"])).to(_device())
    return _product_values(case["d"], case["n"], case["limits"], t).float()


def _interpolant(w, c, d, n, limits, x):
    """The exact sparse-grid interpolant of the product function at x, in 64
    bits: sum over level vectors of prod_k e_k[l_k] with e_k[l] = 1-D surplus
    times hat, as a convolution over the level sum."""
    t = torch.from_numpy(_surplus_tables(w, c, n)).to(x.device)
    lim = _limits(d, n, limits)
    out = torch.empty(x.shape[0], dtype=torch.float64, device=x.device)
    for b in range(0, x.shape[0], 1 << 19):
        xb = x[b:b + (1 << 19)].double()
        acc = None
        for k in range(d):
            e = []
            for l in range(lim[k] + 1):
                y = xb[:, k] * float(1 << l)
                cell = y.floor()
                e.append(t[k][((1 << l) - 1) + cell.long()] * (1.0 - (2.0 * (y - cell) - 1.0).abs()))
            if acc is None:
                acc = e + [None] * (n - len(e))
                continue
            new = []
            for s in range(n):
                v = None
                for l in range(min(s, lim[k]) + 1):
                    if acc[s - l] is not None:
                        v = acc[s - l] * e[l] if v is None else v + acc[s - l] * e[l]
                new.append(v)
            acc = new
        out[b:b + (1 << 19)] = sum(a for a in acc if a is not None)
    return out


def _mixed_shapes(case, pts=(256, 65536)):
    """The shapes of a batch or pool: per grid d in 2..12 and n in 3..9 with at
    most max_points points, and a log-uniform point count; part of the case."""
    r = np.random.RandomState(case["shapes"] % (1 << 31))
    out = []
    for _ in range(case["grids"]):
        while True:
            d, n = int(r.randint(2, 13)), int(r.randint(3, 10))
            if _sizes(d, n)[0] <= case["max_points"]:
                break
        out.append((d, n, int(round(math.exp(r.uniform(math.log(pts[0]), math.log(pts[1])))))))
    return out


def _requests(case):
    """(grid, points) per request."""
    r = np.random.RandomState((case["shapes"] + 1) % (1 << 31))
    return [(int(r.randint(case["grids"])), int(round(math.exp(r.uniform(0.0, math.log(65536))))))
            for _ in range(case["requests"])]


# ---- what a program holds, and one pass ---------------------------------------

def _grid(case):
    return sg.Grid(case["d"], case["n"], _limits(case["d"], case["n"], case["limits"]) if case["limits"] else None)


_STREAMS = []


def _batch_stream():
    """One stream for batched work: graphs cannot be captured on the legacy
    default stream."""
    if not _STREAMS:
        _STREAMS.append(torch.cuda.Stream())
    return _STREAMS[0]


def prepare(case, seed):
    kind, st = case["kind"], {"case": case}
    if kind == "hierarchize":
        st["grid"] = _grid(case)
        st["grid"].precision = "fp64" if case["fp64"] else "fp32"
        st["values"] = _nodal(case, seed)
        st["surplus"] = torch.empty_like(st["values"])
        st["grid"].set_values_device(st["values"])
    elif kind == "refine":
        st["grid"] = _grid(case)
        w, c = _function(seed, case["d"], True)
        st["params"] = (float(c[0]), float(w[0]))
        st["grid"].sample_function(FN_BUMP, st["params"])
        st["surplus"] = torch.empty(st["grid"].num_points, device=_device())
    elif kind in ("evaluate", "host"):
        st["grid"] = _grid(case)
        x = _points(seed, case["points"], case["d"], case["local"])
        v = _nodal(case, seed)
        if kind == "host":
            st["x"], st["values"] = x.cpu().numpy(), v.cpu().numpy()
            st["grid"].set_values(st["values"])
        else:
            st["x"], st["out"] = x, torch.empty(case["points"], device=x.device)
            st["grid"].set_values_device(v)
            st["grid"].hierarchize()
    elif kind == "batch":
        shapes = _mixed_shapes(case)
        st["batch"] = sg.Batch([s[0] for s in shapes], [s[1] for s in shapes])
        st["offsets"] = np.concatenate([[0], np.cumsum([s[2] for s in shapes])]).astype(np.int64)
        st["values"] = torch.cat([_nodal({"d": d, "n": n, "limits": "", "local": False}, seed * 101 + i)
                                  for i, (d, n, _) in enumerate(shapes)])
        st["x"] = torch.cat([_points(seed * 101 + i, m, d, False).reshape(-1) for i, (d, _, m) in enumerate(shapes)])
        st["out"] = torch.empty(int(st["offsets"][-1]), device=st["x"].device)
        st["surplus"] = torch.empty_like(st["values"])
        torch.cuda.synchronize()
        st["batch"].set_values_device(st["values"], _batch_stream())
    elif kind == "serve":
        shapes = _mixed_shapes(case)
        st["server"] = sg.Server(4 << 30, max_batch_points=1 << 20)
        st["ids"] = []
        for i, (d, n, _) in enumerate(shapes):
            st["ids"].append(st["server"].add_grid(d, n, FN_BUMP, _serve_params(seed, i)))
        st["requests"] = [(g, _points(seed * 211 + q, m, shapes[g][0], False).cpu().numpy())
                          for q, (g, m) in enumerate(_requests(case))]
    return st


def _serve_params(seed, i):
    r = np.random.RandomState((seed * 6007 + i) % (1 << 31))
    return float(r.rand()), float(0.3 + r.rand())


def run(st):
    kind = st["case"]["kind"]
    if kind == "hierarchize":
        g = st["grid"]
        g.set_values_device(st["values"])
        g.hierarchize_async()
        g.get_values_device(st["surplus"])
        return st["surplus"]
    if kind == "refine":
        g = st["grid"]
        g.sample_function(FN_BUMP, st["params"])
        g.hierarchize_async()
        g.get_values_device(st["surplus"])
        return [g.subspace_maxabs(), st["surplus"]]
    if kind == "evaluate":
        st["grid"].evaluate_device(st["x"], st["out"])
        return st["out"]
    if kind == "host":
        g = st["grid"]
        g.set_values(st["values"])
        g.hierarchize()
        return g.evaluate(st["x"])
    if kind == "batch":
        b, stream = st["batch"], _batch_stream()
        b.set_values_device(st["values"], stream)
        b.hierarchize_async(stream)
        b.evaluate_device(st["offsets"], st["x"], st["out"], stream)
        b.get_values_device(st["surplus"], stream)
        return [st["out"], st["surplus"]]
    if kind == "serve":
        s = st["server"]
        tickets = [s.submit(st["ids"][g], x) for g, x in st["requests"]]
        return [s.wait(t)[0] for t in tickets]
    raise ValueError(kind)


# ---- the cost of a pass, and its exact result ----------------------------------

def _updates(d, n, limits=""):
    """Points updated by all sweeps together: per dim, those with l_k >= 1."""
    total = _sizes(d, n, limits)[0]
    lim = _limits(d, n, limits)
    out = 0
    for k in range(d):
        rest = lim[:k] + lim[k + 1:]
        out += total - (_sizes(d - 1, n, ",".join(map(str, rest)))[0] if d > 1 else 1)
    return out


def _hier_work(d, n, limits=""):
    return 8 * _sizes(d, n, limits)[0], 3 * _updates(d, n, limits)


def _eval_work(d, n, limits, m):
    p, s = _sizes(d, n, limits)
    return 4 * min(p, s * m) + 4 * m * (d + 1), 2 * s * m


def work(case):
    kind = case["kind"]
    if kind == "hierarchize":
        b, f = _hier_work(case["d"], case["n"], case["limits"])
    elif kind == "refine":
        p, s = _sizes(case["d"], case["n"], case["limits"])
        b, f = 8 * p + 4 * s, _hier_work(case["d"], case["n"], case["limits"])[1] + 3 * case["d"] * p
    elif kind == "evaluate":
        b, f = _eval_work(case["d"], case["n"], case["limits"], case["points"])
    elif kind == "host":
        (b0, f0), (b1, f1) = _hier_work(case["d"], case["n"], case["limits"]), _eval_work(
            case["d"], case["n"], case["limits"], case["points"])
        b, f = b0 + b1, f0 + f1
    else:
        shapes = _mixed_shapes(case)
        asked = [(d, n, m) for d, n, m in shapes] if kind == "batch" else [
            (shapes[g][0], shapes[g][1], m) for g, m in _requests(case)]
        b = f = 0
        for d, n, m in asked:
            e = _eval_work(d, n, "", m)
            b, f = b + e[0], f + e[1]
            if kind == "batch":
                h = _hier_work(d, n)
                b, f = b + h[0], f + h[1]
    return {"bytes": b, "flops": f}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("hierarchize", "refine"):
        d, n, limits = case["d"], case["n"], case["limits"]
        w, c = _function(seed, d, case["local"])
        s = _product_values(d, n, limits, torch.from_numpy(_surplus_tables(w, c, n)).to(_device()))
        if kind == "hierarchize":
            return s
        out, at = [], 0
        for level, count in enumerate(_counts(d, n, limits)):
            out.append(s[at:at + (count << level)].reshape(count, 1 << level).abs().amax(1) if count else s[:0])
            at += count << level
        return [torch.cat(out), s]
    if kind in ("evaluate", "host"):
        w, c = _function(seed, case["d"], case["local"])
        return _interpolant(w, c, case["d"], case["n"], case["limits"],
                            _points(seed, case["points"], case["d"], case["local"]))
    shapes = _mixed_shapes(case)
    if kind == "batch":
        outs, surs = [], []
        for i, (d, n, m) in enumerate(shapes):
            w, c = _function(seed * 101 + i, d, False)
            outs.append(_interpolant(w, c, d, n, "", _points(seed * 101 + i, m, d, False)))
            surs.append(_product_values(d, n, "", torch.from_numpy(_surplus_tables(w, c, n)).to(_device())))
        return [torch.cat(outs), torch.cat(surs)]
    outs = []
    for q, (g, m) in enumerate(_requests(case)):
        d, n, _ = shapes[g]
        center, width = _serve_params(seed, g)
        outs.append(_interpolant(np.full(d, width), np.full(d, center), d, n, "", _points(seed * 211 + q, m, d, False)))
    return outs
