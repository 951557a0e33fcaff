"""What a user of this framework has it do, as cases that can be timed and compared.

Sizes are those of the benchmark's workloads and of the tests: the 250 x 500 x 4 panel, the
1218 x 5000 x 12 panel, stock returns of 1218 dates x 2000 / 5000 stocks, blocks of a
T x 8000 streaming panel, batches of uneven panels (N 300..6000, F = 8), and sections wider than
one CTA's shared memory (N > 16384).  Inputs follow the benchmark's panels: Gaussian, lognormal
and Student-t(3) factors, pre-listing gaps, 1 % missing cells and 5 % rounded (tied) values.
``draw`` gives more cases of the same ranges.
"""
from __future__ import annotations

import ctypes
import math
import pathlib
import sys

import torch

_PKG = str(pathlib.Path(__file__).resolve().parent.parent / "factor-cuda_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import fcb200  # noqa: E402
from fcb200 import _native as nat  # noqa: E402

MIN_VALID = 30
DEV = "cuda"


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # one live date: every stock of today's universe ranked (latency)
        {"name": "rank_one_date", "op": "rank", "T": 1, "N": 5000, "mask": True, "desc": True},
        # the small f64 panel's daily IC, one factor (latency; few CTAs)
        {"name": "ic_small_f64", "op": "ic", "T": 250, "N": 500, "fdt": "f64", "rdt": "f64", "mask": True},
        # one factor plane of the 1218 x 5000 panel, ranked under the listing mask
        {"name": "rank_plane", "op": "rank", "T": 1218, "N": 5000, "mask": True, "desc": False},
        # a universe wider than one CTA's shared memory (odd width)
        {"name": "rank_wide", "op": "rank", "T": 61, "N": 20011, "mask": False, "desc": False},
        # direction x mask scan of a ragged plane, all four groups
        {"name": "scan_plane", "op": "scan", "T": 1001, "N": 4733, "groups": "1111"},
        # daily IC of one f32 factor plane against forward returns, both masks
        {"name": "ic_plane", "op": "ic", "T": 1218, "N": 5000, "fdt": "f32", "rdt": "f32", "mask": True},
        # the headline step: ranks + IC of 12 factors with learned splitters
        {"name": "panel_learned", "op": "panel", "T": 1218, "N": 5000, "F": 12, "learned": True},
        # a block of the wide streaming panel ranked without a model
        {"name": "panel_block", "op": "panel", "T": 250, "N": 8000, "F": 16, "learned": False},
        # pooled factor correlation of the 1218 x 5000 x 12 panel
        {"name": "factor_corr", "op": "fcorr", "T": 1218, "N": 5000, "F": 12, "dt": "f32", "mask": True},
        # stock correlation, the drop-in f64-accurate path
        {"name": "stock_corr", "op": "scorr", "T": 1218, "N": 2000, "dt": "f32", "mask": True},
        # stock correlation, the BF16x3 precision form at full width
        {"name": "stock_corr_bf16x3", "op": "sprec", "T": 1218, "N": 5000},
        # many uneven panels in one replay: ranks, IC and factor correlation
        {"name": "batch_uneven", "op": "batch", "panels": 16, "F": 8, "Nlo": 300, "Nhi": 6000, "Tlo": 60, "Thi": 600,
         "shape": 7, "learned": True},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["rank", "rank", "wide", "ic", "ic", "scan", "panel", "panel", "fcorr", "scorr", "sprec", "batch"])
    if op == "wide":
        return {"op": "rank", "T": _logint(rng, 4, 64), "N": _logint(rng, 16385, 40000), "mask": rng.random() < 0.5,
                "desc": rng.random() < 0.5}
    if op == "rank":
        return {"op": op, "T": _logint(rng, 1, 1500), "N": _logint(rng, 200, 16000), "mask": rng.random() < 0.5,
                "desc": rng.random() < 0.5}
    if op == "ic":
        return {"op": op, "T": _logint(rng, 20, 1300), "N": _logint(rng, 300, 8000), "fdt": rng.choice(["f32", "f64"]),
                "rdt": rng.choice(["f32", "f64"]), "mask": rng.random() < 0.5}
    if op == "scan":
        return {"op": op, "T": _logint(rng, 20, 1300), "N": _logint(rng, 300, 8000),
                "groups": rng.choice(["1111", "1010", "0101", "1001", "1000"])}
    if op == "panel":
        return {"op": op, "T": _logint(rng, 50, 800), "N": _logint(rng, 500, 8000), "F": rng.randint(2, 12),
                "learned": rng.random() < 0.5}
    if op == "fcorr":
        return {"op": op, "T": _logint(rng, 60, 1000), "N": _logint(rng, 200, 3000), "F": _logint(rng, 2, 40),
                "dt": rng.choice(["f32", "f64"]), "mask": rng.random() < 0.5}
    if op == "scorr":
        return {"op": op, "T": _logint(rng, 60, 1300), "N": _logint(rng, 100, 2500), "dt": rng.choice(["f32", "f64"]),
                "mask": rng.random() < 0.7}
    if op == "sprec":
        return {"op": op, "T": _logint(rng, 120, 1218), "N": _logint(rng, 300, 5000)}
    return {"op": "batch", "panels": rng.randint(4, 16), "F": rng.randint(3, 9), "Nlo": 300, "Nhi": rng.randint(1000, 6000),
            "Tlo": 40, "Thi": rng.randint(100, 600), "shape": rng.randint(1, 10 ** 6), "learned": rng.random() < 0.5}


# ---------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float32)


def _student(g, df, *shape):
    chi = torch.zeros(*shape, device=DEV)
    for _ in range(df):
        chi += _normal(g, *shape) ** 2
    return _normal(g, *shape) / torch.sqrt(chi / df)


def _listed_mask(g, T, N, share=0.14):
    start = torch.randint(0, max(1, int(share * T)), (N,), generator=g, device=DEV)
    return torch.arange(T, device=DEV)[:, None] >= start[None, :]


def _widened(g, x, dt):
    """f32 draws as `dt`; in f64 the digits below f32's are drawn too."""
    return x if dt == torch.float32 else x.double() * (1 + 1e-8 * torch.randn(x.shape, generator=g, device=DEV, dtype=dt))


def _factor(g, kind, T, N, listing, dt=torch.float32):
    """One factor plane: Gaussian, lognormal(1) or Student-t(3); 1 % missing, 5 % rounded to 1e-3, gaps before listing."""
    x = _normal(g, T, N) if kind == 0 else torch.exp(_normal(g, T, N)) if kind == 1 else _student(g, 3, T, N)
    x = _widened(g, x, dt)
    u = torch.rand(T, N, generator=g, device=DEV)
    x = torch.where(u < 0.05, torch.round(x * 1000) / 1000, x)
    return torch.where((u > 0.99) | ~listing, torch.nan, x)


def _kind(f, F):
    return 0 if 2 * f < F else 1 if 4 * f < 3 * F else 2


def _panel(g, T, N, F, fdt=torch.float32, rdt=torch.float32):
    """Factor planes (F,T,N), forward returns (T,N), listing and return masks."""
    listing = _listed_mask(g, T, N)
    X = torch.empty(F, T, N, device=DEV, dtype=fdt)
    for f in range(F):
        X[f] = _factor(g, _kind(f, F), T, N, listing, fdt)
    R = _widened(g, 0.03 * torch.nan_to_num(X[0]).float() + _student(g, 4, T, N), rdt)
    R = torch.where(listing, R, torch.nan)
    return X, R, listing, torch.isfinite(R)


def _returns(g, T, N):
    """Daily stock returns: three common factors plus 0.02 * t(4); mask = listed and traded (98 %)."""
    B = 0.5 * _normal(g, N, 3)
    f = 0.01 * _normal(g, T, 3)
    X = 0.02 * _student(g, 4, T, N) + f @ B.T
    mask = _listed_mask(g, T, N, 0.1) & (torch.rand(T, N, generator=g, device=DEV) < 0.98)
    return X, mask


def _dt(name):
    return torch.float64 if name == "f64" else torch.float32


def _batch_shapes(case):
    import random
    r = random.Random(case["shape"])
    return [(_logint(r, case["Tlo"], case["Thi"]), _logint(r, case["Nlo"], case["Nhi"])) for _ in range(case["panels"])]


def _radix_panel(X, R, fm, rm, ranks, ic):
    F, T, N = X.shape
    nat.check(nat.lib().fcb_dev_rank_ic_panel(X.data_ptr(), R.data_ptr(), fm.data_ptr(), rm.data_ptr(), F, T, N,
                                              MIN_VALID, ranks.data_ptr(), ic.data_ptr(), 0,
                                              torch.cuda.current_stream().cuda_stream), "fcb_dev_rank_ic_panel")


def _fitted_model(X, R, fm, rm):
    """A CDF model fitted on the exact ranks of the panel's first (up to 250) dates."""
    F, T, N = X.shape
    t = min(T, 250)
    ranks, ic = torch.empty_like(X), torch.empty(F, T, dtype=torch.float64, device=DEV)
    _radix_panel(X, R, fm, rm, ranks, ic)
    model = fcb200.CdfModel(F)
    model.fit(X, ranks, T, N, 0, t, steps=300, lr=3e-3, stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return model


def prepare(case, seed):
    g = _gen(seed)
    op = case["op"]
    s = {"case": case}
    if op in ("rank", "scan"):
        T, N = case["T"], case["N"]
        listing = _listed_mask(g, T, N)
        s["x"] = _factor(g, seed % 3, T, N, listing)
        mask = listing & (torch.rand(T, N, generator=g, device=DEV) < 0.97)
        if op == "rank":
            s["mask"] = mask if case["mask"] else None
        else:
            s["mask"] = mask.to(torch.uint8)
            s["out"] = [torch.empty(T, N, device=DEV) if c == "1" else None for c in case["groups"]]
    elif op == "ic":
        X, R, fm, rm = _panel(g, case["T"], case["N"], 1, _dt(case["fdt"]), _dt(case["rdt"]))
        s["f"], s["r"] = X[0], R
        s["fm"], s["rm"] = (fm, rm) if case["mask"] else (None, None)
    elif op == "panel":
        X, R, fm, rm = _panel(g, case["T"], case["N"], case["F"])
        s["X"], s["R"], s["fm"], s["rm"] = X, R, fm.to(torch.uint8), rm.to(torch.uint8)
        s["ranks"] = torch.empty_like(X)
        s["ic"] = torch.empty(case["F"], case["T"], dtype=torch.float64, device=DEV)
        if case["learned"]:
            s["model"] = _fitted_model(X, R, s["fm"], s["rm"])
    elif op == "fcorr":
        X, _, fm, _ = _panel(g, case["T"], case["N"], case["F"], _dt(case["dt"]))
        s["x"] = X.permute(1, 2, 0).contiguous()
        s["mask"] = fm if case["mask"] else None
    elif op in ("scorr", "sprec"):
        X, mask = _returns(g, case["T"], case["N"])
        if op == "scorr":
            s["x"], s["mask"] = _widened(g, X, _dt(case["dt"])), mask if case["mask"] else None
        else:
            s["x"], s["mask"] = X, mask.to(torch.uint8)
            s["out"] = torch.empty(case["N"], case["N"], dtype=torch.float64, device=DEV)
            s["ws"] = fcb200.Workspace()
    else:
        F = case["F"]
        panels = []
        for k, (T, N) in enumerate(_batch_shapes(case)):
            X, R, fm, rm = _panel(g, T, N, F)
            p = {"X": X, "R": R, "fmask": fm.to(torch.uint8), "rmask": rm.to(torch.uint8), "ranks": torch.empty_like(X),
                 "ic": torch.empty(F, T, dtype=torch.float64, device=DEV),
                 "corr": torch.empty(F, F, dtype=torch.float64, device=DEV)}
            if case["learned"]:
                p["model"] = _fitted_model(X, R, p["fmask"], p["rmask"]) if k == 0 else panels[0]["model"]
            panels.append(p)
        s["panels"], s["batch"] = panels, fcb200.Batch(panels, min_valid=MIN_VALID)
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    case = s["case"]
    op = case["op"]
    if op == "rank":
        return fcb200.cross_sectional_rank(s["x"], s["mask"], descending=case["desc"])
    if op == "ic":
        return fcb200.rolling_ic(s["f"], s["r"], s["fm"], s["rm"], min_valid=MIN_VALID)
    if op == "scan":
        T, N = s["x"].shape
        outs = (ctypes.c_void_p * 4)(*[nat.ptr(o) for o in s["out"]])
        active = (ctypes.c_int * 4)(*[int(c) for c in case["groups"]])
        status = (ctypes.c_int * 4)()
        nat.check(nat.lib().fcb_dev_parameter_scan_f32(s["x"].data_ptr(), s["mask"].data_ptr(), T, N, outs, status, active,
                                                       torch.cuda.current_stream().cuda_stream), "fcb_dev_parameter_scan_f32")
        return [o for o in s["out"] if o is not None]
    if op == "panel":
        X = s["X"]
        if not case["learned"]:
            _radix_panel(X, s["R"], s["fm"], s["rm"], s["ranks"], s["ic"])
        else:
            F, T, N = X.shape
            nat.check(nat.lib().fcb_dev_rank_ic_panel_learned(
                X.data_ptr(), s["R"].data_ptr(), s["fm"].data_ptr(), s["rm"].data_ptr(), F, T, N, MIN_VALID,
                s["ranks"].data_ptr(), s["ic"].data_ptr(), s["model"].handle, 0, None,
                torch.cuda.current_stream().cuda_stream), "fcb_dev_rank_ic_panel_learned")
        return [s["ranks"], s["ic"]]
    if op == "fcorr":
        return fcb200.factor_corr(s["x"], s["mask"])
    if op == "scorr":
        return fcb200.stock_corr(s["x"], s["mask"])
    if op == "sprec":
        T, N = s["x"].shape
        nat.check(nat.lib().fcb_dev_stock_corr_prec(s["x"].data_ptr(), s["mask"].data_ptr(), T, N, 0, s["out"].data_ptr(),
                                                    s["ws"].handle, torch.cuda.current_stream().cuda_stream),
                  "fcb_dev_stock_corr_prec")
        return s["out"]
    s["batch"].run()
    return [[p["ranks"], p["ic"], p["corr"]] for p in s["panels"]]


# ---------------------------------------------------------------- what it cannot do without
def _panel_work(F, T, N):
    cells = F * T * N
    return {"bytes": 8 * cells + 6 * T * N + 8 * F * T, "flops": 2 * cells}


def work(case):
    op = case["op"]
    if op == "batch":
        w = [_panel_work(case["F"], T, N) for T, N in _batch_shapes(case)]
        pooled = sum(T * N for T, N in _batch_shapes(case))
        return {"bytes": sum(v["bytes"] for v in w), "flops": sum(v["flops"] for v in w) + pooled * case["F"] * (case["F"] + 1)}
    T, N = case["T"], case["N"]
    n = T * N
    if op == "rank":
        return {"bytes": n * (9 if case["mask"] else 8), "flops": n}
    if op == "scan":
        return {"bytes": n * (5 + 4 * case["groups"].count("1")), "flops": n}
    if op == "ic":
        per = sum(8 if case[k] == "f64" else 4 for k in ("fdt", "rdt")) + (2 if case["mask"] else 0)
        return {"bytes": n * per + 8 * T, "flops": 2 * n}
    if op == "panel":
        return _panel_work(case["F"], T, N)
    if op == "fcorr":
        F = case["F"]
        return {"bytes": n * F * (8 if case["dt"] == "f64" else 4) + (n if case["mask"] else 0) + 8 * F * F,
                "flops": n * F * (F + 1)}
    masked = op == "sprec" or case["mask"]
    per = (8 if case.get("dt") == "f64" else 4) + (1 if masked else 0)
    # sum x_i x_j of the upper triangle; with a mask also the count, both sums and both sums of squares of each pair
    return {"bytes": n * per + 8 * N * N, "flops": T * N * N * (6 if masked else 1)}


# ---------------------------------------------------------------- 64-bit values
def _ranks64(x, valid, desc=False):
    """Stable ordinal ranks 1..K of the valid cells of each row, ties by column; NaN elsewhere."""
    out = torch.empty(x.shape, dtype=torch.float64, device=DEV)
    step = max(1, 20_000_000 // x.shape[1])
    for t in range(0, x.shape[0], step):
        v, ok = x[t:t + step].double(), valid[t:t + step]
        v = torch.where(ok, (-v if desc else v) + 0.0, torch.inf)
        order = torch.sort(v, dim=1, stable=True).indices
        pos = torch.arange(1, v.shape[1] + 1, device=DEV, dtype=torch.float64).expand_as(v)
        out[t:t + step].scatter_(1, order, pos)
        out[t:t + step][~ok] = torch.nan
    return out


def _constant(x, joint):
    v = x.double()
    lo, hi = torch.where(joint, v, torch.inf).amin(1), torch.where(joint, v, -torch.inf).amax(1)
    return lo == hi


def _ic64(f, r, fm, rm):
    joint = torch.isfinite(f) & torch.isfinite(r)
    joint &= True if fm is None else fm.bool()
    joint &= True if rm is None else rm.bool()
    m = joint.sum(1).double()
    a, b = (torch.nan_to_num(_ranks64(v, joint)) for v in (f, r))
    mean = (m + 1) / 2
    a, b = (torch.where(joint, v - mean[:, None], 0.0) for v in (a, b))
    ic = (a * b).sum(1) / torch.sqrt((a * a).sum(1)) / torch.sqrt((b * b).sum(1))
    bad = (m < MIN_VALID) | _constant(f, joint) | _constant(r, joint)
    return torch.where(bad, torch.nan, ic)


def _corr64(X, valid):
    """Pairwise-complete Pearson of the columns of X (rows, columns)."""
    v = valid.double()
    x = torch.where(valid, X.double(), 0.0)
    x = torch.where(valid, x - x.sum(0) / v.sum(0), 0.0)
    n, s, q, xy = v.T @ v, x.T @ v, (x * x).T @ v, x.T @ x
    cov, var = xy - s * s.T / n, q - s * s / n
    c = cov / torch.sqrt(var) / torch.sqrt(var.T)
    return torch.where(n >= 2, c, torch.nan).fill_diagonal_(1.0)


def _panel64(X, R, fm, rm):
    ranks = torch.empty(X.shape, dtype=torch.float64, device=DEV)
    for f in range(X.shape[0]):
        ranks[f] = _ranks64(X[f], torch.isfinite(X[f]) & fm.bool())
    return [ranks, torch.stack([_ic64(X[f], R, fm, rm) for f in range(X.shape[0])])]


def exact(case, seed):
    s = prepare(case, seed)
    op = case["op"]
    if op in ("rank", "scan"):
        x, finite = s["x"], torch.isfinite(s["x"])
        if op == "rank":
            return _ranks64(x, finite if s["mask"] is None else finite & s["mask"], case["desc"])
        masked = finite & s["mask"].bool()
        every = [(masked, False), (finite, False), (masked, True), (finite, True)]
        return [_ranks64(x, v, d) for (v, d), c in zip(every, case["groups"]) if c == "1"]
    if op == "ic":
        return _ic64(s["f"], s["r"], s["fm"], s["rm"])
    if op == "panel":
        return _panel64(s["X"], s["R"], s["fm"], s["rm"])
    if op == "fcorr":
        x = s["x"].reshape(-1, case["F"])
        valid = torch.isfinite(x)
        return _corr64(x, valid if s["mask"] is None else valid & s["mask"].reshape(-1, 1))
    if op in ("scorr", "sprec"):
        valid = torch.isfinite(s["x"])
        return _corr64(s["x"], valid if s["mask"] is None else valid & s["mask"].bool())
    out = []
    for p in s["panels"]:
        F = p["X"].shape[0]
        x, fm = p["X"].reshape(F, -1).T, p["fmask"].reshape(-1, 1).bool()
        out.append(_panel64(p["X"], p["R"], p["fmask"], p["rmask"]) + [_corr64(x, torch.isfinite(x) & fm)])
    return out
