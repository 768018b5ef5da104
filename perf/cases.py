"""The work this framework is asked to do, as cases that can be timed and checked.

A case is a dict of plain values: "op" names the public entry point that is called, the
rest are its sizes and options.  Inputs are expression matrices of a sparse regulatory
network (roots N(0,1), each other gene tanh of a weighted sum of its parents plus noise,
min-max scaled per gene) and, for the calls that start from a similarity matrix, a
symmetric MI-like matrix of such data with a zero diagonal.  Both are made on the GPU
with torch alone.
"""
import math

import numpy as np
import torch

import mcpnet_gb300 as M

BINS, ORDER = 10, 3  # the reference's defaults, and every configuration's


def listed():
    return [
        # the smallest call: a pathway's genes, host arrays in and out, default precision
        {"name": "mi_host_64x500", "op": "mi_host", "n": 64, "m": 500, "precision": "fp32"},
        # a 2,000-gene study in plain FP32 with the marginal entropies
        {"name": "mi_fp32_2000x2000", "op": "mi", "n": 2000, "m": 2000, "precision": "fp32"},
        # a whole genome on the tensor cores, the fastest form within 1e-4 nats
        {"name": "mi_bf16f8_20000x2000", "op": "mi", "n": 20000, "m": 2000, "precision": "bf16f8"},
        # the hi+lo split on sizes that fill no tile
        {"name": "mi_bf16x3_4999x1003", "op": "mi", "n": 4999, "m": 1003, "precision": "bf16x3"},
        # adaptive-partitioning MI, the reference applications' default method, with their tie-breaking noise
        {"name": "ap_mi_3001x1000", "op": "ap_mi", "n": 3001, "m": 1000},
        # the ensemble's products and the MCP2/3/4 scores of a 2,000-gene study
        {"name": "ensemble_2000", "op": "ensemble", "n": 2000},
        # MCP2 capacities and scores of a whole genome
        {"name": "mcp2_20000", "op": "mcp", "n": 20000, "path": 2, "symmetrize": False},
        # the DPI filter over a whole genome
        {"name": "dpi_20000", "op": "dpi", "n": 20000, "tol": 0.1, "mask": False},
        # transcription-factor products: 512 factors among 8,192 genes
        {"name": "tf_products_8192x512", "op": "tf", "n": 8192, "t": 512},
        # choosing ensemble coefficients against known edges
        {"name": "combo_eval_4096", "op": "combo_eval", "n": 4096, "rows": 35},
        # the MI adjoint (fitting per-gene parameters)
        {"name": "mi_bwd_2048x1000", "op": "mi_bwd", "n": 2048, "m": 1000},
        # forward and backward of an MCP3 loss over 5 % of the pairs
        {"name": "mcp3_grad_4096x1024", "op": "mcp3_grad", "n": 4096, "m": 1024},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["mi_host", "mi", "mi", "ap_mi", "ensemble", "mcp", "mcp", "dpi", "tf", "combo_eval", "mi_bwd",
                     "mcp3_grad"])
    if op == "mi_host":
        return {"op": op, "n": _log_int(rng, 16, 1000), "m": _log_int(rng, 60, 2000),
                "precision": rng.choice(["fp32", "fp32", "bf16f8"])}
    if op == "mi":
        if rng.random() < 0.5:
            return {"op": op, "n": _log_int(rng, 100, 4000), "m": _log_int(rng, 100, 2000), "precision": "fp32"}
        return {"op": op, "n": _log_int(rng, 500, 20000), "m": _log_int(rng, 200, 2000),
                "precision": rng.choice(["bf16f8", "bf16f8", "bf16x3", "fp16x3", "bf16", "fp16"])}
    if op == "ap_mi":
        return {"op": op, "n": _log_int(rng, 64, 3500), "m": _log_int(rng, 64, 1000)}
    if op == "ensemble":
        return {"op": op, "n": _log_int(rng, 64, 4096)}
    if op == "mcp":
        path = rng.choice([2, 3, 4])
        return {"op": op, "n": _log_int(rng, 200, 20000 if path == 2 else 12000), "path": path,
                "symmetrize": path == 3 and rng.random() < 0.5}
    if op == "dpi":
        return {"op": op, "n": _log_int(rng, 100, 20000), "tol": rng.choice([0.0, 0.1, 0.1, 0.15]),
                "mask": rng.random() < 0.5}
    if op == "tf":
        n = _log_int(rng, 256, 8192)
        return {"op": op, "n": n, "t": _log_int(rng, 8, max(16, n // 4))}
    if op == "combo_eval":
        return {"op": op, "n": _log_int(rng, 128, 4096), "rows": rng.choice([10, 20, 35])}
    if op == "mi_bwd":
        return {"op": op, "n": _log_int(rng, 32, 2048), "m": _log_int(rng, 64, 1000)}
    return {"op": op, "n": _log_int(rng, 64, 4096), "m": _log_int(rng, 64, 1024)}


# ---------------- inputs ----------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 13)
    return g


def _expression(n, m, g):
    """n genes x m samples in [0, 1]: a sparse random DAG (about two parents per gene, weights
    +-U(0.5, 1.5)), built level by level."""
    kw = {"generator": g, "device": "cuda"}
    x = torch.randn(n, m, **kw)
    noise = 0.3 * x
    cut = [0] + [max(1, int(n * f)) for f in (0.05, 0.1, 0.2, 0.4, 0.7)] + [n]
    for a, b in zip(cut[1:-1], cut[2:]):
        if b <= a:
            continue
        parents = torch.randint(0, a, (b - a, 4), **kw)
        w = (0.5 + torch.rand(b - a, 4, **kw)) * torch.where(torch.rand(b - a, 4, **kw) < 0.5, -1.0, 1.0)
        w = torch.where(torch.rand(b - a, 4, **kw) < 0.5, w, torch.zeros_like(w))
        s = torch.zeros(b - a, m, device="cuda")
        for k in range(4):
            s += w[:, k:k + 1] * x[parents[:, k]]
        root = (w == 0).all(1, keepdim=True)
        x[a:b] = torch.where(root, x[a:b], torch.tanh(s) + noise[a:b])
    lo, hi = x.amin(1, keepdim=True), x.amax(1, keepdim=True)
    return ((x - lo) / (hi - lo)).contiguous()


def _similarity(n, g, m=500):
    """A symmetric MI-like n x n matrix (bits) with a zero diagonal: the Gaussian MI of the data's
    linear correlations plus the first higher-order terms, so edges, indirect edges and the
    estimator's noise floor all appear."""
    x = _expression(n, m, g)
    z = x - x.mean(1, keepdim=True)
    z = z / z.norm(dim=1, keepdim=True)
    q = z * z
    q = q - q.mean(1, keepdim=True)
    q = q / q.norm(dim=1, keepdim=True)
    a = (z @ z.T).square_().clamp_(max=0.9999)
    a = torch.log2(1.0 - a).mul_(-0.5)
    c = (z @ q.T).square_()
    a += (0.5 / math.log(2.0)) * (c + c.T)
    del c
    a += (0.5 / math.log(2.0)) * (q @ q.T).square_()
    a = torch.maximum(a, a.T.contiguous())
    a.fill_diagonal_(0.0)
    return a


def _coefficients(rows):
    """The first rows of the grid of convex coefficients in steps of a quarter."""
    grid = [(a, b, c, 4 - a - b - c) for a in range(5) for b in range(5 - a) for c in range(5 - a - b)]
    return np.array(grid[:rows], dtype=np.float64) / 4.0


def _handle():
    h = M.Handle(torch.cuda.current_device())
    h.set_stream(torch.cuda.current_stream().cuda_stream)
    return h


def prepare(case, seed):
    g = _generator(seed)
    op, n = case["op"], case["n"]
    f32 = {"dtype": torch.float32, "device": "cuda"}
    s = {"case": case, "h": _handle()}
    if op == "mi_host":
        s["X"] = _expression(n, case["m"], g).cpu().numpy()
    elif op == "mi":
        s["X"] = _expression(n, case["m"], g)
        s["MI"] = torch.empty(n, n, **f32)
        s["H"] = torch.empty(n, dtype=torch.float64, device="cuda")
    elif op == "ap_mi":
        s["X"] = _expression(n, case["m"], g)
        s["MI"] = torch.empty(n, n, **f32)
    elif op == "ensemble":
        s["A"] = _similarity(n, g)
        s["out"] = {k: torch.empty(n, n, **f32) for k in ("M1", "M2", "M3", "R2", "R3", "R4")}
    elif op == "mcp":
        s["A"] = _similarity(n, g)
        s["M"], s["R"] = torch.empty(n, n, **f32), torch.empty(n, n, **f32)
    elif op == "dpi":
        s["A"] = _similarity(n, g)
        s["out"] = torch.empty(n, n, **f32)
        s["mask"] = torch.empty(n, n, dtype=torch.uint8, device="cuda") if case["mask"] else None
    elif op == "tf":
        s["A"] = _similarity(n, g)
        tfs = np.full(n, -np.inf, dtype=np.float32)
        tfs[torch.randperm(n, generator=g, device="cuda")[:case["t"]].cpu().numpy()] = np.inf
        s["tfs"] = tfs
        s["out"] = {k: torch.empty(case["t"], n, **f32) for k in ("T", "M1", "M2", "M3")}
    elif op == "combo_eval":
        a = _similarity(n, g)
        # stand-ins for the three products: larger than the entry, and correlated with it
        s["m"] = [a] + [torch.maximum(a, (0.02 * k) * torch.rand(n, n, generator=g, **f32) + 0.5 * a)
                        for k in (1, 2, 3)]
        known = torch.rand(n, n, generator=g, **f32)
        s["labels"] = torch.where(a > 0.08, 1, torch.where(known < 0.5, 0, -1)).to(torch.int8)
        s["coeffs"] = _coefficients(case["rows"])
    elif op == "mi_bwd":
        s["X"] = _expression(n, case["m"], g)
        s["G"] = torch.randn(n, n, generator=g, **f32).fill_diagonal_(0.0)
        s["dX"] = torch.empty(n, case["m"], **f32)
    elif op == "mcp3_grad":
        s["X"] = _expression(n, case["m"], g)
        e = max(8, n * n // 20)
        s["rows"] = torch.randint(0, n, (e,), generator=g, device="cuda")
        s["cols"] = torch.randint(0, n, (e,), generator=g, device="cuda")
        s["coef"] = 2.0 * torch.rand(e, generator=g, device="cuda") - 1.0
    else:
        raise ValueError(op)
    return s


def run(s):
    case, h = s["case"], s["h"]
    op = case["op"]
    if op == "mi_host":
        mi, H = h.bspline_mi(s["X"], BINS, ORDER, case["precision"], return_H=True)
        return {"MI": mi, "H": H}
    if op == "mi":
        h.bspline_mi_dev(s["X"], s["MI"], BINS, ORDER, case["precision"], H=s["H"])
        return {"MI": s["MI"], "H": s["H"]}
    if op == "ap_mi":
        h.ap_mi_dev(s["X"], s["MI"], noise=M.AP_NOISE, seed=1)
        return s["MI"]
    if op == "ensemble":
        h.maxmins_dev(s["A"], **s["out"])
        return s["out"]
    if op == "mcp":
        h.mcp_dev(s["A"], case["path"], M=s["M"], R=s["R"], symmetrize=case["symmetrize"])
        return {"M": s["M"], "R": s["R"]}
    if op == "dpi":
        removed = h.dpi_dev(s["A"], s["out"], tol=case["tol"], mask=s["mask"])
        out = {"out": s["out"], "removed": removed}
        return out if s["mask"] is None else dict(out, mask=s["mask"])
    if op == "tf":
        h.maxmins_tf_dev(s["A"], s["tfs"], **s["out"])
        return s["out"]
    if op == "combo_eval":
        aupr, auroc, best = h.combo_eval_dev(*s["m"], s["labels"], s["coeffs"])
        return {"aupr": aupr, "auroc": auroc, "best": best}
    if op == "mi_bwd":
        h.bspline_mi_bwd_dev(s["X"], s["G"], s["dX"], BINS, ORDER)
        return s["dX"]
    loss, dx = h.mcp3_loss_grad_dev(s["X"], s["rows"], s["cols"], s["coef"], bins=BINS, order=ORDER)
    return {"loss": loss, "dX": dx}


def work(case):
    op, n, m = case["op"], case["n"], case.get("m", 0)
    pairs = n * (n + 1) // 2
    # a sample has ORDER nonzero weights per gene; the tensor-core forms contract all BINS
    joint = 2.0 * (ORDER * ORDER if case.get("precision", "fp32") == "fp32" else BINS * BINS) * m
    if op in ("mi", "mi_host"):
        return {"bytes": 4 * n * m + 4 * n * n + 8 * n, "flops": joint * pairs}
    if op == "ap_mi":  # every pair looks at every sample
        return {"bytes": 4 * n * m + 4 * n * n, "flops": 2.0 * m * pairs}
    # the selection products are counted by their matrices: how many candidates have to be
    # compared depends on the data
    if op == "ensemble":
        return {"bytes": 4 * n * n * 7, "flops": 0}
    if op == "mcp":
        return {"bytes": 4 * n * n * 3, "flops": 0}
    if op == "dpi":
        return {"bytes": n * n * (9 if case["mask"] else 8), "flops": 0}
    if op == "tf":
        return {"bytes": 4 * n * n + 16 * case["t"] * n, "flops": 0}
    if op == "combo_eval":  # the labelled half of the lower triangle, read once
        return {"bytes": (4 * 4 + 1) * n * n // 2, "flops": 0}
    if op == "mi_bwd":  # the joint tables, then their weighted contraction with the samples
        return {"bytes": 8 * n * m + 4 * n * n, "flops": joint * pairs + joint * n * n}
    return {"bytes": 4 * n * m * 2 + 4 * n * n * 6, "flops": joint * pairs * 2 + joint * n * n}


# ---------------- the same in 64 bits ----------------
def _basis64(x):
    """B-spline weights (genes x samples x BINS) of the rows of x, each scaled to [0, 1]."""
    lo, hi = x.amin(1, keepdim=True), x.amax(1, keepdim=True)
    t = (x - lo) / (hi - lo)
    inner = BINS - ORDER
    v = [0.0] * ORDER + [(i + 1) / (inner + 1) for i in range(inner)] + [1.0] * ORDER
    d = t.detach()
    last = max(i for i in range(len(v) - 1) if v[i] < v[i + 1])
    b = []
    for i in range(len(v) - 1):
        inside = (d >= v[i]) & (d < v[i + 1]) if v[i] < v[i + 1] else torch.zeros_like(d, dtype=torch.bool)
        if i == last:
            inside = inside | (d >= 1.0)
        b.append(inside.double())
    for p in range(2, ORDER + 1):
        nxt = []
        for i in range(len(v) - p):
            d1, d2 = v[i + p - 1] - v[i], v[i + p] - v[i + 1]
            e = torch.zeros_like(t)
            if d1 > 0:
                e = e + (t - v[i]) / d1 * b[i]
            if d2 > 0:
                e = e + (v[i + p] - t) / d2 * b[i + 1]
            nxt.append(e)
        b = nxt
    return torch.stack(b[:BINS], dim=-1)


def _xlogx(p):
    return torch.where(p > 0, p * torch.log2(torch.where(p > 0, p, torch.ones_like(p))), torch.zeros_like(p))


def _mi64(x, step=128):
    n, m = x.shape
    w = _basis64(x.double())
    h = -_xlogx(w.mean(1)).sum(1)
    flat = w.permute(0, 2, 1).reshape(n * BINS, m).contiguous()
    out = torch.empty(n, n, dtype=torch.float64, device=x.device)
    for i in range(0, n, step):
        k = min(step, n - i)
        p = (flat[i * BINS:(i + k) * BINS] @ flat.T) / m
        e = _xlogx(p).view(k, BINS, n, BINS).sum((1, 3))
        out[i:i + k] = h[i:i + k, None] + h[None, :] + e
    return out, h


def _maxmin64(a, b):
    out = torch.empty(a.shape[0], b.shape[0], dtype=torch.float64, device=a.device)
    for i in range(a.shape[0]):
        out[i] = torch.minimum(a[i][None, :], b).amax(1)
    return out


def _ratio64(a, c):
    eps = torch.finfo(torch.float32).eps
    r = torch.where(c.abs() < eps, torch.full_like(a, torch.finfo(torch.float32).max), a / torch.where(c == 0, 1, c))
    return torch.where(a.abs() < eps, torch.zeros_like(a), r)


def exact(case, seed):
    op, n, m = case["op"], case["n"], case.get("m", 0)
    if op in ("mi", "mi_host", "mi_bwd") and n * n * m > 3e10:
        return None
    if op in ("ensemble", "mcp", "dpi", "tf") and n > 2000:
        return None
    if op in ("ap_mi", "combo_eval", "mcp3_grad"):
        return None
    s = prepare(case, seed)
    if op in ("mi", "mi_host"):
        mi, h = _mi64(torch.as_tensor(s["X"], device="cuda"))
        return {"MI": mi, "H": h}
    if op == "mi_bwd":
        # L = sum G_ij MI_ij; the pairs' tables are formed a few genes at a time
        x = s["X"].double().requires_grad_(True)
        w = _basis64(x)
        leaf = w.detach().requires_grad_(True)
        gsum = s["G"].double().sum(1) + s["G"].double().sum(0)
        hl = (-_xlogx(leaf.mean(1)).sum(1) * gsum).sum()
        hl.backward()
        flat = leaf.detach().permute(0, 2, 1).reshape(n * BINS, m).contiguous()
        sym = s["G"].double() + s["G"].double().T
        dw = torch.empty(n * BINS, m, dtype=torch.float64, device="cuda")
        for i in range(0, n, 64):
            k = min(64, n - i)
            p = (flat[i * BINS:(i + k) * BINS] @ flat.T) / m
            q = torch.where(p > 0, torch.log2(torch.where(p > 0, p, torch.ones_like(p))) + 1.0 / math.log(2.0),
                            torch.zeros_like(p))
            q = (q.view(k, BINS, n, BINS) * sym[i:i + k, None, :, None]).reshape(k * BINS, n * BINS)
            dw[i * BINS:(i + k) * BINS] = (q @ flat) / m
        w.backward(leaf.grad + dw.view(n, BINS, m).permute(0, 2, 1))
        return x.grad
    a = s["A"].double()
    if op == "ensemble":
        m1 = _maxmin64(a, a)
        m2, m3 = _maxmin64(a, m1), _maxmin64(m1, m1)
        return {"M1": m1, "M2": m2, "M3": m3, "R2": _ratio64(a, m1), "R3": _ratio64(a, m2), "R4": _ratio64(a, m3)}
    if op == "mcp":
        c = _maxmin64(a, a)
        if case["path"] == 3:
            c = _maxmin64(a, c)
            c = torch.maximum(c, c.T) if case["symmetrize"] else c
        elif case["path"] == 4:
            c = _maxmin64(c, c)
        return {"M": c, "R": _ratio64(a, c)}
    if op == "tf":
        at = a[:, torch.as_tensor(s["tfs"] > 0, device="cuda")]
        rows = torch.as_tensor(s["tfs"] > 0, device="cuda").nonzero()[:, 0]
        pick = lambda t: t[:, rows]
        m1 = _maxmin64(at[rows], at)
        return {"T": a[rows], "M1": m1, "M2": _maxmin64(pick(m1), at),
                "M3": _maxmin64(pick(m1), pick(_maxmin64(at, at)))}
    mult = 1.0 / (1.0 - float(np.float32(case["tol"])))
    b = a.clone()
    out = torch.empty_like(a)
    for i in range(n):
        c = torch.minimum(a[i][None, :], b)
        c[:, i] = -math.inf
        c.fill_diagonal_(-math.inf)
        gone = c.amax(1) >= (a[i] * mult).float().double()
        out[i] = torch.where(gone, torch.zeros_like(a[i]), a[i])
    out.fill_diagonal_(0.0)
    return {"out": out, "removed": None} if not case["mask"] else {"out": out, "removed": None, "mask": None}
