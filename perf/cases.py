"""Workloads of the transform library, from the smallest call to the largest: what each one is, its
inputs, one pass through the public entry points, the work it cannot do without, and its result in
64-bit arithmetic from plain torch.

A case is a dict: `kind` names the entry points, the other keys their sizes and options.

  memo     the host drop-ins InvFSTSemiMemo and FSTSemiMemo, one function, caller's tables
  conv     the host drop-in ConvOn2SphereSemiMemo, one function and a zonal filter
  f64      Plan.inv_fst and Plan.fst on device buffers (FP64); fly: the plan without tables
  split    Plan.inv_fst_real_f32 and fst_real_f32 (FP32 samples, split tensor-core contraction)
  csplit   the same for COMPLEX data (inv_fst_complex_f32, fst_complex_f32)
  group    Group.fst_inv: functions of uneven bandwidth in one call
  refined  Plan.fst_refined: FP64 samples, split contraction and one FP64-residual step
  host     the queued host-buffer calls (inv_fst_real_f32_host_async, fst_real_f32_host_async)
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from s2kit_gb300 import api

DEV = "cuda" if torch.cuda.is_available() else "cpu"
PREC = {"bf16x3": api.PREC_BF16X3, "bf16x2": api.PREC_BF16X2, "fp16x2": api.PREC_FP16X2}
GROUP_BW = (16, 32, 64, 128, 256)
GROUP_P = (0.3, 0.3, 0.2, 0.15, 0.05)


def listed():
    return [
        # one function through the reference's own calls: a program written for S2kit, relinked
        {"name": "memo_bw64", "kind": "memo", "bw": 64, "cutoff": 64, "complex": False},
        # smoothing one field with a zonal filter, the reference's convolution call
        {"name": "conv_bw256", "kind": "conv", "bw": 256},
        # double-precision analysis of a batch of fields that stay on the GPU
        {"name": "f64_bw256_x64", "kind": "f64", "bw": 256, "cutoff": 256, "complex": False, "fly": False, "batch": 64},
        # complex data at an odd bandwidth with the seminaive/naive split the reference offers
        {"name": "f64_complex_bw101_x16", "kind": "f64", "bw": 101, "cutoff": 64, "complex": True, "fly": False,
         "batch": 16},
        # the family without tables, for programs that cannot hold them
        {"name": "fly_bw256_x16", "kind": "f64", "bw": 256, "cutoff": 256, "complex": False, "fly": True, "batch": 16},
        # the smallest device call: one function at the smallest bandwidth of the split path
        {"name": "split_bw16_x1", "kind": "split", "bw": 16, "batch": 1, "prec": "bf16x3"},
        # many small fields at once (descriptors, patches, features)
        {"name": "split_bw64_x4096", "kind": "split", "bw": 64, "batch": 4096, "prec": "bf16x3"},
        # the benchmark's own batch
        {"name": "split_bw256_x256", "kind": "split", "bw": 256, "batch": 256, "prec": "bf16x3"},
        # complex fields at an odd bandwidth, where 2 bw has no convenient factors
        {"name": "csplit_bw255_x32", "kind": "csplit", "bw": 255, "batch": 32, "prec": "bf16x3"},
        # functions of uneven bandwidth in one captured call
        {"name": "group_512", "kind": "group", "functions": 512, "mix": 3, "prec": "fp16x2"},
        # large fields to near double precision: the split transform with its refinement step
        {"name": "refined_bw1024_x16", "kind": "refined", "bw": 1024, "batch": 16, "prec": "bf16x3"},
        # fields that live in (pinned) host memory, the benchmark's end-to-end step
        {"name": "host_bw256_x256", "kind": "host", "bw": 256, "batch": 256, "prec": "bf16x3"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _split_bw(rng):
    return rng.choice((512, 1024)) if rng.random() < 0.15 else _log_int(rng, 16, 256)


def draw(rng: random.Random):
    kind = rng.choice(("memo", "conv", "f64", "f64", "split", "split", "split", "csplit", "group", "refined", "host"))
    if kind == "memo":
        bw = _log_int(rng, 8, 256)
        return {"kind": kind, "bw": bw, "cutoff": bw if rng.random() < 0.5 else rng.randint((bw + 1) // 2, bw),
                "complex": rng.random() < 0.3}
    if kind == "conv":
        return {"kind": kind, "bw": _log_int(rng, 16, 256)}
    if kind == "f64":
        bw = 512 if rng.random() < 0.1 else _log_int(rng, 8, 300)
        fly = rng.random() < 0.25
        return {"kind": kind, "bw": bw, "cutoff": bw if fly or rng.random() < 0.6 else rng.randint((bw + 1) // 2, bw),
                "complex": rng.random() < 0.35, "fly": fly,
                "batch": _log_int(rng, 1, max(1, min(512, 2 ** 29 // bw ** 3)))}
    if kind in ("split", "csplit", "host"):
        bw = _split_bw(rng)
        most = 2 ** 24 if kind == "split" else 2 ** 22
        return {"kind": kind, "bw": bw, "batch": _log_int(rng, 1, most // bw ** 2),
                "prec": rng.choice(("bf16x3", "bf16x3", "bf16x2", "fp16x2"))}
    if kind == "group":
        return {"kind": kind, "functions": _log_int(rng, 16, 512), "mix": rng.randrange(1 << 16), "prec": "fp16x2"}
    bw = rng.choice((512, 1024)) if rng.random() < 0.3 else _log_int(rng, 16, 256)
    return {"kind": kind, "bw": bw, "batch": _log_int(rng, 1, max(1, min(64, 2 ** 24 // bw ** 2))), "prec": "bf16x3"}


# ---- inputs ---------------------------------------------------------------------------------
def _group_bws(case):
    return random.Random(case["mix"]).choices(GROUP_BW, GROUP_P, k=case["functions"])


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float64)


def _index(m, l, bw):
    """Slot of f(l, m) in the reference layout."""
    if m >= 0:
        return m * bw - m * (m - 1) // 2 + (l - m)
    a, top = -m, bw - 1
    return top * (top + 3) // 2 + 1 + (top - a) * (top - a + 1) // 2 + (l - a)


_slots = {}


def _slot_lm(bw):
    """Degree and order of every slot, on the device."""
    if bw not in _slots:
        ls, ms = np.empty(bw * bw, np.int64), np.empty(bw * bw, np.int64)
        for m in range(-(bw - 1), bw):
            i = _index(m, abs(m), bw)
            ls[i:i + bw - abs(m)] = np.arange(abs(m), bw)
            ms[i:i + bw - abs(m)] = m
        mate = np.arange(bw * bw)  # the slot of f(l, |m|)
        for m in range(1, bw):
            at = _index(-m, m, bw)
            mate[at:at + bw - m] = np.arange(_index(m, m, bw), _index(m, m, bw) + bw - m)
        _slots[bw] = tuple(torch.from_numpy(a).to(DEV) for a in (ls, ms, mate))
    return _slots[bw]


def _coeffs(g, bw, batch, power, real):
    """Coefficients N(0,1) (1+l)^-power; real fields: f(l,-m) = (-1)^m conj f(l,m), f(l,0) real."""
    ls, ms, mate = _slot_lm(bw)
    s = (1.0 + ls.double()) ** -power
    rc, ic = _randn(g, batch, bw * bw) * s, _randn(g, batch, bw * bw) * s
    if real:
        ic = torch.where(ms == 0, torch.zeros_like(ic), ic)
        neg, sign = ms < 0, 1.0 - 2.0 * (ms % 2).double()
        rc = torch.where(neg, sign * rc[:, mate], rc)
        ic = torch.where(neg, -sign * ic[:, mate], ic)
    return rc, ic


def _field(g, bw, batch):
    """Samples of smooth fields: a mean and six plane waves of random direction, |k| up to 0.7 bw."""
    S = 2 * bw
    th = torch.arange(S, device=DEV, dtype=torch.float64).add(0.5).mul(math.pi / S)
    ph = torch.arange(S, device=DEV, dtype=torch.float64).mul(2 * math.pi / S)
    st, ct = torch.sin(th)[:, None], torch.cos(th)[:, None]
    out = _randn(g, batch, 1, 1).expand(batch, S, S).contiguous()
    for _ in range(6):
        k = torch.rand(batch, 1, 1, generator=g, device=DEV, dtype=torch.float64) * (0.7 * bw)
        d = _randn(g, 3, batch, 1, 1)
        d = k * d / d.norm(dim=0)
        a, p = _randn(g, batch, 1, 1) / (1 + k).sqrt(), _randn(g, batch, 1, 1) * 3
        out += a * torch.cos(d[0] * (st * torch.cos(ph)) + d[1] * (st * torch.sin(ph)) + d[2] * ct + p)
    return out.view(batch, S * S)


def _zonal_coeffs(bw):
    l = np.arange(bw)
    return np.exp(-l * (l + 1) / (2 * (0.15 * bw) ** 2))


def _zonal_field(bw):
    """Samples of the zonal filter sum_l h_l Y_l0."""
    S = 2 * bw
    x = np.cos((np.arange(S) + 0.5) * math.pi / S)
    p0, p1, out = np.ones(S), x.copy(), np.zeros(S)
    for l, h in enumerate(_zonal_coeffs(bw)):
        out += h * math.sqrt((2 * l + 1) / (4 * math.pi)) * p0
        p0, p1 = p1, ((2 * l + 3) * x * p1 - (l + 1) * p0) / (l + 2)
    return np.repeat(out[:, None], S, axis=1).reshape(-1).copy()


def _inputs(case, seed):
    """(coefficients, samples) of the case in FP64 on the device; None where the case has no such input."""
    g = _gen(seed)
    kind = case["kind"]
    if kind == "group":
        bws = _group_bws(case)  # one batch per bandwidth, then back to the order of the functions
        grids = {bw: iter(_field(g, bw, bws.count(bw))) for bw in sorted(set(bws))}
        return None, torch.cat([next(grids[bw]) for bw in bws])
    bw = case["bw"]
    if kind == "conv":
        return None, _field(g, bw, 1)
    if kind == "refined":
        return None, _field(g, bw, case["batch"])
    batch = case.get("batch", 1)
    cplx = kind == "csplit" or case.get("complex", False)
    rc, ic = _coeffs(g, bw, batch, 1.0, not cplx)
    if kind == "host":
        return (rc, ic), None
    gr = _field(g, bw, batch)
    return (rc, ic), (gr, _field(g, bw, batch) if cplx else None)


def _pinned(x):
    t = torch.empty(x.shape, dtype=torch.float32, pin_memory=DEV == "cuda")
    t.copy_(x)
    return t.numpy()


def _dev(*shape, dtype=torch.float32):
    return torch.zeros(*shape, dtype=dtype, device=DEV)


_tables = {}


def _memo_tables(bw, cutoff):
    """The caller's tables, built once as the reference's own programs build them."""
    if (bw, cutoff) not in _tables:
        n = api.Reduced_SpharmonicTableSize(bw, cutoff) + api.Reduced_Naive_TableSize(bw, cutoff)
        fwd = api.SemiNaive_Naive_Pml_Table(bw, cutoff, np.zeros(n + 2 * bw))
        inv = api.Transpose_SemiNaive_Naive_Pml_Table(fwd, bw, cutoff, np.zeros(n + 2 * bw))
        w = np.zeros(4 * bw)
        api.GenerateWeightsForDLT(bw, w)
        _tables[bw, cutoff] = fwd, inv, w
    return _tables[bw, cutoff]


def prepare(case, seed):
    kind = case["kind"]
    coeffs, grid = _inputs(case, seed)
    s = dict(case)
    if kind == "memo":
        bw, n = case["bw"], 4 * case["bw"] ** 2
        s["tables"] = _memo_tables(bw, case["cutoff"])
        s["rc"], s["ic"] = (c[0].cpu().numpy().copy() for c in coeffs)
        s["gr"] = grid[0][0].cpu().numpy().copy()
        s["gi"] = np.zeros(n) if grid[1] is None else grid[1][0].cpu().numpy().copy()
        s["out_g"], s["out_c"] = np.zeros((2, n)), np.zeros((2, bw * bw))
    elif kind == "conv":
        bw, n = case["bw"], 4 * case["bw"] ** 2
        s["gr"], s["gi"] = grid[0].cpu().numpy().copy(), np.zeros(n)
        s["fr"], s["fi"], s["out_g"] = _zonal_field(bw), np.zeros(n), np.zeros((2, n))
    elif kind == "f64":
        bw, nb = case["bw"], case["batch"]
        s["plan"] = api.Plan(bw, case["cutoff"], fly=case["fly"])
        s["rc"], s["ic"] = coeffs
        s["gr"], s["gi"] = grid
        s["out_g"] = [_dev(nb, 4 * bw * bw, dtype=torch.float64) for _ in range(2 if case["complex"] else 1)]
        s["out_c"] = [_dev(nb, bw * bw, dtype=torch.float64) for _ in range(2)]
    elif kind in ("split", "csplit"):
        bw, nb = case["bw"], case["batch"]
        s["plan"] = api.Plan(bw, bw)
        s["rc"], s["ic"] = (c.float() for c in coeffs)
        s["gr"], s["gi"] = (None if x is None else x.float() for x in grid)
        s["out_g"] = [_dev(nb, 4 * bw * bw) for _ in range(2 if kind == "csplit" else 1)]
        s["out_c"] = [_dev(nb, bw * bw) for _ in range(2)]
    elif kind == "group":
        s["group"] = api.Group(_group_bws(case), PREC[case["prec"]])
        s["group"].autotune()
        s["gr"], s["out_g"] = grid.float(), _dev(s["group"].grid_total)
        s["out_c"] = [_dev(s["group"].coeff_total) for _ in range(2)]
    elif kind == "refined":
        bw, nb = case["bw"], case["batch"]
        s["plan"], s["gr"] = api.Plan(bw, bw), grid
        s["out_c"] = [_dev(nb, bw * bw, dtype=torch.float64) for _ in range(2)]
    else:
        bw, nb = case["bw"], case["batch"]
        s["plan"] = api.Plan(bw, bw)
        s["rc"], s["ic"] = (_pinned(c) for c in coeffs)
        s["out_g"] = _pinned(torch.zeros(nb, 4 * bw * bw))
        s["out_c"] = [_pinned(torch.zeros(nb, bw * bw)) for _ in range(2)]
    return s


def run(s):
    kind = s["kind"]
    if kind == "memo":
        fwd, inv, w = s["tables"]
        fmt = api.COMPLEX if s["complex"] else api.REAL
        g, c = s["out_g"], s["out_c"]
        api.InvFSTSemiMemo(s["rc"], s["ic"], g[0], g[1], s["bw"], inv, None, fmt, s["cutoff"])
        api.FSTSemiMemo(s["gr"], s["gi"], c[0], c[1], s["bw"], fwd, None, fmt, s["cutoff"], weights=w)
        return {"coeffs": c, "grid": g}
    if kind == "conv":
        g = s["out_g"]
        api.ConvOn2SphereSemiMemo(s["gr"], s["gi"], s["fr"], s["fi"], g[0], g[1], s["bw"])
        return {"grid": g}
    c, p = s["out_c"], s.get("plan")
    if kind == "f64":
        fmt = api.COMPLEX if s["complex"] else api.REAL
        g = s["out_g"]
        p.inv_fst(s["rc"], s["ic"], g[0], g[1] if s["complex"] else None, s["batch"], fmt)
        p.fst(s["gr"], s["gi"], c[0], c[1], s["batch"], fmt)
        return {"coeffs": c, "grid": g}
    if kind == "refined":
        p.fst_refined(s["gr"], c[0], c[1], s["batch"], PREC[s["prec"]])
        return {"coeffs": c}
    g = s["out_g"]
    if kind == "group":
        s["group"].fst_inv(s["gr"], c[0], c[1], g)
    elif kind == "split":
        p.inv_fst_real_f32(s["rc"], s["ic"], g[0], s["batch"], PREC[s["prec"]])
        p.fst_real_f32(s["gr"], c[0], c[1], s["batch"], PREC[s["prec"]])
    elif kind == "csplit":
        p.inv_fst_complex_f32(s["rc"], s["ic"], g[0], g[1], s["batch"], PREC[s["prec"]])
        p.fst_complex_f32(s["gr"], s["gi"], c[0], c[1], s["batch"], PREC[s["prec"]])
    else:
        p.inv_fst_real_f32_host_async(s["rc"], s["ic"], g, s["batch"], PREC[s["prec"]])
        p.fst_real_f32_host_async(g, c[0], c[1], s["batch"], PREC[s["prec"]])
        p.wait()
    return {"coeffs": c, "grid": g}


# ---- the work of one pass -------------------------------------------------------------------------
def _flops(bw):
    """One real function, one direction: row FFTs, per-order DCTs of both parts, triangular contraction."""
    S = 2 * bw
    fft = 2.5 * S * math.log2(S)
    return S * fft + 2 * bw * fft + 2 * 2 * bw ** 3 / 6


def work(case):
    kind = case["kind"]
    if kind == "group":
        bws = _group_bws(case)
        return {"bytes": 4 * sum(2 * 4 * b * b + 2 * b * b for b in bws), "flops": 2 * sum(_flops(b) for b in bws)}
    bw, nb = case["bw"], case.get("batch", 1)
    grid, coef = 4 * bw * bw, 2 * bw * bw
    if kind == "conv":  # data and filter in, field out; two analyses (one zonal) and a synthesis
        return {"bytes": 8 * 2 * (3 * grid), "flops": 2 * _flops(bw)}
    if kind == "refined":  # analysis, synthesis of the residual, its analysis
        return {"bytes": nb * 8 * (grid + coef), "flops": nb * 3 * _flops(bw)}
    two = 2 if kind == "csplit" or case.get("complex") else 1
    per = 8 if kind in ("memo", "f64") else 4
    imag = 2 if kind == "memo" else two  # the drop-ins take and give both parts
    return {"bytes": nb * per * 2 * (imag * grid + coef), "flops": nb * 2 * two * _flops(bw)}


# ---- the same in 64 bits ------------------------------------------------------------------------
# The Legendre functions come from the three-term recurrence in double-double arithmetic (Dekker's
# products, Knuth's sums), so that their own rounding does not show beside the library's.
def _dd(v):
    """A long-double array as a pair of doubles on the device."""
    hi = v.astype(np.float64)
    return tuple(torch.from_numpy(np.ascontiguousarray(p)).to(DEV) for p in (hi, (v - hi).astype(np.float64)))


def _two_prod(a, b):
    p = a * b
    t = a * 134217729.0
    ah = t - (t - a)
    t = b * 134217729.0
    bh = t - (t - b)
    al, bl = a - ah, b - bh
    return p, ((ah * bh - p) + ah * bl + al * bh) + al * bl


def _mul(a, b):
    p, e = _two_prod(a[0], b[0])
    e = e + (a[0] * b[1] + a[1] * b[0])
    s = p + e
    return s, e - (s - p)


def _sub(a, b):
    s = a[0] - b[0]
    t = s - a[0]
    e = (a[0] - (s - t)) - (b[0] + t) + (a[1] - b[1])
    r = s + e
    return r, e - (r - s)


def _legendre(bw):
    """L2-normalised P(m, l) at the 2 bw nodes, degree by degree: (l, [m <= l][nodes])."""
    ld = np.longdouble
    th = (np.arange(2 * bw).astype(ld) * 2 + 1) * (4 * np.arctan(ld(1))) / (4 * bw)
    x, st = _dd(np.cos(th)), _dd(np.sin(th))
    cur, prev = ([torch.zeros(bw, 2 * bw, device=DEV, dtype=torch.float64) for _ in range(2)] for _ in range(2))
    seed = tuple(torch.full((2 * bw,), float(v), device=DEV, dtype=torch.float64)
                 for v in (np.float64(np.sqrt(ld(0.5))), np.sqrt(ld(0.5)) - np.float64(np.sqrt(ld(0.5)))))
    for l in range(bw):
        if l:
            seed = _mul(seed, _mul(_dd(-np.sqrt(ld(2 * l + 1) / (2 * l)).reshape(1)), st))
        n = slice(0, l + 1)
        cur[0][l], cur[1][l] = seed
        yield l, cur[0][n]
        m = np.arange(l + 1).astype(ld)
        r = (2 * l + 3) / ((l + 1 - m) * (l + 1 + m))
        a, c = _dd(np.sqrt(r * (2 * l + 1))[:, None]), _dd(np.sqrt(r * ((l - m) * (l + m)) / max(1, 2 * l - 1))[:, None])
        now = (cur[0][n], cur[1][n])
        nxt = _sub(_mul(a, _mul(x, now)), _mul(c, (prev[0][n], prev[1][n])))
        for k in range(2):
            prev[k][n] = cur[k][n]
            cur[k][n] = nxt[k]


def _nodes(bw):
    return torch.arange(2 * bw, device=DEV, dtype=torch.float64).add(0.5).mul(math.pi / (2 * bw))


def _weights(bw):
    th = _nodes(bw)
    k = torch.arange(bw, device=DEV, dtype=torch.float64).mul(2).add(1)
    return 2 / bw * torch.sin(th) * (torch.sin(th[:, None] * k) / k).sum(dim=1)


def _slots_of(l, bw, sign):
    return torch.tensor([_index(sign * m, l, bw) for m in range(l + 1)], device=DEV)


def _rows(bw, cplx):
    m = torch.arange(bw, device=DEV)
    return m, (-m) % (2 * bw) if cplx else None


def _exact_fwd(gr, gi, bw, cplx):
    """Coefficients of samples [n][(2bw)^2]; real data: the negative orders by symmetry."""
    S, n = 2 * bw, gr.shape[0]
    out = torch.zeros(2, n, bw * bw, device=DEV, dtype=torch.float64)
    step = max(1, 2 ** 26 // (bw * S))
    w = _weights(bw) * (math.sqrt(2 * math.pi) / S)
    for at in range(0, n, step):
        z = gr[at:at + step].double().view(-1, S, S)
        z = torch.complex(z, torch.zeros_like(z) if gi is None else gi[at:at + step].double().view(-1, S, S))
        X = torch.fft.fft(z, dim=2) * w[:, None]
        c = X.shape[0]
        pos, neg = _rows(bw, cplx)
        X = X[:, :, pos if neg is None else torch.cat((pos, neg))]
        X = torch.view_as_real(X.permute(2, 1, 0).contiguous()).reshape(-1, S, 2 * c)
        for l, P in _legendre(bw):
            a = torch.bmm(P[:, None], X[:l + 1]).view(l + 1, c, 2)
            out[:, at:at + c, _slots_of(l, bw, 1)] = a.permute(2, 1, 0)
            sign = (1.0 - 2.0 * (torch.arange(l + 1, device=DEV) % 2)).double()
            if cplx:
                b = torch.bmm(P[:, None], X[bw:bw + l + 1]).view(l + 1, c, 2).permute(2, 1, 0) * sign
            else:
                b = a.permute(2, 1, 0) * torch.stack((sign, -sign))[:, None]
            out[:, at:at + c, _slots_of(l, bw, -1)[1:]] = b[:, :, 1:]
    return out


def _exact_inv(rc, ic, bw, cplx):
    """Samples [2 or 1][n][(2bw)^2] of coefficients [n][bw^2]; real data: from the orders m >= 0."""
    S, n = 2 * bw, rc.shape[0]
    out = torch.zeros(2, n, S * S, device=DEV, dtype=torch.float64)
    step = max(1, 2 ** 26 // (bw * S))
    for at in range(0, n, step):
        c = min(step, n - at)
        a = torch.stack((rc[at:at + c].double(), ic[at:at + c].double()), dim=2)
        F = torch.zeros(2, bw, S, 2 * c, device=DEV, dtype=torch.float64)
        for l, P in _legendre(bw):
            for half, sign in ((0, 1), (1, -1))[:2 if cplx else 1]:
                v = a[:, _slots_of(l, bw, sign)].permute(1, 0, 2).reshape(l + 1, 1, 2 * c)
                torch.baddbmm(F[half, :l + 1], P[:, :, None], v, out=F[half, :l + 1])
        F = torch.view_as_complex(F.view(2, bw, S, c, 2)) / math.sqrt(2 * math.pi)
        full = torch.zeros(c, S, S, device=DEV, dtype=torch.complex128)
        pos = F[0].permute(2, 1, 0)
        full[:, :, :bw] = pos
        if cplx:
            sign = (1.0 - 2.0 * (torch.arange(bw, device=DEV) % 2)).double()
            full[:, :, bw + 1:] = (F[1].permute(2, 1, 0) * sign)[:, :, 1:].flip(2)
        else:
            full[:, :, 0] = full[:, :, 0].real + 0j
            full[:, :, bw + 1:] = pos[:, :, 1:].conj().flip(2)
        g = torch.fft.ifft(full, dim=2) * S
        out[0, at:at + c], out[1, at:at + c] = g.real.reshape(c, -1), g.imag.reshape(c, -1)
    return out


def exact(case, seed):
    kind = case["kind"]
    coeffs, grid = _inputs(case, seed)
    if kind == "group":
        bws, at_g, at_c = _group_bws(case), 0, 0
        off = []
        for bw in bws:
            off.append((at_g, at_c))
            at_g, at_c = at_g + 4 * bw * bw, at_c + bw * bw
        out_g = torch.zeros(at_g, device=DEV, dtype=torch.float64)
        out_c = torch.zeros(2, at_c, device=DEV, dtype=torch.float64)
        for bw in sorted(set(bws)):
            idx = [i for i, b in enumerate(bws) if b == bw]
            g = torch.stack([grid[off[i][0]:off[i][0] + 4 * bw * bw] for i in idx]).float()
            c = _exact_fwd(g, None, bw, False)
            back = _exact_inv(c[0], c[1], bw, False)[0]
            for j, i in enumerate(idx):
                out_g[off[i][0]:off[i][0] + 4 * bw * bw] = back[j]
                out_c[:, off[i][1]:off[i][1] + bw * bw] = c[:, j]
        return {"coeffs": list(out_c), "grid": out_g}
    bw = case["bw"]
    if kind == "conv":
        l = _slot_lm(bw)[0]
        h = torch.from_numpy(_zonal_coeffs(bw)).to(DEV) * torch.sqrt(4 * math.pi / (
            2 * torch.arange(bw, device=DEV, dtype=torch.float64) + 1))
        c = _exact_fwd(grid, None, bw, False) * h[l]
        return {"grid": _exact_inv(c[0], c[1], bw, False)[:, 0]}
    if kind == "refined":
        return {"coeffs": list(_exact_fwd(grid, None, bw, False))}
    cplx = kind == "csplit" or case.get("complex", False)
    rc, ic = coeffs
    gr, gi = grid if grid is not None else (None, None)
    if kind in ("split", "csplit", "host"):
        rc, ic = rc.float(), ic.float()
        gr, gi = (None if x is None else x.float() for x in (gr, gi))
    g = _exact_inv(rc, ic, bw, cplx)
    if kind == "host":  # the forward takes the inverse's samples
        return {"coeffs": list(_exact_fwd(g[0], None, bw, False)), "grid": g[0]}
    c = _exact_fwd(gr, gi, bw, cplx)
    if kind == "memo":
        return {"coeffs": c[:, 0], "grid": g[:, 0]}
    return {"coeffs": list(c), "grid": list(g if cplx else g[:1])}
