"""Performance cases of the SpGEMM engine: what a program asks of it through
its public entry points (the Python binding of the C ABI), over the ranges
those calls are made with.

Inputs are made on the GPU from the seed, with the row-length, column and value
distributions of this repository's benchmark workloads: uniform rows, skewed
lognormal rows around a diagonal band, and the Galerkin chain of a 7-point
operator (seeded cell coefficients) under 2x2x2 aggregation.
"""
from __future__ import annotations

import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
if str(ROOT / "spgemm-hpc-thesis_gb300") not in sys.path:
    sys.path.insert(0, str(ROOT / "spgemm-hpc-thesis_gb300"))

import spgemm_gb300 as sg  # noqa: E402

DEV = "cuda:0"


def listed():
    return [
        # the coarsest level of a multigrid hierarchy: one call of a few thousand products, all latency
        {"name": "galerkin_16", "kind": "galerkin", "nx": 16, "ny": 16, "nz": 16},
        # the smallest request of a batched or served stream, alone: long rows, few of them
        {"name": "uniform_1000", "kind": "uniform", "rows": 1000, "inner": 1000, "cols": 1000, "lo": 4, "hi": 64},
        # the ordinary product: 65,536 rows of 16 entries
        {"name": "uniform_65536", "kind": "uniform", "rows": 65536, "inner": 65536, "cols": 65536, "lo": 16, "hi": 16},
        # skewed rows (a graph or circuit squared) at an odd size
        {"name": "powerlaw_100003", "kind": "powerlaw", "rows": 100003},
        # the same at the benchmark's size, the largest call
        {"name": "powerlaw_1M", "kind": "powerlaw", "rows": 1 << 20},
        # R*A and (R*A)*R^T on the finest grid: millions of very short rows
        {"name": "galerkin_128", "kind": "galerkin", "nx": 128, "ny": 128, "nz": 128},
        # independent uneven products in one call
        {"name": "batch_16", "kind": "batch", "count": 16, "rows_lo": 1000, "rows_hi": 20000, "lo": 4, "hi": 64,
         "sizes": 4},
        # R*A re-formed with new coefficients: one plan, replayed
        {"name": "plan_galerkin", "kind": "plan", "nx": 96, "ny": 80, "nz": 112},
        # a block's partial products summed over the stages of a block algorithm; rows in file order with
        # repeated columns, as a Matrix Market file may hold them
        {"name": "accumulate_4", "kind": "accumulate", "rows": 32771, "inner": 8192, "cols": 40009, "stages": 4,
         "lo": 2, "hi": 14},
        # the layout for products whose upper bound would not fit: rows counted first
        {"name": "exact_131071", "kind": "exact", "rows": 131071},
        # host operands to host result, the drop-in path of a host program
        {"name": "to_host_65539", "kind": "to_host", "rows": 65539},
        # A^T of a skewed matrix
        {"name": "transpose_524287", "kind": "transpose", "rows": 524287, "cols": 524287},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["galerkin", "uniform", "powerlaw", "batch", "plan", "accumulate", "exact", "to_host",
                       "transpose"])
    if kind in ("galerkin", "plan"):
        return {"kind": kind, **{k: 2 * _log(rng, 8, 64) for k in ("nx", "ny", "nz")}}
    if kind == "uniform":
        lo = rng.randint(1, 24)
        return {"kind": kind, "rows": _log(rng, 1000, 200000), "inner": _log(rng, 1000, 200000),
                "cols": _log(rng, 1000, 200000), "lo": lo, "hi": rng.randint(lo, 64),
                "file_order": rng.random() < 0.25}
    if kind == "powerlaw":
        return {"kind": kind, "rows": _log(rng, 4096, 1 << 20)}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(2, 20), "rows_lo": 1000, "rows_hi": _log(rng, 4000, 20000),
                "lo": 4, "hi": 64, "sizes": rng.randint(1, 1 << 20)}
    if kind == "accumulate":
        return {"kind": kind, "rows": _log(rng, 1000, 65536), "inner": _log(rng, 1000, 32768),
                "cols": _log(rng, 1000, 65536), "stages": rng.randint(2, 6), "lo": 2, "hi": rng.randint(4, 20)}
    if kind == "exact":
        return {"kind": kind, "rows": _log(rng, 4096, 262144)}
    if kind == "to_host":
        return {"kind": kind, "rows": _log(rng, 4096, 131072)}
    return {"kind": "transpose", "rows": _log(rng, 4096, 1 << 20), "cols": _log(rng, 4096, 1 << 20)}


# ---------------------------------------------------------------------------
# Inputs (torch, on the GPU)

# A case's sparsity is drawn once for its sizes; a seed then shifts rows and
# columns cyclically (every seed has other rows, and as many stored entries in
# every product) and draws the values.

def _gen(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + salt)


def _shift(seed, salt, n):
    return random.Random(int(seed) * 31 + salt).randrange(n)


def _from_rows(rows, cols, r, c, g, val=None):
    rp = torch.zeros(rows + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(torch.bincount(r, minlength=rows), 0, out=rp[1:])
    if val is None:
        val = torch.rand(c.numel(), dtype=torch.float64, device=DEV, generator=g) * 2 - 1
    return sg.DeviceCsr(rows, cols, rp, c.to(torch.int32), val)


def _placed(rows, cols, r, c, shifts, seed, salt, file_order):
    """Rows and columns shifted; distinct sorted columns in every row, or the
    drawn order with repeated columns."""
    if not file_order:
        key = torch.unique(r * cols + c)
        r = torch.div(key, cols, rounding_mode="floor")
        c = key - r * cols
    r, c = (r + shifts[0]) % rows, (c + shifts[1]) % cols
    at = torch.argsort(r, stable=True) if file_order else torch.argsort(r * cols + c)
    return _from_rows(rows, cols, r[at], c[at], _gen(seed, salt))


def _uniform(rows, cols, lo, hi, seed, salt, shifts, file_order=False):
    """Row lengths uniform in [lo, hi], uniform columns."""
    g = _gen(1, salt)
    lens = torch.randint(lo, hi + 1, (rows,), device=DEV, generator=g)
    r = torch.repeat_interleave(torch.arange(rows, device=DEV), lens)
    c = torch.randint(0, cols, (r.numel(),), device=DEV, generator=g)
    return _placed(rows, cols, r, c, shifts, seed, salt, file_order)


def _pair(case, sizes, seed, salt, outer, file_order=False):
    """A and B of one uniform product; their inner dimension shifts alike."""
    rows, inner, cols = sizes
    k = _shift(seed, salt, inner)
    return (_uniform(rows, inner, case["lo"], case["hi"], seed, salt, (outer[0], k), file_order),
            _uniform(inner, cols, case["lo"], case["hi"], seed, salt + 1, (k, outer[1]), file_order))


def _powerlaw(rows, cols, seed, salt):
    """Lognormal row lengths (mean 24, sigma 1.2, capped at 20,000), 70% of the
    columns within +-2,048 of the diagonal, the rest anywhere."""
    g = _gen(1, salt)
    mu = math.log(24.0) - 0.5 * 1.2 * 1.2
    lens = torch.exp(mu + 1.2 * torch.randn(rows, dtype=torch.float64, device=DEV, generator=g))
    lens = lens.round().clamp(1, min(20000, cols)).to(torch.int64)
    r = torch.repeat_interleave(torch.arange(rows, device=DEV), lens)
    u = torch.rand(r.numel(), dtype=torch.float64, device=DEV, generator=g)
    centre = torch.div(r * cols, rows, rounding_mode="floor")
    first, last = (centre - 2048).clamp(min=0), (centre + 2048).clamp(max=cols - 1)
    band = first + (u * (last - first + 1)).to(torch.int64)
    anywhere = (u * cols).to(torch.int64)
    in_band = torch.rand(r.numel(), device=DEV, generator=g) < 0.7
    k = _shift(seed, salt, rows)
    return _placed(rows, cols, r, torch.where(in_band, band, anywhere), (k, k if rows == cols else k * cols // rows),
                   seed, salt, False)


def _operator(nx, ny, nz, seed):
    """7-point operator on an nx x ny x nz grid: off-diagonals minus the mean of
    two seeded cell coefficients, the diagonal their sum with fixed walls."""
    g = _gen(seed)
    k = torch.rand(nz, ny, nx, dtype=torch.float64, device=DEV, generator=g) + 0.5
    i = torch.arange(nx * ny * nz, device=DEV).reshape(nz, ny, nx)
    n = nx * ny * nz
    rows, cols, vals = [], [], []
    diag = torch.zeros_like(k)
    for d in range(3):
        m = k.shape[d]
        lo, hi = i.narrow(d, 0, m - 1), i.narrow(d, 1, m - 1)
        f = (k.narrow(d, 0, m - 1) + k.narrow(d, 1, m - 1)) * 0.5
        diag.narrow(d, 0, m - 1).add_(f)
        diag.narrow(d, 1, m - 1).add_(f)
        diag.narrow(d, 0, 1).add_(k.narrow(d, 0, 1))
        diag.narrow(d, m - 1, 1).add_(k.narrow(d, m - 1, 1))
        rows += [lo.reshape(-1), hi.reshape(-1)]
        cols += [hi.reshape(-1), lo.reshape(-1)]
        vals += [-f.reshape(-1), -f.reshape(-1)]
    r = torch.cat(rows + [i.reshape(-1)])
    c = torch.cat(cols + [i.reshape(-1)])
    v = torch.cat(vals + [diag.reshape(-1)])
    at = torch.argsort(r * n + c)
    return _from_rows(n, n, r[at], c[at], None, v[at])


def _restriction(nx, ny, nz):
    """2x2x2 aggregation (8 entries of 1/8 per row) and its transpose."""
    n, m = nx * ny * nz, nx * ny * nz // 8
    i = torch.arange(n, device=DEV)
    x, y, z = i % nx, torch.div(i, nx, rounding_mode="floor") % ny, torch.div(i, nx * ny, rounding_mode="floor")
    half = lambda t: torch.div(t, 2, rounding_mode="floor")  # noqa: E731
    coarse = (half(z) * (ny // 2) + half(y)) * (nx // 2) + half(x)
    at = torch.argsort(coarse * n + i)
    eighth = torch.full((n,), 0.125, dtype=torch.float64, device=DEV)
    return (_from_rows(m, n, coarse[at], i[at], None, eighth), _from_rows(n, m, i, coarse, None, eighth.clone()))


def _batch_sizes(case):
    r = random.Random(case["sizes"])
    return [_log(r, case["rows_lo"], case["rows_hi"]) for _ in range(case["count"])]


def _operands(case, seed):
    """The (A, B) products of a pass, in order."""
    kind = case["kind"]
    if kind == "uniform":
        outer = _shift(seed, 5, case["rows"]), _shift(seed, 6, case["cols"])
        return [_pair(case, (case["rows"], case["inner"], case["cols"]), seed, 1, outer, bool(case.get("file_order")))]
    if kind in ("powerlaw", "exact", "to_host"):
        a = _powerlaw(case["rows"], case["rows"], seed, 3)
        return [(a, a)]
    if kind in ("galerkin", "plan"):
        r, rt = _restriction(case["nx"], case["ny"], case["nz"])
        a = _operator(case["nx"], case["ny"], case["nz"], seed)
        return [(r, a), (None, rt)] if kind == "galerkin" else [(r, a)]
    if kind == "batch":
        return [_pair(case, (n, n, n), seed, 10 + 2 * i, (_shift(seed, 100 + i, n), _shift(seed, 200 + i, n)))
                for i, n in enumerate(_batch_sizes(case))]
    if kind == "accumulate":
        outer = _shift(seed, 5, case["rows"]), _shift(seed, 6, case["cols"])
        return [_pair(case, (case["rows"], case["inner"], case["cols"]), seed, 50 + 2 * i, outer, True)
                for i in range(case["stages"])]
    return [(_powerlaw(case["rows"], case["cols"], seed, 90), None)]  # transpose


# ---------------------------------------------------------------------------
# A pass

_engines: dict = {}


def _engine(mode="auto"):
    """The program's engine handle, made once."""
    if mode not in _engines:
        _engines[mode] = sg.Engine(0, mode=mode)
    return _engines[mode]


class _Array:
    """Device memory of a result as torch takes it; keeps the result alive."""

    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (int(n),), "typestr": typestr, "data": (int(ptr or 0), False),
                                         "version": 2}


def _tensor(owner, ptr, n, typestr, dtype):
    if n == 0:
        return torch.empty(0, dtype=dtype, device=DEV)
    return torch.as_tensor(_Array(owner, ptr, n, typestr), device=DEV)


def _arrays(owner, rows, nnz, ptrs):
    return {"row_ptr": _tensor(owner, ptrs[0], rows + 1, "<i8", torch.int64),
            "col": _tensor(owner, ptrs[1], nnz, "<i4", torch.int32),
            "val": _tensor(owner, ptrs[2], nnz, "<f8", torch.float64)}


def _result(res):
    return _arrays(res, res.rows, res.nnz, res.pointers)


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h


def prepare(case, seed):
    kind = case["kind"]
    ops = _operands(case, seed)
    st = {"kind": kind, "ops": ops, "engine": _engine("exact" if kind == "exact" else "auto"), "case": dict(case)}
    if kind == "plan":
        torch.cuda.synchronize()
        st["plan"] = st["engine"].plan(ops)
    if kind == "to_host":
        a = ops[0][0]
        n = int((a.row_ptr[1:] - a.row_ptr[:-1])[a.col.long()].sum())
        st["host"] = sg.Csr(a.rows, a.cols, *(_pinned(t).numpy() for t in (a.row_ptr, a.col, a.val)))
        st["out"] = (torch.empty(a.rows + 1, dtype=torch.int64, pin_memory=True),
                     torch.empty(n, dtype=torch.int32, pin_memory=True),
                     torch.empty(n, dtype=torch.float64, pin_memory=True))
    torch.cuda.synchronize()
    return st


def run(st):
    kind, ops, eng = st["kind"], st["ops"], st["engine"]
    if kind in ("uniform", "powerlaw", "exact"):
        return _result(eng.multiply(*ops[0], out="device"))
    if kind == "galerkin":
        (r, a), (_, rt) = ops
        ra = _result(eng.multiply(r, a, out="device"))
        rar = eng.multiply(sg.DeviceCsr(r.rows, a.cols, ra["row_ptr"], ra["col"], ra["val"]), rt, out="device")
        return {"ra": ra, "rar": _result(rar)}
    if kind == "batch":
        return [_result(r) for r in eng.multiply_batch(ops, out="device")]
    if kind == "plan":
        plan = st["plan"]
        plan.execute()
        res = sg._Result()
        if sg.library().spg_plan_result(plan.p, 0, sg.C.byref(res)) != 0:
            raise RuntimeError("spg_plan_result failed")
        return _arrays(plan, res.rows, res.nnz, (res.row_ptr, res.col, res.val))
    if kind == "accumulate":
        return _result(eng.accumulate(st["case"]["rows"], st["case"]["cols"], ops, out="device"))
    if kind == "to_host":
        rp, ci, va = st["out"]
        nnz = eng.multiply_to_host(st["host"], st["host"], rp, ci, va)
        return {"row_ptr": rp, "col": ci[:nnz], "val": va[:nnz]}
    return _result(eng.transpose(ops[0][0], out="device"))


# ---------------------------------------------------------------------------
# What a pass cannot do without (expected sizes; inputs once, outputs once)

def _uniform_sizes(rows, inner, cols, lo, hi):
    """Entries of A and B, products and stored entries of one uniform product."""
    mean = 0.5 * (lo + hi)
    p = mean * mean
    return rows * mean, inner * mean, rows * p, rows * cols * (1.0 - math.exp(-p / cols))


def _csr_bytes(rows, nnz):
    return 8.0 * (rows + 1) + 12.0 * nnz


def work(case):
    kind = case["kind"]
    if kind in ("uniform", "batch"):
        sizes = [(case["rows"], case["inner"], case["cols"])] if kind == "uniform" else [(n, n, n) for n in _batch_sizes(case)]
        b = f = 0.0
        for rows, inner, cols in sizes:
            na, nb, p, nc = _uniform_sizes(rows, inner, cols, case["lo"], case["hi"])
            b += _csr_bytes(rows, na) + _csr_bytes(inner, nb) + _csr_bytes(rows, nc)
            f += 2 * p
        return {"bytes": b, "flops": f}
    if kind == "accumulate":
        na, nb, p, _ = _uniform_sizes(case["rows"], case["inner"], case["cols"], case["lo"], case["hi"])
        s = case["stages"]
        nc = case["rows"] * case["cols"] * (1.0 - math.exp(-s * p / case["rows"] / case["cols"]))
        return {"bytes": s * (_csr_bytes(case["rows"], na) + _csr_bytes(case["inner"], nb)) + _csr_bytes(case["rows"], nc),
                "flops": 2 * s * p}
    if kind in ("powerlaw", "exact", "to_host"):
        n = case["rows"]
        return {"bytes": _csr_bytes(n, 24.0 * n) + _csr_bytes(n, 0.95 * 576.0 * n), "flops": 2 * 576.0 * n}
    if kind in ("galerkin", "plan"):
        n = case["nx"] * case["ny"] * case["nz"]
        m = n // 8
        b = _csr_bytes(m, n) + _csr_bytes(n, 7.0 * n) + _csr_bytes(m, 32.0 * m)
        f = 2 * 7.0 * n
        if kind == "galerkin":
            b += _csr_bytes(n, n) + _csr_bytes(m, 7.0 * m)
            f += 2 * 32.0 * m
        return {"bytes": b, "flops": f}
    n = 24.0 * case["rows"]
    return {"bytes": _csr_bytes(case["rows"], n) + _csr_bytes(case["cols"], n), "flops": 0.0}


# ---------------------------------------------------------------------------
# The same in plain 64-bit torch

def _exact_sum(rows, cols, pairs):
    """Sum of A*B over the pairs: sorted rows, zeros dropped."""
    total = torch.zeros(rows, dtype=torch.int64, device=DEV)
    for a, b in pairs:
        w = (b.row_ptr[1:] - b.row_ptr[:-1])[a.col.long()]
        c = torch.zeros(a.nnz + 1, dtype=torch.int64, device=DEV)
        torch.cumsum(w, 0, out=c[1:])
        total += c[a.row_ptr[1:]] - c[a.row_ptr[:-1]]
    ends = torch.cumsum(total, 0).cpu().numpy()
    ks, vs, r0 = [], [], 0
    while r0 < rows:
        done = int(ends[r0 - 1]) if r0 else 0
        r1 = max(r0 + 1, int(np.searchsorted(ends, done + 50_000_000, side="right")))
        keys, vals = [], []
        for a, b in pairs:
            p0, p1 = int(a.row_ptr[r0]), int(a.row_ptr[r1])
            ac = a.col[p0:p1].long()
            start, n = b.row_ptr[ac], b.row_ptr[ac + 1] - b.row_ptr[ac]
            e = torch.repeat_interleave(torch.arange(p1 - p0, device=DEV), n)
            q = torch.arange(e.numel(), device=DEV) - (torch.cumsum(n, 0) - n)[e] + start[e]
            lens = a.row_ptr[r0 + 1:r1 + 1] - a.row_ptr[r0:r1]
            row = torch.repeat_interleave(torch.arange(r0, r1, device=DEV), lens)
            keys.append(row[e] * cols + b.col[q])
            vals.append(a.val[p0:p1][e] * b.val[q])
        key, inv = torch.unique(torch.cat(keys), return_inverse=True)
        val = torch.zeros(key.numel(), dtype=torch.float64, device=DEV).index_add_(0, inv, torch.cat(vals))
        ks.append(key[val != 0])
        vs.append(val[val != 0])
        r0 = r1
    key, val = torch.cat(ks), torch.cat(vs)
    r = torch.div(key, cols, rounding_mode="floor")
    m = _from_rows(rows, cols, r, key - r * cols, None, val)
    return m


def _as_dict(m):
    return {"row_ptr": m.row_ptr, "col": m.col, "val": m.val}


def exact(case, seed):
    kind, ops = case["kind"], _operands(case, seed)
    if kind == "galerkin":
        (r, a), (_, rt) = ops
        ra = _exact_sum(r.rows, a.cols, [(r, a)])
        return {"ra": _as_dict(ra), "rar": _as_dict(_exact_sum(ra.rows, rt.cols, [(ra, rt)]))}
    if kind == "accumulate":
        return _as_dict(_exact_sum(case["rows"], case["cols"], ops))
    if kind == "batch":
        return [_as_dict(_exact_sum(a.rows, b.cols, [(a, b)])) for a, b in ops]
    if kind == "transpose":
        a = ops[0][0]
        row = torch.repeat_interleave(torch.arange(a.rows, device=DEV), a.row_ptr[1:] - a.row_ptr[:-1])
        at = torch.argsort(a.col, stable=True)
        return _as_dict(_from_rows(a.cols, a.rows, a.col[at].long(), row[at], None, a.val[at]))
    a, b = ops[0]
    out = _as_dict(_exact_sum(a.rows, b.cols, [(a, b)]))
    return {k: v.cpu() for k, v in out.items()} if kind == "to_host" else out
