"""Workloads of the library's public entry points, as a user's program calls them.

Every case is one call of the Python API on operands that such a program has in
hand: plain products from a few hundred rows to millions, graph (power-law),
uniform and mesh (27-point stencil) matrices, FP64 and FP32, the host entry
point, the Galerkin triple product, the transpose, a planned product replayed
after its values changed, and a packed batch.  Operands are made on the GPU
from the seed alone; ``exact`` gives the same results in 64 bits by expanding,
sorting and summing the products with torch.

A case's fields: ``op`` (product, host, rap, transpose, plan, batch), ``kind``
(uniform, rect, powerlaw, stencil, aggregation, blocks), ``dtype`` (f64, f32),
the sizes that the kind takes and, for random structures, ``graph``, which
says which random structure of that kind it is.  The seed numbers the
structure's rows and columns (a rotation of the indices, so the sizes of a
case's operands and results do not change) and gives the values.
"""
import math

import numpy as np
import torch

from gpuspgemm_b200 import api

DEV = "cuda"
GRAPH = 20261203


def listed():
    return [
        # the smallest calls: a coarse-grid or unit-test sized rectangular product
        {"name": "rect_300x500x200_f64", "op": "product", "kind": "rect", "dtype": "f64",
         "m": 300, "k": 500, "n": 200, "per_row": 4, "graph": GRAPH},
        # a small square product with evenly filled rows (4096 rows of 8)
        {"name": "uniform_4096x8_f64", "op": "product", "kind": "uniform", "dtype": "f64",
         "n": 4096, "per_row": 8, "graph": GRAPH},
        # a medium graph, as a request stream holds them
        {"name": "powerlaw_30k_f32", "op": "product", "kind": "powerlaw", "dtype": "f32",
         "n": 30000, "exponent": 2.0, "cap": 4700, "graph": GRAPH},
        # host operands in, host result out: copies both ways inside the call
        {"name": "host_powerlaw_200k_f64", "op": "host", "kind": "powerlaw", "dtype": "f64",
         "n": 200003, "exponent": 2.0, "cap": 4700, "graph": GRAPH},
        # the benchmark's graph squared, in both value types
        {"name": "powerlaw_1m_f64", "op": "product", "kind": "powerlaw", "dtype": "f64",
         "n": 1000000, "exponent": 2.0, "cap": 4700, "graph": GRAPH},
        {"name": "powerlaw_1m_f32", "op": "product", "kind": "powerlaw", "dtype": "f32",
         "n": 1000000, "exponent": 2.0, "cap": 4700, "graph": GRAPH},
        # a graph with more columns than the narrow (2^20-column) kernels take
        {"name": "powerlaw_wide_2m_f64", "op": "product", "kind": "powerlaw", "dtype": "f64",
         "n": 2097159, "exponent": 2.0, "cap": 4700, "graph": GRAPH},
        # a mesh operator squared: six products fall on each entry of C
        {"name": "stencil_60_f32", "op": "product", "kind": "stencil", "dtype": "f32",
         "nx": 60, "ny": 60, "nz": 60},
        # multigrid setup: R * (A * P) with R = P^T formed on the device
        {"name": "rap_100_f64", "op": "rap", "kind": "aggregation", "dtype": "f64",
         "nx": 100, "ny": 100, "nz": 100, "agg": 3},
        # a graph transposed (skewed column counts)
        {"name": "transpose_powerlaw_1m_f32", "op": "transpose", "kind": "powerlaw", "dtype": "f32",
         "n": 1000000, "exponent": 2.0, "cap": 4700, "graph": GRAPH},
        # a time stepper's A * P: structure planned once, values new at each step
        {"name": "plan_stencil_64_f64", "op": "plan", "kind": "aggregation", "dtype": "f64",
         "nx": 64, "ny": 64, "nz": 64, "agg": 3},
        # independent small products run as one packed batch
        {"name": "batch_20_f32", "op": "batch", "kind": "blocks", "dtype": "f32",
         "count": 20, "rows_lo": 64, "rows_hi": 16384, "lam_lo": 6.0, "lam_hi": 40.0,
         "graph": GRAPH},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    dtype = rng.choice(["f64", "f32"])
    seed = rng.randrange(1 << 30)
    op = rng.choice(["rect", "uniform", "powerlaw", "powerlaw", "powerlaw", "wide", "stencil",
                     "host", "rap", "transpose", "plan", "batch"])
    if op == "rect":
        return {"op": "product", "kind": "rect", "dtype": dtype, "m": _log(rng, 100, 20000),
                "k": _log(rng, 100, 20000), "n": _log(rng, 100, 20000),
                "per_row": rng.randint(2, 16), "graph": seed}
    if op == "uniform":
        return {"op": "product", "kind": "uniform", "dtype": dtype, "n": _log(rng, 500, 200000),
                "per_row": rng.randint(3, 16), "graph": seed}
    graph = {"kind": "powerlaw", "dtype": dtype, "n": _log(rng, 10000, 1000000),
             "exponent": round(rng.uniform(2.0, 2.4), 2), "cap": 4700, "graph": seed}
    if op == "wide":
        return {**graph, "op": "product", "n": rng.randint(1048577, 2097159)}
    if op in ("powerlaw", "host", "transpose"):
        if op == "host":
            graph["n"] = _log(rng, 10000, 200003)
        return {**graph, "op": "product" if op == "powerlaw" else op}
    if op == "batch":
        return {"op": "batch", "kind": "blocks", "dtype": dtype, "count": rng.randint(5, 20),
                "rows_lo": 64, "rows_hi": _log(rng, 1000, 16384), "lam_lo": 6.0,
                "lam_hi": 40.0, "graph": seed}
    hi = {"stencil": 60, "rap": 100, "plan": 64}[op]
    grid = {"nx": rng.randint(20, hi), "ny": rng.randint(20, hi), "nz": rng.randint(20, hi)}
    if op == "stencil":
        return {"op": "product", "kind": "stencil", "dtype": dtype, **grid}
    return {"op": op, "kind": "aggregation", "dtype": dtype, **grid, "agg": rng.choice([2, 3])}


# ---- operands --------------------------------------------------------------
# An operand is (m, n, rpt, col, val): int32 row pointer and columns (sorted
# and distinct per row) and float64 values, rounded to the case's type where
# they are used.

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _uniform(g, n, lo, hi):
    return torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * (hi - lo) + lo


def _from_pairs(m, n, rows, cols, val_of):
    """CSR from (row, column) pairs in any order, duplicates dropped."""
    keys = torch.unique(rows * n + cols)
    rows = keys // n
    rpt = torch.zeros(m + 1, dtype=torch.int64, device=DEV)
    rpt[1:] = torch.cumsum(torch.bincount(rows, minlength=m), 0)
    return m, n, rpt.int(), (keys % n).int(), val_of(keys.numel())


def _random_pairs(g, m, n, per_row):
    """per_row uniform columns (some twice) in each of m rows."""
    rows = torch.arange(m, device=DEV).repeat_interleave(min(per_row, n))
    return rows, torch.randint(0, n, rows.shape, generator=g, device=DEV)


def _power_law_pairs(g, n, exponent, cap, block=2000):
    """Row degrees ~ Zipf(exponent) on [1, cap]; columns by preferential
    attachment (a target is drawn in proportion to 1 + its in-degree before
    the block)."""
    cap = min(cap, n)
    p = torch.arange(1, cap + 1, device=DEV, dtype=torch.float64) ** (-exponent)
    cdf = torch.cumsum(p / p.sum(), 0)
    deg = torch.searchsorted(cdf, _uniform(g, n, 0.0, 1.0), right=True).clamp_(max=cap - 1) + 1
    ends = torch.cumsum(deg, 0)
    stops = ends[block - 1::block].tolist()
    total = int(ends[-1])
    if not stops or stops[-1] != total:
        stops.append(total)
    past = torch.empty(total, dtype=torch.int64, device=DEV)
    at = 0
    for stop in stops:
        idx = torch.randint(0, n + at, (stop - at,), generator=g, device=DEV)
        past[at:stop] = torch.where(idx >= n, past[(idx - n).clamp_(min=0)], idx)
        at = stop
    return torch.arange(n, device=DEV).repeat_interleave(deg, output_size=total), past


def _grid(nx, ny, nz):
    i = torch.arange(nx * ny * nz, device=DEV)
    return i, i % nx, (i // nx) % ny, i // (nx * ny)


def _stencil(g, nx, ny, nz):
    """27-point operator on an nx x ny x nz grid with varying coefficients."""
    i, x, y, z = _grid(nx, ny, nz)
    n = nx * ny * nz
    rows, cols = [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                ok = ((x + dx >= 0) & (x + dx < nx) & (y + dy >= 0) & (y + dy < ny) &
                      (z + dz >= 0) & (z + dz < nz))
                rows.append(i[ok])
                cols.append((i + (dz * ny + dy) * nx + dx)[ok])
    m, _, rpt, col, val = _from_pairs(n, n, torch.cat(rows), torch.cat(cols),
                                      lambda k: _uniform(g, k, -1.5, -0.5))
    rows = i.repeat_interleave((rpt[1:] - rpt[:-1]).long())
    val[rows == col] = _uniform(g, n, 25.0, 27.0)
    return m, n, rpt, col, val


def _aggregation(g, nx, ny, nz, agg):
    """Smoothed aggregation: each fine point reaches its own agg^3 block and the
    blocks one step away along the axes, weights U[0.1, 1]."""
    i, x, y, z = _grid(nx, ny, nz)
    ax, ay, az = (max(v // agg, 1) for v in (nx, ny, nz))
    nc = ax * ay * az
    rows, cols = [], []
    for dx, dy, dz in ((0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1),
                       (0, 0, -1), (1, 1, 0)):
        u, v, w = x + dx, y + dy, z + dz
        ok = (u >= 0) & (u < nx) & (v >= 0) & (v < ny) & (w >= 0) & (w < nz)
        c = ((w // agg).clamp(max=az - 1) * ay + (v // agg).clamp(max=ay - 1)) * ax + \
            (u // agg).clamp(max=ax - 1)
        rows.append(i[ok])
        cols.append(c[ok])
    return _from_pairs(nx * ny * nz, nc, torch.cat(rows), torch.cat(cols),
                       lambda k: _uniform(g, k, 0.1, 1.0))


def _blocks(case, seed):
    """A batch's block-diagonal operands: (row offsets, A, B) of `count`
    square pairs, rows log-uniform, nnz per row ~ Poisson(U[lam_lo, lam_hi])."""
    g, gs = _gen(case["graph"]), _gen(seed)
    u = _uniform(g, 2 * case["count"], 0.0, 1.0).cpu().numpy()
    lo, hi = math.log(case["rows_lo"]), math.log(case["rows_hi"])
    sizes = np.exp(lo + u[:case["count"]] * (hi - lo)).astype(np.int64)
    lams = case["lam_lo"] + u[case["count"]:] * (case["lam_hi"] - case["lam_lo"])
    off = np.concatenate([[0], np.cumsum(sizes)])
    n = int(off[-1])
    block = torch.arange(case["count"], device=DEV).repeat_interleave(
        torch.from_numpy(sizes).to(DEV))
    size = torch.from_numpy(sizes).to(DEV)[block]
    first = torch.from_numpy(off[:-1].copy()).to(DEV)[block]
    lam = torch.from_numpy(lams).to(DEV)[block]
    turn = torch.randint(0, 1 << 30, (case["count"],), generator=gs, device=DEV)[block] % size

    def turned(i):  # an index of a block, rotated inside the block
        return first[i] + (i - first[i] + turn[i]) % size[i]

    def one():
        cnt = torch.minimum(torch.poisson(lam, generator=g).long(), size)
        rows = torch.arange(n, device=DEV).repeat_interleave(cnt)
        cols = first[rows] + (_uniform(g, rows.numel(), 0.0, 1.0) * size[rows]).long()
        return _from_pairs(n, n, turned(rows), turned(cols), lambda k: _uniform(gs, k, -1.0, 1.0))

    return off, one(), one()


def _operands(case, seed):
    """The case's operands in 64 bits: (A, B)."""
    gs = _gen(seed)
    kind = case["kind"]
    if kind in ("stencil", "aggregation"):
        a = _stencil(gs, case["nx"], case["ny"], case["nz"])
        return a, a if kind == "stencil" else _aggregation(gs, case["nx"], case["ny"],
                                                           case["nz"], case["agg"])
    g = _gen(case["graph"])
    if kind == "rect":
        m, k, n = case["m"], case["k"], case["n"]
        ar, ac = _random_pairs(g, m, k, case["per_row"])
        br, bc = _random_pairs(g, k, n, case["per_row"])
        s, t, u = torch.randint(0, 1 << 30, (3,), generator=gs, device=DEV).tolist()
        return (_from_pairs(m, k, (ar + s) % m, (ac + t) % k, lambda c: _uniform(gs, c, -1.0, 1.0)),
                _from_pairs(k, n, (br + t) % k, (bc + u) % n, lambda c: _uniform(gs, c, -1.0, 1.0)))
    n = case["n"]
    if kind == "uniform":
        (rows, cols), lo = _random_pairs(g, n, n, case["per_row"]), -1.0
    else:
        (rows, cols), lo = _power_law_pairs(g, n, case["exponent"], case["cap"]), 0.0
    s = int(torch.randint(0, n, (1,), generator=gs, device=DEV))
    a = _from_pairs(n, n, (rows + s) % n, (cols + s) % n, lambda c: _uniform(gs, c, lo, 1.0))
    return a, a


def _later_values(case, seed, count):
    """A planned product's values of A at a later step."""
    return _uniform(_gen(seed + 1000003), count, -1.5, 1.5)


def _dtype(case):
    return torch.float64 if case["dtype"] == "f64" else torch.float32


def _csr(case, x):
    m, n, rpt, col, val = x
    return api.DeviceCSR(m, n, rpt, col, val.to(_dtype(case)))


def prepare(case, seed):
    op = case["op"]
    if op == "batch":
        off, a, b = _blocks(case, seed)
        off = off.astype(np.int32)
        return {"op": op, "batch": api.PackedBatch(off, off.copy(), off.copy(), _csr(case, a),
                                                   _csr(case, b))}
    a, b = _operands(case, seed)
    A = _csr(case, a)
    B = A if b is a else _csr(case, b)
    if op == "host":
        A = A.to_host()
        return {"op": op, "A": A, "B": A}
    state = {"op": op, "A": A, "B": B}
    if op == "plan":
        state["plan"] = api.plan(A, B)
        A.val.copy_(_later_values(case, seed, A.nnz))
    return state


def _out(c):
    return {"rpt": c.rpt, "col": c.col, "val": c.val}


def run(state):
    op = state["op"]
    if op == "product":
        return _out(api.proposal(state["A"], state["B"]))
    if op == "host":
        return _out(api.proposal_host(state["A"], state["B"]))
    if op == "rap":
        return _out(api.rap(state["A"], state["B"]))
    if op == "transpose":
        return _out(api.transpose(state["A"]))
    if op == "plan":
        state["plan"].execute()
        return _out(state["plan"].result)
    return [_out(c) for c in api.batch(state["batch"])]


# ---- the same in 64 bits, and the work -------------------------------------

def _round(case, x):
    m, n, rpt, col, val = x
    return m, n, rpt, col, val.to(_dtype(case)).double()


def _nip(a, b):
    blen = (b[2][1:] - b[2][:-1]).long()
    return int(blen[a[3].long()].sum())


def _multiply(a, b, limit=1 << 26):
    """a * b: every product expanded, sorted by (row, column) and summed, in
    row chunks of at most `limit` products."""
    m, _, art, acol, aval = a
    _, n, brt, bcol, bval = b
    blen = (brt[1:] - brt[:-1]).long()
    per_entry = blen[acol.long()]
    entry_row = torch.arange(m, device=DEV).repeat_interleave((art[1:] - art[:-1]).long())
    done = torch.cumsum(torch.zeros(m, dtype=torch.int64, device=DEV).index_add_(
        0, entry_row, per_entry), 0)
    rpt = torch.zeros(m + 1, dtype=torch.int64, device=DEV)
    cols, vals = [], []
    r0 = before = 0
    while r0 < m:
        r1 = int(torch.searchsorted(done, before + limit, right=True))
        r1 = min(max(r1, r0 + 1), m)
        e0, e1 = int(art[r0]), int(art[r1])
        cnt = per_entry[e0:e1]
        total = int(cnt.sum())
        first = torch.cumsum(cnt, 0) - cnt
        ent = torch.arange(e0, e1, device=DEV).repeat_interleave(cnt, output_size=total)
        pos = torch.arange(total, device=DEV) - first[ent - e0] + brt[acol[ent].long()].long()
        keys, order = torch.sort(entry_row[ent] * n + bcol[pos].long(), stable=True)
        prod = (aval[ent] * bval[pos])[order]
        keys, inverse = torch.unique_consecutive(keys, return_inverse=True)
        vals.append(torch.zeros(keys.numel(), dtype=torch.float64, device=DEV).index_add_(
            0, inverse, prod))
        cols.append((keys % n).int())
        rpt[1:] += torch.bincount(keys // n, minlength=m)
        before = int(done[r1 - 1])
        r0 = r1
    return m, n, torch.cumsum(rpt, 0).int(), torch.cat(cols), torch.cat(vals)


def _transposed(a):
    m, n, rpt, col, val = a
    rows = torch.arange(m, device=DEV).repeat_interleave((rpt[1:] - rpt[:-1]).long())
    order = torch.sort(col.long() * m + rows)[1]
    out = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    out[1:] = torch.cumsum(torch.bincount(col.long(), minlength=n), 0)
    return n, m, out.int(), rows[order].int(), val[order]


def _as_out(c):
    return {"rpt": c[2], "col": c[3], "val": c[4]}


def _split(c, off):
    """The products of a block-diagonal result, with local indices."""
    parts = []
    for r0, r1 in zip(off[:-1].tolist(), off[1:].tolist()):
        e0, e1 = int(c[2][r0]), int(c[2][r1])
        parts.append({"rpt": c[2][r0:r1 + 1] - e0, "col": c[3][e0:e1] - r0, "val": c[4][e0:e1]})
    return parts


def exact(case, seed):
    op = case["op"]
    if op == "batch":
        off, a, b = _blocks(case, seed)
        return _split(_multiply(_round(case, a), _round(case, b)), off)
    a, b = (_round(case, x) for x in _operands(case, seed))
    if op == "transpose":
        return _as_out(_transposed(a))
    if op == "plan":
        a = _round(case, a[:4] + (_later_values(case, seed, a[4].numel()),))
    if op == "rap":
        return _as_out(_multiply(_transposed(b), _multiply(a, b)))
    c = _as_out(_multiply(a, b))
    return {k: v.cpu().numpy() for k, v in c.items()} if op == "host" else c


def work(case):
    """Each operand read once, each result written once; two operations per
    product."""
    size = 4 + (8 if case["dtype"] == "f64" else 4)  # bytes of an entry

    def bytes_of(*mats):
        return sum(4 * (x[0] + 1) + size * x[3].numel() for x in mats)

    op = case["op"]
    if op == "batch":
        _, a, b = _blocks(case, 1)
    else:
        a, b = _operands(case, 1)
    if op == "transpose":
        return {"bytes": bytes_of(a) + 4 * (a[1] + 1) + size * a[3].numel(), "flops": 0}
    c = _multiply(a, b)
    products = _nip(a, b)
    inputs = [a] if b is a else [a, b]
    if op == "rap":
        # the intermediate A * P and P^T stay inside the call
        r = _transposed(b)
        products += _nip(r, c)
        c = _multiply(r, c)
    return {"bytes": bytes_of(*inputs, c), "flops": 2 * products}
