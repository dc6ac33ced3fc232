"""The sparse products that programs ask of this library, as cases to be timed and compared.

A case is one way a program uses the library: a matrix family, its sizes, the value type and
the call.  ``prepare`` builds the matrices on the GPU and the handle, plan or batch such a
program keeps; ``run`` makes one pass through the public Python entry points.

Families (sizes vary freely in each):
  grid5      5-point operator of a 2-D grid, C = A*A: small finite-difference problems
  grid27     27-point operator of a 3-D grid, C = A*A: finite elements on structured grids
  web        web-like graph, C = A*A: power-law rows, half local and half popular columns
  er         uniform random graph, C = A*B: samples of graph batches, odd and rectangular sizes
  hubs       power-law graph times its transpose's pattern, C = A*B: similarity, with hub rows
  galerkin   27-point operator A, trilinear interpolation P, C = P^T (A P): multigrid set-up

Calls:
  oneshot    Handle.spgemm_oneshot: the library counts, allocates and computes C
  twophase   Handle.spgemm: symbolic and numeric phase, C in torch memory
  numeric    Handle.numeric on a pattern counted before: new values on a known pattern
  train      FixedPatternSpGEMM forward and backward through autograd: C, dA and dB
  batch      Batch: many er problems planned and computed together
  replay     Batch.execute of a planned batch as one graph launch: new values, same patterns
"""
import math

import numpy as np
import torch

import opsparse_gb300 as ops
from opsparse_gb300.autograd import FixedPatternSpGEMM

_DTYPES = {"f64": torch.float64, "f32": torch.float32}
_PATTERNS = 20261203  # seeds the patterns; a case's pattern is the case's, its values the seed's


def listed():
    return [
        # the smallest everyday call: a 128 x 128 finite-difference operator squared; its time
        # is the call's latency
        {"name": "grid5_128", "family": "grid5", "nx": 128, "ny": 128, "dtype": "f64", "call": "oneshot"},
        # a small random graph as graph learning samples them, through the two-phase call
        {"name": "er_small_f32", "family": "er", "rows": 2000, "inner": 2000, "cols": 2000, "deg_a": 8.0,
         "deg_b": 8.0, "dtype": "f32", "call": "twophase"},
        # the headline: a million-row web graph squared
        {"name": "web_1m", "family": "web", "rows": 1000000, "lmax": 4700, "dtype": "f64", "call": "oneshot"},
        # an ordinary web-like graph of odd size in single precision, two-phase
        {"name": "web_300k_f32", "family": "web", "rows": 300007, "lmax": 3000, "dtype": "f32", "call": "twophase"},
        # a large structured finite-element operator squared
        {"name": "grid27_80", "family": "grid27", "nx": 80, "ny": 80, "nz": 80, "dtype": "f64", "call": "oneshot"},
        # the same operator family reassembled with new values on a known pattern, ragged grid
        {"name": "grid27_numeric_f32", "family": "grid27", "nx": 61, "ny": 47, "nz": 53, "dtype": "f32",
         "call": "numeric"},
        # multigrid set-up: the Galerkin coarse operator of a ragged 3-D grid, two products
        {"name": "galerkin_57", "family": "galerkin", "nx": 57, "ny": 61, "nz": 59, "dtype": "f64",
         "call": "twophase"},
        # graph similarity with hub rows: rows of a handful of products beside rows of millions
        {"name": "hubs_200k", "family": "hubs", "rows": 200000, "deg": 16.0, "dtype": "f64", "call": "oneshot"},
        # a training step on that pattern: values forward, gradients of both factors back
        {"name": "train_hubs_200k", "family": "hubs", "rows": 200000, "deg": 16.0, "dtype": "f64", "call": "train"},
        # a training step on a rectangular random pattern in single precision
        {"name": "train_er_f32", "family": "er", "rows": 50021, "inner": 40009, "cols": 30011, "deg_a": 12.0,
         "deg_b": 10.0, "dtype": "f32", "call": "train"},
        # many independent graphs of very different sizes, planned and computed as one batch
        {"name": "batch_256_f32", "family": "er", "problems": 256, "lo": 64, "hi": 65536, "dmin": 4.0, "dmax": 32.0,
         "dtype": "f32", "call": "batch"},
        # a batch of small graphs replayed on new values
        {"name": "replay_100_f64", "family": "er", "problems": 100, "lo": 64, "hi": 4096, "dmin": 4.0, "dmax": 24.0,
         "dtype": "f64", "call": "replay"},
    ]


def _log_int(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))


def draw(rng):
    """One more case of the same families, calls, types and ranges."""
    kind = rng.choice(["grid5", "er", "web", "grid27", "galerkin", "hubs", "train", "batch", "replay"])
    dtype = rng.choice(["f64", "f32"])
    single = rng.choice(["oneshot", "twophase", "numeric"])
    if kind == "grid5":
        return {"family": "grid5", "nx": _log_int(rng, 32, 512), "ny": _log_int(rng, 32, 512), "dtype": dtype,
                "call": single}
    if kind == "er":
        return {"family": "er", "rows": _log_int(rng, 500, 100000), "inner": _log_int(rng, 500, 100000),
                "cols": _log_int(rng, 500, 200000), "deg_a": round(rng.uniform(2, 24), 2),
                "deg_b": round(rng.uniform(2, 24), 2), "dtype": dtype, "call": single}
    if kind == "web":
        return {"family": "web", "rows": _log_int(rng, 20000, 1000000), "lmax": _log_int(rng, 500, 4700),
                "dtype": dtype, "call": single}
    if kind == "grid27":
        return {"family": "grid27", "nx": _log_int(rng, 8, 80), "ny": _log_int(rng, 8, 80),
                "nz": _log_int(rng, 8, 80), "dtype": dtype, "call": single}
    if kind == "galerkin":
        return {"family": "galerkin", "nx": _log_int(rng, 8, 64), "ny": _log_int(rng, 8, 64),
                "nz": _log_int(rng, 8, 64), "dtype": dtype, "call": rng.choice(["oneshot", "twophase"])}
    if kind == "hubs":
        return {"family": "hubs", "rows": _log_int(rng, 5000, 200000), "deg": round(rng.uniform(4, 16), 2),
                "dtype": dtype, "call": single}
    if kind == "train":
        if rng.random() < 0.5:
            return {"family": "hubs", "rows": _log_int(rng, 5000, 200000), "deg": round(rng.uniform(4, 16), 2),
                    "dtype": dtype, "call": "train"}
        return {"family": "er", "rows": _log_int(rng, 2000, 100000), "inner": _log_int(rng, 2000, 100000),
                "cols": _log_int(rng, 2000, 100000), "deg_a": round(rng.uniform(2, 16), 2),
                "deg_b": round(rng.uniform(2, 16), 2), "dtype": dtype, "call": "train"}
    lo = _log_int(rng, 64, 512)
    hi = _log_int(rng, 1024, 32768 if kind == "batch" else 8192)
    return {"family": "er", "problems": _log_int(rng, 10, 160), "lo": lo, "hi": hi, "dmin": 4.0,
            "dmax": round(rng.uniform(8, 28), 2), "dtype": dtype, "call": kind}


# ------------------------------------------------------------------------------ matrices --
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _generator(seed, device):
    return torch.Generator(device=device).manual_seed(int(seed))


def _csr(keys, rows, cols):
    """Row pointers and columns (int32) of sorted unique keys row * cols + col."""
    r = torch.div(keys, cols, rounding_mode="floor")
    rpt = torch.zeros(rows + 1, dtype=torch.int64, device=keys.device)
    rpt[1:] = torch.cumsum(torch.bincount(r, minlength=rows), 0)
    return rpt.to(torch.int32), (keys - r * cols).to(torch.int32)


def _axis(n, device):
    return torch.arange(n, device=device, dtype=torch.int64)


def _grid_keys(dims, offsets, device):
    """Sorted keys of the operator coupling each grid point to the points at `offsets`."""
    n = math.prod(dims)
    idx = _axis(n, device)
    coord, rest = [], idx
    for d in reversed(dims):
        coord.insert(0, rest % d)
        rest = torch.div(rest, d, rounding_mode="floor")
    parts = []
    for off in offsets:
        ok = torch.ones(n, dtype=torch.bool, device=device)
        col = torch.zeros(n, dtype=torch.int64, device=device)
        for x, o, d in zip(coord, off, dims):
            ok &= (x + o >= 0) & (x + o < d)
            col = col * d + x + o
        parts.append(idx[ok] * n + col[ok])
    return torch.sort(torch.cat(parts)).values


def _grid5(case, gen, device):
    dims = (case["nx"], case["ny"])
    n = math.prod(dims)
    rpt, col = _csr(_grid_keys(dims, ((-1, 0), (0, -1), (0, 0), (0, 1), (1, 0)), device), n, n)
    # diffusion coefficients that vary over the grid: negative couplings, dominant diagonal
    val = -0.5 - torch.rand(col.numel(), generator=gen, device=device, dtype=torch.float64)
    rows = torch.repeat_interleave(_axis(n, device), (rpt[1:] - rpt[:-1]).long())
    return rpt, col, torch.where(rows == col, 6.0 - val, val), n, n


def _grid27(case, gen, device):
    dims = (case["nx"], case["ny"], case["nz"])
    n = math.prod(dims)
    offsets = [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)]
    rpt, col = _csr(_grid_keys(dims, offsets, device), n, n)
    return rpt, col, torch.randn(col.numel(), generator=gen, device=device, dtype=torch.float64), n, n


def _interpolation(case, device):
    """Trilinear interpolation from every second grid point: 1, 2, 4 or 8 weights a row."""
    dims = (case["nx"], case["ny"], case["nz"])
    coarse = tuple((d + 1) // 2 for d in dims)
    n, nc = math.prod(dims), math.prod(coarse)
    idx = _axis(n, device)
    x = [torch.div(idx, dims[1] * dims[2], rounding_mode="floor"),
         torch.div(idx, dims[2], rounding_mode="floor") % dims[1], idx % dims[2]]
    keys, vals = [], []
    for up in [(a, b, c) for a in (0, 1) for b in (0, 1) for c in (0, 1)]:
        ok = torch.ones(n, dtype=torch.bool, device=device)
        col = torch.zeros(n, dtype=torch.int64, device=device)
        w = torch.ones(n, dtype=torch.float64, device=device)
        for xi, u, d in zip(x, up, coarse):
            odd = xi % 2 == 1
            c = torch.div(xi, 2, rounding_mode="floor") + u
            ok &= (c < d) & (odd | (u == 0))
            w = w * torch.where(odd, 0.5, 1.0)
            col = col * d + c
        keys.append(idx[ok] * nc + col[ok])
        vals.append(w[ok])
    keys, order = torch.sort(torch.cat(keys))
    rpt, col = _csr(keys, n, nc)
    return rpt, col, torch.cat(vals)[order], n, nc


def _transposed(m):
    rpt, col, val, rows, cols = m
    r = torch.repeat_interleave(_axis(rows, rpt.device), (rpt[1:] - rpt[:-1]).long())
    keys, order = torch.sort(col.long() * rows + r)
    trpt, tcol = _csr(keys, cols, rows)
    return trpt, tcol, val[order], cols, rows


def _web(case, gen, device):
    """Power-law row lengths (exponent 2.1); half the columns within 512 of the row, half by
    popularity (Zipf, exponent 1, over a random ranking).  The thousand most popular pages
    link to at most 16 others: a draw's cost does not hang on the length of one of them."""
    m, lmax = case["rows"], min(case["lmax"], case["rows"])
    values, gen = gen, _generator(_PATTERNS, device)
    cdf = torch.cumsum(torch.arange(1, lmax + 1, device=device, dtype=torch.float64) ** -2.1, 0)
    u = torch.rand(m, generator=gen, device=device, dtype=torch.float64)
    lens = torch.searchsorted(cdf / cdf[-1], u).clamp(max=lmax - 1) + 1
    ranking = torch.randperm(m, generator=gen, device=device)
    lens[ranking[:1000]] = lens[ranking[:1000]].clamp(max=16)
    rows = torch.repeat_interleave(_axis(m, device), lens)
    n = rows.numel()
    near = (rows + torch.randint(-512, 513, (n,), generator=gen, device=device)).clamp(0, m - 1)
    pop = torch.cumsum(torch.arange(1, m + 1, device=device, dtype=torch.float64) ** -1.0, 0)
    u = torch.rand(n, generator=gen, device=device, dtype=torch.float64)
    far = ranking[torch.searchsorted(pop / pop[-1], u).clamp(max=m - 1)]
    local = torch.rand(n, generator=gen, device=device) < 0.5
    rpt, col = _csr(torch.unique(rows * m + torch.where(local, near, far)), m, m)
    return rpt, col, torch.rand(col.numel(), generator=values, device=device, dtype=torch.float64), m, m


def _uniform(rows, cols, deg, gen, values, device):
    """Each row draws Poisson(deg) columns uniformly, duplicates removed, values N(0,1)."""
    lam = torch.full((rows,), float(deg), device=device)
    d = torch.poisson(lam, generator=gen).long().clamp(max=cols)
    r = torch.repeat_interleave(_axis(rows, device), d)
    c = torch.randint(0, cols, (r.numel(),), generator=gen, device=device)
    rpt, col = _csr(torch.unique(r * cols + c), rows, cols)
    return rpt, col, torch.randn(col.numel(), generator=values, device=device, dtype=torch.float64), rows, cols


def _hubs(case, gen, device):
    """Power-law degrees (exponent 2.2) scaled to the mean, uniform columns, values N(0,1)."""
    n = case["rows"]
    values, gen = gen, _generator(_PATTERNS, device)
    u = torch.rand(n, generator=gen, device=device, dtype=torch.float64)
    raw = (1.0 - u) ** (-1.0 / 1.2)
    deg = torch.round(raw * case["deg"] / raw.mean()).long().clamp(1, n)
    deg = deg.clamp(max=max(1, int(0.15 * n)))  # the largest hub knows at most 15% of the nodes
    r = torch.repeat_interleave(_axis(n, device), deg)
    c = torch.randint(0, n, (r.numel(),), generator=gen, device=device)
    rpt, col = _csr(torch.unique(r * n + c), n, n)
    return rpt, col, torch.randn(col.numel(), generator=values, device=device, dtype=torch.float64), n, n


def _sizes(case):
    """Sizes (log-spaced) and mean degrees of a batch's problems, in a mixed order."""
    r = np.random.default_rng(case["problems"])
    t = (np.arange(case["problems"]) + 0.5) / case["problems"]
    sizes = np.floor(case["lo"] * (case["hi"] / case["lo"]) ** t).astype(np.int64)
    degs = case["dmin"] + (case["dmax"] - case["dmin"]) * r.permutation(t)
    order = r.permutation(case["problems"])
    return [int(n) for n in sizes[order]], [float(d) for d in degs[order]]


def _batch_side(sizes, degs, gen, values, device):
    """One factor of every problem: [(rpt, col, val, n, n)], values N(0,1)."""
    ns = torch.tensor(sizes, device=device)
    n_of_row = torch.repeat_interleave(ns, ns)
    lam = torch.repeat_interleave(torch.tensor(degs, device=device, dtype=torch.float32), ns)
    d = torch.minimum(torch.poisson(lam, generator=gen).long(), n_of_row)
    rows = torch.repeat_interleave(_axis(n_of_row.numel(), device), d)
    width = max(sizes)
    u = torch.rand(rows.numel(), generator=gen, device=device, dtype=torch.float64)
    rpt, col = _csr(torch.unique(rows * width + (u * n_of_row[rows]).long()), n_of_row.numel(), width)
    val = torch.randn(col.numel(), generator=values, device=device, dtype=torch.float64)
    first = np.concatenate([[0], np.cumsum(sizes)])
    cut = rpt[torch.as_tensor(first, device=device)].cpu().numpy()
    return [(rpt[first[i]:first[i + 1] + 1] - int(cut[i]), col[cut[i]:cut[i + 1]].clone(),
             val[cut[i]:cut[i + 1]].clone(), n, n) for i, n in enumerate(sizes)]


def _factors(case, seed, device):
    """[(A, B), ...]: the products of the case in order, each factor (rpt, col, val, rows,
    cols) with 64-bit values; a galerkin case gives A and P of its first product."""
    gen, pattern = _generator(seed, device), _generator(_PATTERNS, device)
    family = case["family"]
    if "problems" in case:
        sizes, degs = _sizes(case)
        return list(zip(_batch_side(sizes, degs, pattern, gen, device), _batch_side(sizes, degs, pattern, gen, device)))
    if family == "er":
        return [(_uniform(case["rows"], case["inner"], case["deg_a"], pattern, gen, device),
                 _uniform(case["inner"], case["cols"], case["deg_b"], pattern, gen, device))]
    if family == "hubs":
        a = _hubs(case, gen, device)
        b = _transposed(a)
        return [(a, b[:2] + (torch.randn(b[2].numel(), generator=gen, device=device, dtype=torch.float64),) + b[3:])]
    if family == "galerkin":
        return [(_grid27(case, gen, device), _interpolation(case, device))]
    a = {"grid5": _grid5, "grid27": _grid27, "web": _web}[family](case, gen, device)
    return [(a, a)]


def _typed(m, case):
    """The factor with its values in the case's type (what a program holds)."""
    return m[:2] + (m[2].to(_DTYPES[case["dtype"]]),) + m[3:]


def _matrix(m):
    rpt, col, val, rows, cols = m
    return ops.CsrMatrix(rows, cols, rpt, col, val)


# ---------------------------------------------------------------------------------- passes --
def prepare(case, seed):
    pairs = []
    for a, b in _factors(case, seed, "cuda"):
        ma = _matrix(_typed(a, case))
        pairs.append((ma, ma if b is a else _matrix(_typed(b, case))))
    state = {"case": case, "handle": ops.Handle(), "pairs": pairs}
    A, B = pairs[0]
    call = case["call"]
    if case["family"] == "galerkin":
        state["R"] = _matrix(_typed(_transposed(_interpolation(case, "cuda")), case))
    if call == "numeric":
        state["rpt"], state["nnz"] = state["handle"].symbolic(A, B)
    elif call == "train":
        op = FixedPatternSpGEMM(A, B, state["handle"])
        gen = _generator(seed + 1, "cuda")
        state["op"] = op
        state["dc"] = torch.randn(op.nnz, generator=gen, device="cuda", dtype=torch.float64).to(A.val.dtype)
        state["a"] = A.val.clone().requires_grad_(True)
        state["b"] = B.val.clone().requires_grad_(True)
    elif call == "replay":
        batch = ops.Batch(state["handle"], pairs)
        batch.execute(True)
        batch.check()
        state["batch"] = batch
        state["views"] = [batch.result_device(i) for i in range(batch.n)]
    return state


def _arrays(C):
    return C.rpt, C.col, C.val


def run(state):
    case, h = state["case"], state["handle"]
    A, B = state["pairs"][0]
    call = case["call"]
    if call == "train":
        c = state["op"](state["a"], state["b"])
        return c.detach(), *torch.autograd.grad(c, (state["a"], state["b"]), state["dc"])
    if call == "numeric":
        return h.numeric(A, B, state["rpt"], state["nnz"])
    if call == "batch":
        batch = ops.Batch(h, state["pairs"])
        batch.execute(False)
        batch.check()
        views = [batch.result_device(i) for i in range(batch.n)]
        out = tuple(torch.cat([v[k] for v in views]) for k in range(3))
        torch.cuda.current_stream().synchronize()  # the views are the batch's memory
        batch.close()
        return out
    if call == "replay":
        state["batch"].execute(True)
        state["batch"].check()
        return tuple(torch.cat([v[k] for v in state["views"]]) for k in (1, 2))
    multiply = h.spgemm_oneshot if call == "oneshot" else h.spgemm
    if case["family"] == "galerkin":
        ap = multiply(A, B)
        return _arrays(ap) + _arrays(multiply(state["R"], ap))
    return _arrays(multiply(A, B))


# ------------------------------------------------------------------------- what is needed --
def _expand(a, b):
    """The products of A*B in A's order: A entry, B entry and key row * cols + column."""
    arpt, acol, _, rows, _ = a
    brpt, bcol, _, _, cols = b
    dev = arpt.device
    j = acol.long()
    count = (brpt[j + 1] - brpt[j]).long()
    e = torch.repeat_interleave(_axis(acol.numel(), dev), count)
    first = torch.cumsum(count, 0) - count
    q = brpt[j].long()[e] + _axis(e.numel(), dev) - first[e]
    r = torch.repeat_interleave(_axis(rows, dev), (arpt[1:] - arpt[:-1]).long())
    return e, q, r[e] * cols + bcol[q].long()


def _counts(a, b):
    """(products, entries of C)."""
    _, _, key = _expand(a, b)
    return key.numel(), torch.unique(key).numel()


def _distinct(n, draws):
    """Expected distinct values of `draws` uniform draws from n."""
    return n * -math.expm1(draws * math.log1p(-1.0 / n)) if n > 1 else min(1.0, draws)


def _er_counts(rows, inner, cols, deg_a, deg_b):
    """Expected entries of A and B, products, and entries of C of an er product."""
    da = _distinct(inner, deg_a)
    db = _distinct(cols, deg_b)
    return rows * da, inner * db, rows * da * db, rows * _distinct(cols, da * db)


def _one(rows, inner, nnz_a, nnz_b, nnz_c, vs, same):
    """Bytes of one product: A, B and C, each once (A is B in a square)."""
    a = 4 * (rows + 1) + (4 + vs) * nnz_a
    b = 0 if same else 4 * (inner + 1) + (4 + vs) * nnz_b
    return a + b + 4 * (rows + 1) + (4 + vs) * nnz_c


def work(case):
    vs = 8 if case["dtype"] == "f64" else 4
    family, call = case["family"], case["call"]
    if family == "er":
        if "problems" in case:
            shapes = [(n, n, n, d, d) for n, d in zip(*_sizes(case))]
        else:
            shapes = [(case["rows"], case["inner"], case["cols"], case["deg_a"], case["deg_b"])]
        per = [(s[0], s[1]) + _er_counts(*s) for s in shapes]
    elif family == "grid27":
        dims = (case["nx"], case["ny"], case["nz"])
        n = math.prod(dims)
        nnz, products, entries = (math.prod(max(f(d), 1) for d in dims)
                                  for f in (lambda d: 3 * d - 2, lambda d: 9 * d - 10, lambda d: 5 * d - 6))
        per = [(n, n, nnz, nnz, products, entries)]
    else:
        a, b = _factors(case, 0, _device())[0]
        per = [(a[3], a[4], a[1].numel(), b[1].numel()) + _counts(a, b)]
        if family == "galerkin":
            r, (rpt, col, _) = _transposed(b), _product(a, b)
            ap = (rpt, col, None, a[3], b[4])
            per.append((r[3], r[4], r[1].numel(), col.numel()) + _counts(r, ap))
    same = family in ("grid5", "grid27", "web")
    nbytes = sum(_one(m, k, na, nb, nc, vs, same) for m, k, na, nb, _, nc in per)
    flops = 2.0 * sum(p[4] for p in per)
    if call == "train":  # backward: dC and both factors again, dA and dB out
        nbytes += sum((4 + vs) * nc + 2 * vs * (na + nb) + 4 * (na + nb) for _, _, na, nb, _, nc in per)
        flops *= 3
    return {"bytes": float(nbytes), "flops": float(flops)}


# ---------------------------------------------------------------------------- exact values --
def _product(a, b):
    """Row pointers, columns and 64-bit values of A*B by expanding and sorting."""
    e, q, key = _expand(a, b)
    keys, pos = torch.unique(key, return_inverse=True)
    rpt, col = _csr(keys, a[3], b[4])
    val = torch.zeros(keys.numel(), dtype=torch.float64, device=keys.device)
    val.index_add_(0, pos, a[2][e].double() * b[2][q].double())
    return rpt, col, val


def exact(case, seed):
    call = case["call"]
    pairs = [(_typed(a, case), _typed(b, case)) for a, b in _factors(case, seed, "cuda")]
    if "problems" in case:
        done = [_product(a, b) for a, b in pairs]
        return tuple(torch.cat([d[k] for d in done]) for k in ((1, 2) if call == "replay" else (0, 1, 2)))
    a, b = pairs[0]
    if call == "train":
        e, q, key = _expand(a, b)
        _, pos = torch.unique(key, return_inverse=True)
        n = int(pos.max()) + 1
        dc = torch.randn(n, generator=_generator(seed + 1, "cuda"), device="cuda", dtype=torch.float64)
        dc = dc.to(a[2].dtype).double()[pos]
        av, bv = a[2].double(), b[2].double()
        return (torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, pos, av[e] * bv[q]),
                torch.zeros_like(av).index_add_(0, e, bv[q] * dc), torch.zeros_like(bv).index_add_(0, q, av[e] * dc))
    rpt, col, val = _product(a, b)
    if case["family"] == "galerkin":
        # the second product starts from the computed A P, rounded to the case's type
        ap = (rpt, col, val.to(_DTYPES[case["dtype"]]), a[3], b[4])
        return (rpt, col, val) + _product(_transposed(b), ap)
    return (col, val) if call == "numeric" else (rpt, col, val)
