"""What a program does with this library, as cases that can be timed and checked.

Every case is one call (or one burst of calls) of the public Python entry points on
device-resident inputs made from a seed.  The kinds:

  lu      one delayed-pivoting LU of an m x n matrix (``getrf_device_ex``), factored in place
  ir      mixed-precision factorisation and refined solve (``gesv_ir_device``)
  batch   independent LUs of uneven orders in one persistent launch (``Batch.getrf_graph``)
  solve   a refined solve with resident factors (``Factor.solve``)
  ldlt    delayed Bunch-Kaufman LDL^T of a symmetric matrix (``sytrf_device``)
  front   partial LU of a multifrontal front (``front_factor``)
  serve   a burst of factor + solve requests and follow-up solves through a ``Server``

Factorisations work in place, so a pass of ``lu``, ``batch``, ``ldlt`` and ``front`` copies the
matrix first, as a program that still needs A (for residuals, for refinement) does.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "delayed-pivoting_b200"))
import delayed_pivoting as dp  # noqa: E402

DEV = "cuda"
F64 = torch.float64
TINY = 1e-18


def listed():
    return [
        # a small dense block, as a caller's inner loop factors: launches and latency
        {"name": "lu_100", "kind": "lu", "m": 100, "n": 100, "lda": 104, "tiny": 0, "zero": 0},
        # the known-answer workload: tiny columns and exact-zero columns, delays and fallbacks
        {"name": "lu_1024_delayed", "kind": "lu", "m": 1024, "n": 1024, "lda": 1024, "tiny": 16, "zero": 4},
        # a ragged tall block with padded columns (a front's fully-summed columns)
        {"name": "lu_3001x1537", "kind": "lu", "m": 3001, "n": 1537, "lda": 3008, "tiny": 2, "zero": 1},
        # the largest order of the served stream
        {"name": "lu_8192", "kind": "lu", "m": 8192, "n": 8192, "lda": 8192, "tiny": 8, "zero": 0},
        # the single-matrix benchmark: 0.1 % tiny and 0.02 % zero columns
        {"name": "lu_16384_delayed", "kind": "lu", "m": 16384, "n": 16384, "lda": 16384, "tiny": 16, "zero": 3},
        # mixed-precision factorisation with FP64 refinement, a few right-hand sides
        {"name": "ir_10000", "kind": "ir", "n": 10000, "nrhs": 4, "log_kappa": 3.0, "terms": 3},
        # the batched benchmark: 8192 matrices of orders log-uniform in [32, 512]
        {"name": "batch_8192", "kind": "batch", "count": 8192, "lo": 32, "hi": 512, "shape_seed": 1},
        # follow-up solves on resident factors: one vector, and a block of them
        {"name": "solve_4096_rhs1", "kind": "solve", "n": 4096, "nrhs": 1, "log_kappa": 2.0},
        {"name": "solve_2311_rhs32", "kind": "solve", "n": 2311, "nrhs": 32, "log_kappa": 4.0},
        # a symmetric indefinite system of ordinary size with two empty nodes
        {"name": "ldlt_3000", "kind": "ldlt", "n": 3000, "zero": 2},
        # a front half of whose rows are fully summed
        {"name": "front_4096", "kind": "front", "m": 4096, "n": 4096, "p": 2048, "zero": 1},
        # a served burst: requests of mixed orders arriving together
        {"name": "serve_48", "kind": "serve", "count": 48, "lo": 64, "hi": 4096, "shape_seed": 1},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["lu", "lu", "lu", "ir", "batch", "batch", "solve", "solve", "ldlt", "front", "serve"])
    if kind == "lu":
        n = log_int(64, 12000)
        m = n if rng.random() < 0.6 else max(64, min(12000, int(n * rng.uniform(0.5, 2.0))))
        return {"kind": kind, "m": m, "n": n, "lda": m + rng.choice([0, 0, 1, 8]),
                "tiny": rng.randrange(4), "zero": rng.choice([0, 0, 1, 2])}
    if kind == "ir":
        return {"kind": kind, "n": log_int(600, 10000), "nrhs": rng.choice([1, 3, 8, 33, 64]),
                "log_kappa": round(rng.uniform(1.5, 3.5), 2), "terms": rng.choice([2, 3, 3])}
    if kind == "batch":
        lo = log_int(16, 96)
        return {"kind": kind, "count": log_int(48, 6000), "lo": lo, "hi": min(512, lo * rng.choice([2, 4, 16])),
                "shape_seed": rng.randrange(1 << 20)}
    if kind == "solve":
        return {"kind": kind, "n": log_int(520, 9000), "nrhs": rng.choice([1, 2, 5, 16, 32, 64]),
                "log_kappa": round(rng.uniform(1.5, 4.0), 2)}
    if kind == "ldlt":
        return {"kind": kind, "n": log_int(200, 6000), "zero": rng.randrange(3)}
    if kind == "front":
        m = log_int(500, 6000)
        n = m if rng.random() < 0.7 else int(m * rng.uniform(0.8, 1.0))
        return {"kind": kind, "m": m, "n": n, "p": max(1, int(min(m, n) * rng.uniform(0.2, 0.8))),
                "zero": rng.randrange(2)}
    return {"kind": kind, "count": rng.randrange(16, 64), "lo": 64, "hi": log_int(600, 4096),
            "shape_seed": rng.randrange(1 << 20)}


# ---- inputs ---------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape):
    return torch.randn(*shape, dtype=F64, device=DEV, generator=g)


def _dct(x):
    """Orthonormal DCT-II along the last dimension."""
    n = x.shape[-1]
    v = torch.cat([x[..., ::2], x[..., 1::2].flip(-1)], -1)
    k = torch.arange(n, dtype=F64, device=x.device)
    y = (torch.fft.fft(v) * torch.polar(torch.ones_like(k), -math.pi * k / (2 * n))).real
    y *= math.sqrt(2.0 / n)
    y[..., 0] *= math.sqrt(0.5)
    return y


def _conditioned(g, n, log_kappa):
    """n x n matrix U diag(sigma) V^T with orthogonal U, V (permuted and signed cosine
    transforms) and sigma geometric from 1 to 10^-log_kappa."""
    s = torch.logspace(0, -log_kappa, n, dtype=F64, device=DEV)
    signs = torch.randint(0, 2, (2, n), device=DEV, generator=g).to(F64) * 2 - 1
    p, q = (torch.randperm(n, device=DEV, generator=g) for _ in range(2))
    a = torch.zeros(n, n, dtype=F64, device=DEV)
    a[p, q] = s
    a = _dct(a) * signs[0]
    return (_dct(a.T.contiguous()) * signs[1]).contiguous()


def _planted(g, m, n, lda, tiny, zero):
    """Storage of an m x n N(0, 1) matrix, column-major: row j of the (n, lda) tensor is column
    j.  `tiny` columns scaled by 1e-18 and `zero` columns cleared, at seeded places."""
    a = _randn(g, n, lda)
    at = torch.randperm(n, device=DEV, generator=g)
    a[at[:tiny]] *= TINY
    a[at[tiny:tiny + zero]] = 0.0
    return a


def _batch_shapes(case):
    """Orders, and per matrix the columns that are exactly zero (0-2 of them)."""
    r = np.random.default_rng(case["shape_seed"])
    lo, hi = case["lo"], case["hi"]
    ns = np.floor(np.exp(r.uniform(math.log(lo), math.log(hi + 1), case["count"])))
    ns = np.clip(ns, lo, hi).astype(np.int32)
    zeros = (r.random((2, case["count"])) < 0.3).sum(0)
    return ns, [r.choice(n, min(z, n), replace=False) if z else [] for n, z in zip(ns, zeros)]


def _serve_shapes(case):
    """(order, right-hand sides of the first solve, right-hand sides of its follow-ups)."""
    r = np.random.default_rng(case["shape_seed"])
    out = []
    for _ in range(case["count"]):
        n = int(round(math.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        out.append((n, int(r.integers(1, 33)), [int(v) for v in r.integers(1, 33, r.integers(0, 5))]))
    return out


def _inputs(case, seed):
    g, kind = _gen(seed), case["kind"]
    if kind == "lu":
        return {"a": _planted(g, case["m"], case["n"], case["lda"], case["tiny"], case["zero"])}
    if kind in ("ir", "solve"):
        n = case["n"]
        a = _conditioned(g, n, case["log_kappa"])
        x = _randn(g, case["nrhs"], n)
        return {"a": a, "b": x @ a}  # a's storage is the transpose: B^T = X^T A^T
    if kind == "batch":
        ns, zeros = _batch_shapes(case)
        offsets = np.concatenate([[0], np.cumsum((ns.astype(np.int64) ** 2 + 3) & ~3)])
        base = _randn(g, int(offsets[-1]))
        clear = []
        for n, first, columns in zip(ns.astype(np.int64), offsets, zeros):
            clear += [np.arange(first + c * n, first + (c + 1) * n) for c in columns]
        if clear:
            base[torch.from_numpy(np.concatenate(clear)).to(DEV)] = 0.0
        return {"ns": ns, "offsets": offsets, "base": base}
    if kind == "ldlt":
        n = case["n"]
        a = _randn(g, n, n).tril_()
        a = a + a.tril(-1).T
        at = torch.randperm(n, device=DEV, generator=g)[:case["zero"]]
        a[at] = 0.0
        a[:, at] = 0.0
        return {"a": a.contiguous()}
    if kind == "front":
        a = _randn(g, case["n"], case["m"])
        p = case["p"]
        at = torch.randperm(p, device=DEV, generator=g)[:case["zero"]]
        a[at, :p] = 0.0  # a fully-summed column with no pivot in its block
        return {"a": a}
    mats, rhs = [], []
    for n, first, more in _serve_shapes(case):
        a = _conditioned(g, n, 2.0 + 2.0 * float(torch.rand(1, generator=g, device=DEV)))
        mats.append(a)
        rhs.append([_randn(g, k, n) @ a for k in [first] + more])
    return {"mats": mats, "rhs": rhs}


def prepare(case, seed):
    s = dict(_inputs(case, seed), case=case, kind=case["kind"])
    kind = s["kind"]
    if kind in ("lu", "ldlt", "front"):
        s["work"] = torch.empty_like(s["a"])
    if kind in ("ir", "solve"):
        s["x"] = torch.empty_like(s["b"])
    if kind == "lu":
        k = min(case["m"], case["n"])
        s["ipiv"], s["jpiv"] = np.zeros(k, dtype=np.int32), np.zeros(k, dtype=np.int32)
    if kind == "solve":
        s["factor"] = dp.Factor(case["n"], s["a"], case["n"], precision=dp.PRECISION_FP64)
    if kind == "batch":
        s["plan"] = dp.Batch(s["ns"])
        assert np.array_equal(s["plan"].offsets, s["offsets"][:-1])
        s["work"] = torch.empty_like(s["base"])
        s["ipiv"] = torch.empty(s["plan"].total_records, dtype=torch.int32, device=DEV)
        s["jpiv"] = torch.empty_like(s["ipiv"])
        s["info"] = torch.empty(case["count"], dtype=torch.int32, device=DEV)
    if kind == "serve":
        s["server"] = dp.Server()
        flat = torch.cat([b.reshape(-1) for bs in s["rhs"] for b in bs])
        s["flat"], s["work"] = flat, torch.empty_like(flat)
        calls, at, rid = [], 0, 1
        for (n, first, more), a in zip(_serve_shapes(case), s["mats"]):
            head = rid
            for j, k in enumerate([first] + more):
                calls.append((rid, n, a if j == 0 else None, s["work"][at:at + n * k], k,
                              len(more) if j == 0 else 0, 0 if j == 0 else head))
                at += n * k
                rid += 1
        s["calls"] = calls
    return s


# ---- one pass -------------------------------------------------------------


def _ok(status):
    if status != dp.SUCCESS:
        raise RuntimeError(dp.delayed_getrf_cuda_status_string(status))


def run(s):
    case, kind = s["case"], s["kind"]
    if kind == "lu":
        s["work"].copy_(s["a"])
        st, info = dp.getrf_device_ex(case["m"], case["n"], s["work"], case["lda"], s["ipiv"], s["jpiv"])
        _ok(st)
        return {"lu": s["work"], "ipiv": s["ipiv"], "jpiv": s["jpiv"], "info": info}
    if kind == "ir":
        s["x"].copy_(s["b"])
        precision = dp.PRECISION_MIXED_BF16X3 if case["terms"] == 2 else dp.PRECISION_MIXED_BF16X6
        st, res = dp.gesv_ir_device(case["n"], case["nrhs"], s["a"], case["n"], s["x"], case["n"],
                                    precision=precision)
        _ok(st)
        return {"x": s["x"], "info": res.info, "converged": res.converged}
    if kind == "batch":
        s["work"].copy_(s["base"])
        _ok(s["plan"].getrf_graph(s["work"], s["ipiv"], s["jpiv"], s["info"]))
        return {"lu": s["work"], "ipiv": s["ipiv"], "jpiv": s["jpiv"], "info": s["info"]}
    if kind == "solve":
        s["x"].copy_(s["b"])
        st, res = s["factor"].solve(s["x"], case["n"], case["nrhs"])
        _ok(st)
        return {"x": s["x"], "converged": res.converged}
    if kind == "ldlt":
        s["work"].copy_(s["a"])
        st, perm, piv, info = dp.sytrf_device(case["n"], s["work"], case["n"])
        _ok(st)
        return {"ld": s["work"], "perm": perm, "piv": piv, "info": info}
    if kind == "front":
        s["work"].copy_(s["a"])
        rows = np.arange(case["m"], dtype=np.int32)
        cols = np.arange(case["n"], dtype=np.int32)
        st, npiv, ipiv, jpiv = dp.front_factor(case["m"], case["n"], case["p"], s["work"], case["m"], rows, cols)
        _ok(st)
        return {"front": s["work"], "ipiv": ipiv, "jpiv": jpiv, "npiv": npiv, "rows": rows, "cols": cols}
    # the server works on streams of its own: the right-hand sides are in place before it is called
    s["work"].copy_(s["flat"])
    torch.cuda.current_stream().synchronize()
    srv = s["server"]
    for rid, n, a, b, k, followups, head in s["calls"]:
        _ok(srv.submit(rid, n, a, n, b, n, k, followups=followups, factor_id=head))
    left, info = len(s["calls"]), 0
    while left:
        for r in srv.poll(256, wait_ms=1000):
            _ok(r.status)
            info += r.info
            left -= 1
    return {"x": s["work"], "info": info}


# ---- the work of a pass ---------------------------------------------------


def _lu_flops(m, n, k):
    """Multiplications and additions of k elimination steps on an m x n matrix."""
    return 2.0 * (m * n * k - (m + n) * k * k / 2.0 + k ** 3 / 3.0)


def work(case):
    kind = case["kind"]
    if kind == "lu":
        m, n = case["m"], case["n"]
        return {"bytes": 16.0 * m * n, "flops": _lu_flops(m, n, min(m, n))}
    if kind == "ir":
        n, r = case["n"], case["nrhs"]
        return {"bytes": 24.0 * n * n + 16.0 * n * r, "flops": _lu_flops(n, n, n) + 4.0 * n * n * r}
    if kind == "batch":
        sq = cube = 0.0
        lo, hi, c = case["lo"], case["hi"], case["count"]
        span = math.log(hi / lo) if hi > lo else 1.0
        sq = c * ((hi ** 2 - lo ** 2) / (2 * span) if hi > lo else lo ** 2)
        cube = c * ((hi ** 3 - lo ** 3) / (3 * span) if hi > lo else lo ** 3)
        return {"bytes": 16.0 * sq, "flops": 2.0 / 3.0 * cube}
    if kind == "solve":
        n, r = case["n"], case["nrhs"]
        return {"bytes": 16.0 * n * n + 16.0 * n * r, "flops": 4.0 * n * n * r}
    if kind == "ldlt":
        n = case["n"]
        return {"bytes": 8.0 * n * n, "flops": n ** 3 / 3.0}
    if kind == "front":
        m, n = case["m"], case["n"]
        return {"bytes": 16.0 * m * n, "flops": _lu_flops(m, n, case["p"])}
    by = fl = 0.0
    for n, first, more in _serve_shapes(case):
        by += 24.0 * n * n + 16.0 * n * (first + sum(more))
        fl += _lu_flops(n, n, n) + 2.0 * n * n * (first + sum(more))
    return {"bytes": by, "flops": fl}


# ---- the same results in plain torch --------------------------------------


def _eliminate(a, rows, cols):
    """Delayed-pivoting elimination of a[i] (a: [count, M, N]) with pivots among the first rows[i]
    rows and cols[i] columns: column partial pivoting; where a column has no nonzero entry left,
    the largest entry of the whole remaining block takes its place; where there is none either,
    the rest is delayed.  In place; returns (ipiv, jpiv, info)."""
    count, steps = a.shape[0], int(torch.minimum(rows, cols).max())
    lim = torch.minimum(rows, cols)
    at = torch.arange(count, device=a.device)
    row_id = torch.arange(a.shape[1], device=a.device)
    ipiv = torch.arange(steps, device=a.device).repeat(count, 1)
    jpiv = ipiv.clone()
    info = lim.clone()
    uneven = bool((rows < a.shape[1]).any())
    for k in range(steps):
        c = a[:, k:, k].abs()
        if uneven:
            c = torch.where(row_id[k:] < rows[:, None], c, -1.0)
        best, p = c.max(1)
        p = p + k
        live = info > k
        none = live & ~(best > 0)
        if bool(none.any()):
            for i in none.nonzero()[:, 0].tolist():
                r, q = int(rows[i]), int(cols[i])
                sub = a[i, k:r, k:q].abs()
                big = sub.max()
                if not bool(big > 0):
                    info[i] = k
                    continue
                flat = int(sub.T.reshape(-1).argmax())
                pr, pc = k + flat % (r - k), k + flat // (r - k)
                p[i], jpiv[i, k] = pr, pc
                if pc != k:
                    a[i][:, [k, pc]] = a[i][:, [pc, k]]
            live = info > k
        p = torch.where(live, p, k)
        ipiv[:, k] = p
        top, low = a[at, k].clone(), a[at, p].clone()
        a[at, p] = top
        a[at, k] = low
        piv = torch.where(live, a[:, k, k], 1.0)
        m = torch.where(live[:, None], a[:, k + 1:, k] / piv[:, None], 0.0)
        a[:, k + 1:, k] = torch.where(live[:, None], m, a[:, k + 1:, k])
        if count == 1:
            a[0, k + 1:, k + 1:].addcmul_(m[0, :, None], a[0, k, None, k + 1:], value=-1)
        else:
            a[:, k + 1:, k + 1:].baddbmm_(m[:, :, None], a[:, k, None, k + 1:], alpha=-1)
    return ipiv, jpiv, info


def _ldlt(a):
    """Delayed Bunch-Kaufman LDL^T of the full symmetric matrix a, in place (lower triangle);
    returns (perm, piv_size, info)."""
    n, alpha = a.shape[0], (1 + math.sqrt(17.0)) / 8
    upper = a.triu(1)
    perm, size = list(range(n)), [0] * n

    def swap(x, y):
        if x != y:
            a[[x, y]] = a[[y, x]]
            a[:, [x, y]] = a[:, [y, x]]
            perm[x], perm[y] = perm[y], perm[x]

    k, e = 0, n
    while k < e:
        c = a[k:e, k].abs()
        if e - k > 1:
            v, i = c[1:].max(0)
            akk, colmax, p = torch.stack([c[0], v, i.to(F64)]).tolist()
            p = int(p) + k + 1
        else:
            akk, colmax, p = float(c[0]), 0.0, k
        one = two = False
        piv = k
        if max(akk, colmax) > 0:
            if akk >= alpha * colmax:
                one = True
            else:
                r = a[k:e, p].abs()
                app = r[p - k].clone()
                r[p - k] = 0.0
                rowmax, app, d0, d1, d2 = torch.stack([r.max(), app, a[k, k], a[p, k], a[p, p]]).tolist()
                if akk >= alpha * colmax * (colmax / rowmax):
                    one = True
                elif app >= alpha * rowmax:
                    one, piv = True, p
                else:
                    s = max(abs(d0), abs(d1), abs(d2))
                    x, y, z = d0 / s, d1 / s, d2 / s
                    nrm = max(abs(x) + abs(y), abs(y) + abs(z))
                    two = s > 0 and abs(x * z - y * y) > 64 * 2.0 ** -52 * nrm * nrm
                    piv = p
        if not one and not two:
            swap(k, e - 1)
            e -= 1
            continue
        w = 2 if two else 1
        swap(k + w - 1, piv)
        b = a[k + w:, k:k + w].clone()
        d = a[k:k + w, k:k + w].clone()
        low = b / d if one else torch.linalg.solve(d, b.T).T
        a[k + w:, k + w:].addmm_(low, b.T, alpha=-1)
        a[k + w:, k:k + w] = low
        a[k:k + w, k + w:] = 0.0
        size[k] = w
        k += w
    a.tril_().add_(upper)
    return np.array(perm, dtype=np.int32), np.array(size, dtype=np.int32), e


def _exact_lu(a, rows, cols):
    """a: the column-major storage ([columns, rows]) of one matrix."""
    x = a.T.contiguous()[None]
    lim = [torch.tensor([v], device=DEV) for v in (rows, cols)]
    ipiv, jpiv, info = _eliminate(x, *lim)
    return (x[0].T.contiguous(), ipiv[0].to(torch.int32).cpu().numpy(), jpiv[0].to(torch.int32).cpu().numpy(),
            int(info[0]))


def exact(case, seed):
    kind, s = case["kind"], _inputs(case, seed)
    if kind == "lu":
        m, n = case["m"], case["n"]
        lu, ipiv, jpiv, info = _exact_lu(s["a"][:, :m].contiguous(), m, n)
        s["a"][:, :m] = lu
        return {"lu": s["a"], "ipiv": ipiv, "jpiv": jpiv, "info": info}
    if kind in ("ir", "solve"):
        x = torch.linalg.solve(s["a"].T, s["b"].T).T.contiguous()
        return {"x": x, "info": case["n"], "converged": 1} if kind == "ir" else {"x": x, "converged": 1}
    if kind == "batch":
        ns, offsets, base = s["ns"], s["offsets"], s["base"]
        order, out = np.argsort(ns, kind="stable"), base.clone()
        for at in range(0, len(order), 256):  # matrices of nearby orders together, padded with zeros
            part = order[at:at + 256]
            top = int(ns[part].max())
            x = torch.zeros(len(part), top, top, dtype=F64, device=DEV)
            for j, i in enumerate(part):
                n, o = int(ns[i]), int(offsets[i])
                x[j, :n, :n] = base[o:o + n * n].view(n, n).T
            lim = torch.from_numpy(ns[part].astype(np.int64)).to(DEV)
            _eliminate(x, lim, lim)
            for j, i in enumerate(part):
                n, o = int(ns[i]), int(offsets[i])
                out[o:o + n * n] = x[j, :n, :n].T.reshape(-1)
        return {"lu": out, "ipiv": None, "jpiv": None, "info": None}
    if kind == "ldlt":
        x = s["a"].clone()  # symmetric: its own transpose
        perm, piv, info = _ldlt(x)
        return {"ld": x.T.contiguous(), "perm": perm, "piv": piv, "info": info}
    if kind == "front":
        p = case["p"]
        f, ipiv, jpiv, npiv = _exact_lu(s["a"], p, p)
        return {"front": f, "ipiv": ipiv, "jpiv": jpiv, "npiv": npiv, "rows": None, "cols": None}
    x = [torch.linalg.solve(a.T, b.T).T.reshape(-1) for a, bs in zip(s["mats"], s["rhs"]) for b in bs]
    return {"x": torch.cat(x), "info": None}
