"""The work whose speed is measured: what users of this library have it do, through its public
entry points, over the sizes of its own workloads (the banded, Poisson, IC(0) and random-band
generators of ``synth``, the many-system group, the serving loop's batches, the drop-in calls).

A case is a dict of plain values:

    kind    "solve"   one right-hand side, device arrays (spk_solve_device)
            "host"    one right-hand side, page-locked host arrays (spk_solve, the drop-in's form)
            "batch"   k right-hand sides, device arrays (spk_solve_batch), FP64 or FP32 + refinement
            "pair"    L, then L^T: the application of an incomplete-Cholesky factor (TriangularPair)
            "group"   many systems in one captured launch sequence (Group)
            "oneshot" preprocessing and one solve (spike_pstrsv), device arrays
    matrix  "banded"  `per_row` off-diagonals at random places of the `band` columns before the row
            "random"  the same with Poisson(`per_row`) off-diagonals per row
            "poisson" lower triangle of the 5-point Laplacian on a grid x grid mesh
            "ic0"     IC(0)-like factor of the 7-point Laplacian on a grid^3 mesh
    uplo    "L", or "U": the transpose, whose rows have unequal lengths
    parts   partitions (the drop-in's nthreads)

Matrices and right-hand sides are made on the GPU from the seed: off-diagonals N(0,1)/16, diagonal
1 + sum of absolute off-diagonals (banded, random), x_true uniform in [-1, 1], b = A x_true.
"""
import numpy as np
import torch

import spike_pstrsv_b200 as spk
from spike_pstrsv_b200 import synth
from spike_pstrsv_b200.group import Group
from spike_pstrsv_b200.pair import TriangularPair

M_FULL = 4194304


def listed():
    return [
        # the smallest calls, where latency is all: a 2-D Poisson factor (coupled over the whole
        # mesh: its spikes never decay), and a small member of a pool of random-band systems
        {"name": "poisson128", "kind": "solve", "matrix": "poisson", "grid": 128, "uplo": "L", "parts": 4},
        {"name": "small_random", "kind": "solve", "matrix": "random", "m": 5003, "per_row": 8, "band": 48,
         "uplo": "U", "parts": 4},
        # ordinary sizes: a banded factor of a quarter million rows, backward solve, ragged; and a
        # band wider than the chain solver's limit of 128 columns
        {"name": "banded_mid_u", "kind": "solve", "matrix": "banded", "m": 262147, "per_row": 16, "band": 64,
         "uplo": "U", "parts": 64},
        {"name": "wide_band", "kind": "solve", "matrix": "random", "m": 100003, "per_row": 8, "band": 200,
         "uplo": "L", "parts": 48},
        # the headline workload and its transpose
        {"name": "banded_full_l", "kind": "solve", "matrix": "banded", "m": M_FULL, "per_row": 16, "band": 64,
         "uplo": "L", "parts": 1024},
        {"name": "banded_full_u", "kind": "solve", "matrix": "banded", "m": M_FULL, "per_row": 16, "band": 64,
         "uplo": "U", "parts": 1024},
        # the reference's own phases with nothing truncated (SPK_EXACT), reduced system and all
        {"name": "exact_mode", "kind": "solve", "matrix": "banded", "m": 524288, "per_row": 16, "band": 64,
         "uplo": "L", "parts": 128, "exact": True},
        # the drop-in's form: host arrays in, host arrays out
        {"name": "host_arrays", "kind": "host", "matrix": "banded", "m": 1048576, "per_row": 16, "band": 64,
         "uplo": "L", "parts": 256},
        # many right-hand sides on the headline matrix, FP64
        {"name": "batch32_fp64", "kind": "batch", "matrix": "banded", "m": M_FULL, "per_row": 16, "band": 64,
         "uplo": "L", "parts": 1024, "k": 32, "mode": 0},
        # a serving loop's batch: FP32 solve, one FP64-residual correction, checked residual
        {"name": "served_ir", "kind": "batch", "matrix": "random", "m": 300007, "per_row": 8, "band": 96,
         "uplo": "L", "parts": 73, "k": 21, "mode": 1},
        # a preconditioner's two sweeps (three couplings per row, the widest grid^2 away)
        {"name": "ic0_pair", "kind": "pair", "matrix": "ic0", "grid": 32, "uplo": "L", "parts": 8},
        # a pool of systems of many sizes and bands, one graph replay
        {"name": "group", "kind": "group", "matrix": "random", "count": 32, "m_lo": 1024, "m_hi": 131072,
         "per_row": 8, "band_lo": 32, "band_hi": 256, "uplo": "L", "rows": 1024, "mode": 0},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["solve"] * 7 + ["host", "batch", "batch", "batch", "group", "pair", "oneshot"])
    uplo = rng.choice("LU")
    if kind == "pair":
        return {"kind": kind, "matrix": "ic0", "grid": rng.randint(12, 32), "uplo": "L", "parts": rng.choice([4, 8])}
    if kind == "group":
        return {"kind": kind, "matrix": "random", "count": rng.randint(8, 32), "m_lo": 1024,
                "m_hi": _log_uniform(rng, 8192, 131072), "per_row": 8, "band_lo": 32, "band_hi": 256, "uplo": uplo,
                "rows": rng.choice([512, 1024, 2048]), "mode": rng.choice([0, 1])}
    matrix = rng.choice(["banded", "banded", "random", "poisson"] if kind == "solve" else ["banded", "random"])
    if matrix == "poisson":
        return {"kind": kind, "matrix": matrix, "grid": rng.randint(32, 160), "uplo": uplo,
                "parts": rng.choice([1, 2, 4, 8])}
    if matrix == "banded":
        c = {"kind": kind, "matrix": matrix, "m": _log_uniform(rng, 2048, M_FULL), "per_row": 16, "band": 64}
    else:
        c = {"kind": kind, "matrix": matrix, "m": _log_uniform(rng, 1024, 500000), "per_row": 8,
             "band": rng.randint(32, 256)}
    c["uplo"] = uplo
    c["parts"] = max(2, min(1024, c["m"] // rng.choice([1024, 2048, 4096])))
    if kind == "solve" and rng.random() < 0.2 and c["m"] <= 524288:
        c["exact"] = True
    if kind == "oneshot":
        c["m"] = min(c["m"], 524288)
        c["parts"] = max(2, min(c["parts"], c["m"] // 1024))
    if kind == "batch":
        c["k"] = rng.randint(2, 32)
        c["mode"] = rng.choice([0, 1])
    return c


# ---- matrices, on the GPU ---------------------------------------------------------


def _rows(m, per_row, band, poisson, g):
    """Lower triangle: per row the distances (columns before the row), ascending columns, and a mask."""
    parts = []
    for r0 in range(0, m, 1 << 18):
        r = torch.arange(r0, min(m, r0 + (1 << 18)), device="cuda")
        d = torch.arange(1, band + 1, device="cuda")
        keys = torch.rand(len(r), band, device="cuda", generator=g)
        keys.masked_fill_(d[None, :] > r[:, None], 2.0)
        if poisson:
            cnt = torch.poisson(torch.full((len(r),), float(per_row), device="cuda"), generator=g).long()
        else:
            cnt = torch.full((len(r),), per_row, device="cuda")
        cnt = torch.minimum(cnt, r).clamp(max=band)
        w = max(int(cnt.max()), 1)
        dist = torch.topk(keys, w, dim=1, largest=False, sorted=True).indices + 1
        dist.masked_fill_(torch.arange(w, device="cuda")[None, :] >= cnt[:, None], 0)
        dist = dist.sort(dim=1, descending=True).values  # ascending columns, unused last
        val = torch.randn(len(r), w, device="cuda", dtype=torch.float64, generator=g) / 16
        parts.append((r, cnt, dist, val))
    return parts


def _coo(case, seed):
    """(m, rows, columns, values) of the lower triangle without its diagonal, and the diagonal."""
    g = torch.Generator("cuda").manual_seed(seed)
    if case["matrix"] in ("poisson", "ic0"):
        n = case["grid"]
        dims = 2 if case["matrix"] == "poisson" else 3
        m = n ** dims
        i = torch.arange(m, device="cuda")
        rows, cols = [], []
        for k in range(dims):
            has = (i // n ** k) % n > 0
            rows.append(i[has])
            cols.append(i[has] - n ** k)
        rows, cols = torch.cat(rows), torch.cat(cols)
        order = torch.argsort(rows * m + cols)
        rows, cols = rows[order], cols[order]
        if dims == 2:
            return m, rows, cols, torch.full((len(rows),), -1.0, device="cuda", dtype=torch.float64), \
                torch.full((m,), 4.0, device="cuda", dtype=torch.float64)
        u = torch.rand(len(rows), device="cuda", dtype=torch.float64, generator=g)
        return m, rows, cols, -(0.9 + 0.2 * u) / 6 ** 0.5, torch.full((m,), 6 ** 0.5, device="cuda", dtype=torch.float64)
    m = case["m"]
    rows, cols, vals = [], [], []
    diag = torch.empty(m, device="cuda", dtype=torch.float64)
    for r, cnt, dist, val in _rows(m, case["per_row"], case["band"], case["matrix"] == "random", g):
        used = dist > 0
        rows.append(r[:, None].expand_as(dist)[used].int())
        cols.append((r[:, None] - dist)[used].int())
        vals.append(val[used])
        diag[r] = 1 + (val.abs() * used).sum(1)
    return m, torch.cat(rows), torch.cat(cols), torch.cat(vals), diag


def _csr(m, rows, cols, vals, diag, uplo):
    """The triangle as the library takes it: int32 CSR, sorted columns, the diagonal in the row."""
    if uplo == "U":  # the transpose: stable by column keeps rows ascending
        order = torch.argsort(cols, stable=True)
        rows, cols, vals = cols[order], rows[order], vals[order]
    cnt = torch.bincount(rows, minlength=m)
    ia = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    ia[1:] = torch.cumsum(cnt + 1, 0)
    at = torch.arange(len(rows), device="cuda") + rows  # each earlier row has put one diagonal before
    own = torch.arange(m, device="cuda")
    if uplo == "U":
        at, dat = at + 1, ia[:-1]
    else:
        dat = ia[1:] - 1
    ja = torch.empty(len(rows) + m, dtype=torch.int32, device="cuda")
    a = torch.empty(len(rows) + m, dtype=torch.float64, device="cuda")
    ja[at], a[at] = cols.int(), vals
    ja[dat], a[dat] = own.int(), diag
    return a, ia.int(), ja




def _product(m, rows, cols, vals, diag, uplo, X):
    """A X, the same bits each time: torch's sparse product in CSR."""
    a, ia, ja = _csr(m, rows, cols, vals, diag, uplo)
    A = torch.sparse_csr_tensor(ia.long(), ja.long(), a, size=(m, m), check_invariants=False)
    return torch.stack([A @ x for x in X]).contiguous()


def _make(case, seed):
    """(m, coo parts, b): the matrix, and k right-hand sides of random solutions."""
    coo = _coo(case, seed)
    g = torch.Generator("cuda").manual_seed(seed + 1)
    x = torch.rand(case.get("k", 1), coo[0], device="cuda", dtype=torch.float64, generator=g) * 2 - 1
    if case["kind"] == "pair":  # b = L L^T x
        x = _product(*coo, "U", x)
    return coo, _product(*coo, case["uplo"], x)


def _members(case, seed):
    """The group's systems: sizes log-uniform, bands and right-hand-side counts as in synth.batch_pool."""
    rng = np.random.default_rng(case["count"] + case["m_hi"])  # sizes belong to the case, numbers to the seed
    for i in range(case["count"]):
        m = int(np.exp(rng.uniform(np.log(case["m_lo"]), np.log(case["m_hi"]))))
        band = int(rng.integers(case["band_lo"], case["band_hi"] + 1))
        k = int(rng.choice([1, 2, 4, 8, 16, 32]))
        yield {"kind": "batch", "matrix": "random", "m": m, "per_row": case["per_row"], "band": band,
               "uplo": case["uplo"], "k": k, "parts": max(1, min(1024, m // case["rows"]))}, seed + 1000 * (i + 1)


def _system(case, coo):
    csr = _csr(*coo, case["uplo"])
    torch.cuda.synchronize()  # preprocessing reads them on a stream of its own
    s = spk.System()
    if case.get("exact"):
        s.set_truncation(-1.0)
    return s.preproc(*csr, coo[0], case["parts"], case["uplo"])


def prepare(case, seed):
    state = {"kind": case["kind"]}
    if case["kind"] == "group":
        B, systems = [], []
        for c, sd in _members(case, seed):
            coo, b = _make(c, sd)
            B.append(b)
            systems.append(_system(c, coo))
        X = [torch.zeros_like(b) for b in B]
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        state.update(group=Group(systems, B, X, mode=case["mode"], iters=case["mode"], stream=stream.cuda_stream),
                     X=X, stream=stream)
        return state
    coo, b = _make(case, seed)
    if case["kind"] == "pair":
        csr = [synth.CSR(coo[0], *(t.cpu().numpy() for t in (ia, ja, a)))
               for a, ia, ja in (_csr(*coo, "L"), _csr(*coo, "U"))]
        state.update(pair=TriangularPair(csr[0], case["parts"], csr[1]), b=b, x=torch.zeros_like(b),
                     y=torch.zeros_like(b))
    elif case["kind"] == "oneshot":
        state.update(csr=_csr(*coo, case["uplo"]), b=b[0], x=torch.zeros_like(b[0]), case=case)
    elif case["kind"] == "host":
        state.update(system=_system(case, coo), b=b[0].cpu().pin_memory().numpy(),
                     x=torch.zeros(coo[0], dtype=torch.float64).pin_memory().numpy())
    elif case["kind"] == "batch":
        state.update(system=_system(case, coo), b=b, x=torch.zeros_like(b), mode=case["mode"])
    else:
        state.update(system=_system(case, coo), b=b[0].contiguous(), x=torch.zeros_like(b[0]))
    return state


def run(state):
    kind = state["kind"]
    if kind == "group":
        state["group"].solve()
        return state["X"]
    stream = torch.cuda.current_stream().cuda_stream
    b, x = state["b"], state["x"]
    if kind == "solve":
        state["system"].solve_device(b.data_ptr(), x.data_ptr(), stream)
    elif kind == "host":
        state["system"].solve(b, x)
    elif kind == "batch":
        # the serving loop's call: a fixed correction step, and the residual of what it returns
        state["system"].solve_batch(b, x, mode=state["mode"], tol=-1.0, maxit=1, stream=stream,
                                    want_resid=state["mode"] == 1)
    elif kind == "pair":
        state["pair"].solve(b, x, mode=0, tol=-1.0, maxit=0, stream=stream, Y=state["y"], want_resid=False)
        return {"y": state["y"], "x": x}
    else:
        c = state["case"]
        spk.spike_pstrsv(c["uplo"], x.numel(), *state["csr"], b, x, c["parts"])
    return x


def _nnz(case):
    if case["matrix"] in ("poisson", "ic0"):
        n, dims = case["grid"], 2 if case["matrix"] == "poisson" else 3
        return n ** dims, n ** dims + dims * (n ** dims - n ** (dims - 1))
    return case["m"], case["m"] * (case["per_row"] + 1)


def work(case):
    """The matrix read once (12 bytes a nonzero, the row pointers), b and x once; a multiply and an add a nonzero."""
    if case["kind"] == "group":
        each = [work(c) for c, _ in _members(case, 0)]
        return {key: sum(w[key] for w in each) for key in ("bytes", "flops")}
    m, nnz = _nnz(case)
    k, sweeps = case.get("k", 1), 2 if case["kind"] == "pair" else 1
    return {"bytes": sweeps * (12 * nnz + 4 * (m + 1) + 16 * m * k), "flops": sweeps * 2 * nnz * k}


def _substitute(coo, uplo, b):
    """x of A x = b by x <- (b - N x) / d, until it stands still (the diagonal is dominant)."""
    m, rows, cols, vals, diag = coo
    if uplo == "U":
        order = torch.argsort(cols, stable=True)
        rows, cols, vals = cols[order], rows[order], vals[order]
    ia = torch.zeros(m + 1, dtype=torch.int64, device=b.device)
    ia[1:] = torch.cumsum(torch.bincount(rows, minlength=m), 0)
    N = torch.sparse_csr_tensor(ia, cols.long(), vals, size=(m, m), check_invariants=False)
    out = []
    for c in b:
        x = c / diag
        for _ in range(400):
            new = (c - N @ x) / diag
            still = torch.equal(new, x)
            x = new
            if still:
                break
        out.append(x)
    return torch.stack(out)


def exact(case, seed):
    if case["kind"] == "group":
        return [_substitute(coo, c["uplo"], b) for c, (coo, b) in ((c, _make(c, sd)) for c, sd in _members(case, seed))]
    coo, b = _make(case, seed)
    if case["kind"] == "pair":
        y = _substitute(coo, "L", b)
        return {"y": y, "x": _substitute(coo, "U", y)}
    x = _substitute(coo, case["uplo"], b)
    return x if case["kind"] == "batch" else x[0].cpu().numpy() if case["kind"] == "host" else x[0]
