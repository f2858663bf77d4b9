"""What this library is used for, as timed cases.

Each case is one call (or one resident-state step) a user's program makes through the Python
package: Lloyd steps of resident jobs over dense and CSR rows, whole ``hcluster`` and
``scluster`` calls, k-means++ seeding, the coreset sampler, and requests served by the
continuous-batching server.  Sizes follow the configurations of ``bench.py``.

``listed()`` names the cases, ``draw(rng)`` gives one more of the same ranges, ``prepare``
makes the inputs, ``run`` makes one pass, ``work`` counts what a pass cannot do without and
``exact`` gives the outputs in 64 bits.
"""
import math

import numpy as np
import torch

import minicore_gb300 as mc

MSR = {"l1": mc.L1, "sqrl2": mc.SQRL2, "jsd": mc.JSD, "mkl": mc.MKL, "hellinger": mc.HELLINGER}
DEV = "cuda"


def listed():
    return [
        # the small configuration: a whole hcluster call of a notebook user, host rows, 20
        # Lloyd updates of a 10,000 x 50 mixture (launches and latency count)
        {"name": "hcluster_small", "kind": "hcluster", "n": 10000, "d": 50, "k": 25, "msr": "sqrl2", "updates": 20},
        # the headline configuration: one Lloyd update of a resident job on the tensor cores
        {"name": "lloyd_bf16_4m", "kind": "lloyd", "n": 4000000, "d": 128, "k": 1024, "msr": "sqrl2",
         "precision": "bf16"},
        # the default precision (FP32) on a mid-sized job with ragged sizes
        {"name": "lloyd_fp32", "kind": "lloyd", "n": 300001, "d": 100, "k": 200, "msr": "sqrl2", "precision": "fp32"},
        # k-medians over dense rows: L1 assignment and coordinate-wise medians
        {"name": "lloyd_l1", "kind": "lloyd", "n": 100000, "d": 64, "k": 50, "msr": "l1", "precision": "fp32"},
        # D^2 seeding of the coreset configuration: 2M x 64, 100 centers
        {"name": "seed_dense", "kind": "seed", "n": 2000000, "d": 64, "k": 100, "msr": "sqrl2", "nnz_row": 0},
        # D^2 seeding over sparse counts (single-cell sized columns), 50 centers, MKL
        {"name": "seed_csr", "kind": "seed", "n": 100000, "d": 20000, "k": 50, "msr": "mkl", "nnz_row": 1500},
        # Bregman Lloyd update over sparse counts: the CSR configuration at a fifth of its rows
        {"name": "csr_mkl", "kind": "csr_lloyd", "n": 200000, "d": 20000, "k": 50, "msr": "mkl", "nnz_row": 1500},
        # the same rows' shape under Jensen-Shannon divergence
        {"name": "csr_jsd", "kind": "csr_lloyd", "n": 50000, "d": 20000, "k": 50, "msr": "jsd", "nnz_row": 1500},
        # one request to the server, nothing else running: pinned host rows, seeding, 10 updates
        {"name": "serve_one", "kind": "serve", "jobs": 1, "slots": 1, "n": 60000, "d": 128, "k": 40, "csr": 0},
        # a burst of requests of the serving stream: half dense BF16, half 1%-dense CSR MKL
        {"name": "serve_mix", "kind": "serve", "jobs": 8, "slots": 8, "n": 90000, "d": 512, "k": 60, "csr": 2},
        # coreset sampler: LBK sensitivities, alias table and 50,000 draws from 2M points
        {"name": "coreset", "kind": "coreset", "n": 2000000, "k": 100, "m": 50000, "sens": mc.LBK},
        # soft clustering of 200k x 32, 20 centers, 8 iterations
        {"name": "soft", "kind": "soft", "n": 200000, "d": 32, "k": 20, "msr": "sqrl2", "iters": 8},
    ]


# ------------------------------------------------------------------------------------
# drawn cases
# ------------------------------------------------------------------------------------
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["hcluster", "lloyd", "lloyd", "seed", "seed", "csr_lloyd", "csr_lloyd", "serve", "coreset",
                       "soft"])
    if kind == "hcluster":
        return {"kind": kind, "n": _log(rng, 1000, 200000), "d": _log(rng, 8, 128), "k": _log(rng, 5, 64),
                "msr": rng.choice(["sqrl2", "sqrl2", "hellinger"]), "updates": rng.randint(5, 25)}
    if kind == "lloyd":
        prec = rng.choice(["bf16", "tf32", "fp32", "fp32"])
        msr = rng.choice(["sqrl2", "l1", "hellinger", "mkl"]) if prec == "fp32" else "sqrl2"
        d = rng.choice([_log(rng, 16, 256), rng.choice([32, 64, 128, 256])])
        k = _log(rng, 8, 1024)
        most = 4e6 * 128 * 1024 if prec != "fp32" else 1e10 if msr == "sqrl2" else 3e9
        n = _log(rng, 20000, max(20001, min(4e6, 5e8 / d, most / (d * k))))
        return {"kind": kind, "n": n, "d": d, "k": k, "msr": msr, "precision": prec}
    if kind == "seed":
        if rng.random() < 0.5:
            d = rng.choice([16, 50, 64, 100, 128, _log(rng, 8, 256)])
            return {"kind": kind, "n": _log(rng, 5000, min(2e6, 1.28e8 / d)), "d": d, "k": _log(rng, 5, 100),
                    "msr": rng.choice(["sqrl2", "sqrl2", "mkl"]), "nnz_row": 0}
        if rng.random() < 0.5:  # 1%-dense rows of the serving stream
            d = rng.choice([64, 128, 512, _log(rng, 64, 2048)])
            return {"kind": kind, "n": _log(rng, 5000, 200000), "d": d, "k": _log(rng, 5, 100), "msr": "mkl",
                    "nnz_row": max(1, d // 100)}
        nnz = _log(rng, 100, 1500)
        return {"kind": kind, "n": _log(rng, 10000, min(200000, 1.5e8 / nnz)), "d": _log(rng, 4000, 20000),
                "k": _log(rng, 5, 50), "msr": rng.choice(["mkl", "jsd"]), "nnz_row": nnz}
    if kind == "csr_lloyd":
        msr = rng.choice(["mkl", "mkl", "jsd", "hellinger", "sqrl2"])
        nnz = _log(rng, 50, 1500)
        return {"kind": kind, "n": _log(rng, 10000, min(200000, (7e7 if msr == "jsd" else 3e8) / nnz)),
                "d": _log(rng, max(2000, 3 * nnz), 20000), "k": rng.choice([_log(rng, 5, 100), 50]), "msr": msr,
                "nnz_row": nnz}
    if kind == "serve":
        jobs = rng.choice([1, 4, 8])
        return {"kind": kind, "jobs": jobs, "slots": jobs, "n": _log(rng, 1000, 120000 if jobs == 1 else 80000),
                "d": rng.choice([32, 64, 128, 512]), "k": _log(rng, 5, 100), "csr": rng.choice([0, 1, 2])}
    if kind == "coreset":
        return {"kind": kind, "n": _log(rng, 10000, 2000000), "k": _log(rng, 10, 200), "m": _log(rng, 1000, 50000),
                "sens": rng.choice([mc.BFL, mc.VX, mc.LBK])}
    return {"kind": kind, "n": _log(rng, 5000, 200000), "d": _log(rng, 8, 64), "k": _log(rng, 4, 32),
            "msr": rng.choice(["sqrl2", "sqrl2", "hellinger"]), "iters": rng.randint(3, 10)}


# ------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) + 1)


def _prior(msr):
    return 0.0 if msr in ("sqrl2", "l1") else 1.0


def _mixture(n, d, k, msr, g):
    """n x d rows of a k-component Gaussian mixture (means ~ N(0, 4I)); row i < k belongs to
    component i, so the first k rows are one seed per component, as a good seeding gives.
    The divergences (mkl, jsd, hellinger) take its magnitudes: non-negative rows."""
    mu = torch.randn(k, d, generator=g, device=DEV) * 2.0
    lab = torch.randint(0, k, (n,), generator=g, device=DEV)
    lab[:k] = torch.arange(k, device=DEV)
    X = torch.randn(n, d, generator=g, device=DEV)
    for r0 in range(0, n, 1 << 20):
        X[r0:r0 + (1 << 20)] += mu[lab[r0:r0 + (1 << 20)]]
    return X.abs_() if msr in ("mkl", "jsd", "hellinger") else X


def _counts(n, d, nnz_row, g):
    """CSR counts: columns taken with Zipf(1.1) rank weights (about nnz_row of them a row, ranks
    in a random order of the columns; rows of 1% density: uniform weights), values negative
    binomial (mean 3, dispersion 0.5) without zeros.  Every row has at least one entry."""
    zipf = nnz_row * 50 > d
    rank = torch.randperm(d, generator=g, device=DEV).double() + 1.0
    w = rank ** -1.1 if zipf else torch.ones(d, dtype=torch.float64, device=DEV)
    lo, hi = 0.0, 1e12
    for _ in range(100):  # inclusion probabilities 1 - exp(-lam w) that sum to nnz_row
        mid = math.sqrt((lo + 1e-12) * hi)
        if float((1 - torch.exp(-mid * w)).sum()) < nnz_row:
            lo = mid
        else:
            hi = mid
    p = (1 - torch.exp(-hi * w)).float()
    r, q = 2.0, 0.6  # P(v) ~ C(v + 1, v) q^v, v >= 1
    v = torch.arange(1, 65, dtype=torch.float64, device=DEV)
    cdf = torch.cumsum((v + 1) * q ** v, 0)
    cdf = (cdf / cdf[-1]).float()
    chunk = max(1, (1 << 27) // d)
    idx, cnt = [], []
    for r0 in range(0, n, chunk):
        m = min(chunk, n - r0)
        mask = torch.rand(m, d, generator=g, device=DEV) < p
        none = (~mask.any(1)).nonzero().squeeze(1)
        mask[none, torch.randint(0, d, (none.numel(),), generator=g, device=DEV)] = True
        cnt.append(mask.sum(1))
        idx.append(mask.nonzero()[:, 1].int())
    idx = torch.cat(idx)
    indptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    indptr[1:] = torch.cumsum(torch.cat(cnt), 0)
    u = torch.rand(idx.numel(), generator=g, device=DEV)
    val = (torch.searchsorted(cdf, u) + 1).clamp_(max=64).float()
    return val, idx, indptr


def _csr(case, seed):
    val, idx, indptr = _counts(case["n"], case["d"], case["nnz_row"], _gen(seed))
    return mc.CSparseMatrix(data=val, indices=idx, indptr=indptr, shape=(case["n"], case["d"]))


def _csr_seeds(X, k):
    """The first k rows as dense centers."""
    C = torch.zeros(k, X.shape[1], device=DEV)
    e = int(X.indptr[k])
    rows = torch.repeat_interleave(torch.arange(k, device=DEV), torch.diff(X.indptr[:k + 1]))
    C[rows, X.indices[:e].long()] = X.data[:e]
    return C


def _pinned(t):
    return t.cpu().pin_memory()


def _serve_specs(case, seed):
    """The requests: sizes fall from the case's n, every other one CSR where csr is 2."""
    out = []
    for i in range(case["jobs"]):
        n = max(1000, int(case["n"] * (1.0 - 0.11 * i)))
        d, k = case["d"], max(2, case["k"] - 3 * i)
        g = _gen(seed * 1000 + i)
        if case["csr"] == 1 or (case["csr"] == 2 and i % 2):
            val, idx, indptr = _counts(n, d, max(1, d // 100), g)
            X = mc.CSparseMatrix(data=_pinned(val), indices=_pinned(idx), indptr=_pinned(indptr), shape=(n, d))
            out.append(dict(matrix=X, k=k, msr=mc.MKL, prior=1.0, precision="fp32", eps=1e-4, maxiter=10, seed=100 + i))
        else:
            X = _pinned(_mixture(n, d, 200, "sqrl2", g))
            out.append(dict(matrix=X, k=k, msr=mc.SQRL2, prior=0.0, precision="bf16", eps=1e-4, maxiter=10,
                            seed=100 + i))
    return out


def prepare(case, seed):
    kind, s = case["kind"], {"case": case}
    if kind in ("lloyd", "csr_lloyd"):
        n, d, k = case["n"], case["d"], case["k"]
        if kind == "lloyd":
            X = _mixture(n, d, k, case["msr"], _gen(seed))
            C, prec = X[:k].clone(), case["precision"]
        else:
            X = _csr(case, seed)
            C, prec = _csr_seeds(X, k), "fp32"
        torch.cuda.synchronize()  # the job launches on its context's own stream
        # a resident job, assigned to its seeds: what a program keeps between Lloyd updates
        s["job"] = mc.Job(X, C, msr=MSR[case["msr"]], prior=_prior(case["msr"]), precision=prec, seed=7)
        s["job"].assign()
        s["centers"] = torch.empty(k, d, device=DEV)
        s["asn"] = torch.empty(n, dtype=torch.int32, device=DEV)
        s["costs"] = torch.empty(n, dtype=torch.float64, device=DEV)
    elif kind == "hcluster":
        s["X"] = _mixture(case["n"], case["d"], case["k"], case["msr"], _gen(seed)).cpu().numpy()
        s["C"] = s["X"][:case["k"]].copy()
    elif kind == "seed":
        s["X"] = _csr(case, seed) if case["nnz_row"] else _mixture(case["n"], case["d"], 200, case["msr"], _gen(seed))
        torch.cuda.synchronize()
    elif kind == "serve":
        s["specs"] = _serve_specs(case, seed)
        s["server"] = mc.Server(slots=case["slots"])
    elif kind == "coreset":
        g = _gen(seed)
        asn = torch.randint(0, case["k"], (case["n"],), generator=g, device=DEV)
        cost = torch.rand(case["n"], generator=g, device=DEV).log_().neg_() * (1.0 + asn % 7)
        s["costs"], s["asn"] = cost.float().cpu().numpy(), asn.cpu().numpy().astype(np.uint32)
        s["sampler"] = mc.CoresetSampler()
    else:
        s["X"] = _mixture(case["n"], case["d"], case["k"], case["msr"], _gen(seed))
        s["C"] = s["X"][:case["k"]].cpu().numpy()
        torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("lloyd", "csr_lloyd"):
        state["job"].lloyd_step()
        state["job"].read(state["centers"], state["asn"], state["costs"])
        return {"centers": state["centers"], "asn": state["asn"], "costs": state["costs"]}
    if kind == "hcluster":
        # eps 0: the given number of updates
        r = mc.hcluster(state["X"], state["C"], msr=MSR[case["msr"]], prior=_prior(case["msr"]), eps=0.0,
                        maxiter=case["updates"] - 1, seed=7)
        return {"centers": r["centers"], "asn": r["asn"], "costs": r["costs"], "numiter": int(r["numiter"])}
    if kind == "seed":
        ids, asn, costs = mc.kmeanspp(state["X"], case["k"], msr=MSR[case["msr"]], prior=_prior(case["msr"]), seed=11)
        return {"ids": ids, "asn": asn, "costs": costs}
    if kind == "serve":
        tickets = [state["server"].submit(**spec) for spec in state["specs"]]
        res = [state["server"].wait(t) for t in tickets]
        return [{k: r[k] for k in ("center_ids", "centers", "asn", "costs", "numiter")} for r in res]
    if kind == "coreset":
        s = state["sampler"]
        s.make_sampler(case["k"], state["costs"], state["asn"], sens=case["sens"])
        w, idx = s.sample(case["m"], seed=5)
        return {"probs": s.get_probs(), "weights": w, "indices": idx}
    r = mc.scluster(state["X"], state["C"], msr=MSR[case["msr"]], prior=_prior(case["msr"]), temp=1.0,
                    maxiter=case["iters"])
    return {"centers": r["centers"], "costs": r["costs"], "asn": r["asn"], "numiter": int(r["numiter"])}


def work(case):
    """Inputs read once, outputs written once; per (row entry, center) the arithmetic of the
    measure (2 for a product or a squared difference, 4 where a logarithm is taken)."""
    kind, n, k = case["kind"], case["n"], case["k"]
    if kind == "coreset":
        return {"bytes": 8.0 * n + 4.0 * n + 12.0 * case["m"], "flops": 10.0 * n}
    d = case["d"]
    per = 4.0 if case.get("msr") == "jsd" else 2.0
    if kind == "lloyd":
        return {"bytes": 4.0 * n * d + 12.0 * n + 8.0 * k * d, "flops": per * n * k * d + 1.0 * n * d}
    if kind == "csr_lloyd":
        nnz = float(n) * case["nnz_row"]
        return {"bytes": 8.0 * nnz + 20.0 * n + 8.0 * k * d, "flops": per * nnz * k + nnz}
    if kind == "hcluster":
        return {"bytes": 4.0 * n * d + 8.0 * n + 8.0 * k * d, "flops": (per * n * k * d + n * d) * case["updates"]}
    if kind == "seed":
        ent = float(n) * (case["nnz_row"] or d)
        return {"bytes": (8.0 if case["nnz_row"] else 4.0) * ent + 12.0 * n, "flops": per * ent * k}
    if kind == "serve":
        b = f = 0.0
        for i in range(case["jobs"]):
            m, c = max(1000, int(n * (1.0 - 0.11 * i))), max(2, k - 3 * i)
            csr = case["csr"] == 1 or (case["csr"] == 2 and i % 2)
            ent = float(m) * (max(1, d // 100) if csr else d)
            b += (8.0 if csr else 4.0) * ent + 12.0 * m
            f += 2.0 * ent * c * 11
        return {"bytes": b, "flops": f}
    return {"bytes": 4.0 * n * d + 8.0 * n * k, "flops": (per * n * k * d + 2.0 * n * k * d) * case["iters"]}


# ------------------------------------------------------------------------------------
# 64-bit values
# ------------------------------------------------------------------------------------
def _pair_term(msr, a, b):
    """One column's term of the measure for center value a and row value b (both transformed)."""
    if msr == "sqrl2":
        return (a - b) ** 2
    if msr == "l1":
        return (a - b).abs()
    if msr == "hellinger":
        return (a.sqrt() - b.sqrt()) ** 2
    if msr == "mkl":
        return a * (a.log() - b.log())
    m = a + b
    return 0.5 * (a * a.log() + b * b.log() - m * (m * 0.5).log())


def _finish(msr, s):
    return (s.clamp(min=0) * 0.5).sqrt() if msr == "hellinger" else s.clamp(min=0)


def _norm(V, msr):
    """Rows as the measure sees them: (v + 1) / (sum v + d) for the divergences (prior 1)."""
    return V if msr in ("sqrl2", "l1") else (V + 1.0) / (V.sum(1, keepdim=True) + V.shape[1])


def _dense_dist(X, C, msr):
    """Distances of float64 rows to float64 centers, n x k."""
    A, B = _norm(C, msr), _norm(X, msr)
    if msr == "sqrl2":
        return ((B * B).sum(1, keepdim=True) - 2.0 * B @ A.t() + (A * A).sum(1)).clamp_(min=0)
    if msr == "mkl":
        return ((A * A.log()).sum(1) - B.log() @ A.t()).clamp_(min=0)
    return torch.stack([_finish(msr, _pair_term(msr, a, B).sum(1)) for a in A], 1)


def _dense_nearest(X, C, msr):
    asn, cost = [], []
    step = max(1, (1 << 27) // max(C.shape[0], C.shape[1]))
    for r0 in range(0, X.shape[0], step):
        x = X[r0:r0 + step].double()
        a = _dense_dist(x, C, msr).argmin(1)
        asn.append(a)
        cost.append(_finish(msr, _pair_term(msr, _norm(C, msr)[a], _norm(x, msr)).sum(1)))
    return torch.cat(asn), torch.cat(cost)


def _dense_centers(X, asn, C, msr):
    """Means of the clusters (medians for l1); a cluster without rows keeps its center."""
    k = C.shape[0]
    out = C.clone()
    if msr == "l1":
        order = torch.argsort(asn, stable=True)
        cnt = torch.bincount(asn, minlength=k).tolist()
        b = 0
        for c in range(k):
            if cnt[c]:
                v = X[order[b:b + cnt[c]]].double().sort(0).values
                out[c] = 0.5 * (v[(cnt[c] - 1) // 2] + v[cnt[c] // 2])
            b += cnt[c]
        return out
    tot = torch.zeros_like(out)
    for r0 in range(0, X.shape[0], 1 << 20):
        tot.index_add_(0, asn[r0:r0 + (1 << 20)], X[r0:r0 + (1 << 20)].double())
    cnt = torch.bincount(asn, minlength=k).double()
    full = cnt > 0
    out[full] = tot[full] / cnt[full, None]
    return out


def _csr_nearest(X, C, msr):
    """Per center: the column terms as if every entry were zero (one value per distinct zero
    entry of the rows), corrected at the stored entries."""
    n, d = X.shape
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), torch.diff(X.indptr))
    val, idx = X.data.double(), X.indices.long()
    A = _norm(C, msr)
    if msr == "sqrl2":
        r = torch.zeros(n, dtype=torch.float64, device=DEV)
        b = val
    else:
        tot = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, rows, val) + d
        r = 1.0 / tot
        b = (val + 1.0) / tot[rows]
    ru, inv = torch.unique(r, return_inverse=True)
    best, asn = torch.full((n,), math.inf, dtype=torch.float64, device=DEV), torch.zeros(n, dtype=torch.long, device=DEV)
    for c in range(C.shape[0]):
        z = torch.cat([_pair_term(msr, A[c][None, :], q[:, None]).sum(1) for q in ru.split(4096)])
        s = z[inv]
        for e0 in range(0, val.numel(), 1 << 26):
            e = slice(e0, e0 + (1 << 26))
            a = A[c][idx[e]]
            s.index_add_(0, rows[e], _pair_term(msr, a, b[e]) - _pair_term(msr, a, r[rows[e]]))
        s = _finish(msr, s)
        m = s < best
        best, asn = torch.where(m, s, best), torch.where(m, c, asn)
    return asn, best


def _csr_centers(X, asn, C):
    n, d = X.shape
    k = C.shape[0]
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), torch.diff(X.indptr))
    tot = torch.zeros(k * d, dtype=torch.float64, device=DEV)
    tot.index_add_(0, asn[rows] * d + X.indices.long(), X.data.double())
    cnt = torch.bincount(asn, minlength=k).double()
    out = tot.view(k, d) / cnt.clamp(min=1)[:, None]
    return torch.where((cnt > 0)[:, None], out, C)


def exact(case, seed):
    kind = case["kind"]
    msr = case.get("msr")
    if kind == "lloyd":
        X = _mixture(case["n"], case["d"], case["k"], msr, _gen(seed))
        C = X[:case["k"]].double()
        C = _dense_centers(X, _dense_nearest(X, C, msr)[0], C, msr)
        return {"centers": C, "asn": None, "costs": _dense_nearest(X, C, msr)[1]}
    if kind == "csr_lloyd":
        if float(case["n"]) * case["nnz_row"] * case["k"] > 6e9:
            return None  # minutes in 64 bits
        X = _csr(case, seed)
        C = _csr_seeds(X, case["k"]).double()
        C = _csr_centers(X, _csr_nearest(X, C, msr)[0], C)
        return {"centers": C, "asn": None, "costs": _csr_nearest(X, C, msr)[1]}
    if kind == "hcluster":
        X = _mixture(case["n"], case["d"], case["k"], msr, _gen(seed))
        C = X[:case["k"]].double()
        asn, _ = _dense_nearest(X, C, msr)
        for _ in range(case["updates"]):
            C = _dense_centers(X, asn, C, msr)
            asn, cost = _dense_nearest(X, C, msr)
        return {"centers": C, "asn": None, "costs": cost, "numiter": None}
    if kind == "soft":
        X = _mixture(case["n"], case["d"], case["k"], msr, _gen(seed)).double()
        C = X[:case["k"]].clone()
        D, old = _dense_dist(X, C, msr), None
        for _ in range(case["iters"]):
            P = torch.softmax(-D, 1)
            cost = float((P * D).sum())
            new = (P.t() @ X) / P.sum(0)[:, None]
            D = _dense_dist(X, new, msr)
            better = old is None or old >= cost
            C = new if better else C
            if old is not None and old - cost <= 1e-8 * max(old, cost):
                break
            old = cost
        return {"centers": C, "costs": D, "asn": P, "numiter": None}
    if kind == "coreset":
        s = prepare(case, seed)
        c, a, n, k = s["costs"].astype(np.float64), s["asn"], case["n"], case["k"]
        cnt, tot = np.bincount(a, minlength=k).astype(np.float64), float(c.sum())
        if case["sens"] == mc.BFL:
            p = 0.5 * (c / tot + 1.0 / (cnt * cnt)[a])
        elif case["sens"] == mc.VX:
            p = c / tot + 1.0 / cnt[a]
        else:
            alpha, avg = 16.0 * math.log(k) + 32.0, tot / n
            per = np.bincount(a, weights=c, minlength=k)
            p = alpha / avg * c + (2.0 * alpha * per / (cnt * avg) + 4.0 * n / cnt)[a]
        return {"probs": p / p.sum(), "weights": None, "indices": None}
    # seeding and whole served requests follow random draws from the distances: an exact run
    # would choose other rows after the first difference in the last bit
    return None
