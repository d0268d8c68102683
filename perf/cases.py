"""Timed cases of the skeleton-discovery framework: whole calls a user's program makes.

Kinds of case (the field "kind"):

gauss   samples on the device -> correlation -> level loop -> skeleton, separation sets, pmax
batch   many uneven Gaussian instances bound to one GaussianBatch, solved by one run()
disc    ordinal codes on the device -> discrete level loop -> results on the host
api     NumPy samples -> discover_skeleton_gpu_discrete (the drop-in call) -> NumPy results
encode  categorical samples on the device -> ordinal codes and cardinalities
orient  skeleton and separation sets on the device -> CPDAG

Sizes are those of the repository's workloads (gpucsl_gb300/workloads.py, synthetic.py and
bench.py) or odd numbers inside their ranges.  Samples follow the same laws as
gpucsl_gb300/synthetic.py, drawn on the device from the seed.
"""
import itertools
import math
from statistics import NormalDist

import numpy as np
import torch

from gpucsl_gb300 import engine
from gpucsl_gb300.batch import GaussianBatch
from gpucsl_gb300.orient import orient_edges_device
from gpucsl_gb300.pc.discover_skeleton_discrete import discover_skeleton_gpu_discrete
from gpucsl_gb300.synthetic import batch_instance_sizes

DEV = "cuda"
DTYPES = {"f64": torch.float64, "f32": torch.float32, "i64": torch.int64, "i32": torch.int32, "u8": torch.uint8}


def listed():
    return [
        # the smallest problem: a few dozen variables, where launches and latency are all there is
        {"name": "gauss_p20_n1000", "kind": "gauss", "p": 20, "n": 1000, "deg": 2.0, "alpha": 0.05, "level": 3,
         "dtype": "f64"},
        # an ordinary request of the serving mix: a few hundred variables, FP32 samples, odd sizes
        {"name": "gauss_p211_n7919_f32", "kind": "gauss", "p": 211, "n": 7919, "deg": 3.0, "alpha": 0.01, "level": 4,
         "dtype": "f32"},
        # the headline problem: FP64 samples, levels until no edge has enough neighbours (they end below 12)
        {"name": "gauss_p1000_n10000", "kind": "gauss", "p": 1000, "n": 10000, "deg": 3.0, "alpha": 0.01, "level": 12,
         "dtype": "f64"},
        # the largest Gaussian request of the serving mix, ragged
        {"name": "gauss_p1999_n49999_f32", "kind": "gauss", "p": 1999, "n": 49999, "deg": 3.0, "alpha": 0.01,
         "level": 3, "dtype": "f32"},
        # many variables, few samples (gene expression): the p x p matrices exceed the L2
        {"name": "gauss_p5000_n2000", "kind": "gauss", "p": 5000, "n": 2000, "deg": 3.0, "alpha": 0.01, "level": 1,
         "dtype": "f64"},
        # bootstrap-like batches of uneven problems, in split precision and in FP64
        {"name": "batch_256_split", "kind": "batch", "count": 256, "alpha": 0.01, "level": 4, "precision": "split"},
        {"name": "batch_24_f64", "kind": "batch", "count": 24, "alpha": 0.01, "level": 4, "precision": "f64"},
        # a small categorical survey through the drop-in call, host arrays in and out
        {"name": "api_disc_p23_n10007", "kind": "api", "p": 23, "n": 10007, "card": 4, "alpha": 0.05, "level": 3},
        # the named discrete problem, and the largest discrete request of the serving mix, ragged
        {"name": "disc_p200_n50000", "kind": "disc", "p": 200, "n": 50000, "card": 5, "alpha": 0.05, "level": 3},
        {"name": "disc_p299_n99991", "kind": "disc", "p": 299, "n": 99991, "card": 6, "alpha": 0.05, "level": 3},
        # encoding of integer categories, as a discrete solve does first
        {"name": "encode_p200_n50000", "kind": "encode", "p": 200, "n": 50000, "card": 5, "dtype": "i64"},
        # orientation of the headline problem's skeleton, the last stage of a whole PC run
        {"name": "orient_p1000", "kind": "orient", "p": 1000, "n": 10000, "deg": 3.0, "alpha": 0.01, "level": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gauss", "gauss", "gauss", "wide", "batch", "batch", "disc", "disc", "api", "encode", "orient"])
    if kind == "gauss":
        return {"kind": "gauss", "p": _log_int(rng, 20, 1990), "n": _log_int(rng, 1000, 49990),
                "deg": round(rng.uniform(2.0, 3.0), 2), "alpha": rng.choice([0.01, 0.05]), "level": rng.choice([2, 3, 4]),
                "dtype": rng.choice(["f64", "f32"])}
    if kind == "wide":
        return {"kind": "gauss", "p": _log_int(rng, 2000, 4990), "n": _log_int(rng, 500, 2000),
                "deg": round(rng.uniform(2.0, 3.0), 2), "alpha": 0.01, "level": 1, "dtype": rng.choice(["f64", "f32"])}
    if kind == "batch":
        return {"kind": "batch", "count": _log_int(rng, 4, 128), "alpha": 0.01, "level": rng.choice([3, 4]),
                "precision": rng.choice(["split", "f64"])}
    if kind == "disc":
        return {"kind": "disc", "p": rng.randint(20, 290), "n": _log_int(rng, 10000, 99000), "card": rng.randint(3, 6),
                "alpha": rng.choice([0.01, 0.05]), "level": rng.choice([2, 3])}
    if kind == "api":
        return {"kind": "api", "p": _log_int(rng, 10, 60), "n": _log_int(rng, 1000, 20000), "card": rng.randint(2, 5),
                "alpha": 0.05, "level": rng.choice([1, 2, 3])}
    if kind == "encode":
        return {"kind": "encode", "p": rng.randint(20, 300), "n": _log_int(rng, 10000, 100000),
                "card": rng.randint(2, 12), "dtype": rng.choice(["i64", "i32", "u8", "f64"])}
    return {"kind": "orient", "p": _log_int(rng, 50, 1500), "n": _log_int(rng, 1000, 20000),
            "deg": round(rng.uniform(2.0, 3.0), 2), "alpha": rng.choice([0.01, 0.05]), "level": rng.choice([2, 3, 4])}


# ------------------------------------------------------------------ inputs
def _dag(rng, p, deg):
    """Parents (p, k) in topological positions, padded with 0, their validity, the depth of
    each position and the position of each variable."""
    order = rng.permutation(p)
    prob = 0.0 if p < 2 else min(1.0, deg / (p - 1))
    parents = [np.nonzero(rng.random(b) < prob)[0] for b in range(p)]
    depth = np.zeros(p, np.int64)
    for b in range(p):
        if parents[b].size:
            depth[b] = depth[parents[b]].max() + 1
    return order, parents, depth


def _gaussian(p, n, deg, seed):
    """(n, p) FP64 samples of a linear-Gaussian DAG on the device: weights +-U[0.1, 1], N(0, 1) noise."""
    rng = np.random.default_rng(seed)
    order, parents, depth = _dag(rng, p, deg)
    k = max(1, max(len(x) for x in parents))
    idx, w = np.zeros((p, k), np.int64), np.zeros((p, k))
    for b, x in enumerate(parents):
        idx[b, :len(x)] = x
        w[b, :len(x)] = rng.uniform(0.1, 1.0, len(x)) * rng.choice([-1.0, 1.0], len(x))
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    Z = torch.randn((p, n), generator=gen, dtype=torch.float64, device=DEV)
    for d in range(1, int(depth.max()) + 1):
        rows = np.nonzero(depth == d)[0]
        at = torch.from_numpy(rows).to(DEV)
        for c in range(max(len(parents[b]) for b in rows)):
            Z[at] += torch.from_numpy(w[rows, c]).to(DEV)[:, None] * Z[torch.from_numpy(idx[rows, c]).to(DEV)]
    pos = np.empty(p, np.int64)
    pos[order] = np.arange(p)  # position b holds variable order[b]
    return Z[torch.from_numpy(pos).to(DEV)].t().contiguous()


def _categorical(p, n, card, seed, deg=2.0, max_in=3):
    """(n, p) uint8 samples of a discrete Bayesian network on the device: cardinalities
    U{2..card}, at most max_in parents, probability rows from Dirichlet(1)."""
    rng = np.random.default_rng(seed)
    order, parents, _ = _dag(rng, p, deg)
    cards = rng.integers(2, card + 1, size=p)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    Z = torch.empty((p, n), dtype=torch.int64, device=DEV)
    u = torch.rand((p, n), generator=gen, dtype=torch.float64, device=DEV)
    for b in range(p):
        pa = parents[b] if len(parents[b]) <= max_in else np.sort(rng.choice(parents[b], max_in, replace=False))
        cfg = torch.zeros(n, dtype=torch.int64, device=DEV)
        mult = 1
        for x in pa:
            cfg += Z[int(x)] * mult
            mult *= int(cards[x])
        cdf = torch.from_numpy(np.cumsum(rng.dirichlet(np.ones(cards[b]), size=mult), axis=1)).to(DEV)
        Z[b] = torch.clamp((u[b][:, None] > cdf[cfg]).sum(1), max=int(cards[b]) - 1)
    pos = np.empty(p, np.int64)
    pos[order] = np.arange(p)
    return Z[torch.from_numpy(pos).to(DEV)].t().to(torch.uint8).contiguous()


def _categories(case, seed):
    """Category labels as a table holds them: not zero-based, with gaps."""
    X = _categorical(case["p"], case["n"], case["card"], seed).to(torch.int64) * 3 + 1
    return X.to(DTYPES[case["dtype"]]).contiguous()


def _instances(case, seed):
    sizes = batch_instance_sizes(case["count"], base_seed=1000)  # sizes of the case, data of the seed
    return [s[0] for s in sizes], [s[1] for s in sizes], \
        [_gaussian(p, n, deg, seed * 1009 + k) for k, (p, n, deg, _) in enumerate(sizes)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "gauss":
        X = _gaussian(case["p"], case["n"], case["deg"], seed).to(DTYPES[case["dtype"]])
        return {"case": case, "X": X, "solver": engine.GaussianSolver(case["p"], case["level"], dense_sepsets=True),
                "thr": engine.gaussian_thresholds(case["n"], case["alpha"])}
    if kind == "batch":
        ps, ns, Xs = _instances(case, seed)
        batch = GaussianBatch(ps, ns, case["alpha"], case["level"], case["precision"])
        batch.bind_samples(Xs)
        batch.capture()  # the graph that later runs replay
        return {"case": case, "batch": batch}
    if kind == "api":
        return {"case": case, "data": _categorical(case["p"], case["n"], case["card"], seed).cpu().numpy()}
    if kind == "disc":
        codes, dims = engine.ordinal_encode_device(_categorical(case["p"], case["n"], case["card"], seed))
        solver = engine.DiscreteSolver(case["p"], case["n"], case["level"], int(dims.max()))
        solver.load(codes_dev=codes[:, :case["n"]], dims_dev=dims)
        return {"case": case, "solver": solver}
    if kind == "encode":
        return {"case": case, "X": _categories(case, seed)}
    # orient: the skeleton and sets of a solve
    solver = engine.GaussianSolver(case["p"], case["level"], dense_sepsets=True)
    solver.run(engine.correlation(_gaussian(case["p"], case["n"], case["deg"], seed)), case["n"],
               engine.gaussian_thresholds(case["n"], case["alpha"]))
    return {"case": case, "G": solver.G, "sep": solver.sep_dense}


def _whole(views):
    """The one buffer that a batch's per-instance results are consecutive views of."""
    return torch.as_strided(views[0], (sum(v.numel() for v in views),), (1,), 0)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "gauss":
        solver = state["solver"]
        C = engine.correlation(state["X"])
        solver.run(C, case["n"], state["thr"])
        return {"C": C, "skeleton": solver.G, "sepsets": solver.sep_dense, "pmax": solver.pmax}
    if kind == "batch":
        batch = state["batch"]
        results = batch.run()
        return {"skeletons": _whole(batch.G), "pmax": _whole(batch.pmax),
                "records": np.array([r.n_records for r in results]), "tests": np.array([r.tests for r in results])}
    if kind == "api":
        r = discover_skeleton_gpu_discrete(None, state["data"], case["alpha"], case["level"], case["p"], case["n"]).result
        return {"skeleton": r.skeleton.astype(np.int32), "sepsets": r.seperation_sets, "pmax": r.pmax}
    if kind == "disc":
        state["solver"].run(case["alpha"])
        G, sep, pmax = state["solver"].to_host()
        return {"skeleton": G.astype(np.int32), "sepsets": sep, "pmax": pmax}
    if kind == "encode":
        codes, dims = engine.ordinal_encode_device(state["X"])
        return {"codes": codes, "dims": dims}
    D, passes = orient_edges_device(state["G"], state["sep"])
    return {"cpdag": D, "passes": passes}


def work(case):
    """Inputs read once, outputs written once; one multiply-add per sample and pair of
    variables for a correlation, one count per sample and pair for the discrete tests."""
    kind = case["kind"]
    if kind == "batch":
        sizes = batch_instance_sizes(case["count"], base_seed=1000)
        return {"bytes": sum(8 * n * p + 18 * p * p for p, n, _, _ in sizes), "flops": sum(n * p * (p + 1) for p, n, _, _ in sizes)}
    p, n = case["p"], case["n"]
    if kind == "gauss":
        return {"bytes": (8 if case["dtype"] == "f64" else 4) * n * p + (18 + 4 * case["level"]) * p * p,
                "flops": n * p * (p + 1)}
    if kind in ("api", "disc"):
        return {"bytes": n * p + (10 + 4 * case["level"]) * p * p, "flops": n * p * (p - 1) / 2}
    if kind == "encode":
        return {"bytes": (torch.empty(0, dtype=DTYPES[case["dtype"]]).element_size() + 1) * n * p, "flops": n * p}
    return {"bytes": (3 + 4 * case["level"]) * p * p, "flops": p * p}


# ------------------------------------------------------------ 64-bit results
def _corrcoef(X):
    """Correlation matrix in 64 bits, summed over blocks of samples to keep the rounding small."""
    X = X.double()
    Xc = X - X.mean(0)
    Xc = Xc - Xc.mean(0)
    S = sum(Xc[t:t + 512].t() @ Xc[t:t + 512] for t in range(0, X.shape[0], 512))
    sd = S.diagonal().sqrt()
    return (S / sd[:, None] / sd[None, :]).clamp(-1.0, 1.0)


def _z(rho):
    return (0.5 * ((1 + rho).abs().log() - (1 - rho).abs().log())).abs()


def _rho(C, vi, vj, S):
    """Partial correlations of (vi, vj) given the columns of S, one per row, by elimination."""
    L = S.shape[1]
    V = torch.cat([S, vi[:, None], vj[:, None]], 1)
    A = C[V[:, :, None], V[:, None, :]]
    for j in range(L):
        A = A - A[:, :, j:j + 1] * A[:, j:j + 1, :] / A[:, j:j + 1, j:j + 1]
    return A[:, L, L + 1] / (A[:, L, L].abs().sqrt() * A[:, L + 1, L + 1].abs().sqrt())


def _gauss_skeleton(C, n, alpha, max_level):
    """PC-stable skeleton, separation sets and largest p-values in 64 bits.  Tests of a pair
    run in the order (rank, direction) up to the first that removes it."""
    p = C.shape[0]
    q = abs(NormalDist().inv_cdf(alpha / 2))
    zmin = _z(C - torch.eye(p, dtype=C.dtype, device=C.device))
    G = zmin >= q / math.sqrt(n - 4)
    G.fill_diagonal_(False)
    sep = torch.full((p, p, max(max_level, 1)), -1, dtype=torch.int32, device=C.device)
    for L in range(1, max_level + 1):
        deg = G.sum(1)
        top = int(deg.max())
        if top - 1 < L:
            break
        tau = q / math.sqrt(n - L - 4)
        nbr = torch.sort(torch.where(G, torch.arange(p, device=C.device), p), 1).values[:, :top]
        lo, hi = torch.nonzero(torch.triu(G), as_tuple=True)
        jobs = []  # (edge, key, z) of all tests
        for K in range(L, top):
            combos = torch.from_numpy(np.array(list(itertools.combinations(range(K), L)), np.int64)).to(C.device)
            for d, (a, b) in enumerate(((lo, hi), (hi, lo))):
                edges = torch.nonzero(deg[a] - 1 == K).flatten()
                for part in edges.split(max(1, 1_500_000 // (len(combos) * (L + 2)))):
                    vi, vj = a[part], b[part]
                    row = nbr[vi][:, :K + 1]
                    rest = row[row != vj[:, None]].view(-1, K)
                    S = rest[:, combos]
                    m, r = S.shape[:2]
                    z = _z(_rho(C, vi.repeat_interleave(r), vj.repeat_interleave(r), S.view(m * r, L)))
                    jobs.append((part.repeat_interleave(r), (2 * torch.arange(r, device=C.device) + d).repeat(m), z,
                                 S.view(m * r, L)))
        if not jobs:
            break
        e, key, z = (torch.cat([j[i] for j in jobs]) for i in range(3))
        S = torch.cat([j[3] for j in jobs])
        none = 1 << 62
        gone = z < tau
        first = torch.full((len(lo),), none, device=C.device).scatter_reduce(0, e[gone], key[gone], "amin")
        seen = (key <= first[e]) & ~z.isnan()
        low = torch.full((len(lo),), math.inf, dtype=C.dtype, device=C.device).scatter_reduce(0, e[seen], z[seen], "amin")
        zmin[lo, hi] = torch.minimum(zmin[lo, hi], low)
        at = torch.nonzero(key == first[e]).flatten()
        a, b = lo[e[at]], hi[e[at]]
        sep[a, b, :L] = sep[b, a, :L] = S[at].int()
        G[a, b] = G[b, a] = False
    pmax = torch.special.erfc(math.sqrt(n - 3) * zmin / math.sqrt(2.0))
    pmax = torch.where(torch.ones_like(G).triu(1), pmax, -1.0)
    return G.to(torch.int16), sep[:, :, :max_level], pmax


def _chi2_pvalue(codes, dims, i, j, S):
    """p-value of the chi-squared test of i and j given the set S, in 64 bits."""
    s, ds = torch.zeros_like(codes[0]), 1
    for v in S:
        s = s + codes[v] * ds
        ds *= dims[v]
    T = torch.bincount((s * dims[i] + codes[i]) * dims[j] + codes[j], minlength=ds * dims[i] * dims[j])
    T = T.view(ds, dims[i], dims[j]).double()
    E = T.sum(2, keepdim=True) * T.sum(1, keepdim=True) / T.sum((1, 2), keepdim=True)
    x = torch.where(E > 0, (T - E) ** 2 / E, 0.0).sum()
    df = (dims[i] - 1) * (dims[j] - 1) * ds
    return 1.0 if df < 1 else float(torch.special.gammaincc(torch.tensor(df / 2, dtype=torch.float64), (x / 2).cpu()))


def _disc_skeleton(data, alpha, max_level):
    cols = [torch.unique(data[:, v], return_inverse=True) for v in range(data.shape[1])]
    codes, dims = [c[1].long() for c in cols], [len(c[0]) for c in cols]
    p = len(codes)
    G, pmax, sep = np.zeros((p, p), np.int32), np.full((p, p), -1.0), np.full((p, p, max_level), -1, np.int32)
    for i, j in itertools.combinations(range(p), 2):
        pmax[i, j] = _chi2_pvalue(codes, dims, i, j, ())
        G[i, j] = G[j, i] = pmax[i, j] < alpha
    for L in range(1, max_level + 1):
        nbrs = [list(np.nonzero(G[v])[0]) for v in range(p)]
        if max(map(len, nbrs)) - 1 < L:
            break
        for i, j in itertools.combinations(range(p), 2):
            if j not in nbrs[i]:
                continue
            best = None
            for d, (a, b) in enumerate(((i, j), (j, i))):
                for rank, S in enumerate(itertools.combinations([v for v in nbrs[a] if v != b], L)):
                    pv = _chi2_pvalue(codes, dims, a, b, S)
                    pmax[i, j] = max(pmax[i, j], pv)
                    if pv >= alpha and (best is None or (rank, d) < best[0]):
                        best = ((rank, d), S)
            if best:
                G[i, j] = G[j, i] = 0
                sep[i, j, :L] = sep[j, i, :L] = best[1]
    return G, sep, pmax


def exact(case, seed):
    kind = case["kind"]
    if kind == "gauss":
        C = _corrcoef(_gaussian(case["p"], case["n"], case["deg"], seed).to(DTYPES[case["dtype"]]))
        G, sep, pmax = _gauss_skeleton(C, case["n"], case["alpha"], case["level"])
        return {"C": C, "skeleton": G, "sepsets": sep, "pmax": pmax}
    if kind == "batch" and case["count"] <= 24:
        ps, ns, Xs = _instances(case, seed)
        got = [_gauss_skeleton(_corrcoef(X), n, case["alpha"], case["level"]) for X, n in zip(Xs, ns)]
        return {"skeletons": torch.cat([g[0].flatten() for g in got]), "pmax": torch.cat([g[2].flatten() for g in got]),
                "records": None, "tests": None}
    if kind == "api" and case["p"] <= 30:
        data = _categorical(case["p"], case["n"], case["card"], seed)
        G, sep, pmax = _disc_skeleton(data, case["alpha"], case["level"])
        return {"skeleton": G, "sepsets": sep, "pmax": pmax}
    return None  # tens of thousands of separate tests, or whole numbers only
