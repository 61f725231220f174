"""The work this library is measured on: calls a user makes, through the public entry points.

A case is a dict of plain values.  ``listed()`` names the fixed ones, ``draw(rng)`` gives one more of the
same ranges, ``prepare`` makes a user's inputs from a seed, ``run`` is one pass, ``exact`` the same
result in 64 bits from plain torch, ``work`` the bytes and operations a pass cannot do without.

Graphs are UMAP fuzzy-kNN graphs of Gaussian mixtures with uniform background points, as the repository's
benchmark and tests use them: 10 to 30 neighbours, tens of clusters, nodes either in cluster order or
shuffled (data sets that come in no order).  Solves that iterate ask for a residual of 1e-10, at which the
embedding no longer depends on the path that the iteration took.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import spectral_init_b200 as si
from spectral_init_b200 import synthetic
from spectral_init_b200._lib import SiCsrF32, SiReport
from spectral_init_b200.warm_start import DeviceLaplacian, WarmStartModel

DEV = "cuda"
GROUP = 16384       # consecutive points that search one another when n is too large for brute force
BRUTE = 50_000      # largest n whose neighbours are searched exactly
SOLVE_TOL = 1e-10


# ---- what is measured ----------------------------------------------------------------------------
def _init(name, n, nc, *, k=15, dims=50, clusters=10, precision="fp64", where="host", order="cluster"):
    c = {"kind": "init", "n": n, "nc": nc, "k": k, "dims": dims, "clusters": clusters, "precision": precision,
         "where": where, "order": order}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a few hundred points embedded inside an interactive loop: the smallest call, latency only
        _init("init_150", 150, 2, k=10, dims=8, clusters=3),
        # a small data set with a 3-D embedding, just below the dense limit (2000 nodes), odd size
        _init("init_1873_nc3", 1873, 3, dims=16, clusters=8),
        # an ordinary small data set through the host call: launches and the host's part count
        _init("init_5003", 5003, 2, dims=16, clusters=8),
        # a mid-size data set in mixed precision, host arrays, ragged size
        _init("init_60013_mixed", 60013, 2, clusters=10, precision="mixed"),
        # an ordinary large data set in no particular order, graph already on the device
        _init("init_200k_shuffled", 200_000, 2, clusters=6, where="device", order="shuffled"),
        # the repository's headline size, mixed precision, host arrays in and the embedding out
        _init("init_1m_mixed", 1_000_000, 2, clusters=100, precision="mixed"),
        # many embedding dimensions: 16-wide blocks, denser graph
        _init("init_100k_nc8", 100_003, 8, k=30, clusters=20, where="device"),
        # a graph that falls apart: components of 20 to 12 000 nodes embedded and laid out together
        {"name": "components_60", "kind": "components", "parts": 60, "size_max": 12_000, "nc": 2},
        # the prepared operator applied in a user's own iteration: f32 blocks of four columns
        {"name": "apply_f32_1m_k4", "kind": "apply", "n": 1_000_000, "cols": 4, "dtype": "float32", "k": 15,
         "clusters": 100, "order": "cluster"},
        # the same in f64 on n_components + 1 columns, nodes in no order
        {"name": "apply_f64_300k_k3", "kind": "apply", "n": 300_007, "cols": 3, "dtype": "float64", "k": 15,
         "clusters": 40, "order": "shuffled"},
        # one training step's loss and gradient of the warm-start network (forward and backward)
        {"name": "train_60k", "kind": "train", "n": 60_000, "nc": 2, "k": 15, "clusters": 20},
        # points to fuzzy graph: exact neighbours, calibration, union, pruning
        {"name": "fuzzy_20k", "kind": "fuzzy", "n": 20_011, "dims": 50, "k": 15},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dense", "dense", "init", "init", "init", "wide", "components", "apply", "apply", "train", "fuzzy"])
    order = rng.choice(["cluster", "shuffled"])
    if kind == "dense":
        n = _log_int(rng, 120, 1990)
        return _init(None, n, rng.randint(1, 5), k=rng.choice([10, 15]), dims=rng.choice([8, 16]),
                     clusters=rng.randint(2, 8), order=order)
    if kind in ("init", "wide"):
        n = _log_int(rng, 2500, 400_000 if kind == "init" else 100_000)
        return _init(None, n, rng.choice([1, 2]) if kind == "init" else rng.choice([4, 5, 6, 8, 10]),
                     k=rng.choice([15, 20, 30]), dims=16 if n < 10_000 else 50, clusters=min(rng.choice([4, 5, 6, 10, 30]), max(4, n // 3000)),
                     precision=rng.choice(["fp64", "mixed"]), where=rng.choice(["host", "device"]), order=order)
    if kind == "components":
        return {"kind": "components", "parts": rng.randint(5, 60), "size_max": _log_int(rng, 500, 12_000), "nc": 2}
    if kind == "apply":
        n = _log_int(rng, 1000, 800_000)
        return {"kind": "apply", "n": n, "cols": rng.choice([1, 2, 3, 4, 5, 8, 9, 16]),
                "dtype": rng.choice(["float32", "float64"]), "k": rng.choice([10, 15, 30]),
                "clusters": max(2, min(80, n // 5000)), "order": order}
    if kind == "train":
        n = _log_int(rng, 3000, 100_000)
        return {"kind": "train", "n": n, "nc": rng.choice([1, 2, 3]), "k": rng.choice([10, 15, 30]),
                "clusters": max(4, min(40, n // 3000))}
    return {"kind": "fuzzy", "n": _log_int(rng, 200, 20_000), "dims": rng.choice([2, 10, 16, 50, 100]),
            "k": rng.choice([10, 15, 30])}


# ---- inputs ----------------------------------------------------------------------------------------
def _knn(x, k, seed):
    """Neighbours within groups of consecutive points plus a random sample of all points: what an
    approximate index finds (column 0 is the point itself)."""
    n = x.shape[0]
    if n <= BRUTE:
        return synthetic.knn_gpu(x, k)
    prev = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    try:
        g = torch.Generator(device=x.device)
        g.manual_seed(seed + 17)
        sq = (x * x).sum(1)
        idx = torch.empty(n, k, dtype=torch.int64, device=x.device)
        dist = torch.empty(n, k, dtype=torch.float32, device=x.device)
        for s in range(0, n, GROUP):
            e = min(n, s + GROUP)
            far = torch.randperm(n, generator=g, device=x.device)[:GROUP]
            far = far[(far < s) | (far >= e)]
            cand = torch.cat([torch.arange(s, e, device=x.device), far])
            xc, sc = x[cand], sq[cand]
            for a in range(s, e, 4096):
                b = min(e, a + 4096)
                d = torch.addmm(sc[None, :] + sq[a:b, None], x[a:b], xc.T, alpha=-2.0)
                r = torch.arange(b - a, device=x.device)
                d[r, r + (a - s)] = -1.0
                v, i = torch.topk(d, k, dim=1, largest=False, sorted=True)
                v[:, 0] = 0.0
                idx[a:b] = cand[i]
                dist[a:b] = v.clamp_min(0.0).sqrt()
        return idx, dist
    finally:
        torch.backends.cuda.matmul.allow_tf32 = prev


def _graph(n, k, clusters, dims, order, seed):
    """(indptr i64, indices i32, data f32) of a fuzzy-kNN graph, on the device."""
    # centres of the benchmark's spread in 50-D; closer in few dimensions, where the background is thin
    std = 2.0 if dims >= 50 else 1.0
    x = synthetic.gaussian_mixture_gpu(n, clusters, dims, seed % (1 << 31), center_std=std, background_frac=0.05,
                                       device=DEV)
    idx, dist = _knn(x, k, seed % (1 << 31))
    if order == "shuffled":
        g = torch.Generator(device=DEV)
        g.manual_seed(seed % (1 << 31) + 1)
        p = torch.randperm(n, generator=g, device=DEV)   # new node i is old node p[i]
        inv = torch.empty_like(p)
        inv[p] = torch.arange(n, device=DEV)
        idx, dist = inv[idx[p]], dist[p]
    sigma, rho = synthetic.smooth_knn_gpu(dist, k)
    return synthetic.fuzzy_graph_gpu(idx, dist, sigma, rho)


def _part_sizes(case):
    """Component sizes, even over their logarithm from 20 to size_max (the repository's size law, without its luck)."""
    return np.geomspace(20, case["size_max"], case["parts"]).astype(int).tolist()


def _parts_graph(case, seed):
    """Block-diagonal union of independent fuzzy-kNN graphs (1 to 10 overlapping clusters each) and their points."""
    rng = np.random.default_rng(seed)
    ips, ixs, dvs, xs, nodes, entries = [], [], [], [], 0, 0
    for c, size in enumerate(_part_sizes(case)):
        x = synthetic.gaussian_mixture_gpu(size, int(rng.integers(1, 11)), 20, (seed * 1009 + c) % (1 << 31),
                                           center_std=1.0, device=DEV)
        x = x + torch.from_numpy(rng.normal(0.0, 100.0, 20).astype(np.float32)).to(DEV)
        k = min(15, size - 1)
        idx, dist = synthetic.knn_gpu(x, k)
        sigma, rho = synthetic.smooth_knn_gpu(dist, k)
        ip, ix, dv = synthetic.fuzzy_graph_gpu(idx, dist, sigma, rho, prune=False)
        ips.append(ip[:-1] + entries)
        ixs.append(ix + nodes)
        dvs.append(dv)
        xs.append(x)
        nodes += size
        entries += ix.numel()
    ips.append(torch.tensor([entries], dtype=torch.int64, device=DEV))
    return (torch.cat(ips), torch.cat(ixs).contiguous(), torch.cat(dvs).contiguous()), torch.cat(xs)


def _host(t):
    return tuple(a.cpu().numpy() for a in t)


def _values64(indptr, indices, data, n):
    """Off-diagonal entries of the normalised Laplacian in f64, and the row of each entry."""
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), indptr[1:] - indptr[:-1])
    w = data.double()
    deg = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, rows, w)
    inv = torch.where(deg > 0, deg.rsqrt(), torch.zeros_like(deg))
    cols = indices.long()
    return rows, cols, -inv[rows] * w * inv[cols]


def _config(case):
    return si.SpectralInitConfig(precision=si.Precision.MIXED if case.get("precision") == "mixed" else si.Precision.FP64,
                                 tol=SOLVE_TOL)


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case, "seed": int(seed) % (1 << 31), "ctx": si.get_context()}
    if kind == "init":
        g = _graph(case["n"], case["k"], case["clusters"], case["dims"], case["order"], seed)
        if case["where"] == "host":
            state["graph"] = _host(g) + (case["n"],)
        else:
            state["graph"] = g
            state["out"] = torch.empty(case["n"], case["nc"], dtype=torch.float32, device=DEV)
        state["config"] = _config(case)
    elif kind == "components":
        (ip, ix, dv), x = _parts_graph(case, state["seed"])
        state["graph"] = _host((ip, ix, dv)) + (x.shape[0],)
        state["data"] = x.cpu().numpy()
        state["config"] = _config(case)
    elif kind == "apply":
        n = case["n"]
        ip, ix, dv = _graph(n, case["k"], case["clusters"], 50 if n >= 10_000 else 16, case["order"], seed)
        v = _values64(ip, ix, dv, n)[2]
        f32 = case["dtype"] == "float32"
        state["op"] = si.CsrOperator(_host((ip, ix, v)) + (n,), diag=1.0, with_f32=f32).prepare()
        g = torch.Generator(device=DEV)
        g.manual_seed(state["seed"] + 2)
        state["x"] = torch.randn(n, case["cols"], generator=g, device=DEV, dtype=getattr(torch, case["dtype"]))
        state["y"] = torch.empty_like(state["x"])
    elif kind == "train":
        n = case["n"]
        g = _graph(n, case["k"], case["clusters"], 50 if n >= 10_000 else 16, "cluster", seed)
        state["lap"] = DeviceLaplacian(g + (n,))
        state["model"] = WarmStartModel(seed=state["seed"])
        gen = torch.Generator(device=DEV)
        gen.manual_seed(state["seed"] + 3)
        # orthonormal targets, smooth over the graph as eigenvectors are
        t = torch.randn(n, case["nc"] + 1, generator=gen, device=DEV, dtype=torch.float64)
        state["target"] = torch.linalg.qr(t)[0].contiguous()
    else:
        rng = np.random.default_rng(state["seed"])
        centres = rng.normal(0.0, 2.0, (10, case["dims"]))
        x = centres[rng.integers(0, 10, case["n"])] + rng.normal(size=(case["n"], case["dims"]))
        n, k = case["n"], case["k"]
        state["points"] = torch.from_numpy(x).to(DEV)
        cap = 2 * n * k
        state["out"] = {"indptr": torch.zeros(n + 1, dtype=torch.int64, device=DEV),
                        "indices": torch.zeros(cap, dtype=torch.int32, device=DEV),
                        "data": torch.zeros(cap, dtype=torch.float32, device=DEV),
                        "idx": torch.zeros(n, k, dtype=torch.int32, device=DEV),
                        "dist": torch.zeros(n, k, dtype=torch.float32, device=DEV),
                        "sigma": torch.zeros(n, dtype=torch.float32, device=DEV),
                        "rho": torch.zeros(n, dtype=torch.float32, device=DEV)}
    torch.cuda.synchronize()
    return state


# ---- one pass ---------------------------------------------------------------------------------------
def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "init" and case["where"] == "device":
        ip, ix, dv = state["graph"]
        g = SiCsrF32(case["n"], ix.numel(), ip.data_ptr(), ix.data_ptr(), dv.data_ptr())
        rep, cfg = SiReport(), state["config"].to_c()
        ctx.check(ctx.lib.si_spectral_init_device(ctx.ptr, C.byref(g), case["nc"], state["seed"], None, 0, C.byref(cfg),
                                                  state["out"].data_ptr(), C.byref(rep)), case["n"], case["nc"])
        return {"embedding": state["out"], "eigenvalues": np.array(rep.eigenvalues[:case["nc"] + 1])}
    if kind == "init":
        emb, rep = si.spectral_init(state["graph"], case["nc"], state["seed"], config=state["config"], return_report=True)
        return {"embedding": emb, "eigenvalues": np.array(rep.eigenvalues)}
    if kind == "components":
        return si.spectral_init(state["graph"], case["nc"], state["seed"], data=state["data"], config=state["config"])
    if kind == "apply":
        return state["op"].apply_prepared(state["x"], state["y"])
    if kind == "train":
        loss, grad = state["model"].gradient(state["lap"], state["target"], seed=state["seed"])
        return {"loss": loss, "grad": grad}
    o, x, nnz = state["out"], state["points"], C.c_uint64(0)
    ctx.check(ctx.lib.si_fuzzy_graph(ctx.ptr, x.data_ptr(), case["n"], case["dims"], case["k"], o["idx"].data_ptr(),
                                     o["dist"].data_ptr(), o["sigma"].data_ptr(), o["rho"].data_ptr(),
                                     o["indptr"].data_ptr(), o["indices"].data_ptr(), o["data"].data_ptr(),
                                     o["data"].numel(), C.byref(nnz)))
    return dict(o, nnz=nnz.value)


# ---- the same in 64 bits ------------------------------------------------------------------------------
def _philox_normals(seed, stream, count):
    """`count` pairs of the library's documented noise stream: Philox4x32-10 (Salmon et al., SC'11), Box-Muller."""
    i = np.arange(count, dtype=np.uint64)
    m32 = np.uint64(0xFFFFFFFF)
    c = [i & m32, i >> np.uint64(32), np.full(count, stream & 0xFFFFFFFF, np.uint64), np.full(count, stream >> 32, np.uint64)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & m32, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    u = [((((a << np.uint64(21)) ^ (b >> np.uint64(11))) & np.uint64((1 << 53) - 1)).astype(np.float64) + 0.5) * 2.0 ** -53
         for a, b in ((c[0], c[1]), (c[2], c[3]))]
    r = np.sqrt(-2.0 * np.log(u[0]))
    return np.stack([r * np.cos(2 * np.pi * u[1]), r * np.sin(2 * np.pi * u[1])], 1).reshape(-1)


def _exact_fuzzy(x, k):
    n, d = x.shape
    idx = torch.empty(n, k, dtype=torch.int64, device=DEV)
    dist = torch.empty(n, k, dtype=torch.float64, device=DEV)
    step = max(1, (1 << 27) // (n * d))
    for s in range(0, n, step):
        e = min(n, s + step)
        d2 = (x[s:e, None, :] - x[None, :, :]).square().sum(2)
        r = torch.arange(e - s, device=DEV)
        d2[r, r + s] = float("inf")
        v, i = torch.topk(d2, k, dim=1, largest=False, sorted=True)
        dist[s:e], idx[s:e] = v.sqrt(), i
    rho = torch.where(dist > 0, dist, torch.full_like(dist, float("inf"))).min(1).values
    rho = torch.where(torch.isinf(rho), torch.zeros_like(rho), rho)
    return {"indptr": None, "indices": None, "data": None, "idx": None, "dist": dist.cpu().numpy(), "sigma": None,
            "rho": rho.cpu().numpy(), "nnz": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "init" and case["n"] <= 6000:
        n, nc = case["n"], case["nc"]
        ip, ix, dv = _graph(n, case["k"], case["clusters"], case["dims"], case["order"], seed)
        rows, cols, v = _values64(ip, ix, dv, n)
        lap = torch.zeros(n, n, dtype=torch.float64, device=DEV)
        lap[rows, cols] = v
        lap.diagonal().add_(1.0)
        lam, vec = torch.linalg.eigh(lap)
        emb = vec[:, 1:nc + 1]
        top = emb.gather(0, emb.abs().argmax(0, keepdim=True))
        emb = emb * torch.where(top < 0, -1.0, 1.0)
        emb = (emb * (10.0 / emb.abs().max())).cpu().numpy()
        noise = _philox_normals(int(seed) % (1 << 31), 0x5CA1E, (n * nc + 1) // 2)[:n * nc].reshape(n, nc)
        return {"embedding": emb + 1e-4 * noise, "eigenvalues": lam[:nc + 1].cpu().numpy()}
    if kind == "apply":
        n = case["n"]
        ip, ix, dv = _graph(n, case["k"], case["clusters"], 50 if n >= 10_000 else 16, case["order"], seed)
        rows, cols, v = _values64(ip, ix, dv, n)
        g = torch.Generator(device=DEV)
        g.manual_seed(int(seed) % (1 << 31) + 2)
        x = torch.randn(n, case["cols"], generator=g, device=DEV, dtype=getattr(torch, case["dtype"])).double()
        return x.clone().index_add_(0, rows, v[:, None] * x[cols])
    if kind == "fuzzy":
        return _exact_fuzzy(prepare(case, seed)["points"], case["k"])
    return None


# ---- what a pass cannot do without ----------------------------------------------------------------------
def _entries(case):
    return int(case["n"] * case["k"] * 1.62)  # stored entries of the symmetric graph, as measured


def work(case):
    kind = case["kind"]
    if kind == "components":
        n = sum(_part_sizes(case))
        return {"bytes": n * (15 * 1.7 * 8 + 8 + 20 * 4 + 4 * case["nc"]), "flops": 0}
    n = case["n"]
    if kind == "init":
        return {"bytes": 8 * _entries(case) + 8 * n + 4 * n * case["nc"], "flops": 0}
    if kind == "apply":
        s = 4 if case["dtype"] == "float32" else 8
        return {"bytes": _entries(case) * (4 + s) + 8 * n + 2 * n * case["cols"] * s,
                "flops": 2 * _entries(case) * case["cols"]}
    if kind == "train":
        # forward and backward of three 128 x 64 layers and the 128 x 16 head over n rows
        return {"bytes": 8 * _entries(case) + 8 * n * (case["nc"] + 2), "flops": 6 * n * 128 * (3 * 64 + 16)}
    return {"bytes": 8 * n * case["dims"] + n * case["k"] * (8 + 16) + 16 * n, "flops": 3 * n * n * case["dims"]}
