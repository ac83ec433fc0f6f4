"""The work a user has this library do, as timed cases: kNN graphs of cytometry- and scRNA-like data.

Every case goes through a public entry point: the drop-in module `costal_gb300._costal` on host arrays
(what the reference's Python package calls), or the C ABI on host arrays or on data that already lies
on the GPU. Edge lists go to arrays that the program keeps (room for n k edges, as the C ABI asks for,
zero beyond the edges found), so that every pass returns arrays of one size. Sizes and distributions
are those of `costal_gb300.workloads`, of the tests and of the published reference runs; inputs are
drawn on the GPU from the seed alone.
"""

from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from costal_gb300 import _costal as ext
from costal_gb300 import _lib as L


def listed():
    return [
        # One gate or one small sample through the reference's package (costal.find_communities calls
        # _knn_exact, _reweight, _fuzzy_union in turn, with the default backend): latency.
        dict(name="dropin_small", op="dropin", data="mixture", clusters=8, n=1511, d=25, k=10),
        # A usual cytometry sample the same way (the mixture_20k workload).
        dict(name="dropin_20k", op="dropin", data="mixture", clusters=20, n=20_000, d=32, k=10),
        # Levine_32dim without its duplicate events has 161,443 rows: the reference's own full run.
        dict(name="dropin_161k", op="dropin", data="zipf", clusters=24, n=161_443, d=32, k=10),
        # Deep rows (highly variable genes) on the default backend, sizes of no round number.
        dict(name="knn_genes_10k", op="knn", data="scrna", clusters=15, n=10_007, d=501, k=15),
        # Tanimoto selection, where the norm of a cell counts too.
        dict(name="knn_tanimoto_100k", op="knn", data="rare", clusters=12, n=100_003, d=15, k=10, select="tanimoto"),
        # A small sample on the tensor-core backend (COSTAL_GB300_MATMUL=bf16 moves every call there).
        dict(name="graph_small", op="graph", data="mixture", clusters=8, n=5003, d=17, k=7, matmul="bf16"),
        # X to the Leiden's CSR with Jaccard weights, k = 30, noise and exact duplicates (dense_dup_160k).
        dict(name="csr_dup_160k", op="csr", data="dup", clusters=24, n=160_000, d=32, k=30, matmul="bf16",
             weight="jaccard"),
        # X to the edge list from host memory with a rare population (rare_400k).
        dict(name="graph_rare_400k", op="graph", data="rare", clusters=12, n=400_000, d=15, k=10, margin=8, matmul="bf16"),
        # Device-resident data, clusters of very different sizes.
        dict(name="device_600k", op="device", data="zipf", clusters=50, n=600_001, d=40, k=10, matmul="bf16"),
        # The benchmark's workload in its configuration: 2,000,000 x 40 with the learned block threshold.
        dict(name="device_2m_learned", op="device", data="zipf", clusters=50, n=2_000_000, d=40, k=10, matmul="bf16",
             learned=True),
        # scRNA-seq over 2,000 genes (scrna_100k), device-resident.
        dict(name="device_scrna_100k", op="device", data="scrna", clusters=15, n=100_000, d=2000, k=15, matmul="bf16"),
        # Training the block threshold: labels, features, Adam steps.
        dict(name="train_200k", op="train", data="zipf", clusters=50, n=200_000, d=40, k=10, sample=32_768, epochs=4),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["dropin", "dropin", "knn_deep", "tanimoto", "graph", "graph", "csr", "device", "device",
                       "device_deep", "train"])
    k = rng.choice([5, 7, 10, 10, 12, 15, 20, 30])
    data = rng.choice(["mixture", "zipf", "rare", "dup"])
    clusters = rng.randint(6, 50)
    if kind == "dropin":
        return dict(op="dropin", data=data, clusters=clusters, n=log_int(600, 200_000), d=rng.randint(6, 50), k=k)
    if kind == "knn_deep":
        return dict(op="knn", data="scrna", clusters=15, n=log_int(2000, 14_000), d=log_int(70, 2000), k=k)
    if kind == "tanimoto":
        return dict(op="knn", data=data, clusters=clusters, n=log_int(2000, 150_000), d=rng.randint(6, 50), k=k,
                    select="tanimoto")
    if kind in ("graph", "csr"):
        return dict(op=kind, data=data, clusters=clusters, n=log_int(1500, 500_000), d=rng.randint(6, 50), k=k,
                    matmul="bf16", weight=rng.choice(["tanimoto", "tanimoto", "jaccard", "cosine"]))
    if kind == "device":
        return dict(op="device", data=data, clusters=clusters, n=log_int(5000, 1_500_000), d=rng.randint(6, 40),
                    k=min(k, 15), matmul="bf16", learned=rng.random() < 0.25)
    if kind == "device_deep":
        return dict(op="device", data="scrna", clusters=15, n=log_int(3000, 90_000), d=log_int(130, 2000), k=k,
                    matmul="bf16")
    return dict(op="train", data=data, clusters=clusters, n=log_int(20_000, 200_000), d=rng.randint(6, 40), k=10,
                sample=rng.choice([8192, 20_000, 32_768]), epochs=rng.randint(2, 6))


# ---- inputs ----------------------------------------------------------------------------------------

_DEV = "cuda"


def _rows(case, seed):
    """The case's (n, d) float32 matrix on the GPU: the distributions of costal_gb300.workloads."""
    g = torch.Generator(device=_DEV)
    g.manual_seed(seed * 7919 + 17)
    n, d, kc = case["n"], case["d"], case["clusters"]

    def normal(*shape):
        return torch.randn(*shape, generator=g, device=_DEV)

    def uniform(*shape):
        return torch.rand(*shape, generator=g, device=_DEV)

    def some(m):  # m different rows
        return torch.randperm(n, generator=g, device=_DEV)[:m]

    if case["data"] == "scrna":  # negative-binomial counts of log-normal profiles, library size, log1p
        profiles = torch.exp(normal(kc, d) * 1.6 - 3.0)
        out = torch.empty(n, d, device=_DEV)
        for a in range(0, n, 8192):
            m = min(8192, n - a)
            mu = profiles[(uniform(m) * kc).long().clamp_(max=kc - 1)] * torch.exp(0.3 * normal(m, 1))
            gamma = -torch.log((1 - uniform(m, d)) * (1 - uniform(m, d)))  # shape 2: dispersion 0.5
            counts = torch.poisson(gamma * (mu / 2.0), generator=g)
            lib = counts.sum(1, keepdim=True).clamp_(min=1.0)
            out[a:a + m] = torch.log1p(counts / lib * 1e4)
        return out
    means, stds = normal(kc, d) * 2.0, 0.3 + 0.7 * uniform(kc, d)
    w = torch.ones(kc, device=_DEV)
    if case["data"] == "zipf":
        w = 1.0 / torch.arange(1, kc + 1, device=_DEV) ** 1.2
    cum = torch.cumsum(w / w.sum(), 0)
    lab = torch.searchsorted(cum, uniform(n)).clamp_(max=kc - 1)
    x = means[lab] + stds[lab] * normal(n, d)
    if case["data"] == "rare":  # one cell in a thousand in a tight population 3 sd off a cluster
        dirn = normal(d)
        m = max(1, n // 1000)
        x[some(m)] = means[0] + 3.0 * stds[0] * dirn / dirn.norm() + 0.5 * stds[0] * normal(m, d)
    if case["data"] == "dup":  # a tenth uniform noise, one row in a hundred an exact copy of another
        lo, hi = x.amin(0), x.amax(0)
        m = max(1, n // 10)
        x[some(m)] = lo + (hi - lo) * uniform(m, d)
        m = max(1, n // 100)
        x[some(m)] = x[some(m)]
    return torch.asinh(x / 5.0)


def prepare(case, seed):
    x = _rows(case, seed)
    n, k = case["n"], case["k"]
    state = {"case": case}
    if case["op"] != "device" or case.get("learned"):
        state["x"] = np.ascontiguousarray(x.cpu().numpy())
    if case.get("learned"):  # a model trained once and kept by the program
        ext._mlp_train(state.pop("x"), k, sample=min(n, 100_000), epochs=40, quantile=0.01)
        state["model"] = ext._mlp_get()
    most = (2 if case["op"] == "csr" else 1) * n * k
    if case["op"] == "device":
        state["x"] = x
        state["rows"] = torch.zeros(most, dtype=torch.int32, device=_DEV)
        state["cols"] = torch.zeros(most, dtype=torch.int32, device=_DEV)
        state["w"] = torch.zeros(most, dtype=torch.float64, device=_DEV)
    elif case["op"] in ("dropin", "graph", "csr"):
        # (a CSR's row pointers are u64 and its neighbours u32, all far below their signed types' limits)
        state["rows"] = np.full(n + 1, 0, np.int64) if case["op"] == "csr" else np.full(most, 0, np.int32)
        state["cols"] = np.full(most, 0, np.int32)
        state["w"] = np.full(most, 0.0, np.float64)
    return state


def _ptr(a):
    return C.c_void_p(a.data_ptr() if isinstance(a, torch.Tensor) else a.ctypes.data)


def _call(fn, *args):
    err, size = L.errbuf()
    L.check(fn(*args, err, size), err)


def _opts(case, learned):
    return L.KnnOpts(margin=case.get("margin", 0xFFFFFFFF), select=L.SELECT["cosine"],
                     backend={"fp32": L.BACKEND_FP32, "bf16": L.BACKEND_BF16}[case["matmul"]], sort_by_norm=1, prune=1,
                     learned_prune=int(learned))


def _build(state):
    case, x = state["case"], state["x"]
    n, d = x.shape
    if "model" in state:
        ext._mlp_set(*state["model"])
    m, st, o = C.c_uint64(0), L.KnnStats(), _opts(case, "model" in state)
    edges = (state["rows"], state["cols"], state["w"])
    args = (_ptr(x), n, d, case["k"], C.byref(o), L.WEIGHT[case.get("weight", "tanimoto")]) + tuple(map(_ptr, edges))
    if case["op"] == "device":
        _call(L.lib().costal_build_graph_device, *args, C.byref(m), C.byref(st),
              C.c_void_p(torch.cuda.current_stream().cuda_stream))
    elif case["op"] == "csr":
        _call(L.lib().costal_build_graph_csr, *args, C.byref(m), C.byref(st))
    else:
        _call(L.lib().costal_build_graph, *args, C.byref(m), None, None, None, C.byref(st))
    return edges + (m.value,)


def run(state):
    case, x = state["case"], state["x"]
    op, k = case["op"], case["k"]
    if op == "dropin":
        (idx, cos, norms), _ = ext._knn_exact(x, k)
        w = ext._reweight(idx, cos, norms, "tanimoto")
        m, edges = C.c_uint64(0), (state["rows"], state["cols"], state["w"])
        _call(L.lib().costal_fuzzy_union, case["n"], k, _ptr(idx), _ptr(w), *map(_ptr, edges), C.byref(m))
        return (idx, cos, norms, w) + edges + (m.value,)
    if op == "knn":
        return ext._knn_exact(x, k, select=case.get("select"), matmul=case.get("matmul"))[0]
    if op == "train":
        st = ext._mlp_train(x, k, sample=case["sample"], epochs=case["epochs"])
        params, _, _, _ = ext._mlp_get()
        return {"params": params, "loss": st["loss"], "mae": st["mae"], "coverage": st["coverage"]}
    return _build(state)


def work(case):
    """Every input read once and every output written once; two operations a dimension for every pair of
    rows (the similarities; the pair (i, j) and the pair (j, i) are one), and for training the network's
    forward and backward products."""
    n, d, k, op = case["n"], case["d"], case["k"], case["op"]
    flops = float(n) * n * d
    nbytes = 4.0 * n * d
    if op == "train":
        F = d + 64
        nets = 128 * F + 128 * 128 + 128
        m = min(n, case["sample"])
        return {"bytes": nbytes + 4.0 * (nets + 257), "flops": 2.0 * m * n * d + 6.0 * m * nets * case["epochs"]}
    if op in ("dropin", "knn"):
        nbytes += n * k * 12.0 + n * 8.0
    if op == "dropin":
        nbytes += n * k * 8.0
    if op != "knn":  # about 0.85 n k edges, 16 bytes each (CSR: 12 bytes in both directions)
        nbytes += 0.85 * n * k * (24.0 if op == "csr" else 16.0)
    return {"bytes": nbytes, "flops": flops}


# ---- the same outputs in 64 bits, without the library ----------------------------------------------

def _exact_knn(x, k, select):
    """(idx, cos, norms) of the rows of x (float64, on the GPU): every pair, ties by index."""
    n = x.shape[0]
    norms = x.norm(dim=1)
    xn = x / norms.clamp(min=1e-300)[:, None]
    more = min(n - 1, k + 24)
    idx = torch.empty(n, k, dtype=torch.int64, device=x.device)
    cos = torch.empty(n, k, dtype=torch.float64, device=x.device)
    step = max(1, min(4096, (1 << 28) // n))
    for a in range(0, n, step):
        b = min(n, a + step)
        s = xn[a:b] @ xn.T
        if select == "tanimoto":
            ab = norms[a:b, None] * norms[None, :] * s
            s = ab / (norms[a:b, None] ** 2 + norms[None, :] ** 2 - ab)
        s[torch.arange(b - a, device=x.device), torch.arange(a, b, device=x.device)] = -math.inf
        cand = s.topk(more, dim=1).indices.sort(dim=1).values
        c = torch.empty(b - a, more, dtype=torch.float64, device=x.device)
        for r in range(0, b - a, 512):  # the same sum for equal rows, whatever their place
            q = min(b - a, r + 512)
            c[r:q] = (x[cand[r:q]] * x[a + r:a + q, None, :]).sum(-1)
        c = c / (norms[a:b, None] * norms[cand]).clamp(min=1e-300)
        t = c
        if select == "tanimoto":
            ab = norms[a:b, None] * norms[cand] * c
            t = ab / (norms[a:b, None] ** 2 + norms[cand] ** 2 - ab)
        o = t.sort(dim=1, descending=True, stable=True).indices[:, :k]
        idx[a:b], cos[a:b] = cand.gather(1, o), c.gather(1, o)
    return idx, cos, norms


def _exact_weights(idx, cos, norms, weight):
    if weight == "cosine":
        return cos
    if weight == "tanimoto":
        ab = norms[:, None] * norms[idx] * cos
        return ab / (norms[:, None] ** 2 + norms[idx] ** 2 - ab)
    n, k = idx.shape
    srt = idx.sort(dim=1).values
    w = torch.empty(n, k, dtype=torch.float64, device=idx.device)
    for a in range(0, n, 4096):
        b = min(n, a + 4096)
        other = srt[idx[a:b]]  # (rows, k, k)
        at = torch.searchsorted(srt[a:b, None, :].expand(-1, k, -1).contiguous(), other).clamp(max=k - 1)
        s = (srt[a:b, None, :].expand(-1, k, -1).gather(2, at) == other).sum(2).double()
        w[a:b] = s / (2.0 * k - s)
    return w


def _exact_union(idx, w):
    """Upper-triangular (lo * n + hi ascending) edge keys and weights a + b - a b."""
    n, k = idx.shape
    i = torch.arange(n, device=idx.device).repeat_interleave(k)
    j, w = idx.reshape(-1), w.reshape(-1)
    key, o = (torch.minimum(i, j) * n + torch.maximum(i, j)).sort(stable=True)
    w = w[o]
    first = torch.ones_like(key, dtype=torch.bool)
    first[1:] = key[1:] != key[:-1]
    at = torch.nonzero(first).flatten()
    v = w[at].clone()
    two = torch.zeros_like(at, dtype=torch.bool)
    two[:-1] = at[1:] - at[:-1] == 2
    two[-1] = len(key) - at[-1] == 2
    b = w[at[two] + 1]
    v[two] = v[two] + b - v[two] * b
    keep = v != 0
    return key[at][keep], v[keep]


def exact(case, seed):
    n, d, k, op = case["n"], case["d"], case["k"], case["op"]
    if op == "train" or float(n) * n * (d + 100) > 6e12:
        return None  # (training in f32 steps has no such value; the others would take too long)
    x = _rows(case, seed).double()
    idx, cos, norms = _exact_knn(x, k, case.get("select") or "cosine")
    if op == "knn":
        return None, cos.cpu().numpy(), norms.cpu().numpy()
    weight = case.get("weight", "tanimoto")
    w = _exact_weights(idx, cos, norms, weight)
    key, v = _exact_union(idx, w)
    if op == "csr":
        src = torch.cat([key // n, key % n])
        dst = torch.cat([key % n, key // n])
        v = torch.cat([v, v])[(src * n + dst).sort().indices]
    edges = np.zeros((2 if op == "csr" else 1) * n * k)
    edges[:len(v)] = v.cpu().numpy()
    if op == "dropin":
        return None, cos.cpu().numpy(), norms.cpu().numpy(), w.cpu().numpy(), None, None, edges, None
    return None, None, edges, None
