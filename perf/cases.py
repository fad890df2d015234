"""What a user of this package has it do, as cases whose time can be taken.

Each case goes through a public entry point: ``pp.neighbors`` on an AnnData
(host arrays in and out), the device-pointer graph and kNN calls of the C ABI
on embeddings that already sit in HBM, a batch plan, the query service, and
the steps before and after the neighbour graph (PCA, UMAP, Leiden).  The
embeddings are Gaussian mixtures with a decaying spectrum, 1% duplicated
cells and about one cluster per 2,500-5,000 cells, the shape PCA gives.

listed()            the named cases
draw(rng)           another case of the same ranges
prepare(case, seed) inputs and handles, on the GPU unless the call takes host
                    arrays
run(state)          one pass, all its outputs; a graph's entries go into arrays
                    the caller keeps, sized for the 2 n k entries a union of n
                    rows of k can have, with zeros after the last one
work(case)          bytes and operations a pass cannot do without
exact(case, seed)   the computed numbers in 64 bits, where they have a value
"""

from __future__ import annotations

import ctypes
import math
import weakref

import numpy as np
import torch

from mrustsc_gb300 import _lib, _scrust, pp, serving, tl
from mrustsc_gb300.anndata_lite import AnnData

DEVICE = "cuda"
ATLAS_CELLS = 1_000_000  # cells of the atlas that the query service holds


def listed() -> list[dict]:
    return [
        # A first look at a small experiment (the 2,638-cell set every tutorial
        # of this field starts with): one call on host arrays, latency-bound.
        {"name": "neighbors_2638", "kind": "neighbors", "n": 2638, "d": 50, "n_neighbors": 15, "metric": "euclidean"},
        # One tissue sample, cosine metric as latent spaces of generative
        # models are often compared, with the wider neighbourhood.
        {"name": "neighbors_30011_cosine", "kind": "neighbors", "n": 30_011, "d": 50, "n_neighbors": 31,
         "metric": "cosine"},
        # A study: 100k cells, 30 neighbours, the embedding left in HBM by PCA.
        {"name": "graph_100k_k30", "kind": "graph", "n": 100_000, "d": 50, "k": 30, "metric": "euclidean"},
        # An atlas: the headline size, a million cells and the default 15.
        {"name": "graph_1m_k15", "kind": "graph", "n": 1_000_000, "d": 50, "k": 15, "metric": "euclidean"},
        # A smooth, large neighbourhood (k above 32) of a 30-wide latent space.
        {"name": "knn_50021_k50", "kind": "knn", "n": 50_021, "d": 30, "k": 50, "metric": "euclidean"},
        # All 100 components a PCA kept rather than the first 50.
        {"name": "knn_30007_d100", "kind": "knn", "n": 30_007, "d": 100, "k": 15, "metric": "euclidean"},
        # Sixteen donors, each its own graph, rebuilt by one plan launch.
        {"name": "batch_16_samples", "kind": "batch", "samples": 16, "lo": 500, "hi": 20_000, "d": 50, "k": 15},
        # One cell looked up in a resident atlas: the shortest request.
        {"name": "query_1", "kind": "query", "q": 1, "d": 50, "k": 15},
        # A sample mapped onto the atlas.
        {"name": "query_5000", "kind": "query", "q": 5000, "d": 50, "k": 15},
        # The layout of the graph, the reference's default 200 epochs.
        {"name": "umap_30000", "kind": "umap", "n": 30_000, "k": 15, "epochs": 200},
        # PCA of a log-normalised count matrix restricted to 2,000 variable genes.
        {"name": "pca_30000_x2000", "kind": "pca", "n": 30_000, "genes": 2000, "density": 0.1, "components": 50},
        # Leiden communities of the graph, default resolution and iterations.
        {"name": "leiden_60000", "kind": "leiden", "n": 60_000, "k": 15, "resolution": 1.0},
    ]


def draw(rng) -> dict:
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["neighbors", "neighbors", "graph", "graph", "graph", "knn", "knn", "wide", "batch", "query",
                       "query", "umap", "pca", "leiden"])
    metric = rng.choice(["euclidean", "euclidean", "cosine"])
    if kind == "neighbors":
        return {"kind": kind, "n": log(400, 60_000), "d": rng.randint(10, 61), "n_neighbors": rng.randint(5, 33),
                "metric": metric}
    if kind == "graph":
        return {"kind": kind, "n": log(2000, 500_000), "d": rng.randint(10, 60), "k": rng.randint(5, 32),
                "metric": metric}
    if kind == "knn":
        return {"kind": kind, "n": log(3000, 60_000), "d": rng.randint(10, 60), "k": rng.randint(33, 100),
                "metric": metric}
    if kind == "wide":
        return {"kind": "knn", "n": log(2000, 60_000), "d": rng.randint(62, 104), "k": rng.randint(5, 30),
                "metric": metric}
    if kind == "batch":
        return {"kind": kind, "samples": rng.randint(3, 24), "lo": rng.randint(200, 1000), "hi": rng.randint(5000, 20_000),
                "d": rng.randint(20, 60), "k": rng.randint(8, 30)}
    if kind == "query":
        return {"kind": kind, "q": log(1, 20_000), "d": rng.randint(20, 60), "k": rng.randint(5, 30)}
    if kind == "umap":
        return {"kind": kind, "n": log(3000, 30_000), "k": rng.randint(8, 15), "epochs": rng.randint(100, 200)}
    if kind == "pca":
        return {"kind": kind, "n": log(3000, 30_000), "genes": rng.randint(1000, 2000),
                "density": round(rng.uniform(0.04, 0.1), 3), "components": rng.randint(20, 50)}
    return {"kind": kind, "n": log(3000, 60_000), "k": rng.randint(8, 15), "resolution": round(rng.uniform(0.5, 1.5), 2)}


# --------------------------------------------------------------------------- inputs

def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device=DEVICE).manual_seed(int(seed) * 7919 + 17)


def _clusters(n: int) -> int:
    return max(4, min(200, n // 2500))


def _mixture(n: int, d: int, clusters: int, gen: torch.Generator, centres=None, dup: float = 0.01) -> torch.Tensor:
    """(n, d) float32: cluster centres uniform in [-5, 5]^d, standard deviation
    2 / sqrt(i) in dimension i, and `dup` of the rows copies of other rows."""
    if centres is None:
        centres = torch.rand((clusters, d), generator=gen, device=DEVICE) * 10 - 5
    std = 2.0 / torch.arange(1, d + 1, device=DEVICE, dtype=torch.float32).sqrt()
    x = torch.randn((n, d), generator=gen, device=DEVICE) * std
    x += centres[torch.randint(len(centres), (n,), generator=gen, device=DEVICE)]
    copies = int(round(dup * n))
    if copies:
        rows = torch.randperm(n, generator=gen, device=DEVICE)[: 2 * copies]
        x[rows[:copies]] = x[rows[copies:]]
    return x.contiguous()


def _embedding(case: dict, seed: int) -> torch.Tensor:
    return _mixture(case["n"], case["d"], _clusters(case["n"]), _generator(seed))


def _batch_sizes(case: dict) -> list[int]:
    """Sample sizes, spread over [lo, hi] by their logarithm; the case's own."""
    r = np.random.RandomState(case["samples"])
    return [int(v) for v in np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]), case["samples"]))]


def _atlas(case: dict, seed: int):
    gen = _generator(seed)
    centres = torch.rand((_clusters(ATLAS_CELLS), case["d"]), generator=gen, device=DEVICE) * 10 - 5
    atlas = _mixture(ATLAS_CELLS, case["d"], 0, gen, centres, dup=0.0)
    queries = _mixture(case["q"], case["d"], 0, gen, centres, dup=0.0)
    queries += 0.1 * torch.randn(queries.shape, generator=gen, device=DEVICE)
    return atlas, queries


def _graph(n: int, k: int, seed: int):
    """A symmetric weighted kNN graph (host CSR, sorted columns) of a 20-wide
    mixture: exp weights from each row's mean neighbour distance, fuzzy union."""
    x = _mixture(n, 20, _clusters(n), _generator(seed))
    sq = (x * x).sum(1)
    rows, cols, vals = [], [], []
    for a in range(0, n, 4096):
        b = min(n, a + 4096)
        d2 = sq[a:b, None] + sq[None, :] - 2.0 * (x[a:b] @ x.T)
        d2[torch.arange(b - a, device=DEVICE), torch.arange(a, b, device=DEVICE)] = math.inf
        v, j = torch.topk(d2, k, dim=1, largest=False)
        dist = v.clamp_min(0).sqrt()
        rho = dist[:, :1]
        w = torch.exp(-(dist - rho) / (dist - rho).mean(1, keepdim=True).clamp_min(1e-6))
        rows.append(torch.arange(a, b, device=DEVICE).repeat_interleave(k))
        cols.append(j.reshape(-1))
        vals.append(w.reshape(-1))
    i, j, w = torch.cat(rows), torch.cat(cols), torch.cat(vals)
    both = torch.cat([i * n + j, j * n + i])
    key, slot = torch.unique(both, return_inverse=True)
    forward = torch.zeros(len(key), device=DEVICE)
    backward = torch.zeros(len(key), device=DEVICE)
    m = len(i)
    forward[slot[:m]] = w
    backward[slot[m:]] = w
    value = forward + backward - forward * backward
    keep = value > 0
    key, value = key[keep], value[keep]
    indptr = torch.zeros(n + 1, dtype=torch.int64, device=DEVICE)
    indptr[1:] = torch.cumsum(torch.bincount(key // n, minlength=n), 0)
    return (indptr.cpu().numpy().astype(np.uint32), (key % n).cpu().numpy().astype(np.uint32),
            value.cpu().numpy().astype(np.float32))


def _counts(case: dict, seed: int):
    """A cells x genes CSR of log-normalised counts: 60 expression programmes
    with falling strengths on top of gene-wise rates, `density` of it non-zero."""
    gen = _generator(seed)
    n, g = case["n"], case["genes"]
    strength = 3.0 * 0.93 ** torch.arange(60, device=DEVICE)
    programme = torch.randn((60, g), generator=gen, device=DEVICE) * strength[:, None] / math.sqrt(g) * 4
    usage = torch.randn((n, 60), generator=gen, device=DEVICE)
    dense = usage @ programme + 0.5 * torch.randn((n, g), generator=gen, device=DEVICE)
    dense += 0.3 * torch.randn(g, generator=gen, device=DEVICE)
    cut = torch.quantile(dense.reshape(-1)[:1_000_000], 1.0 - case["density"])
    dense = torch.log1p((dense - cut).clamp_min(0) * 3)
    csr = dense.to_sparse_csr()
    return (csr.crow_indices().cpu().numpy().astype(np.uint32), csr.col_indices().cpu().numpy().astype(np.uint32),
            csr.values().cpu().numpy().astype(np.float32))


# --------------------------------------------------------------------------- states

class _DeviceView:
    """A library-owned device array, for torch.as_tensor."""

    def __init__(self, ptr: int, count: int, typestr: str):
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 2}


def _stream():
    """The library's stream, for torch work ordered with it."""
    return torch.cuda.ExternalStream(_lib.lib().scrust_cuda_context_stream(_lib.context(0)))


class _DeviceGraph:
    """The caller's own arrays for a graph's CSR, in HBM."""

    def __init__(self, n: int, k: int):
        self.indptr = torch.zeros(n + 1, dtype=torch.int32, device=DEVICE)
        self.columns = torch.zeros(2 * n * k, dtype=torch.int32, device=DEVICE)
        self.weights = torch.zeros(2 * n * k, dtype=torch.float32, device=DEVICE)

    def take(self, indptr: int, columns: int, weights: int, nnz: int) -> dict:
        """Copies a CSR the library owns; on the library's stream."""
        self.indptr.copy_(torch.as_tensor(_DeviceView(indptr, len(self.indptr), "<i4"), device=DEVICE))
        for mine, ptr, kind in ((self.columns, columns, "<i4"), (self.weights, weights, "<f4")):
            if nnz:
                mine[:nnz].copy_(torch.as_tensor(_DeviceView(ptr, nnz, kind), device=DEVICE))
            mine[nnz:].zero_()
        return {"indptr": self.indptr, "columns": self.columns, "weights": self.weights}


class _HostGraph:
    """The same on the host."""

    def __init__(self, n: int, entries: int):
        self.columns = np.zeros(entries, dtype=np.uint32)
        self.weights = np.zeros(entries, dtype=np.float32)

    def take(self, indptr, columns, weights) -> dict:
        nnz = len(columns)
        self.columns[:nnz], self.columns[nnz:] = columns, 0
        self.weights[:nnz], self.weights[nnz:] = weights, 0
        return {"indptr": indptr, "columns": self.columns, "weights": self.weights}


class _DeviceSolve:
    """An embedding in HBM and the output arrays."""

    def __init__(self, case: dict, seed: int):
        self.x = _embedding(case, seed)
        self.n, self.d, self.k = case["n"], case["d"], case["k"]
        self.idx = torch.empty((self.n, self.k), dtype=torch.int32, device=DEVICE)
        self.dist = torch.empty((self.n, self.k), dtype=torch.float32, device=DEVICE)
        self.options = _lib.options(metric=case["metric"])
        self.ctx = _lib.context(0)
        self.mine = _DeviceGraph(self.n, self.k) if case["kind"] == "graph" else None
        self.status = _lib.Status()
        torch.cuda.synchronize()

    def knn(self):
        L = _lib.lib()
        st = ctypes.byref(self.status)
        _lib.check(L.scrust_cuda_knn_device(self.ctx, self.x.data_ptr(), self.n, self.d, self.k,
                                            ctypes.byref(self.options), self.idx.data_ptr(), self.dist.data_ptr(), st),
                   self.status)
        return {"indices": self.idx, "distances": self.dist}

    def graph(self):
        L = _lib.lib()
        st = ctypes.byref(self.status)
        out = ctypes.c_void_p()
        _lib.check(L.scrust_cuda_neighbors_graph_device(self.ctx, self.x.data_ptr(), self.n, self.d, self.k,
                                                        ctypes.byref(self.options), self.idx.data_ptr(),
                                                        self.dist.data_ptr(), ctypes.byref(out), st), self.status)
        try:
            # The entry count of a device CSR is known once the stream is idle.
            _lib.check(L.scrust_cuda_synchronize(self.ctx, st), self.status)
            with torch.cuda.stream(_stream()):
                graph = self.mine.take(L.scrust_csr_indptr(out), L.scrust_csr_indices(out), L.scrust_csr_values(out),
                                       int(L.scrust_csr_nnz(out)))
        finally:
            L.scrust_csr_free(out)
        return {"indices": self.idx, "distances": self.dist, **graph}


class _BatchPlan:
    """Samples concatenated in HBM and the plan that builds all their graphs."""

    def __init__(self, case: dict, seed: int):
        sizes = _batch_sizes(case)
        gen = _generator(seed)
        self.n, self.k = sum(sizes), case["k"]
        self.x = torch.cat([_mixture(s, case["d"], max(4, s // 1000), gen) for s in sizes])
        self.idx = torch.empty((self.n, self.k), dtype=torch.int32, device=DEVICE)
        self.dist = torch.empty((self.n, self.k), dtype=torch.float32, device=DEVICE)
        offsets = np.zeros(len(sizes) + 1, dtype=np.uint64)
        offsets[1:] = np.cumsum(sizes)
        torch.cuda.synchronize()
        L = _lib.lib()
        self.status = _lib.Status()
        self.ctx = _lib.context(0)
        options = _lib.options(form="tensor")
        self.plan = L.scrust_cuda_batch_plan_create_graphs(self.ctx, _lib.ptr(offsets), len(sizes), case["d"], self.k,
                                                           ctypes.byref(options), self.x.data_ptr(),
                                                           self.idx.data_ptr(), self.dist.data_ptr(),
                                                           ctypes.byref(self.status))
        if not self.plan:
            _lib.check(self.status.code or _lib.KERNEL, self.status)
        weakref.finalize(self, L.scrust_cuda_batch_plan_destroy, self.plan)
        self.mine = _DeviceGraph(self.n, self.k)
        ip, ix, vl = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
        L.scrust_cuda_batch_plan_graph(self.plan, ctypes.byref(ip), ctypes.byref(ix), ctypes.byref(vl))
        self.csr = (ip.value, ix.value, vl.value)

    def launch(self):
        L = _lib.lib()
        st = ctypes.byref(self.status)
        _lib.check(L.scrust_cuda_batch_plan_launch(self.plan, st), self.status)
        _lib.check(L.scrust_cuda_synchronize(self.ctx, st), self.status)
        with torch.cuda.stream(_stream()):
            nnz = int(torch.as_tensor(_DeviceView(self.csr[0] + 4 * self.n, 1, "<i4"), device=DEVICE).item())
            graph = self.mine.take(*self.csr, nnz)
        return {"indices": self.idx, "distances": self.dist, **graph}


class _Service:
    """The query service over an atlas, and one request's cells."""

    def __init__(self, case: dict, seed: int):
        atlas, queries = _atlas(case, seed)
        self.queries = queries.cpu().numpy()
        self.server = serving.Server(atlas.cpu().numpy(), case["k"])
        self.mine = _HostGraph(case["q"], case["q"] * case["k"])
        weakref.finalize(self, self.server.close)

    def query(self):
        idx, dist, csr, _ = self.server.query(self.queries)
        return {"indices": idx, "distances": dist, **self.mine.take(*csr)}


def _scipy_csr(parts, n_cols: int):
    import scipy.sparse as sp

    indptr, indices, values = parts
    return sp.csr_matrix((values, indices.astype(np.int32), indptr.astype(np.int32)), shape=(len(indptr) - 1, n_cols))


def prepare(case: dict, seed: int):
    kind = case["kind"]
    if kind == "neighbors":
        x = _embedding(case, seed).cpu().numpy()
        k = case["n_neighbors"] - 1
        return (kind, AnnData(obsm={"X_pca": x}), dict(n_neighbors=case["n_neighbors"], metric=case["metric"]),
                _HostGraph(case["n"], 2 * case["n"] * k))
    if kind in ("graph", "knn"):
        return kind, _DeviceSolve(case, seed)
    if kind == "batch":
        return kind, _BatchPlan(case, seed)
    if kind == "query":
        return kind, _Service(case, seed)
    if kind == "umap":
        adata = AnnData(n_obs=case["n"])
        adata.obsp["connectivities"] = _scipy_csr(_graph(case["n"], case["k"], seed), case["n"])
        return kind, adata, dict(n_epochs=case["epochs"], random_state=int(seed) % 1000)
    if kind == "pca":
        adata = AnnData(_scipy_csr(_counts(case, seed), case["genes"]))
        return kind, adata, dict(n_comps=case["components"])
    if kind == "leiden":
        return kind, _graph(case["n"], case["k"], seed), case["n"], case["resolution"]
    raise ValueError(f"unknown kind {kind!r}")


def run(state):
    kind = state[0]
    if kind == "neighbors":
        adata = state[1]
        pp.neighbors(adata, **state[2])
        d, c = adata.obsp["distances"], adata.obsp["connectivities"]
        return {"indices": d.indices, "distances": d.data, **state[3].take(c.indptr, c.indices, c.data)}
    if kind == "graph":
        return state[1].graph()
    if kind == "knn":
        return state[1].knn()
    if kind == "batch":
        return state[1].launch()
    if kind == "query":
        return state[1].query()
    if kind == "umap":
        tl.umap(state[1], **state[2])
        return state[1].obsm["X_umap"]
    if kind == "pca":
        adata = state[1]
        pp.pca(adata, **state[2])
        return {"embedding": adata.obsm["X_pca"], "components": adata.varm["PCs"],
                "variance": adata.uns["pca"]["variance"], "variance_ratio": adata.uns["pca"]["variance_ratio"]}
    (indptr, indices, values), n, resolution = state[1], state[2], state[3]
    labels, modularity, count = _scrust.leiden(indptr, indices, values, n, resolution, 2, 0, "auto")
    return {"labels": labels, "modularity": modularity, "communities": count}


def work(case: dict) -> dict:
    """Inputs read once and outputs written once; for exact neighbours the
    operations of the k reported distances (which columns those are can be
    known from bounds without a product with every one), for the rest the
    arithmetic the method is made of."""
    kind = case["kind"]
    if kind in ("neighbors", "graph", "knn"):
        n, d = case["n"], case["d"]
        k = case["n_neighbors"] - 1 if kind == "neighbors" else case["k"]
        graph = kind != "knn"
        # A union has between n k and 2 n k entries: 1.5 n k of 8 bytes.
        return {"bytes": 4.0 * n * d + 8.0 * n * k + (12.0 * n * k + 4.0 * n if graph else 0.0),
                "flops": 3.0 * n * k * d + (60.0 * n * k if graph else 0.0)}
    if kind == "batch":
        n, d, k = sum(_batch_sizes(case)), case["d"], case["k"]
        return {"bytes": 4.0 * n * d + 20.0 * n * k + 4.0 * n, "flops": 3.0 * n * k * d + 60.0 * n * k}
    if kind == "query":
        q, d, k = case["q"], case["d"], case["k"]
        return {"bytes": 4.0 * q * d + 16.0 * q * k + 4.0 * q + 4.0 * q * k * d, "flops": 3.0 * q * k * d + 60.0 * q * k}
    if kind == "umap":
        n, edges = case["n"], 1.5 * case["n"] * case["k"]
        # Each epoch reads and writes the layout; about a third of the edges fires in one,
        # each with five negative samples of about 20 operations.
        return {"bytes": 8.0 * edges + 16.0 * n * case["epochs"], "flops": case["epochs"] * edges / 3.0 * 6.0 * 20.0}
    if kind == "pca":
        nnz = case["n"] * case["genes"] * case["density"]
        width = case["components"] + 24
        return {"bytes": 8.0 * nnz + 4.0 * (case["n"] + case["genes"]) * case["components"],
                "flops": 2.0 * nnz * width * 2 * 5 + 4.0 * case["n"] * width * width * 5}
    edges = 1.5 * case["n"] * case["k"]
    # Ten sweeps over the edges bring the moves of two iterations to rest.
    return {"bytes": 8.0 * edges + 4.0 * case["n"], "flops": 10.0 * 4.0 * edges}


# --------------------------------------------------------------------------- in 64 bits

def _nearest(q: torch.Tensor, x: torch.Tensor, k: int, own: bool, cosine: bool):
    """k nearest rows of x for each row of q in float64 (row i itself left out
    when `own`): (ids, distances), nearest first, ties to the smaller id."""
    q, x = q.double(), x.double()
    if cosine:
        q, x = q / q.norm(dim=1, keepdim=True), x / x.norm(dim=1, keepdim=True)
    more = min(len(x), k + 24)
    sq = (x * x).sum(1)
    ids, dists = [], []
    rows = max(16, min(4096, 400_000_000 // len(x)))
    for a in range(0, len(q), rows):
        p = q[a:a + rows]
        d2 = sq[None, :] - 2.0 * (p @ x.T)
        if own:
            i = torch.arange(len(p), device=DEVICE)
            d2[i, i + a] = math.inf
        near = torch.topk(d2, more, dim=1, largest=False).indices.sort(dim=1).values
        if cosine:
            d = (1.0 - torch.einsum("rd,rcd->rc", p, x[near])).clamp_min(0)
        else:
            d = (p[:, None, :] - x[near]).square().sum(2).sqrt()
        if own:
            d = torch.where(near == torch.arange(a, a + len(p), device=DEVICE)[:, None], math.inf, d)
        d, order = torch.sort(d, dim=1, stable=True)
        ids.append(torch.gather(near, 1, order)[:, :k])
        dists.append(d[:, :k])
    return torch.cat(ids), torch.cat(dists)


def _directed(dist: torch.Tensor, mean=None) -> torch.Tensor:
    """umap's smooth_knn_dist weights of each row's neighbours, in float64."""
    n, k = dist.shape
    target = math.log2(k + 1)
    rho = torch.where(dist > 0, dist, math.inf).min(1).values
    rho = torch.where(torch.isinf(rho), 0.0, rho)
    offset = dist - rho[:, None]
    low, high = torch.zeros(n, device=DEVICE, dtype=torch.float64), torch.full((n,), math.inf, device=DEVICE, dtype=torch.float64)
    mid = torch.ones(n, device=DEVICE, dtype=torch.float64)
    open_ = torch.ones(n, device=DEVICE, dtype=torch.bool)
    for _ in range(64):
        total = torch.where(offset > 0, torch.exp(-offset / mid[:, None]), 1.0).sum(1)
        open_ &= (total - target).abs() >= 1e-5
        over = total > target
        high = torch.where(open_ & over, mid, high)
        low = torch.where(open_ & ~over, mid, low)
        step = torch.where(torch.isinf(high), mid * 2, (low + high) / 2)
        mid = torch.where(open_, step, mid)
    mean = dist.mean() if mean is None else mean
    reference = torch.where(rho > 0, dist.sum(1) / (k + 1), mean)
    sigma = torch.maximum(mid, 1e-3 * reference)
    return torch.where(offset <= 0, 1.0, torch.exp(-offset / sigma[:, None]))


def _union(ids: torch.Tensor, weights: torch.Tensor) -> torch.Tensor:
    """Values of the fuzzy union A + A^T - A o A^T in CSR order."""
    n, k = ids.shape
    i = torch.arange(n, device=DEVICE).repeat_interleave(k)
    j, w = ids.reshape(-1), weights.reshape(-1)
    keep = w.float() != 0
    i, j, w = i[keep], j[keep], w[keep]
    key, slot = torch.unique(torch.cat([i * n + j, j * n + i]), return_inverse=True)
    a = torch.zeros(len(key), device=DEVICE, dtype=torch.float64)
    b = torch.zeros(len(key), device=DEVICE, dtype=torch.float64)
    a[slot[:len(i)]] = w
    b[slot[len(i):]] = w
    return a + b - a * b


def _padded(values: torch.Tensor, entries: int) -> torch.Tensor:
    return torch.cat([values, values.new_zeros(entries - len(values))])


def _exact_self(x: torch.Tensor, k: int, cosine: bool, graph: bool) -> dict:
    ids, dist = _nearest(x, x, k, True, cosine)
    out = {"indices": None, "distances": dist}
    if graph:
        # A copied cell's cosine distance is a rounding error or zero, and the
        # weights of its row hang on which: no value to hold them to.
        out.update(indptr=None, columns=None, weights=None if cosine else _union(ids, _directed(dist)))
    return out


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("neighbors", "graph", "knn"):
        if case["n"] > 150_000:
            return None  # minutes of float64 products
        k = case["n_neighbors"] - 1 if kind == "neighbors" else case["k"]
        out = _exact_self(_embedding(case, seed), k, case["metric"] == "cosine", kind != "knn")
        if out.get("weights") is not None:
            out["weights"] = _padded(out["weights"], 2 * case["n"] * k)
        if kind == "neighbors":
            out["distances"] = out["distances"].reshape(-1)
        return out
    if kind == "batch":
        gen = _generator(seed)
        parts = []
        for s in _batch_sizes(case):
            parts.append(_exact_self(_mixture(s, case["d"], max(4, s // 1000), gen), case["k"], False, True))
        return {"indices": None, "distances": torch.cat([p["distances"] for p in parts]), "indptr": None,
                "columns": None,
                "weights": _padded(torch.cat([p["weights"] for p in parts]), 2 * sum(_batch_sizes(case)) * case["k"])}
    if kind == "query":
        atlas, queries = _atlas(case, seed)
        ids, dist = _nearest(queries, atlas, case["k"], False, False)
        order = ids.argsort(1)
        weights = torch.gather(_directed(dist), 1, order).reshape(-1)
        return {"indices": None, "distances": dist, "indptr": None, "columns": None,
                "weights": _padded(weights[weights.float() != 0], case["q"] * case["k"])}
    if kind == "pca":
        indptr, indices, values = _counts(case, seed)
        x = torch.from_numpy(_scipy_csr((indptr, indices, values), case["genes"]).toarray()).to(DEVICE).double()
        n, m = x.shape[0], case["components"]
        x -= x.mean(0)
        variance, vectors = torch.linalg.eigh(x.T @ x / (n - 1))
        variance, vectors = variance.flip(0)[:m], vectors.flip(1)[:, :m]
        total = x.square().sum() / (n - 1)
        # A component's sign is free; the mean of its loadings' signs is not known here.
        return {"embedding": None, "components": None, "variance": variance, "variance_ratio": variance / total}
    # A layout by stochastic gradient steps and a greedy partition have no
    # value that plain 64-bit arithmetic would give.
    return None
