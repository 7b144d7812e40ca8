"""The work that users of the package have it do, as cases that can be timed and compared.

A case is one stage or one stretch of the embedding path (count matrix -> filter and
feature selection -> normalise -> scale -> irlba PCA -> neighbours -> SNN graph) called
through the package's public functions.  Counts are seeded negative-binomial draws with
the parameters of the benchmark's workloads: gene means LogNormal(-1.2, 1.6), cell size
factors LogNormal(0, 0.3), dispersion 0.2, and clusters with log-fold-changes
Normal(0, 0.8) on 5% of the genes, the depth set so that a cell has `nnz` detected genes.
Where the size of an output follows from the data (the entries of a matrix or a graph), the
seed gives the order of one sample's cells and genes; elsewhere it gives the counts.
"""
import functools
import math

import numpy as np
import torch

import __graft_entry__

DISPERSION = 0.2
PRUNE = 1.0 / 15.0


@functools.lru_cache(maxsize=None)
def package():
    return __graft_entry__.load_package()


def listed():
    return [
        # Normalising one small sample in the reference's default type and taking the values
        # back: what an interactive session does first, and the smallest count matrices.
        dict(name="normalize_small", kind="normalize", cells=2000, genes=20000, nnz=1000, dtype="float64",
             method="lognormalize"),
        # Normalise and scale an ordinary sample (FP32) over its variable features: the stage before
        # every PCA, both copies of the counts streamed once.
        dict(name="scale_plain", kind="scale", cells=100000, genes=33538, nnz=2500, dtype="float32", nf=3000),
        # Quality control and variable-feature selection on the raw counts of one sample.
        dict(name="prep_sample", kind="prep", cells=30000, genes=33538, nnz=2000, nf=2000),
        # A host's sparse matrix (a Julia SparseMatrixCSC: 1-based Int64) handed over, and the cell-major
        # arrays that the device built of it taken back, as a program does that writes them to a file.
        dict(name="upload_csc", kind="upload", cells=12000, genes=27998, nnz=2000, index="int64"),
        # A 10X MatrixMarket file in host memory to a count matrix.
        dict(name="reader_mtx", kind="reader", cells=4001, genes=27998, nnz=2000),
        # PCA at the smallest size in use, FP64: launch and latency bound.
        dict(name="pca_small_f64", kind="pca", cells=2000, genes=20000, nnz=1000, dtype="float64", nf=2000,
             npcs=15),
        # PCA of an ordinary sample, FP32 values.
        dict(name="pca_plain_f32", kind="pca", cells=50000, genes=33538, nnz=2500, dtype="float32", nf=3000,
             npcs=30),
        # The mixed-precision path of an atlas in one go: normalise, scale, PCA.  The largest case.
        dict(name="atlas_bf16", kind="embed", cells=500000, genes=27998, nnz=2000, dtype="bfloat16", nf=3000,
             npcs=30),
        # The graph that clustering starts from, in one call with the default FP32 search: odd size.
        dict(name="snn_plain", kind="snn", n=30011, d=50, k=20, dtype="float32", metric="euclidean"),
        # The neighbour search of an atlas on the tensor cores.
        dict(name="ann_large_bf16", kind="ann", n=300000, d=50, k=30, dtype="float32", metric="euclidean",
             include_self=True),
        # The SNN graph from neighbour lists that a program holds.
        dict(name="jaccard_lists", kind="jaccard", n=150001, d=50, k=20, dtype="float64"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["normalize", "scale", "prep", "upload", "reader", "pca", "pca", "embed", "snn", "ann",
                       "jaccard"])
    genes = _log_int(rng, 8000, 33538)
    c = dict(kind=kind)
    if kind == "normalize":
        c.update(cells=_log_int(rng, 300, 20000), genes=genes, nnz=_log_int(rng, 300, 2500),
                 dtype=rng.choice(["float64", "float64", "float32"]),
                 method=rng.choice(["lognormalize", "lognormalize", "relativecounts"]))
    elif kind == "scale":
        c.update(cells=_log_int(rng, 2000, 100000), genes=genes, nnz=_log_int(rng, 500, 2500),
                 dtype=rng.choice(["float64", "float32", "bfloat16"]), nf=_log_int(rng, 500, 4000))
    elif kind == "prep":
        c.update(cells=_log_int(rng, 1000, 40000), genes=genes, nnz=_log_int(rng, 500, 2000),
                 nf=_log_int(rng, 500, 3000))
    elif kind == "upload":
        c.update(cells=_log_int(rng, 500, 16000), genes=genes, nnz=_log_int(rng, 500, 2000),
                 index=rng.choice(["int64", "int32"]))
    elif kind == "reader":
        c.update(cells=_log_int(rng, 300, 5000), genes=genes, nnz=_log_int(rng, 500, 2000))
    elif kind == "pca" and rng.random() < 0.5:
        c.update(cells=_log_int(rng, 1500, 6000), genes=genes, nnz=_log_int(rng, 800, 1500), dtype="float64",
                 nf=_log_int(rng, 800, 3000), npcs=rng.randint(5, 15))
    elif kind == "pca":
        c.update(cells=_log_int(rng, 8000, 60000), genes=genes, nnz=_log_int(rng, 1000, 2500),
                 dtype=rng.choice(["float32", "bfloat16"]), nf=_log_int(rng, 1500, 3500),
                 npcs=rng.randint(10, 30))
    elif kind == "embed":
        c.update(cells=_log_int(rng, 60000, 400000), genes=genes, nnz=_log_int(rng, 1000, 2000),
                 dtype=rng.choice(["bfloat16", "bfloat16", "float32"]), nf=_log_int(rng, 1500, 3000),
                 npcs=rng.randint(10, 30))
    elif kind == "snn":
        c.update(n=_log_int(rng, 300, 40000), d=rng.randint(5, 64), k=rng.randint(5, 32),
                 dtype=rng.choice(["float64", "float32"]), metric=rng.choice(["euclidean", "cosine"]))
    elif kind == "ann":
        c.update(n=_log_int(rng, 5000, 300000), d=rng.randint(10, 64), k=rng.randint(5, 32),
                 dtype=rng.choice(["float64", "float32"]), metric=rng.choice(["euclidean", "cosine"]),
                 include_self=rng.random() < 0.7)
    else:
        c.update(n=_log_int(rng, 500, 250000), d=50, k=rng.randint(5, 32),
                 dtype=rng.choice(["float64", "float32"]))
    return c


# ---- inputs ---------------------------------------------------------------------------------------------

def _model(case, n_cells, seed):
    """Parameters of the count model for n_cells cells and the depth that gives case["nnz"] a cell."""
    rng = np.random.default_rng(seed)
    genes, ncl = case["genes"], 40
    m = dict(mu_g=rng.lognormal(-1.2, 1.6, genes).astype(np.float32),
             s_c=rng.lognormal(0.0, 0.3, n_cells).astype(np.float32),
             cluster=rng.integers(0, ncl, n_cells).astype(np.int32), lfc=np.zeros((ncl, genes), np.float32))
    for c in range(ncl):
        sel = rng.random(genes) < 0.05
        m["lfc"][c, sel] = rng.normal(0.0, 0.8, int(sel.sum()))
    pick = rng.choice(n_cells, min(256, n_cells), replace=False)
    m["pick"] = pick
    base = _rates(m, pick)
    lo, hi = 1e-4, 1e4
    for _ in range(40):
        mid = math.sqrt(lo * hi)
        detected = genes - (1.0 + DISPERSION * mid * base).pow(-1.0 / DISPERSION).sum(1).mean().item()
        lo, hi = (mid, hi) if detected < min(case["nnz"], 0.9 * genes) else (lo, mid)
    m["depth"] = mid
    return m


def _rates(m, cells):
    dev = "cuda"
    r = torch.from_numpy(m["s_c"][cells]).to(dev)[:, None] * torch.from_numpy(m["mu_g"]).to(dev)[None, :]
    return r * torch.from_numpy(m["lfc"]).to(dev)[torch.from_numpy(m["cluster"][cells]).to(dev).long()].exp()


def _features(m, nf, seed):
    """The nf genes (1-based, ascending) of largest variance of the log-normalised values in a sample of
    cells: what feature selection hands to the PCA."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    rate = _rates(m, m["pick"]) * m["depth"]
    x = torch.poisson(rate * torch._standard_gamma(torch.full_like(rate, 1 / DISPERSION), generator=g) * DISPERSION,
                      generator=g)
    x = torch.log1p(1e4 * x / x.sum(1, keepdim=True).clamp(min=1))
    return np.sort(torch.argsort(-x.var(0), stable=True)[:nf].cpu().numpy()) + 1


def _counts(m, seed):
    return package().CountMatrix.generate(len(m["s_c"]), len(m["mu_g"]), m["mu_g"], m["s_c"], m["cluster"],
                                          m["lfc"], depth=m["depth"], dispersion=DISPERSION, seed=seed)


def _reordered(counts, seed):
    """Cell-major arrays (GPU tensors: row pointers, columns, counts) of the same counts with the cells and the
    genes in an order of the seed."""
    X = counts.to_csr()
    g = torch.Generator(device="cuda").manual_seed(seed)
    row = torch.repeat_interleave(torch.arange(X.shape[0], device="cuda"),
                                  torch.from_numpy(X.indptr.astype(np.int64)).cuda().diff())
    row = torch.randperm(X.shape[0], generator=g, device="cuda")[row]
    col = torch.randperm(X.shape[1], generator=g, device="cuda")[torch.from_numpy(X.indices).cuda().long()]
    return _compressed(row, col, torch.from_numpy(X.data).cuda(), X.shape)


def _compressed(row, col, val, shape):
    key, order = (row * shape[1] + col).sort()
    ptr = torch.zeros(shape[0] + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.bincount(row, minlength=shape[0]).cumsum(0)
    return ptr, key % shape[1], val[order]


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.from_numpy(a[:0]).dtype, pin_memory=True).numpy()
    t[...] = a
    return t


def _points(case, seed, order):
    """PCA-like coordinates: a mixture of 60 components, the scale of dimension i falling as 1/sqrt(i)."""
    n, d = case["n"], case["d"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    scale = 1.0 / torch.arange(1, d + 1, device="cuda", dtype=torch.float64).sqrt()
    mean = 4.0 * torch.randn(60, d, generator=g, device="cuda", dtype=torch.float64)
    X = mean[torch.randint(0, 60, (n,), generator=g, device="cuda")] * scale
    X += scale * torch.randn(n, d, generator=g, device="cuda", dtype=torch.float64)
    X = X[torch.randperm(n, generator=torch.Generator(device="cuda").manual_seed(order), device="cuda")]
    X = X.to(getattr(torch, case["dtype"]))
    return np.asfortranarray(X.cpu().numpy())


def _mtx(rowptr, cols, vals, shape):
    """MatrixMarket text, features x barcodes, of cell-major arrays."""
    rows = torch.repeat_interleave(torch.arange(shape[0], device="cuda"), rowptr.diff())
    text = []
    for f, end in zip([cols + 1, rows + 1, vals.long()], b"  \n"):
        width = len(str(int(f.max())))
        p = 10 ** torch.arange(width - 1, -1, -1, device="cuda")
        digits = (f[:, None] // p % 10 + 48).to(torch.uint8)
        digits[f[:, None] < p] = 0
        text += [digits, torch.full((len(f), 1), end, dtype=torch.uint8, device="cuda")]
    text = torch.cat(text, 1).reshape(-1)
    body = text[text != 0].cpu().numpy().tobytes()
    return b"%%%%MatrixMarket matrix coordinate integer general\n%d %d %d\n" % (shape[1], shape[0], len(vals)) + body


def prepare(case, seed):
    sv, kind = package(), case["kind"]
    st = dict(case=case)
    if kind == "jaccard":
        nn = sv.ann(_points(dict(case, dtype="float32"), 4, 4), case["k"], precision="bf16")[0]
        to = torch.randperm(case["n"], generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")
        lists = to[torch.from_numpy(nn).cuda().long() - 1]
        st["nn"] = np.asfortranarray((lists[to.argsort()] + 1).int().cpu().numpy())
        return st
    if kind in ("snn", "ann"):
        st["X"] = _points(case, seed if kind == "ann" else 4, seed)
        return st
    if kind in ("normalize", "upload", "reader"):
        m = _model(case, case["cells"], 4)
        shape = (case["cells"], case["genes"])
        ptr, col, val = _reordered(_counts(m, 4), seed)
        if kind == "reader":
            st["text"] = _mtx(ptr, col, val, shape)
        elif kind == "normalize":
            st["counts"] = sv.CountMatrix.upload_csr(*(a.cpu().numpy() for a in (ptr, col, val)), shape)
        else:
            t = getattr(torch, case["index"])
            row = torch.repeat_interleave(torch.arange(shape[0], device="cuda"), ptr.diff())
            ptr, row, val = _compressed(col, row, val, shape[::-1])
            st["csc"] = [_pinned(a.to(t).cpu().numpy()) for a in (ptr + 1, row + 1, val)]
            st["shape"] = shape
        return st
    m = _model(case, case["cells"], seed)
    if kind != "prep":
        st["features"] = _features(m, case["nf"], seed)
    counts = st["counts"] = _counts(m, seed)
    if kind == "pca":
        st["S"] = sv.scale_features(sv.normalize_cells(counts, scale_factor=1e4, dtype=case["dtype"]),
                                    scale_max=10.0, features=st["features"])
    if kind in ("pca", "embed"):
        # coordinates land in one pinned array that the program keeps
        k = min(case["cells"], case["nf"], case["npcs"])
        st["Z"] = torch.empty((k, case["cells"]), dtype=torch.float64, pin_memory=True).numpy().T
    return st


# ---- one pass -------------------------------------------------------------------------------------------

def _kept(a, case):
    """Embeddings of FP32 and BF16 values are kept in FP32, as AnnData keeps them."""
    return a if case["dtype"] == "float64" else torch.from_numpy(a).to(torch.float32)


def run(st):
    sv, case, kind = package(), st["case"], st["case"]["kind"]
    if kind == "normalize":
        return sv.normalize_cells(st["counts"], method=case["method"], scale_factor=1e4,
                                  dtype=case["dtype"]).values_csc()
    if kind == "scale":
        D = sv.normalize_cells(st["counts"], scale_factor=1e4, dtype=case["dtype"])
        mu, mean, std = sv.scale_features(D, scale_max=10.0, features=st["features"]).stats()
        return {"mu": mu, "mean": mean, "std": std}
    if kind == "prep":
        X, cells = sv.filter_cells(st["counts"], min_features=200)
        features, metric = sv.find_variable_features(X, case["nf"])
        return {"cells": cells, "features": features, "metric": metric}
    if kind == "upload":
        X = sv.CountMatrix.upload(*st["csc"], st["shape"], index_base=1).to_csr()
        return {"indptr": X.indptr, "indices": X.indices, "data": X.data}
    if kind == "reader":
        X = sv.CountMatrix.parse_mtx(st["text"]).to_csc()
        return {"indptr": X.indptr, "indices": X.indices, "data": X.data}
    if kind in ("pca", "embed"):
        S = st.get("S")
        if S is None:
            S = sv.scale_features(sv.normalize_cells(st["counts"], scale_factor=1e4, dtype=case["dtype"]),
                                  scale_max=10.0, features=st["features"])
        em = sv.pca(S, case["npcs"], out=st["Z"])
        return {"coordinates": _kept(em.coordinates, case), "stdev": _kept(em.stdev, case),
                "basis": _kept(em.basis, case)}
    if kind == "snn":
        G = sv.shared_nearest_neighbours(st["X"], case["k"], metric=case["metric"])
        return {"indptr": G.indptr, "indices": G.indices, "data": G.data}
    if kind == "ann":
        idx, dist = sv.ann(st["X"], case["k"], metric=case["metric"], include_self=case["include_self"],
                           precision="bf16")
        return {"idx": idx, "dist": dist}
    G = sv.jaccard_index(st["nn"], case["k"], dtype=case["dtype"])
    return {"indptr": G.indptr, "indices": G.indices, "data": G.data}


# ---- what a pass cannot do without ----------------------------------------------------------------------

def work(case):
    """Bytes: each input read once, each output (device copies that later stages read among them) written
    once.  Flops: a PCA's products for one Lanczos basis; a search's distances."""
    kind = case["kind"]
    if kind in ("snn", "ann", "jaccard"):
        n, d, k = case["n"], case["d"], case["k"]
        es = 8 if case["dtype"] == "float64" else 4
        if kind == "jaccard":
            return {"bytes": n * k * 4 + n * k * (8 + es), "flops": n * k * k}
        b = n * d * es + n * k * (4 + es)
        return {"bytes": b + (n * k * (8 + es) if kind == "snn" else 0), "flops": 2 * n * n * d}
    cells = case["cells"]
    nnz = cells * case["nnz"]
    v = {"float64": 8, "float32": 4, "bfloat16": 2}.get(case.get("dtype"), 0)
    both = nnz * (4 + 4 + v) + nnz * (4 + v)      # normalisation of the gene-major and the cell-major copy
    if kind == "normalize":
        return {"bytes": both + nnz * v, "flops": 2 * nnz}
    if kind == "prep":
        return {"bytes": 4 * nnz * 8, "flops": 6 * nnz}
    if kind == "upload":
        i = np.dtype(case["index"]).itemsize
        return {"bytes": nnz * (2 * i + 8 + 8 + 8), "flops": 0}
    if kind == "reader":
        return {"bytes": nnz * (13 + 8 + 8 + 8), "flops": 0}
    nnz_f = 0.5 * nnz                              # entries of the selected features
    copies = nnz_f * (2 + v) + nnz_f * (1 + v)     # the cell-major and the row-blocked copy
    products = 2 * (case.get("npcs", 0) + 7)
    if kind == "scale":
        return {"bytes": both + 2 * nnz_f * v + copies, "flops": 4 * nnz}
    b = products / 2 * copies + cells * case["npcs"] * 8
    if kind == "embed":
        b += both + 2 * nnz_f * v + copies
    return {"bytes": b, "flops": 2 * products * nnz_f}


# ---- the same in 64 bits --------------------------------------------------------------------------------

def _dense(counts, features, rows=None):
    """log1p(1e4 x / total) of the features in FP64 (cells x features, on the GPU)."""
    X = counts.to_csr()
    ptr = torch.from_numpy(X.indptr.astype(np.int64)).cuda()
    col = torch.from_numpy(X.indices).cuda().long()
    val = torch.from_numpy(X.data).cuda().double()
    row = torch.repeat_interleave(torch.arange(X.shape[0], device="cuda"), ptr.diff())
    total = torch.zeros(X.shape[0], dtype=torch.float64, device="cuda").index_add_(0, row, val)
    where = torch.full((X.shape[1],), -1, device="cuda")
    where[torch.from_numpy(features - 1).cuda()] = torch.arange(len(features), device="cuda")
    keep = where[col] >= 0
    row, col, val = row[keep], where[col[keep]], val[keep]
    out = torch.zeros((X.shape[0], len(features)), dtype=torch.float64, device="cuda")
    out[row, col] = torch.log1p(1e4 * val / total[row])
    return out


def _stdev(A, npcs):
    std, mean = torch.std_mean(A, 0)
    mu = mean / std
    A = torch.minimum(A / std, 10.0 + mu) - mu
    G = A.T @ A if A.shape[0] >= A.shape[1] else A @ A.T
    ev = torch.linalg.eigvalsh(G).flip(0)[:min(npcs, *A.shape)]
    return (ev.clamp(min=0).sqrt() / math.sqrt(max(1, A.shape[0] - 1))).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("prep", "upload", "reader"):
        return None                                # whole numbers, and a metric of smoothed fits
    st = prepare(case, seed)
    if kind == "normalize":
        X = st["counts"].to_csc()
        total = np.bincount(X.indices, X.data, minlength=X.shape[0])
        v = 1e4 * X.data / total[X.indices]
        return np.log1p(v) if case["method"] == "lognormalize" else v
    if kind == "scale":
        std, mean = (t.cpu().numpy() for t in torch.std_mean(_dense(st["counts"], st["features"]), 0))
        return {"mu": mean / std, "mean": mean, "std": std}
    if kind in ("pca", "embed"):
        return {"coordinates": None, "stdev": _stdev(_dense(st["counts"], st["features"]), case["npcs"]),
                "basis": None}                     # singular vectors: up to sign
    if kind == "ann":
        return {"idx": None, "dist": _distances(st["X"], case)}
    if kind == "snn":
        st["nn"] = _neighbours(st["X"], case)[0].cpu().numpy() + 1
    return {"indptr": None, "indices": None, "data": _jaccard(st["nn"], case["k"])}


def _neighbours(X, case, self_first=True):
    """Exact neighbours: FP32 products shortlist 2k + 16 points, FP64 differences order them."""
    X = torch.from_numpy(X).cuda().double()
    if case["metric"] == "cosine":
        X = X / X.norm(dim=1, keepdim=True)
    n, k = len(X), case["k"]
    F = X.float()
    half = 0.5 * F.square().sum(1)
    idx, dist = [], []
    short = min(n, 2 * k + 16)
    for a in range(0, n, 4096):
        near = (F[a:a + 4096] @ F.T - half).topk(short, dim=1).indices
        d2 = (X[near] - X[a:a + 4096, None]).square().sum(2)
        own = torch.arange(a, a + len(near), device="cuda")[:, None]
        d2[near == own] = -1.0 if self_first else math.inf
        d2, at = d2.sort(1)
        idx.append(near.gather(1, at)[:, :k])
        dist.append(d2[:, :k].clamp(min=0))
    d2 = torch.cat(dist)
    return torch.cat(idx), 0.5 * d2 if case["metric"] == "cosine" else d2.sqrt()


def _distances(X, case):
    return _neighbours(X, case, case["include_self"])[1].cpu().numpy()


def _jaccard(nn, k):
    """Weights c / (2k - c) > 1/15 of the shared neighbours, column by column, rows ascending."""
    nn = torch.from_numpy(np.ascontiguousarray(nn)).cuda().long() - 1
    n = len(nn)
    i = torch.arange(n, device="cuda").repeat_interleave(nn.shape[1])
    r = nn.reshape(-1)
    order = r.argsort()
    i, count = i[order], torch.bincount(r, minlength=n)
    start = count.cumsum(0) - count
    keys = []
    for a in range(0, n, 1 << 14):
        cols = torch.arange(a, min(n, a + (1 << 14)), device="cuda")
        q = nn[cols].reshape(-1)
        c = count[q]
        j = cols.repeat_interleave(nn.shape[1]).repeat_interleave(c)
        at = start[q].repeat_interleave(c) + torch.arange(int(c.sum()), device="cuda") - (
            c.cumsum(0) - c).repeat_interleave(c)
        _, shared = torch.unique(j * n + i[at], return_counts=True)
        keys.append(shared.double())
    c = torch.cat(keys)
    w = c / (k + (k - c))
    return w[w > PRUNE].cpu().numpy()
