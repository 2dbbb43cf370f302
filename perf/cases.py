"""Timed cases of the framework's public paths, each at several scales.

A case is a dict: ``kind`` names the path, the other keys are its sizes and
options. ``listed()`` holds the fixed cases, ``draw()`` gives further ones of
the same ranges, ``prepare()`` builds what a program holds before the call (on
the GPU, from the seed alone), ``run()`` makes one pass through the public
entry points and returns its outputs whole, ``work()`` says what a pass cannot
do without, ``exact()`` computes the outputs in 64 bits with plain torch.

Kinds:

- ``solve``     one PCA solve of a resident count matrix (``DeviceMatrix.solve``)
- ``products``  X.(v/sd), (X^T.u)/sd and the gene scaling of a resident matrix
- ``rotate``    the restart rotation of a tall basis (``bgpu_rotate_basis``)
- ``knn``       neighbour search over clustered PCs (``knn_self``)
- ``kmeans``    k-means of PCs (``kmeans``)
- ``harmony``   row normalisation and Harmony of batched PCs
- ``hvg``       the gene statistics of highly-variable-gene selection
- ``prepare``   size factors, materialised normalisation and the transpose
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from brisc_gb300 import DeviceMatrix
from brisc_gb300 import _lib as L
from brisc_gb300 import harmony as harmony_module
from brisc_gb300 import hvg as hvg_module
from brisc_gb300 import knn as knn_module

DEV = "cuda"


def listed():
    return [
        # one small sample, the default 50 PCs: launches and latency
        dict(name="solve_3k", kind="solve", n=2700, g=2000, density=0.08, k=50, m=100,
             norm="logCP10k"),
        # the atlas-sized solve that the benchmark quotes
        dict(name="solve_1m", kind="solve", n=1_000_000, g=2000, density=0.05, k=50, m=100,
             norm="logCP10k"),
        # both sparse products of a solve, counts with the fused normalisation
        dict(name="products_counts_300k", kind="products", n=300_007, g=2000, density=0.05,
             norm="PFlog1pPF"),
        # the same for already normalised float32 values (the drop-in's input)
        dict(name="products_f32_50k", kind="products", n=50_000, g=2000, density=0.08,
             norm="none"),
        # a restart's rotation on its own
        dict(name="rotate_400k", kind="rotate", n=400_000, K=100, ncols=75),
        # neighbours of one small sample, and of a mid-sized atlas
        dict(name="knn_3k", kind="knn", n=2700, d=50, k=20),
        dict(name="knn_300k", kind="knn", n=300_000, d=50, k=20),
        # the clustering before the neighbour search (2 iterations, its default)
        dict(name="kmeans_300k", kind="kmeans", n=300_000, d=50, iterations=2),
        # batch correction of four pooled samples
        dict(name="harmony_100k", kind="harmony", n=100_000, d=50, batches=4),
        # gene statistics before gene selection: every gene of one study, CSR
        dict(name="hvg_all_genes", kind="hvg", n=40_000, g=20_000, density=0.05, form="csr",
             values="float32", subset=False),
        # the same of a larger CSC matrix, the cells that passed QC only
        dict(name="hvg_csc_400k", kind="hvg", n=400_000, g=2000, density=0.05, form="csc",
             values="uint16", subset=True),
        # raw counts to normalised values and their transpose
        dict(name="prepare_200k", kind="prepare", n=200_003, g=2000, density=0.05,
             norm="logCP10k"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "products", "products", "rotate", "knn", "knn",
                       "kmeans", "harmony", "hvg", "hvg", "prepare"])
    if kind == "solve":
        k = rng.choice([10, 20, 30, 50])
        n, g = _log_uniform(rng, 1500, 700_000), rng.randint(600, 2500)
        return dict(kind=kind, n=n, g=g, density=round(rng.uniform(0.04, 0.08), 3), k=k, m=2 * k,
                    norm=rng.choice(["logCP10k", "log1pPF", "PFlog1pPF"]))
    if kind == "products":
        norm = rng.choice(["none", "logCP10k", "PFlog1pPF"])
        return dict(kind=kind, n=_log_uniform(rng, 2000, 800_000), g=rng.randint(500, 3500),
                    density=round(rng.uniform(0.03, 0.08), 3), norm=norm)
    if kind == "rotate":
        K = rng.randint(20, 200)
        return dict(kind=kind, n=_log_uniform(rng, 2000, 1_000_000), K=K,
                    ncols=rng.randint(K // 2, K - 1))
    if kind == "knn":
        return dict(kind=kind, n=_log_uniform(rng, 1500, 400_000), d=rng.randint(10, 100),
                    k=rng.randint(10, 60))
    if kind == "kmeans":
        return dict(kind=kind, n=_log_uniform(rng, 2000, 600_000), d=rng.randint(10, 100),
                    iterations=rng.choice([2, 2, 5]))
    if kind == "harmony":
        return dict(kind=kind, n=_log_uniform(rng, 4000, 200_000), d=rng.randint(20, 60),
                    batches=rng.randint(2, 12))
    if kind == "hvg":
        g = rng.choice([rng.randint(1000, 4000), rng.randint(15_000, 30_000)])
        n = _log_uniform(rng, 2000, 500_000 if g <= 4000 else 50_000)
        return dict(kind=kind, n=n, g=g, density=round(rng.uniform(0.03, 0.08), 3),
                    form=rng.choice(["csr", "csc"]),
                    values=rng.choice(["float32", "uint16", "int32"]),
                    subset=rng.choice([False, True]))
    return dict(kind=kind, n=_log_uniform(rng, 2000, 500_000), g=rng.randint(500, 3500),
                density=round(rng.uniform(0.03, 0.08), 3),
                norm=rng.choice(["logCP10k", "PFlog1pPF"]))


# ---------------------------------------------------------------------------
# inputs
def _generator(seed, salt):
    return torch.Generator(device=DEV).manual_seed(1_000_003 * (int(seed) + 1) + salt)


def _counts(n, g, density, seed):
    """Negative-binomial counts of cells of 12 types, as a CSR matrix: lognormal
    gene means, lognormal library sizes, per-type gene factors (sizes of the
    types uneven), dispersion 0.3. Returns indptr (int64), indices (int32),
    counts (int32). A cell without counts gets one of its first gene."""
    gen = _generator(seed, 1)

    def normal(*shape):
        return torch.randn(*shape, generator=gen, device=DEV)

    means = torch.exp(1.5 * normal(g))
    factors = torch.exp(0.8 * normal(12, g))
    weights = torch.exp(torch.linspace(0, -2.0, 12, device=DEV))
    share = weights / weights.sum()
    # the scale that gives the density: P(count > 0) = 1 - (1 + 0.3 mean)^(-1/0.3)
    lo, hi = -12.0, 6.0
    for _ in range(40):
        mid = 0.5 * (lo + hi)
        p = 1 - torch.pow(1 + 0.3 * math.exp(mid) * means[None, :] * factors, -1 / 0.3)
        lo, hi = (mid, hi) if float((share @ p).mean()) < density else (lo, mid)
    means = means * math.exp(0.5 * (lo + hi))
    rows = max(1, min(n, 40_000_000 // g))
    counts, indices, lengths = [], [], []
    shape = torch.full((1,), 1 / 0.3, device=DEV)
    for r0 in range(0, n, rows):
        r = min(rows, n - r0)
        kind = torch.multinomial(weights, r, replacement=True, generator=gen)
        lib = torch.exp(0.4 * normal(r, 1))
        lam = torch._standard_gamma(shape.expand(r, g), generator=gen)
        lam *= factors[kind]
        lam *= means[None, :] * 0.3
        lam *= lib
        c = torch.poisson(lam, generator=gen)
        c[:, 0] += (c.sum(1) == 0).float()
        flat = c.view(-1).nonzero().view(-1)
        counts.append(c.view(-1)[flat].to(torch.int32))
        indices.append((flat % g).to(torch.int32))
        lengths.append((c != 0).sum(1))
    indptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(torch.cat(lengths), 0, out=indptr[1:])
    return indptr, torch.cat(indices), torch.cat(counts)


def _counts_of_size(n, g, density, seed):
    """_counts() with a number of stored entries that the sizes alone give:
    surplus entries, evenly spread and never a row's first, are left out."""
    indptr, indices, counts = _counts(n, g, 1.08 * density, seed)
    size = int(0.95 * density * n * g)
    free = torch.ones(counts.numel(), dtype=torch.bool, device=DEV)
    free[indptr[:-1]] = False
    free = free.nonzero().view(-1)
    surplus = counts.numel() - size
    at = torch.arange(surplus, device=DEV) * free.numel() // surplus
    keep = torch.ones(counts.numel(), dtype=torch.bool, device=DEV)
    keep[free[at]] = False
    lengths = torch.bincount(_row_ids(indptr)[keep], minlength=n)
    indptr = torch.cat([torch.zeros(1, dtype=torch.int64, device=DEV), lengths.cumsum(0)])
    return indptr, indices[keep], counts[keep]


def _row_ids(indptr):
    n = indptr.numel() - 1
    return torch.repeat_interleave(torch.arange(n, device=indptr.device), indptr[1:] - indptr[:-1])


def _row_sums(indptr, values):
    """Sums of the rows' stored values (a difference of exact prefix sums)."""
    z = torch.zeros(1, dtype=torch.float64, device=DEV)
    c = torch.cat([z, torch.cumsum(values.double(), 0)])
    return c[indptr[1:]] - c[indptr[:-1]]


def _factors(indptr, counts, norm):
    """Per-cell factors as normalize() defines them, rounded to float32."""
    s = _row_sums(indptr, counts)
    if norm == "logCP10k":
        return (1e4 / s).float(), None
    isf = (s.mean() / s).float()
    if norm == "log1pPF":
        return isf, None
    v = torch.log1p(counts.double() * isf[_row_ids(indptr)].double())
    t = _row_sums(indptr, torch.round(v * 2**20) / 2**20)  # exact sums, whatever their order
    return isf, (t.mean() / t).float()


def _values64(indptr, counts, isf, post):
    v = torch.log1p(counts.double() * isf.double()[_row_ids(indptr)])
    return v if post is None else v * post.double()[_row_ids(indptr)]


def _pcs(n, d, seed, batches=0):
    """PC-like coordinates: a Gaussian mixture whose scale falls over the
    dimensions as a PCA spectrum does; with batches, an offset per batch."""
    gen = _generator(seed, 2)
    scale = 10.0 / torch.sqrt(1.0 + torch.arange(d, device=DEV, dtype=torch.float32))
    centres = torch.randn(40, d, generator=gen, device=DEV) * scale
    X = centres[torch.randint(0, 40, (n,), generator=gen, device=DEV)]
    X = X + 0.35 * scale * torch.randn(n, d, generator=gen, device=DEV)
    if not batches:
        return X.contiguous(), None
    labels = torch.randint(0, batches, (n,), generator=gen, device=DEV)
    labels[:batches] = torch.arange(batches, device=DEV)
    X = X + (2.0 * torch.randn(batches, d, generator=gen, device=DEV))[labels]
    return X.contiguous(), labels.to(torch.int32)


def _num_clusters(n):
    """neighbors()'s default number of k-means clusters."""
    return max(1, math.ceil(min(4 * math.sqrt(n), n / 100)))


def _assign(X, C):
    out = []
    cn = (C * C).sum(1)
    for part in X.split(max(1, 40_000_000 // C.shape[0])):
        out.append((cn[None, :] - 2 * (part @ C.T)).argmin(1))
    return torch.cat(out)


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


class _State:
    def __init__(self, case, **kw):
        self.case = case
        self.__dict__.update(kw)


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    if kind in ("solve", "products"):
        indptr, indices, counts = _counts(n, case["g"], case["density"], seed)
        norm = None if case["norm"] == "none" else case["norm"]
        isf, post = _factors(indptr, counts, norm or "logCP10k")
        if norm is None:
            values = _values64(indptr, counts, isf, post).float()
            isf = None
        else:
            values = counts.clamp(max=65535).to(torch.uint16)
        M = DeviceMatrix(indptr.to(torch.int32), indices, values, n, case["g"], norm=norm,
                         inv_size_factors=isf, post_factors=post)
        if kind == "solve":
            pcs = torch.empty(n, case["k"], device=DEV)
            return _State(case, M=M, pcs=pcs)
        gen = _generator(seed, 3)
        v = torch.randn(case["g"], generator=gen, device=DEV)
        u = torch.randn(n, generator=gen, device=DEV)
        return _State(case, M=M, v=v / v.norm(), u=(u - u.mean()) / u.norm(),
                      sd=torch.empty(case["g"], device=DEV), y=torch.empty(n, device=DEV),
                      z=torch.empty(case["g"], device=DEV))
    if kind == "rotate":
        A, B, lda = _rotation(case, seed)
        return _State(case, A=A, B=B, lda=lda, C=torch.zeros(case["ncols"], lda, device=DEV))
    if kind == "knn":
        X, so, cent, sizes, norms, cs = _knn_inputs(case, seed)
        k = case["k"]
        return _State(case, X=X, so=so, cent=cent, sizes=sizes, norms=norms, cs=cs,
                      nbr=torch.empty(n, k, dtype=torch.int32, device=DEV),
                      dist=torch.empty(n, k, device=DEV),
                      cd=torch.empty(n, cs, device=DEV),
                      near=torch.empty(n, cs, dtype=torch.int32, device=DEV))
    if kind == "kmeans":
        X, _ = _pcs(n, case["d"], seed)
        nc = _num_clusters(n)
        i32 = dict(dtype=torch.int32, device=DEV)
        return _State(case, X=X, nc=nc, labels=torch.empty(n, **i32),
                      c0=torch.empty(nc, case["d"], device=DEV),
                      c1=torch.empty(nc, case["d"], device=DEV), sizes=torch.empty(nc, **i32),
                      mind=torch.empty(n, device=DEV), norms=torch.empty(n, device=DEV))
    if kind == "harmony":
        X, labels, Y0 = _harmony_inputs(case, seed)
        return _State(case, X=X, labels=labels, Y0=Y0, Y=torch.empty_like(Y0),
                      Z=torch.empty_like(X), R=torch.empty(n, Y0.shape[0], device=DEV))
    if kind == "hvg":
        data, indices, indptr, cells, clip, used = _hvg_inputs(case, seed)
        g = case["g"]
        f = {k: torch.empty(g, device=DEV) for k in ("mean", "var", "sums", "squares")}
        return _State(case, data=data, indices=indices, indptr=indptr, cells=cells, clip=clip,
                      used=used, nonzero=torch.empty(g, dtype=torch.int32, device=DEV), **f)
    indptr, indices, counts = _counts_of_size(n, case["g"], case["density"], seed)
    nnz = counts.numel()
    f = dict(device=DEV)
    return _State(case, indptr=indptr.to(torch.int32), indices=indices, counts=counts.float(),
                  isf=torch.empty(n, **f), post=torch.empty(n, **f),
                  norm=torch.empty(nnz, **f), Bx=torch.empty(nnz, **f),
                  Bp=torch.empty(case["g"] + 1, dtype=torch.int32, **f),
                  Bi=torch.empty(nnz, dtype=torch.int32, **f))


def _rotation(case, seed):
    """An orthonormal-like basis and a rotation near those of a restart: part of
    the Ritz vectors has converged (one dominant entry), the others mix."""
    n, K = case["n"], case["K"]
    gen = _generator(seed, 4)
    lda = (n + 63) // 64 * 64
    A = torch.zeros(K, lda, device=DEV)
    A[:, :n] = torch.randn(K, n, generator=gen, device=DEV) / math.sqrt(n)
    mix = torch.randn(K, K, generator=gen, device=DEV, dtype=torch.float64)
    mix[: K // 2] *= 0.05
    mix[:, : K // 2] *= 0.05
    Q = torch.linalg.qr(torch.eye(K, device=DEV, dtype=torch.float64) * 2 + mix)[0]
    return A, Q.T.contiguous().float(), lda  # column-major


def _knn_inputs(case, seed):
    """What neighbors() hands to knn_self: the cells sorted by cluster, the
    clusters by their first PC, empty ones left out."""
    n = case["n"]
    X, _ = _pcs(n, case["d"], seed)
    nc = _num_clusters(n)
    gen = _generator(seed, 5)
    C = X[torch.randperm(n, generator=gen, device=DEV)[:nc]]
    for _ in range(2):
        lab = _assign(X, C)
        sizes = torch.bincount(lab, minlength=C.shape[0])
        # sums over the sorted cells, of values whose sums are exact
        o = torch.sort(lab, stable=True)[1]
        ends = torch.cumsum(sizes, 0)
        z = torch.zeros(1, X.shape[1], dtype=torch.float64, device=DEV)
        cum = torch.cat([z, torch.cumsum(torch.round(X[o].double() * 2**16) / 2**16, 0)])
        keep = sizes > 0
        C = ((cum[ends] - cum[ends - sizes])[keep] / sizes[keep, None]).float()
    lab = _assign(X, C)
    keep = torch.bincount(lab, minlength=C.shape[0]) > 0
    C = C[keep]
    C = C[torch.sort(C[:, 0], stable=True)[1]].contiguous()
    lab = _assign(X, C)
    sizes = torch.bincount(lab, minlength=C.shape[0])
    so = torch.sort(lab, stable=True)[1]
    X = X[so].contiguous()
    cs = min(64, C.shape[0])
    order = torch.sort(sizes)[0].cumsum(0)
    need = int(torch.searchsorted(order, case["k"] + 1)) + 1
    cs = min(max(cs, need), C.shape[0])
    return X, so.to(torch.int32), C, sizes.to(torch.int32), (X * X).sum(1), cs


def _harmony_inputs(case, seed):
    X, labels = _pcs(case["n"], case["d"], seed, case["batches"])
    nc = max(min(100, int(round(case["n"] / 30))), 1)
    Z = X / X.norm(dim=1, keepdim=True)
    gen = _generator(seed, 6)
    C = Z[torch.randperm(case["n"], generator=gen, device=DEV)[:nc]]
    for _ in range(3):
        lab = _assign(Z, C)
        one = torch.nn.functional.one_hot(lab, nc).double()
        size = one.sum(0)
        C = torch.where(size[:, None] > 0, (one.T @ Z.double()) / size.clamp(min=1)[:, None],
                        C.double()).float()
    return X, labels, C.contiguous()


def _hvg_inputs(case, seed):
    n, g = case["n"], case["g"]
    indptr, indices, counts = _counts(n, g, case["density"], seed)
    gen = _generator(seed, 7)
    cells, used = None, n
    if case["subset"]:
        mask = torch.rand(n, generator=gen, device=DEV) < 0.9
        mask[0] = mask[1] = True
        cells, used = mask, int(mask.sum())
    if case["form"] == "csc":
        order = torch.sort(indices.long() * n + _row_ids(indptr))[1]
        rows = _row_ids(indptr)[order].to(torch.int32)
        counts = counts[order]
        sizes = torch.bincount(indices, minlength=g)
        indptr = torch.cat([torch.zeros(1, dtype=torch.int64, device=DEV), sizes.cumsum(0)])
        indices = rows
        cells = torch.empty(0, dtype=torch.int8, device=DEV) if cells is None \
            else cells.to(torch.int8)
    else:
        cells = torch.empty(0, dtype=torch.int64, device=DEV) if cells is None \
            else cells.nonzero().view(-1)
    data = counts.to(getattr(torch, case["values"]))
    # a clip value between the bulk of the counts and their tail, as the
    # standardised-variance step sets it
    clip = 2.0 + 6.0 * torch.rand(g, generator=gen, device=DEV)
    return data, indices, indptr.to(torch.int32), cells, clip, used


# ---------------------------------------------------------------------------
# one pass
def run(s):
    c = s.case
    kind = c["kind"]
    if kind == "solve":
        r = s.M.solve(c["k"], c["m"], PCs=s.pcs)
        return [s.pcs, r.singular_values]
    if kind == "products":
        s.M.gene_stddev(s.sd)
        s.M.matvec(s.v, s.sd, s.y)
        s.M.rmatvec(s.u, s.sd, s.z)
        return [s.sd, s.y, s.z]
    if kind == "rotate":
        L.call("bgpu_rotate_basis", s.A.data_ptr(), s.lda, c["n"], c["K"], s.B.data_ptr(), c["K"],
               c["ncols"], s.C.data_ptr(), s.lda, 2, _stream())
        return [s.C]
    if kind == "knn":
        knn_module.knn_self(X=s.X, sorted_order=s.so, centroids=s.cent,
                            num_cells_per_cluster=s.sizes, neighbors=s.nbr, distances=s.dist,
                            cell_norms=s.norms, centroid_distances=s.cd,
                            nearest_clusters=s.near, num_neighbors=c["k"],
                            num_clusters_searched=s.cs)
        return [s.nbr, s.dist, s.near, s.cd]
    if kind == "kmeans":
        it = knn_module.kmeans(X=s.X, cluster_labels=s.labels, centroids=s.c0,
                               centroids_new=s.c1, num_cells_per_cluster=s.sizes,
                               min_distances=s.mind, cell_norms=s.norms,
                               num_kmeans_iterations=c["iterations"])
        return [it, s.labels, s.c0, s.c1, s.sizes, s.mind, s.norms]
    if kind == "harmony":
        harmony_module.normalize_rows(s.X, s.Z)
        s.Y.copy_(s.Y0)  # updated in place by the call
        it = harmony_module.harmony(PCs=s.X, Z=s.Z, Y=s.Y, R=s.R, batch_labels=s.labels,
                                    num_batches=c["batches"])
        return [it, s.Z, s.Y, s.R]
    if kind == "hvg":
        if c["form"] == "csr":
            hvg_module.gene_mean_and_variance_csr(s.data, s.indices, s.indptr, s.cells, s.used,
                                                  c["g"], s.mean, s.var, s.nonzero)
            hvg_module.clipped_sum_csr(s.data, s.indices, s.indptr, s.used, c["g"], s.cells,
                                       s.clip, s.sums, s.squares)
        else:
            hvg_module.gene_mean_and_variance_csc(s.data, s.indices, s.indptr, s.cells, s.used,
                                                  c["g"], s.mean, s.var, s.nonzero)
            hvg_module.clipped_sum_csc(s.data, s.indices, s.indptr, s.cells, s.clip, s.sums,
                                       s.squares)
        return [s.mean, s.var, s.nonzero, s.sums, s.squares]
    n, post = c["n"], s.post if c["norm"] == "PFlog1pPF" else None
    method = {"logCP10k": 0, "PFlog1pPF": 2}[c["norm"]]
    pp = post.data_ptr() if post is not None else None
    L.call("bgpu_size_factors", s.indptr.data_ptr(), L.INDEX_I32, s.counts.data_ptr(),
           L.VALUE_F32, n, method, None, s.isf.data_ptr(), pp, None, _stream())
    L.call("bgpu_normalize_csr", s.indptr.data_ptr(), L.INDEX_I32, s.counts.data_ptr(),
           L.VALUE_F32, n, s.isf.data_ptr(), pp, s.norm.data_ptr(), _stream())
    L.call("bgpu_csr_tocsc", n, c["g"], s.indptr.data_ptr(), s.indices.data_ptr(),
           s.norm.data_ptr(), L.INDEX_I32, s.Bp.data_ptr(), s.Bi.data_ptr(), s.Bx.data_ptr(),
           _stream())
    return [s.isf, s.norm, s.Bp, s.Bi, s.Bx] + ([post] if post is not None else [])


# ---------------------------------------------------------------------------
def work(case):
    kind, n = case["kind"], case["n"]
    nnz = n * case.get("g", 0) * case.get("density", 0.0)
    if kind == "solve":
        # one cycle of m Lanczos steps (more restarts only add to it): both
        # products, one Gram-Schmidt pass per step, the PCs
        m, g = case["m"], case["g"]
        return {"bytes": m * (2 * 2 * nnz + 16 * n) + 4.0 * n * m * m + 4 * n * case["k"],
                "flops": m * 4 * nnz + 2.0 * n * m * m + 2.0 * g * m * m}
    if kind == "products":
        size = 8 if case["norm"] == "none" else 2
        return {"bytes": 3 * size * nnz + 12 * n, "flops": 7 * nnz}
    if kind == "rotate":
        return {"bytes": 4.0 * n * (case["K"] + case["ncols"]),
                "flops": 2.0 * n * case["K"] * case["ncols"]}
    if kind == "knn":
        nc, d = _num_clusters(n), case["d"]
        cs = min(64, nc)
        return {"bytes": 4.0 * n * (d + 2 * case["k"] + 2 * cs + 1) + 4.0 * nc * d,
                "flops": 2.0 * d * n * (nc + n * cs / nc)}
    if kind == "kmeans":
        nc, d, it = _num_clusters(n), case["d"], case["iterations"]
        return {"bytes": 4.0 * n * d * (it + 1) + 12.0 * n + 8.0 * nc * d,
                "flops": 2.0 * n * nc * d * (it + 1)}
    if kind == "harmony":
        # one correction round of five clustering passes (more rounds only add)
        C, d = max(min(100, int(round(n / 30))), 1), case["d"]
        return {"bytes": 4.0 * n * (5 * (2 * C + 2 * d) + C + 3 * d),
                "flops": 2.0 * n * C * d * (2 * 5 + 3)}
    if kind == "hvg":
        # the counts twice: the clip values come from the first statistics
        size = 2 if case["values"] == "uint16" else 4
        return {"bytes": 2 * nnz * (size + 4) + 8 * n + 20 * case["g"], "flops": 6 * nnz}
    return {"bytes": 4 * nnz * (1 + 2 + 2 + 1) + 12 * n, "flops": 3 * nnz}


# ---------------------------------------------------------------------------
# 64-bit values
def _srand(seed):
    state = (seed + 1442695040888963407) & 0xFFFFFFFFFFFFFFFF
    return _rand(state)[1]


def _rand(x):
    s = ((x ^ (x >> 18)) >> 27) & 0xFFFFFFFF
    rot = x >> 59
    out = ((s >> rot) | (s << (-rot & 31))) & 0xFFFFFFFF
    return out, (x * 6364136223846793005 + 1442695040888963407) & 0xFFFFFFFFFFFFFFFF


def _randint(bound, state):
    r, state = _rand(state)
    m = r * bound
    if (m & 0xFFFFFFFF) < bound:
        limit = ((1 << 32) - bound) % bound
        while (m & 0xFFFFFFFF) < limit:
            r, state = _rand(state)
            m = r * bound
    return m >> 32, state


def exact(case, seed):
    return {"solve": _exact_solve, "products": _exact_products, "rotate": _exact_rotate,
            "knn": _exact_knn, "kmeans": _exact_kmeans, "harmony": _exact_harmony,
            "hvg": _exact_hvg, "prepare": _exact_prepare}[case["kind"]](case, seed)


def _sparse64(case, seed):
    indptr, indices, counts = _counts(case["n"], case["g"], case["density"], seed)
    isf, post = _factors(indptr, counts, "logCP10k" if case["norm"] == "none" else case["norm"])
    v = _values64(indptr, counts, isf, post)
    return indptr, indices.long(), v.float().double() if case["norm"] == "none" else v


def _moments64(n, g, indices, v):
    one = torch.zeros(g, dtype=torch.float64, device=DEV).index_add_(0, indices, v)
    two = torch.zeros(g, dtype=torch.float64, device=DEV).index_add_(0, indices, v * v)
    sd = torch.sqrt(((two - one * one / n) / (n - 1)).clamp(min=0))
    return one / n, sd.clamp(min=1e-8)


def _exact_solve(case, seed):
    """The singular values, from the Gram matrix of the centred, scaled matrix.
    The PCs have no such value: their signs come with the start vector."""
    n, g = case["n"], case["g"]
    indptr, indices, v = _sparse64(case, seed)
    mean, sd = _moments64(n, g, indices, v)
    rows = max(1, 200_000_000 // g)
    G = torch.zeros(g, g, dtype=torch.float64, device=DEV)
    ip = indptr.tolist() if n <= rows else indptr[::rows].tolist() + [int(indptr[-1])]
    bounds = [(0, n, 0, ip[-1])] if n <= rows else [
        (i * rows, min(n, (i + 1) * rows), ip[i], int(indptr[min(n, (i + 1) * rows)]))
        for i in range((n + rows - 1) // rows)]
    for r0, r1, e0, e1 in bounds:
        D = torch.zeros(r1 - r0, g, dtype=torch.float64, device=DEV)
        r = torch.repeat_interleave(torch.arange(r1 - r0, device=DEV),
                                    indptr[r0 + 1:r1 + 1] - indptr[r0:r1])
        D[r, indices[e0:e1]] = v[e0:e1]
        G += D.T @ D
    G = (G - n * mean[:, None] * mean[None, :]) / (sd[:, None] * sd[None, :])
    w = torch.linalg.eigvalsh(G).flip(0)[: case["k"]]
    return [None, torch.sqrt(w)]


def _exact_products(case, seed):
    n, g = case["n"], case["g"]
    indptr, indices, v = _sparse64(case, seed)
    gen = _generator(seed, 3)
    a = torch.randn(g, generator=gen, device=DEV)
    u = torch.randn(n, generator=gen, device=DEV)
    a, u = (a / a.norm()).double(), ((u - u.mean()) / u.norm()).double()
    _, sd = _moments64(n, g, indices, v)
    rows = _row_ids(indptr)
    y = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, rows, v * (a / sd)[indices])
    z = torch.zeros(g, dtype=torch.float64, device=DEV).index_add_(0, indices, v * u[rows])
    return [sd, y, z / sd]


def _exact_rotate(case, seed):
    A, B, _ = _rotation(case, seed)
    return [B.double()[: case["ncols"]] @ A.double()]


def _exact_knn(case, seed):
    X, _, C, sizes, _, cs = _knn_inputs(case, seed)
    k = case["k"]
    X, C, sizes = X.double(), C.double(), sizes.long()
    cn = (C * C).sum(1)
    cd, near = [], []
    for part in X.split(max(1, 40_000_000 // C.shape[0])):
        p = torch.topk(cn[None, :] - 2 * (part @ C.T), cs, dim=1, largest=False)
        cd.append(p[0])
        near.append(p[1])
    cd, near = torch.cat(cd), torch.cat(near)
    norms = (X * X).sum(1)
    start = torch.cat([torch.zeros(1, dtype=torch.int64, device=DEV), sizes.cumsum(0)])
    dist = torch.empty(X.shape[0], k, dtype=torch.float64, device=DEV)
    host = start.tolist()
    cluster = torch.repeat_interleave(torch.arange(C.shape[0], device=DEV), sizes)
    for c in range(C.shape[0]):  # the queries of one cluster share their candidates
        a, b = host[c], host[c + 1]
        searched = torch.zeros(b - a, C.shape[0], dtype=torch.bool, device=DEV)
        searched.scatter_(1, near[a:b], True)
        cells = searched.any(0)[cluster].nonzero().view(-1)
        D = norms[a:b, None] + norms[cells][None, :] - 2 * (X[a:b] @ X[cells].T)
        D = D.masked_fill(~searched[:, cluster[cells]], math.inf)
        D = D.masked_fill(cells[None, :] == torch.arange(a, b, device=DEV)[:, None], math.inf)
        dist[a:b] = torch.topk(D, k, dim=1, largest=False)[0]
    return [None, dist, None, cd]


def _assign64(X, C):
    lab, mind = [], []
    cn = (C * C).sum(1)
    for part in X.split(max(1, 40_000_000 // C.shape[0])):
        v, i = (cn[None, :] - 2 * (part @ C.T)).min(1)
        lab.append(i)
        mind.append(v)
    return torch.cat(lab), torch.cat(mind)


def _exact_kmeans(case, seed):
    n, nc = case["n"], _num_clusters(case["n"])
    X = _pcs(n, case["d"], seed)[0].double()
    state, seen, first = _srand(0), set(), []
    while len(first) < nc:
        j, state = _randint(n, state)
        if j not in seen:
            seen.add(j)
            first.append(j)
    buffers = [X[torch.tensor(first, device=DEV)], None]
    it, old = 0, 0.0
    while True:
        lab, mind = _assign64(X, buffers[it & 1])
        size = torch.bincount(lab, minlength=nc)
        if int(size.min()) == 0:
            return None  # a cluster without cells: its new centre is a cell
        sums = torch.zeros(nc, case["d"], dtype=torch.float64, device=DEV).index_add_(0, lab, X)
        buffers[(it + 1) & 1] = sums / size[:, None]
        it += 1
        if it == case["iterations"]:
            break
        total = float((X * X).sum() + mind.sum())
        if it > 1 and old - total < 1e-2 * old:
            break
        old = total
    lab, mind = _assign64(X, buffers[it & 1])
    return [None, None, buffers[0], buffers[1], None, mind, (X * X).sum(1)]


def _exact_harmony(case, seed):
    """Harmony with its defaults: blocks of 5 % of the cells in the seeded
    order, chunks of 256 cells, theta 2, alpha 0.2, sigma 0.1."""
    n, d, B = case["n"], case["d"], case["batches"]
    X, labels, Y = _harmony_inputs(case, seed)
    X, Y, lab = X.double(), Y.double(), labels.long()
    C, chunk, sigma, theta, alpha = Y.shape[0], min(256, n), 0.1, 2.0, 0.2
    sigma = float(np.float32(sigma))
    alpha, tol = float(np.float32(alpha)), float(np.float32(0.01))
    tos = 2.0 / sigma
    Z = X / X.norm(dim=1, keepdim=True)
    count = torch.bincount(lab, minlength=B).double()
    Pr = count / n
    block = math.ceil(float(np.float32(n) * np.float32(0.05)))
    order, state = [0] * n, _srand(0)
    for i in range(n):
        j, state = _randint(i + 1, state)
        order[i] = order[j]
        order[j] = i
    order = torch.tensor(order, device=DEV)
    zeros = lambda *shape: torch.zeros(*shape, dtype=torch.float64, device=DEV)  # noqa: E731

    def objective(R, dots, E, O):
        ent = torch.where(R > 0, R * torch.log(R.clamp(min=1e-300)), zeros(1)).sum()
        pen = (O * torch.log((O + E + 1) / (E + 1)) * theta).sum()
        return float(2 * (R * (1 - dots)).sum() + sigma * ent + sigma * pen)

    dots = Z @ Y.T
    R = torch.exp(tos * (dots - 1))
    R = R / R.sum(1, keepdim=True)
    O = zeros(B, C).index_add_(0, lab, R)
    E = Pr[:, None] * R.sum(0)[None, :]
    prev = objective(R, dots, E, O)
    it = 0
    for it in range(1, 11):
        for _ in range(5):
            Y = R.T @ Z
            Y = Y / Y.norm(dim=1, keepdim=True)
            for b0 in range(0, n, block):
                cells = order[b0:b0 + block]
                m = cells.numel()
                ch = torch.arange(m, device=DEV) // chunk
                nch = (m + chunk - 1) // chunk
                key = ch * B + lab[cells]
                old = zeros(nch * B, C).index_add_(0, key, R[cells]).view(nch, B, C)
                Ei = E[None] - Pr[None, :, None] * old.sum(1, keepdim=True)
                Oi = O[None] - old
                ratio = math.exp(-tos) * torch.pow((Ei + 1) / (Oi + Ei + 1), theta)
                r = torch.exp(tos * (Z[cells] @ Y.T)) * ratio.view(nch * B, C)[key]
                r = r / r.sum(1, keepdim=True)
                R[cells] = r
                new = zeros(nch * B, C).index_add_(0, key, r).view(nch, B, C)
                E = E + (Pr[None, :, None] * (new - old).sum(1, keepdim=True)).sum(0)
                O = O + (new - old).sum(0)
        value = objective(R, Z @ Y.T, E, O)
        sums = zeros(B, C, d)
        for b in range(B):
            at = (lab == b).nonzero().view(-1)
            sums[b] = R[at].T @ X[at]
        W = zeros(C, B, d)
        few = O < 1e-5 * count[:, None]
        factor = torch.where(few, zeros(1), 1 / (O + E * alpha))
        last = torch.where(few, zeros(1), -O * factor)  # last row of the elimination
        norm = 1 / torch.where(few, zeros(1), O * (1 + last)).sum(0)
        rs = torch.where(few[:, :, None], zeros(1), sums)
        # rows 0..B-1 of inv1^T inv2 times the right-hand sides
        tail = (last[:, :, None] * rs).sum(0) + rs.sum(0)
        W = factor.T[:, :, None] * rs.permute(1, 0, 2) \
            + (last * norm[None, :]).T[:, :, None] * tail[:, None, :]
        done = prev - value < tol * abs(prev)
        Z = X.clone()
        for b in range(B):
            at = (lab == b).nonzero().view(-1)
            Z[at] -= R[at] @ W[:, b]
        if done:
            break
        Z = Z / Z.norm(dim=1, keepdim=True)
        prev = value
    return [None, Z, Y, R]


def _exact_hvg(case, seed):
    g = case["g"]
    data, indices, indptr, cells, clip, used = _hvg_inputs(case, seed)
    v = data.double()
    if case["form"] == "csr":
        gene, row = indices.long(), _row_ids(indptr)
        keep = None if cells.numel() == 0 else torch.zeros(
            case["n"], dtype=torch.bool, device=DEV).index_fill_(0, cells, True)
    else:
        gene, row = _row_ids(indptr), indices.long()
        keep = None if cells.numel() == 0 else cells.bool()
    if keep is not None:
        at = keep[row]
        gene, v = gene[at], v[at]

    def total(x):
        return torch.zeros(g, dtype=torch.float64, device=DEV).index_add_(0, gene, x)

    s, s2, n = total(v), total(v * v), float(used)
    w = torch.minimum(v, clip.double()[gene])
    return [s / n, (n * s2 - s * s) / (n * (n - 1)), None, total(w), total(w * w)]


def _exact_prepare(case, seed):
    n, g = case["n"], case["g"]
    indptr, indices, counts = _counts_of_size(n, g, case["density"], seed)
    s = _row_sums(indptr, counts)
    rows = _row_ids(indptr)
    isf = (1e4 if case["norm"] == "logCP10k" else s.mean()) / s
    v = torch.log1p(counts.double() * isf[rows])
    post = None
    if case["norm"] == "PFlog1pPF":
        t = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, rows, v)
        post = t.mean() / t
        v = v * post[rows]
    order = torch.sort(indices.long() * n + rows)[1]
    return [isf, v, None, None, v[order]] + ([post] if post is not None else [])
