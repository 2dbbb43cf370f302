"""knn_self on the GPU (brisc_gb300/knn.py over csrc/knn.cu) against the
reference's own outputs (tests/golden/knn.npz, from brisc/knn.pyx:13 after
brisc/kmeans.pyx:889) and the NumPy oracle (oracle/knn.py).

Tolerance: the same nearest clusters and neighbour sets except at near-ties
within FP32 rounding of the squared norms (2e-6 relative, doubled), distances
within that rounding, run-to-run bit identity."""
import numpy as np
import pytest

from knn_cases import case, check_against

pytestmark = pytest.mark.gpu


def _run(c, **kw):
    from brisc_gb300 import knn
    n, k, cs = c["X"].shape[0], c["num_neighbors"], c["num_clusters_searched"]
    out = dict(neighbors=np.zeros((n, k), np.uint32), distances=np.zeros((n, k), np.float32),
               centroid_distances=np.zeros((n, cs), np.float32),
               nearest_clusters=np.zeros((n, cs), np.uint32))
    knn.knn_self(X=c["X"], sorted_order=c["sorted_order"], centroids=c["centroids"],
                 num_cells_per_cluster=c["num_cells_per_cluster"],
                 cell_norms=c["cell_norms"], num_neighbors=k,
                 num_clusters_searched=cs, chunk_size_kmeans=min(4096, n),
                 chunk_size_search=min(256, n), is_mac=False, num_threads=1, **out, **kw)
    return out


@pytest.mark.parametrize("name", ["knn_a", "knn_b"])
def test_knn_self_matches_reference(cuda, golden, name):
    c = case(golden("knn"), name)
    o = _run(c)
    check_against(c, o["neighbors"], o["distances"], o["nearest_clusters"],
                  o["centroid_distances"])


def test_knn_self_bit_identical_and_device_tensors(cuda, golden):
    """Two runs from host arrays and one on CUDA tensors (int32 holding the
    uint32 arrays) give the same bits."""
    import torch
    from brisc_gb300 import knn
    c = case(golden("knn"), "knn_a")
    a, b = _run(c), _run(c)
    for key in a:
        np.testing.assert_array_equal(a[key], b[key])
    T = lambda x: torch.from_numpy(np.ascontiguousarray(  # noqa: E731
        x.view(np.int32) if x.dtype == np.uint32 else x)).to(cuda)
    n, k, cs = c["X"].shape[0], c["num_neighbors"], c["num_clusters_searched"]
    dev = dict(neighbors=torch.zeros((n, k), dtype=torch.int32, device=cuda),
               distances=torch.zeros((n, k), dtype=torch.float32, device=cuda),
               centroid_distances=torch.zeros((n, cs), dtype=torch.float32, device=cuda),
               nearest_clusters=torch.zeros((n, cs), dtype=torch.int32, device=cuda))
    knn.knn_self(X=T(c["X"]), sorted_order=T(c["sorted_order"]),
                 centroids=T(c["centroids"]),
                 num_cells_per_cluster=T(c["num_cells_per_cluster"]),
                 cell_norms=T(c["cell_norms"]), num_neighbors=k,
                 num_clusters_searched=cs, **dev)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(dev["neighbors"].cpu().numpy().view(np.uint32),
                                  a["neighbors"])
    np.testing.assert_array_equal(dev["distances"].cpu().numpy(), a["distances"])


def _lloyd(X, nc, iters=3, seed=0):
    """A small deterministic k-means (random init + Lloyd steps) standing in
    for the reference's, to make knn_self inputs at sizes with no fixture."""
    rng = np.random.default_rng(seed)
    C = X[rng.choice(len(X), nc, replace=False)].astype(np.float64)
    X64 = X.astype(np.float64)
    for _ in range(iters):
        lab = np.argmin(-2 * X64 @ C.T + (C * C).sum(1), 1)
        for j in range(nc):
            if np.any(lab == j):
                C[j] = X64[lab == j].mean(0)
    lab = np.argmin(-2 * X64 @ C.T + (C * C).sum(1), 1)
    keep = np.unique(lab)
    remap = np.zeros(nc, np.int64)
    remap[keep] = np.arange(len(keep))
    lab, C = remap[lab], C[keep]
    order = np.argsort(C[:, 0])
    inv = np.empty_like(order)
    inv[order] = np.arange(len(order))
    lab, C = inv[lab], C[order]
    so = np.argsort(lab, kind="stable").astype(np.uint32)
    Xs = np.ascontiguousarray(X[so])
    norms = np.einsum("ij,ij->i", Xs, Xs).astype(np.float32)
    counts = np.bincount(lab, minlength=len(C)).astype(np.uint32)
    return Xs, so, np.ascontiguousarray(C.astype(np.float32)), counts, norms


@pytest.mark.parametrize("n,d,nc,k,cs", [(15000, 50, 120, 20, 24), (4000, 100, 40, 64, 40),
                                         (3000, 13, 30, 33, 30), (2500, 7, 250, 128, 200)])
def test_knn_self_matches_oracle(cuda, n, d, nc, k, cs):
    """Shapes beyond the fixtures: 50 and 100 dimensions, 33/64/128
    neighbours, up to 200 clusters searched, empty-ish clusters."""
    from knn_cases import knn_pcs
    from oracle import knn as oknn
    X = knn_pcs(n, d, 30, seed=n + d)
    Xs, so, C, counts, norms = _lloyd(X, nc)
    cs = min(cs, len(C))
    c = dict(X=Xs, sorted_order=so, centroids=C, num_cells_per_cluster=counts,
             cell_norms=norms, num_neighbors=k, num_clusters_searched=cs)
    nbr, dist, near, cdist = oknn.knn_self(Xs, so, C, counts, norms, k, cs)
    c.update(ref_neighbors=nbr, ref_distances=dist, ref_nearest=near, ref_cdist=cdist)
    o = _run(c)
    check_against(c, o["neighbors"], o["distances"], o["nearest_clusters"],
                  o["centroid_distances"])


@pytest.mark.parametrize("name", ["knn_a", "knn_b"])
def test_kmeans_matches_reference(cuda, golden, name):
    """GPU k-means (random initialisation, the reference's M-step order)
    against the reference's kmeans on the same PCs: the same iteration count,
    labels identical except at FP32 near-ties of the E step, centroids and
    cluster sizes accordingly."""
    from brisc_gb300 import knn
    from knn_cases import knn_pcs
    z = golden("knn")
    n, d, comps, seed, k, cs = (int(v) for v in z[f"{name}_shape"])
    X = knn_pcs(n, d, comps, seed)
    ref_c = z[f"{name}_km_final_centroids"]
    nc = ref_c.shape[0]
    out = dict(cluster_labels=np.zeros(n, np.uint32), min_distances=np.zeros(n, np.float32),
               cell_norms=np.zeros(n, np.float32),
               centroids=np.zeros((nc, d), np.float32),
               centroids_new=np.zeros((nc, d), np.float32),
               num_cells_per_cluster=np.zeros(nc, np.uint32))
    it = knn.kmeans(X=X, seed=0, chunk_size=min(4096, n), **out)
    assert it == int(z[f"{name}_km_iterations"])
    C = out["centroids_new"] if it & 1 else out["centroids"]
    same = (out["cluster_labels"] == z[f"{name}_km_cluster_labels"]).mean()
    assert same >= 0.999, same
    scale = np.abs(ref_c).max()
    if same == 1.0:  # same assignments: the reference's summation order
        np.testing.assert_allclose(C, ref_c, rtol=0, atol=2e-6 * scale)
        np.testing.assert_array_equal(out["num_cells_per_cluster"],
                                      z[f"{name}_km_num_cells_per_cluster"])
    else:
        np.testing.assert_allclose(C, ref_c, rtol=0, atol=1e-2 * scale)
    np.testing.assert_allclose(out["cell_norms"], z[f"{name}_cell_norms"][
        np.argsort(z[f"{name}_sorted_order"])], rtol=2e-6)


@pytest.mark.parametrize("name", ["knn_a", "knn_b"])
def test_neighbors_pipeline_matches_reference(cuda, golden, name):
    """brisc_gb300.knn.neighbors (GPU k-means, neighbors()'s preparation, GPU
    knn_self) against the reference's neighbours, both in the original cell
    order: the same sets except at near-ties."""
    from brisc_gb300 import knn
    from knn_cases import knn_pcs
    from oracle import knn as oknn
    z = golden("knn")
    n, d, comps, seed, k, cs = (int(v) for v in z[f"{name}_shape"])
    X = knn_pcs(n, d, comps, seed)
    so = z[f"{name}_sorted_order"]
    ref = np.empty_like(z[f"{name}_neighbors"])
    ref[so] = z[f"{name}_neighbors"]
    nbr, dist = knn.neighbors(X, num_neighbors=k,
                              num_clusters_searched=None if name == "knn_b" else cs)
    ident = np.arange(n, dtype=np.uint32)
    norms = np.einsum("ij,ij->i", X, X).astype(np.float32)
    same, worst = oknn.compare(X, ident, norms, nbr, ref)
    assert same >= 0.99 and worst <= 1.0, (same, worst)


def _chain(X, C):
    """x.c for every pair as the FP32 fused-multiply-add chain over the
    dimensions in order (each step's product and sum rounded once: the sum
    is formed in extended precision)."""
    acc = np.zeros((len(X), len(C)), np.float32)
    for j in range(X.shape[1]):
        p = np.multiply.outer(X[:, j].astype(np.longdouble), C[:, j].astype(np.longdouble))
        acc = (p + acc).astype(np.float32)
    return acc


def _fma(a, b, c):
    return (np.longdouble(a) * b + c).astype(np.float32)


def _lists(dist, order, size):
    """Each row's list after offering the columns of `order[row]` in order, a
    column replacing the first worst entry when strictly closer."""
    n = len(dist)
    out_d = np.full((n, size), np.finfo(np.float32).max, np.float32)
    out_i = np.full((n, size), 0xFFFFFFFF, np.uint32)
    for i in range(n):
        for c in order[i]:
            w = int(np.argmax(out_d[i]))
            if dist[i, c] < out_d[i, w]:
                out_d[i, w], out_i[i, w] = dist[i, c], c
        o = np.lexsort((out_i[i], out_d[i]))
        out_d[i], out_i[i] = out_d[i, o], out_i[i, o]
    return out_i, out_d


@pytest.mark.parametrize("n,d,nc,k,cs", [
    (33, 1, 3, 4, 2), (129, 13, 5, 32, 5), (300, 50, 9, 33, 4), (257, 61, 40, 20, 12),
    (200, 62, 7, 65, 7), (260, 128, 33, 128, 33), (700, 8, 620, 5, 256), (90, 4, 1, 10, 1)])
def test_knn_self_bit_exact_with_ties(cuda, n, d, nc, k, cs):
    """The tensor cores only select candidates: neighbours, distances and
    nearest clusters are bit for bit those of the exhaustive FP32 loop, also
    where rows repeat (equal distances, the reference's tie rule), clusters are
    empty or start inside an 8-row group, more than 512 clusters are searched
    by one CTA's cells, and one cell is far larger than the rest."""
    rng = np.random.default_rng(n * d)
    X = rng.standard_normal((n, d)).astype(np.float32) * np.float32(3)
    X[rng.integers(0, n, n // 3)] = X[rng.integers(0, n, n // 3)]
    X[n // 2] *= 50
    C = rng.standard_normal((nc, d)).astype(np.float32) * np.float32(3)
    if nc > 2:
        C[-1] = C[0]
    lab = np.sort(rng.integers(0, max(1, nc - 1), n))
    counts = np.bincount(lab, minlength=nc).astype(np.uint32)
    norms = np.einsum("ij,ij->i", X, X).astype(np.float32)
    so = rng.permutation(n).astype(np.uint32)
    c = dict(X=X, sorted_order=so, centroids=C, num_cells_per_cluster=counts,
             cell_norms=norms, num_neighbors=k, num_clusters_searched=cs)
    o = _run(c)
    cn = C[:, 0] * C[:, 0]
    for j in range(1, d):
        cn = _fma(C[:, j], C[:, j], cn)
    pd = _fma(np.float32(-2), _chain(X, C), cn[None, :])
    near, cdist = _lists(pd, [range(nc)] * n, cs)
    np.testing.assert_array_equal(o["nearest_clusters"], near)
    np.testing.assert_array_equal(o["centroid_distances"], cdist)
    start = np.concatenate([[0], np.cumsum(counts)]).astype(int)
    dist = norms[:, None] + _fma(np.float32(-2), _chain(X, X), norms[None, :])
    order = [[r for u in np.sort(near[i]) for r in range(start[u], start[u + 1]) if r != i]
             for i in range(n)]
    want_i, want_d = _lists(dist, order, k)
    have = want_i != 0xFFFFFFFF
    np.testing.assert_array_equal(o["distances"], want_d)
    np.testing.assert_array_equal(o["neighbors"] != 0xFFFFFFFF, have)
    np.testing.assert_array_equal(o["neighbors"][have], so[want_i[have]])


@pytest.mark.parametrize("n,d,nc,chunk", [(5, 1, 2, 3), (700, 50, 700, 256), (9000, 33, 1, 4096),
                                          (20000, 7, 300, 4096), (20000, 5, 40, 20000),
                                          (3000, 20, 2500, 1000)])
def test_kmeans_m_step_order(cuda, n, d, nc, chunk):
    """Centroids after one iteration, bit for bit: each chunk's cells of a
    cluster added in order, the chunks in order, times the float of 1 / count;
    chunks that end inside the cells, one cluster, a cluster per cell, and a
    chunk longer than the sorted path takes."""
    from brisc_gb300 import knn
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, d)).astype(np.float32)
    out = dict(cluster_labels=np.zeros(n, np.uint32), min_distances=np.zeros(n, np.float32),
               cell_norms=np.zeros(0, np.float32), centroids=np.zeros((nc, d), np.float32),
               centroids_new=np.zeros((nc, d), np.float32),
               num_cells_per_cluster=np.zeros(nc, np.uint32))
    assert knn.kmeans(X=X, chunk_size=chunk, num_kmeans_iterations=1, **out) == 1
    C0 = out["centroids"]  # the initial centroids: cells
    pd = _fma(np.float32(-2), _chain(X, C0), _norm_chain(C0)[None, :])
    lab = np.argmin(pd, 1)
    want = np.zeros((nc, d), np.float32)
    for c0 in range(0, n, chunk):
        part = np.zeros((nc, d), np.float32)
        for i in range(c0, min(n, c0 + chunk)):
            part[lab[i]] += X[i]
        want += part
    count = np.bincount(lab, minlength=nc)
    assert count.min() > 0
    want *= (1.0 / count).astype(np.float32)[:, None]
    np.testing.assert_array_equal(out["centroids_new"], want)


def _norm_chain(C):
    cn = C[:, 0] * C[:, 0]
    for j in range(1, C.shape[1]):
        cn = _fma(C[:, j], C[:, j], cn)
    return cn


def _kmeans_of(X, nc, seed):
    from brisc_gb300 import knn
    n, d = X.shape
    out = dict(cluster_labels=np.zeros(n, np.uint32), min_distances=np.zeros(n, np.float32),
               cell_norms=np.zeros(0, np.float32), centroids=np.zeros((nc, d), np.float32),
               centroids_new=np.zeros((nc, d), np.float32),
               num_cells_per_cluster=np.zeros(nc, np.uint32))
    assert knn.kmeans(X=X, chunk_size=n, num_kmeans_iterations=1, seed=seed, **out) == 1
    return out


def _nan_and_equal_cells(nan, equal, seed_of):
    """`nan` cells of NaN first, then `equal` equal cells, then one far away, and a
    seed whose random initial centroids leave that one out."""
    from oracle import clib
    n = nan + equal + 1
    X = np.full((n, 3), np.nan, np.float32)
    X[nan:] = 1.0
    X[-1] = 50.0
    seed = next(s for s in range(10_000) if n - 1 not in clib.kmeans_init(n, seed_of, s))
    return X, seed


def test_kmeans_relocation_never_takes_an_unlabelled_cell(cuda):
    """61 empty clusters, one cell at a positive distance and 60 at zero: the
    clusters take those 61, never one of the NaN cells in front of them, which
    have no label."""
    X, seed = _nan_and_equal_cells(3, 60, 62)
    out = _kmeans_of(X, 62, seed)
    assert (out["cluster_labels"][:3] == 0xFFFFFFFF).all()
    assert (out["cluster_labels"][3:] < 62).all()
    assert out["num_cells_per_cluster"].sum() == 61
    assert np.isfinite(out["centroids_new"]).all()
    np.testing.assert_array_equal(out["centroids_new"][out["cluster_labels"][-1]], X[-1])


def test_kmeans_refuses_more_empty_clusters_than_labelled_cells(cuda):
    """59 empty clusters, 34 cells with a label."""
    X, seed = _nan_and_equal_cells(30, 33, 60)
    with pytest.raises(ValueError, match="more empty clusters than cells"):
        _kmeans_of(X, 60, seed)


def _refused_call(cuda, n, d, nc, k, cs, offset):
    """knn_self with a cluster one cell short; the outputs, filled with 7."""
    import torch
    from brisc_gb300 import knn
    gen = torch.Generator(device=cuda).manual_seed(1)
    X = torch.randn(n, d, generator=gen, device=cuda) + offset
    sizes = torch.full((nc,), n // nc, dtype=torch.int32, device=cuda)
    sizes[3] -= 1
    out = dict(neighbors=torch.full((n, k), 7, dtype=torch.int32, device=cuda),
               distances=torch.full((n, k), 7.0, device=cuda),
               nearest_clusters=torch.full((n, cs), 7, dtype=torch.int32, device=cuda),
               centroid_distances=torch.full((n, cs), 7.0, device=cuda))
    with pytest.raises(ValueError, match="does not sum to the number of cells"):
        knn.knn_self(X=X, sorted_order=torch.arange(n, dtype=torch.int32, device=cuda),
                     centroids=X[:nc].contiguous(), num_cells_per_cluster=sizes,
                     cell_norms=(X * X).sum(1), num_neighbors=k, num_clusters_searched=cs, **out)
    return out


@pytest.mark.parametrize("k,cs", [(5, 4), (70, 70)])
def test_knn_self_refusal_leaves_the_outputs(cuda, k, cs):
    """Cluster sizes that do not sum to the number of cells: refused, and
    nothing is written (lists on both sides of 64 entries)."""
    for name, t in _refused_call(cuda, 400, 6, 80, k, cs, 0.0).items():
        assert (t == 7).all(), name



def _norms_of(X):
    return np.einsum("ij,ij->i", X, X).astype(np.float32)


@pytest.mark.parametrize("queries,d,nc,k,cs,kind", [
    (64, 4, 60, 20, 3, "repeat"), (64, 3, 60, 64, 5, "offset"), (64, 2, 700, 5, 256, "offset"),
    (64, 6, 90, 65, 66, "offset"), (128, 5, 150, 33, 40, "repeat"), (128, 4, 90, 1, 2, "repeat"),
    (128, 2, 150, 128, 130, "repeat"), (128, 7, 200, 24, 64, "plain"), (128, 50, 300, 40, 9, "plain"),
    (128, 8, 90, 100, 70, "plain")])
def test_knn_self_bit_exact_at_full_tiles(cuda, queries, d, nc, k, cs, kind):
    """The exhaustive loop's bits where a CTA takes 64 or 128 queries (that many
    per SM, and a ragged last CTA), for every class of list lengths; with rows
    that repeat (most lists end in a tie) and rows far from the origin (margins
    wider than the spread), which whole groups of queries compute again. First,
    last and random rows are compared."""
    import torch
    n = queries * torch.cuda.get_device_properties(cuda).multi_processor_count + 37
    rng = np.random.default_rng(n + d)
    X = rng.standard_normal((n, d)).astype(np.float32)
    if kind == "repeat":
        at = rng.integers(0, n, 6 * n // 10)
        X[at] = X[rng.integers(0, 40, len(at))]
    if kind == "offset":
        X += np.float32(300)
    C = X[rng.choice(n, nc, replace=False)] + np.float32(0.1)
    counts = np.bincount(np.sort(rng.integers(0, nc, n)), minlength=nc).astype(np.uint32)
    norms = _norms_of(X)
    so = rng.permutation(n).astype(np.uint32)
    o = _run(dict(X=X, sorted_order=so, centroids=C, num_cells_per_cluster=counts,
                  cell_norms=norms, num_neighbors=k, num_clusters_searched=cs))
    rows = np.unique(np.concatenate([np.arange(12), np.arange(n - 40, n),
                                     rng.choice(n, 40, replace=False)]))
    pd = _fma(np.float32(-2), _chain(X[rows], C), _norm_chain(C)[None, :])
    near, cdist = _lists(pd, [range(nc)] * len(rows), cs)
    np.testing.assert_array_equal(o["nearest_clusters"][rows], near)
    np.testing.assert_array_equal(o["centroid_distances"][rows], cdist)
    start = np.concatenate([[0], np.cumsum(counts)]).astype(int)
    for i, row in enumerate(rows):
        ids = np.concatenate([np.arange(start[u], start[u + 1]) for u in np.sort(near[i])])
        ids = ids[ids != row]
        dist = norms[row] + _fma(np.float32(-2), _chain(X[row:row + 1], X[ids]), norms[ids])
        at, want = _lists(dist, [range(len(ids))], k)
        have = at[0] != 0xFFFFFFFF
        np.testing.assert_array_equal(o["distances"][row], want[0])
        np.testing.assert_array_equal(o["neighbors"][row][have], so[ids[at[0][have]]])
        assert (o["neighbors"][row][~have] == 0xFFFFFFFF).all()


def test_kmeans_e_step_far_from_the_origin(cuda):
    """Labels and distances of cells whose margins are wider than the centroids'
    spread, bit for bit the first nearest centroid's."""
    import torch
    n = 64 * torch.cuda.get_device_properties(cuda).multi_processor_count + 5
    rng = np.random.default_rng(3)
    X = (rng.standard_normal((n, 6)) + 400).astype(np.float32)
    out = _kmeans_of(X, 300, 1)
    rows = np.unique(np.concatenate([np.arange(40), np.arange(n - 40, n),
                                     rng.choice(n, 100, replace=False)]))
    C = out["centroids_new"]
    pd = _fma(np.float32(-2), _chain(X[rows], C), _norm_chain(C)[None, :])
    np.testing.assert_array_equal(out["cluster_labels"][rows], pd.argmin(1))
    np.testing.assert_array_equal(out["min_distances"][rows], pd.min(1))


@pytest.mark.parametrize("k,cs", [(5, 20), (70, 66)])
def test_knn_self_refusal_of_wide_margins(cuda, k, cs):
    """The same where every list would be computed again."""
    for name, t in _refused_call(cuda, 16000, 6, 400, k, cs, 300.0).items():
        assert (t == 7).all(), name
