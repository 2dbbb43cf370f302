"""GPU HVG statistics (brisc_gb300.hvg, brisc/hvg.pyx) against the reference's
own outputs (tests/golden/hvg.npz) and the oracle, bit for bit."""
import numpy as np
import pytest
import scipy.sparse as sp

from brisc_gb300 import hvg
from oracle import hvg as oh
from test_oracle import HVG_TAGS, hvg_case

pytestmark = pytest.mark.gpu


def _run(form, d, ix, ip, cells, mask, nc, g, clip, device):
    """The four entry points on host arrays, or on CUDA tensors."""
    import torch

    def put(a):
        return torch.from_numpy(np.ascontiguousarray(a)).cuda() if device else a

    def out(n, dt):
        a = np.zeros(n, dt)
        return put(a)

    def back(a):
        return a.cpu().numpy() if device else a

    # nonzero counts: uint32 on the host; an int32 CUDA tensor holds the same
    # 32-bit words on the device
    m, v = out(g, np.float32), out(g, np.float32)
    c = out(g, np.int32 if device else np.uint32)
    b, q = out(g, np.float32), out(g, np.float32)
    D, IX, IP, CL = put(d), put(ix), put(ip), put(clip)
    if form == "csr":
        hvg.gene_mean_and_variance_csr(D, IX, IP, put(cells), nc, g, m, v, c, 8)
        hvg.clipped_sum_csr(D, IX, IP, nc, g, put(cells), CL, b, q, 8)
    else:
        hvg.gene_mean_and_variance_csc(D, IX, IP, put(mask), nc, g, m, v, c, 8)
        hvg.clipped_sum_csc(D, IX, IP, put(mask), CL, b, q, 8)
    if device:
        torch.cuda.synchronize()
    cc = back(c)
    return back(m), back(v), cc.view(np.uint32), back(b), back(q)


@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("sub", ["all", "sub"])
@pytest.mark.parametrize("form", ["csr", "csc"])
@pytest.mark.parametrize("tag", HVG_TAGS)
def test_hvg_matches_reference(cuda, golden, tag, form, sub, device):
    z = golden("hvg")
    n, g = int(z["n"]), int(z["g"])
    d, ix, ip = hvg_case(z, form, tag)
    if device and d.dtype == np.uint32:
        pytest.skip("torch keeps no uint32 CUDA tensors on every version")
    cells = z["cells"] if sub == "sub" else np.zeros(0, np.int64)
    mask = z["mask"] if sub == "sub" else np.zeros(0, np.int8)
    nc = len(cells) if sub == "sub" else n
    got = _run(form, d, ix, ip, cells, mask, nc, g, z["clip"], device)
    key = f"{form}_{tag}_{sub}"
    for a, name in zip(got, ("mean", "var", "nnz", "bsum", "bsq")):
        assert np.array_equal(a, z[f"{key}_{name}"]), name


def _random(n, g, dtype, itype, seed):
    rng = np.random.default_rng(seed)
    X = (rng.random((n, g)) < 0.08) * rng.integers(1, 300, (n, g))
    X[rng.random((n, g)) < 0.001] = 40000  # above every clip value
    A = sp.csr_matrix(X)
    B = sp.csc_matrix(X)
    A.sort_indices()
    B.sort_indices()
    return ((A.data.astype(dtype), A.indices.astype(itype), A.indptr.astype(itype)),
            (B.data.astype(dtype), B.indices.astype(itype), B.indptr.astype(itype)))


@pytest.mark.parametrize("itype", [np.int32, np.int64])
@pytest.mark.parametrize("dtype", [np.uint16, np.int32, np.uint32, np.int64,
                                   np.uint64, np.float32, np.float64])
def test_hvg_every_value_type(cuda, dtype, itype):
    n, g = 1500, 300
    csr, csc = _random(n, g, dtype, itype, 7)
    rng = np.random.default_rng(8)
    cells = np.sort(rng.choice(n, 500, replace=False)).astype(np.int64)
    mask = np.zeros(n, np.int8)
    mask[cells] = 1
    clip = (rng.random(g) * 200 + 1).astype(np.float32)
    for sub in (False, True):
        c = cells if sub else np.zeros(0, np.int64)
        mk = mask if sub else np.zeros(0, np.int8)
        nc = len(cells) if sub else n
        for form, (d, ix, ip) in (("csr", csr), ("csc", csc)):
            got = _run(form, d, ix, ip, c, mk, nc, g, clip, False)
            if form == "csr":
                want = (*oh.gene_mean_and_variance_csr(d, ix, ip, c, nc, g),
                        *oh.clipped_sum_csr(d, ix, ip, nc, g, c, clip))
            else:
                want = (*oh.gene_mean_and_variance_csc(d, ix, ip, mk, nc, g),
                        *oh.clipped_sum_csc(d, ix, ip, mk, clip))
            for a, w, name in zip(got, want, ("mean", "var", "nnz", "bsum", "bsq")):
                assert np.array_equal(a, w), (form, sub, name)


def test_hvg_many_genes_global_accumulators(cuda):
    """More genes than one CTA's shared accumulators hold (4096): the CSR
    kernels add straight into global memory."""
    n, g = 800, 6000
    csr, csc = _random(n, g, np.uint32, np.int32, 9)
    d, ix, ip = csr
    clip = np.full(g, 150.5, np.float32)
    got = _run("csr", d, ix, ip, np.zeros(0, np.int64), np.zeros(0, np.int8), n, g,
               clip, False)
    want = (*oh.gene_mean_and_variance_csr(d, ix, ip, np.zeros(0, np.int64), n, g),
            *oh.clipped_sum_csr(d, ix, ip, n, g, np.zeros(0, np.int64), clip))
    for a, w in zip(got, want):
        assert np.array_equal(a, w)


def test_hvg_out_of_range_index_rejected(cuda):
    """A gene index past num_dataset_genes is skipped by the kernel and
    reported as a ValueError (the reference would write out of bounds)."""
    ip = np.array([0, 2, 3], np.int32)
    ix = np.array([0, 5, 1], np.int32)  # gene 5 of 3
    d = np.array([1, 2, 3], np.uint32)
    m, v, c = np.zeros(3, np.float32), np.zeros(3, np.float32), np.zeros(3, np.uint32)
    with pytest.raises(ValueError, match="out of bounds"):
        hvg.gene_mean_and_variance_csr(d, ix, ip, np.zeros(0, np.int64), 2, 3, m, v, c, 1)
    mask = np.ones(1, np.int8)  # cell 1 is past the mask
    with pytest.raises(ValueError, match="out of bounds"):
        hvg.gene_mean_and_variance_csc(d, np.array([0, 1, 0], np.int32), ip, mask, 2, 2,
                                       m, v, c, 1)


def test_hvg_called_as_single_cell_calls_it(cuda, golden):
    """The keyword calls of SingleCell's HVG step (brisc/single_cell.py:
    11320-11395): CSR with an int64 cell list and num_cells = its length,
    CSC with a boolean cell mask."""
    z = golden("hvg")
    n, g = int(z["n"]), int(z["g"])
    cells = z["cells"]
    for form in ("csr", "csc"):
        d, ix, ip = hvg_case(z, form, "float32_int32")
        mean, var = np.zeros(g, np.float32), np.zeros(g, np.float32)
        nz = np.zeros(g, np.uint32)
        b, q = np.empty(g, np.float32), np.empty(g, np.float32)
        if form == "csr":
            hvg.gene_mean_and_variance_csr(
                data=d, indices=ix, indptr=ip, cell_indices=cells,
                num_cells=len(cells), num_dataset_genes=g, mean=mean, var=var,
                nonzero_count=nz, num_threads=4)
            hvg.clipped_sum_csr(
                data=d, indices=ix, indptr=ip, num_cells=len(cells),
                num_dataset_genes=g, cell_indices=cells, clip_val=z["clip"],
                batch_counts_sum=b, squared_batch_counts_sum=q, num_threads=4)
        else:
            mask = z["mask"].astype(bool)
            hvg.gene_mean_and_variance_csc(
                data=d, indices=ix, indptr=ip, cell_mask=mask,
                num_cells=int(mask.sum()), num_dataset_genes=g, mean=mean, var=var,
                nonzero_count=nz, num_threads=4)
            hvg.clipped_sum_csc(
                data=d, indices=ix, indptr=ip, cell_mask=mask, clip_val=z["clip"],
                batch_counts_sum=b, squared_batch_counts_sum=q, num_threads=4)
        key = f"{form}_float32_int32_sub"
        for a, name in ((mean, "mean"), (var, "var"), (nz, "nnz"), (b, "bsum"),
                        (q, "bsq")):
            assert np.array_equal(a, z[f"{key}_{name}"]), (form, name)


def _skewed_csc(lengths, n, dtype, seed):
    """A CSC matrix whose gene j stores lengths[j] counts (<= n cells)."""
    rng = np.random.default_rng(seed)
    ix = [np.sort(rng.choice(n, m, replace=False)) for m in lengths]
    ip = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    d = rng.integers(1, 40, int(ip[-1]))
    d[rng.random(d.size) < 0.01] = 60000
    return d.astype(dtype), np.concatenate(ix).astype(np.int32), ip


@pytest.mark.parametrize("lengths", [
    [1], [0, 0, 4096, 0, 4096, 0], [4095, 1, 4097, 0, 8192, 3], [0] * 70 + [9000] + [1] * 70,
    [31, 32, 33, 255, 256, 257] * 20, [20000, 0, 19999]])
def test_hvg_csc_entries_split_across_genes(cuda, lengths):
    """Genes that start, end and straddle the chunks of entries the CSC kernel
    splits the matrix into, empty genes between them, with and without a
    mask: every statistic bit-identical to the oracle's."""
    n, g = 20000, len(lengths)
    d, ix, ip = _skewed_csc(lengths, n, np.uint16, sum(lengths))
    rng = np.random.default_rng(3)
    clip = (rng.random(g) * 30 + 1).astype(np.float32)
    for mask in (np.zeros(0, np.int8), (rng.random(n) < 0.7).astype(np.int8)):
        nc = int(mask.sum()) if mask.size else n
        got = _run("csc", d, ix, ip, None, mask, nc, g, clip, False)
        want = (*oh.gene_mean_and_variance_csc(d, ix, ip, mask, nc, g),
                *oh.clipped_sum_csc(d, ix, ip, mask, clip))
        for a, w, name in zip(got, want, ("mean", "var", "nnz", "bsum", "bsq")):
            assert np.array_equal(a, w), name


@pytest.mark.parametrize("n,g", [(1, 1), (700, 31), (5000, 4097), (300, 18910), (300, 37900),
                                 (64, 160000)])
def test_hvg_csr_gene_slices(cuda, n, g):
    """Gene counts around what one, two and more CTAs hold in shared memory and
    past what they hold at all, with zeros and counts on both sides of the
    32-bit accumulators' limit, whole and by cell list (repeated cells, and a
    row that repeats genes): bit-identical to the oracle's."""
    rng = np.random.default_rng(g)
    lens = rng.integers(0, min(g, 400) + 1, n)
    lens[0] = min(g, 400)
    ip = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    ix = np.concatenate([rng.choice(g, m, replace=False) for m in lens]).astype(np.int64)
    d = rng.choice([0, 1, 1, 1, 2, 3, 14, 15, 16, 17, 300, 65535, 65536], ix.size).astype(np.float32)
    if n > 1:  # the last row holds one gene more often than there are genes
        extra = min(g, 500) + 7
        ip[-1] += extra
        ix = np.concatenate([ix, np.full(extra, g - 1)])
        d = np.concatenate([d, np.ones(extra, np.float32)])
    clip = rng.choice(np.float32([0.5, 2, 14.5, 15, 299]), g)
    cells = np.concatenate([np.arange(n), np.arange(n)[::-2], [n - 1, n - 1]]).astype(np.int64)
    for c in (np.zeros(0, np.int64), cells):
        nc = len(c) if len(c) else n
        got = _run("csr", d, ix, ip, c, None, nc, g, clip, False)
        want = (*oh.gene_mean_and_variance_csr(d, ix, ip, c, nc, g),
                *oh.clipped_sum_csr(d, ix, ip, nc, g, c, clip))
        for a, w, name in zip(got, want, ("mean", "var", "nnz", "bsum", "bsq")):
            assert np.array_equal(a, w, equal_nan=True), name


LARGE_COUNTS = [
    (np.uint16, [60000, 65535, 65533]),           # every few additions wrap a word
    (np.float32, [16, 17, 300, 2.75, 0.5, 5000]), (np.float64, [40, 7e4, 1e6, 3]),
    (np.int64, [20, 65535, 65536, 2**33, 1]), (np.int32, [1] * 19 + [500]),  # below the line
    (np.uint32, [1] * 12 + [500])]                # above it


@pytest.mark.parametrize("n,g,dtype,values", [
    (n, g, t, v) for n, g in ((1, 3), (9000, 3), (2500, 700)) for t, v in LARGE_COUNTS] +
    [(900, 38000, *LARGE_COUNTS[1]), (3000, 150000, *LARGE_COUNTS[0])])
def test_hvg_csr_of_large_counts(cuda, n, g, dtype, values):
    """Counts that are mostly or partly above the 32-bit accumulators' limit, few
    and many per gene, whole and by cell list (150,000 genes: the words are taken
    out within a chunk): bit-identical to the oracle's integers."""
    rng = np.random.default_rng(n + g)
    lens = rng.integers(1, min(g, 60) + 1, n)
    ip = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    ix = np.concatenate([rng.choice(min(g, 400), m, replace=False) for m in lens]).astype(np.int64)
    ix = ix * (g // min(g, 400))
    d = rng.choice(np.array(values, np.float64), ix.size).astype(dtype)
    clip = rng.choice(np.float32([0.5, 15, 299, 64000, 1e9]), g)
    for c in (np.zeros(0, np.int64), np.concatenate([np.arange(n), np.arange(n)[::-3]])):
        c = c.astype(np.int64)
        nc = len(c) if len(c) else n
        got = _run("csr", d, ix, ip, c, None, nc, g, clip, False)
        want = (*oh.gene_mean_and_variance_csr(d, ix, ip, c, nc, g),
                *oh.clipped_sum_csr(d, ix, ip, nc, g, c, clip))
        for a, w, name in zip(got, want, ("mean", "var", "nnz", "bsum", "bsq")):
            assert np.array_equal(a, w, equal_nan=True), name
