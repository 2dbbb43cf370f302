// k-nearest-neighbour search over cluster-sorted principal components: the
// reference's knn_self (brisc/knn.pyx:13-515), the search half of
// SingleCell.neighbors() (brisc/single_cell.py:12139-12665). Its inputs are
// the k-means results neighbors() prepares: the PCs grouped by cluster, the
// centroids, the cluster sizes and each cell's squared norm.
//
// Same search as the reference, the same candidates in the same order:
//  1. nearest clusters: for each cell, the num_clusters_searched centroids
//     with the smallest partial distance |c|^2 - 2 x.c, candidates visited in
//     ascending centroid order and kept while strictly smaller than the
//     current worst (the reference's max-heap of knn.pyx:150-185);
//  2. neighbours: for each cell, every cell of those clusters except itself,
//     visited by ascending cluster label and then ascending position, with
//     distance |x|^2 + (|c|^2 - 2 x.c) and the same strict-improvement rule
//     (knn.pyx:186-290); the lists come out sorted by ascending distance and
//     the neighbour ids are mapped through sorted_order.
// The dot products are FP32 fused multiply-adds in dimension order; the
// reference's come from sgemm, so distances agree to FP32 rounding of the
// norms and neighbours can differ only where two candidates' distances do.
//
// The inner loops of both, and of the k-means E step below, are knn_tc.cu: the
// tensor cores select the candidates that can enter a list, and those are
// evaluated and offered exactly as above.
// No atomics on floating-point data and no order-dependent reductions: the
// result depends only on the inputs.
#include <algorithm>
#include <cfloat>
#include <vector>

#include "common.cuh"
#include "knn_tc.cuh"
#include "pcg.h"

namespace bgpu {

namespace {

constexpr uint32_t kMaxDims = 128;
constexpr uint32_t kMaxSearched = 256;
constexpr uint32_t kMaxNeighbors = 128;
constexpr uint32_t kMaxClusters = 32768;

__global__ void k_knn_centroid_norms(const float* __restrict__ C, uint32_t nc,
                                     uint32_t d, float* __restrict__ cn) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nc) return;
  const float* c = C + (uint64_t)i * d;
  float s = c[0] * c[0];
  for (uint32_t j = 1; j < d; ++j) s = fmaf(c[j], c[j], s);
  cn[i] = s;
}

// Cluster offsets (exclusive prefix sum of the sizes) and their total, by one
// block: a run of clusters per thread, then a scan of the runs (2,191 clusters:
// 57 us for one thread, 5 us). Sizes that do not sum to n set err, behind which
// the searches write nothing.
constexpr int kOffThreads = 1024;
__global__ void __launch_bounds__(kOffThreads)
k_knn_offsets(const uint32_t* __restrict__ sizes, uint32_t nc, uint64_t n,
              uint64_t* __restrict__ off, int* __restrict__ err) {
  __shared__ uint64_t wsum[kOffThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t per = (nc + kOffThreads - 1) / kOffThreads;
  const uint32_t a = min(nc, threadIdx.x * per), b = min(nc, a + per);
  uint64_t mine = 0;
  for (uint32_t i = a; i < b; ++i) mine += sizes[i];
  uint64_t incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) wsum[wid] = incl;
  __syncthreads();
  uint64_t pre = incl - mine, total = 0;
  for (int w = 0; w < kOffThreads / 32; ++w) {
    if (w < wid) pre += wsum[w];
    total += wsum[w];
  }
  const bool good = total == n;
  for (uint32_t i = a; i < b; ++i) {
    off[i] = good ? pre : 0ull;
    pre += sizes[i];
  }
  if (threadIdx.x == 0) {
    off[nc] = good ? total : 0ull;
    if (!good) atomicOr(err, kKnnErrSizes);
  }
}

// A refusal that callers may rely on: the shared memory that a table of all
// clusters next to tiles of the cells would take.
size_t search_table_bytes(uint32_t d, uint32_t nc, uint32_t cs, uint32_t k) {
  uint32_t st = (d + 3u) & ~3u;
  if (((st >> 2) & 1u) == 0u) st += 4u;
  const uint32_t R = k <= 32 ? 1 : k <= 64 ? 2 : 4;
  return ((size_t)64 * st + (size_t)32 * st + 64) * 4 + (size_t)nc * 4 + (size_t)32 * cs * 4 +
         (size_t)8 * 32 * R * 8;
}

// The device error word of a call's kernels, read after the stream's wait.
int knn_status(const int* err, cudaStream_t s) {
  int h = 0;
  BGPU_CUDA(cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, s));
  BGPU_CUDA(cudaStreamSynchronize(s));
  BGPU_REQUIRE((h & kKnnErrSizes) == 0, BGPU_ERR_INVALID,
               "knn_self: num_cells_per_cluster does not sum to the number of cells");
  BGPU_REQUIRE(h == 0, BGPU_ERR_DEVICE,
               "nearest rows: a tensor-core wait did not complete within its time limit");
  return BGPU_OK;
}

}  // namespace

}  // namespace bgpu

using namespace bgpu;

extern "C" int bgpu_knn_self(const float* X, const uint32_t* sorted_order,
                             const float* centroids,
                             const uint32_t* num_cells_per_cluster, uint32_t* neighbors,
                             float* distances, const float* cell_norms,
                             float* centroid_distances, uint32_t* nearest_clusters,
                             uint64_t num_cells, uint32_t num_dimensions,
                             uint32_t num_clusters, uint32_t num_neighbors,
                             uint32_t num_clusters_searched, void* stream) {
  BGPU_REQUIRE(X && sorted_order && centroids && num_cells_per_cluster && neighbors &&
                   distances && cell_norms && centroid_distances && nearest_clusters,
               BGPU_ERR_INVALID, "knn_self: NULL argument");
  BGPU_REQUIRE(num_cells >= 2 && num_dimensions >= 1 && num_clusters >= 1,
               BGPU_ERR_INVALID, "knn_self: needs >= 2 cells, >= 1 dimension and cluster");
  BGPU_REQUIRE(num_neighbors >= 1 && num_neighbors < num_cells, BGPU_ERR_INVALID,
               "knn_self: num_neighbors must be >= 1 and less than the number of cells");
  BGPU_REQUIRE(num_clusters_searched >= 1 && num_clusters_searched <= num_clusters,
               BGPU_ERR_INVALID,
               "knn_self: num_clusters_searched must be >= 1 and <= the number of clusters");
  BGPU_REQUIRE(num_dimensions <= kMaxDims, BGPU_ERR_UNSUPPORTED,
               "knn_self: at most 128 dimensions");
  BGPU_REQUIRE(num_clusters_searched <= kMaxSearched, BGPU_ERR_UNSUPPORTED,
               "knn_self: num_clusters_searched must be <= 256");
  BGPU_REQUIRE(num_neighbors <= kMaxNeighbors, BGPU_ERR_UNSUPPORTED,
               "knn_self: num_neighbors must be <= 128");
  BGPU_REQUIRE(num_clusters <= kMaxClusters, BGPU_ERR_UNSUPPORTED,
               "knn_self: at most 32768 clusters");
  cudaStream_t s = (cudaStream_t)stream;
  const uint64_t n = num_cells;
  const uint32_t d = num_dimensions, nc = num_clusters, cs = num_clusters_searched,
                 k = num_neighbors;
  BGPU_REQUIRE(search_table_bytes(d, nc, cs, k) <= (size_t)device_smem_optin() - 256,
               BGPU_ERR_UNSUPPORTED,
               "knn_self: too many clusters for the search's shared-memory cluster table");
  // one allocation: operands of the cells and the centroids, centroid norms,
  // cluster offsets, the queries to replay, the error word
  const size_t xb = round_up(knn_operand_bytes(n, d), 256);
  const size_t cb = round_up(knn_operand_bytes(nc, d), 256);
  const size_t nb = round_up((size_t)nc * 4, 256), ob = round_up(((size_t)nc + 1) * 8, 256);
  unsigned char* mem = nullptr;
  const size_t rb = round_up(knn_replay_bytes(n), 256);
  BGPU_CUDA(scratch_alloc((void**)&mem, xb + cb + nb + ob + rb + 256, s));
  float* cn = (float*)(mem + xb + cb);
  uint64_t* coff = (uint64_t*)(mem + xb + cb + nb);
  uint32_t* replay = (uint32_t*)(mem + xb + cb + nb + ob);
  int* err = (int*)(mem + xb + cb + nb + ob + rb);
  auto run = [&]() -> int {
    BGPU_CUDA(cudaMemsetAsync(err, 0, sizeof(int), s));
    k_knn_centroid_norms<<<(unsigned)ceil_div(nc, 256), 256, 0, s>>>(centroids, nc, d, cn);
    BGPU_CHECK_LAUNCH();
    k_knn_offsets<<<1, kOffThreads, 0, s>>>(num_cells_per_cluster, nc, n, coff, err);
    BGPU_CHECK_LAUNCH();
    KnnOperand x, c;
    BGPU_TRY(knn_prepare(&x, X, cell_norms, n, d, mem, s));
    BGPU_TRY(knn_prepare(&c, centroids, cn, nc, d, mem + xb, s));
    BGPU_TRY(knn_tc_nearest(x, c, d, cs, coff, replay, nearest_clusters, centroid_distances,
                            err, s));
    BGPU_TRY(knn_tc_search(x, d, coff, nc, nearest_clusters, cs, k, sorted_order, replay,
                           neighbors, distances, err, s));
    return knn_status(err, s);
  };
  const int rc = run();
  cudaFreeAsync(mem, s);
  return rc;
}

// ---------------------------------------------------------------------------
// k-means: the reference's kmeans (brisc/kmeans.pyx:889-1433), random
// initialisation (its default, kmeans_random_init, kmeans.pyx:13-38), for
// neighbors() to cluster the PCs on the device before knn_self.
//  - init: num_clusters distinct random cells, drawn with PCG32 + Lemire's
//    bounded integers from srand(seed) exactly as the reference draws them
//    (host), gathered on the device;
//  - |x|^2 per cell (kmeans.pyx:954-965), a dimension-ordered float sum;
//  - E step: the nearest centroid by partial distance |c|^2 - 2 x.c, first
//    minimum in centroid order wins (kmeans.pyx:1016-1041) -- a list of one
//    centroid per cell (knn_tc.cu);
//  - M step: the sums of each chunk of chunk_size cells per cluster, each a
//    sequence over the chunk's cells in order, then the chunks added in
//    chunk order (kmeans.pyx:1043-1064): the reference's own order, so with
//    the same assignments the centroids are bit-identical; empty clusters
//    take the cells farthest from their centroids (kmeans.pyx:747-820, on
//    the host: it is rare and sequential); the sums are scaled by
//    (float)(1.0 / count);
//  - stop after num_kmeans_iterations, or when the float total of |x|^2 +
//    min distance falls by less than tolerance (kmeans.pyx:1082-1098, summed
//    in cell order on the host);
//  - a final E step for the labels, min distances and counts.
// The centroid buffers swap every iteration as the reference's do: the
// final centroids are in centroids_new when the returned count is odd.
namespace bgpu {
namespace {

__global__ void k_km_cell_norms(const float* __restrict__ X, uint64_t n, uint32_t d,
                                float* __restrict__ out) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float* x = X + i * d;
  float s = x[0] * x[0];
  for (uint32_t j = 1; j < d; ++j) s = fmaf(x[j], x[j], s);
  out[i] = s;
}

__global__ void k_km_gather(const float* __restrict__ X, const uint32_t* __restrict__ idx,
                            uint32_t nc, uint32_t d, float* __restrict__ C) {
  const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (t >= (uint64_t)nc * d) return;
  const uint32_t c = (uint32_t)(t / d), j = (uint32_t)(t % d);
  C[t] = X[(uint64_t)idx[c] * d + j];
}

// sums[chunk][label][dim] over the chunk's cells in order. A CTA per chunk
// sorts the cells by label, stably (per-warp counts of consecutive cells in
// shared memory, their starts label by label, ranks among equal labels of 32
// cells by warp matches), then a thread per (label, dimension) adds its
// label's cells in order. The additions of one label are as sequential as
// before, but those of different labels no longer wait for one another:
// 300k cells, 2,191 clusters, 50 dimensions: 1.83 ms with a thread per
// dimension walking the chunk (a chain of 4,096 loads and stores), 0.09 ms.
constexpr int kSumThreads = 1024;
constexpr uint32_t kSumMaxChunk = 16384;
constexpr size_t kSumSmem = 200 * 1024;

// Warps that count separately: as many (up to 32) as fit; 0: none does.
uint32_t sum_warps(uint32_t chunk, uint32_t nc) {
  if (chunk > kSumMaxChunk) return 0;
  for (uint32_t w = kSumThreads / 32; w >= 1; w /= 2)
    if ((size_t)w * nc * 4 + ((size_t)nc + 1) * 4 + (size_t)chunk * 4 <= kSumSmem) return w;
  return 0;
}

__global__ void __launch_bounds__(kSumThreads)
k_km_chunk_sums(const float* __restrict__ X, uint64_t n, uint32_t d,
                const uint32_t* __restrict__ labels, uint32_t chunk, uint32_t nc,
                uint32_t warps, float* __restrict__ sums) {
  extern __shared__ uint32_t km[];
  uint32_t* cnt = km;                  // [warps][nc]: counts, then next places
  uint32_t* start = cnt + warps * nc;  // [nc + 1]
  uint32_t* order = start + nc + 1;    // [chunk]: cells of the chunk by label
  __shared__ uint32_t wsum[kSumThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint64_t c0 = (uint64_t)blockIdx.x * chunk;
  const uint32_t len = (uint32_t)min_u64(chunk, n - c0);
  const uint32_t per = (len + warps - 1) / warps;
  const uint32_t a = min(len, (uint32_t)wid * per), b = min(len, a + per);
  const bool counts = (uint32_t)wid < warps;
  for (uint32_t t = threadIdx.x; t < warps * nc; t += kSumThreads) cnt[t] = 0u;
  __syncthreads();
  uint32_t* my = cnt + (size_t)(counts ? wid : 0) * nc;
  if (counts)
    for (uint32_t i = a + lane; i < b; i += 32)
      if (labels[c0 + i] < nc) atomicAdd(&my[labels[c0 + i]], 1u);
  __syncthreads();
  // start of every label: a run of labels per thread, a scan over the threads
  const uint32_t run = (nc + kSumThreads - 1) / kSumThreads;
  const uint32_t l0 = min(nc, threadIdx.x * run), l1 = min(nc, l0 + run);
  uint32_t mine = 0;
  for (uint32_t l = l0; l < l1; ++l)
    for (uint32_t w = 0; w < warps; ++w) mine += cnt[w * nc + l];
  uint32_t incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) wsum[wid] = incl;
  __syncthreads();
  uint32_t at = incl - mine;
  for (int w = 0; w < wid; ++w) at += wsum[w];
  for (uint32_t l = l0; l < l1; ++l) {
    start[l] = at;
    for (uint32_t w = 0; w < warps; ++w) {
      const uint32_t t = cnt[w * nc + l];
      cnt[w * nc + l] = at;
      at += t;
    }
  }
  if (l1 == nc && l0 < nc) start[nc] = at;  // the thread of the last label
  __syncthreads();
  if (counts)
    for (uint32_t i0 = a; i0 < b; i0 += 32) {
      const uint32_t i = i0 + lane;
      const uint32_t l = i < b ? labels[c0 + i] : 0xFFFFFFFFu;
      const uint32_t lab = l < nc ? l : 0xFFFFFFFFu;
      const uint32_t peers = __match_any_sync(0xffffffffu, lab);
      const int leader = __ffs(peers) - 1;
      uint32_t slot = 0;
      if (lane == leader && lab < nc) {
        slot = my[lab];
        my[lab] = slot + __popc(peers);
      }
      slot = __shfl_sync(0xffffffffu, slot, leader) + __popc(peers & ((1u << lane) - 1u));
      if (lab < nc) order[slot] = i;
      __syncwarp();
    }
  __syncthreads();
  float* out = sums + (uint64_t)blockIdx.x * nc * d;
  const float* x = X + c0 * d;
  constexpr int U = 4;  // independent (label, dimension) sums per thread
  for (uint32_t t0 = threadIdx.x; t0 < nc * d; t0 += kSumThreads * U) {
    uint32_t s[U], e[U], j[U];
    float acc[U];
    uint32_t longest = 0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t t = t0 + u * kSumThreads, l = t / d;
      j[u] = t % d;
      s[u] = t < nc * d ? start[l] : 0u;
      e[u] = t < nc * d ? start[l + 1] : 0u;
      acc[u] = 0.f;
      longest = max(longest, e[u] - s[u]);
    }
    for (uint32_t k = 0; k < longest; ++k) {
      float v[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        v[u] = s[u] + k < e[u] ? x[(uint64_t)order[s[u] + k] * d + j[u]] : 0.f;
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (s[u] + k < e[u]) acc[u] = acc[u] + v[u];
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (t0 + u * kSumThreads < nc * d) out[t0 + u * kSumThreads] = acc[u];
  }
}

// The same for chunks or cluster counts past that: a thread per dimension
// walks the chunk (sums zeroed beforehand).
__global__ void k_km_chunk_walk(const float* __restrict__ X, uint64_t n, uint32_t d,
                                const uint32_t* __restrict__ labels, uint32_t chunk,
                                uint32_t nc, float* __restrict__ sums) {
  const uint64_t c0 = (uint64_t)blockIdx.x * chunk;
  const uint64_t c1 = c0 + chunk < n ? c0 + chunk : n;
  float* base = sums + (uint64_t)blockIdx.x * nc * d;
  for (uint32_t j = threadIdx.x; j < d; j += blockDim.x)
    for (uint64_t i = c0; i < c1; ++i) {
      if (labels[i] >= nc) continue;
      float* p = base + (uint64_t)labels[i] * d + j;
      *p = *p + X[i * d + j];
    }
}

// centroids_new[c][j] = 0 + the chunk sums in chunk order.
__global__ void k_km_reduce(const float* __restrict__ sums, uint32_t nchunks, uint32_t nc,
                            uint32_t d, float* __restrict__ Cn) {
  const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t per = (uint64_t)nc * d;
  if (t >= per) return;
  float s = 0.f;
  for (uint32_t ch = 0; ch < nchunks; ++ch) s += sums[ch * per + t];
  Cn[t] = s;
}

// A cell whose distances are all NaN has no label (0xFFFFFFFF) and counts
// nowhere.
__global__ void k_km_counts(const uint32_t* __restrict__ labels, uint64_t n, uint32_t nc,
                            uint32_t* __restrict__ counts) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i < n && labels[i] < nc) atomicAdd(&counts[labels[i]], 1u);  // integer: order-free
}

__global__ void k_km_normalize(float* __restrict__ Cn, const uint32_t* __restrict__ counts,
                               uint32_t nc, uint32_t d) {
  const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (t >= (uint64_t)nc * d) return;
  const uint32_t cnt = counts[t / d];
  if (cnt > 0) Cn[t] *= (float)(1.0 / (double)cnt);  // kmeans.pyx:1070-1074
}

// Squared distance of each cell to its assigned centroid, a dimension-ordered
// float sum (relocate_empty_clusters, kmeans.pyx:785-791); -1 for a cell without
// a label, whose distances are all NaN.
__global__ void k_km_assigned(const float* __restrict__ X, const uint32_t* __restrict__ lab,
                              const float* __restrict__ C, uint64_t n, uint32_t d,
                              uint32_t nc, float* __restrict__ out) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float* x = X + i * d;
  if (lab[i] >= nc) {
    out[i] = -1.f;
    return;
  }
  const float* c = C + (uint64_t)lab[i] * d;
  float diff = x[0] - c[0];
  float s = diff * diff;
  for (uint32_t j = 1; j < d; ++j) {
    diff = x[j] - c[j];
    s = fmaf(diff, diff, s);
  }
  out[i] = s;
}

// E step: labels, min distances (= partial distances) and, when counts is
// given, the cluster sizes. cmem: the centroids' operand.
int km_estep(const KnnOperand& x, uint32_t d, const float* C, float* cn, uint32_t nc, void* cmem,
             uint32_t* replay, uint32_t* labels, float* mind, uint32_t* counts, int* err,
             cudaStream_t s) {
  const uint64_t n = x.n;
  k_knn_centroid_norms<<<(unsigned)ceil_div(nc, 256), 256, 0, s>>>(C, nc, d, cn);
  BGPU_CHECK_LAUNCH();
  KnnOperand c;
  BGPU_TRY(knn_prepare(&c, C, cn, nc, d, cmem, s));
  BGPU_TRY(knn_tc_nearest(x, c, d, 1, nullptr, replay, labels, mind, err, s));
  if (counts) {
    BGPU_CUDA(cudaMemsetAsync(counts, 0, (size_t)nc * 4, s));
    k_km_counts<<<(unsigned)ceil_div(n, 256), 256, 0, s>>>(labels, n, nc, counts);
    BGPU_CHECK_LAUNCH();
  }
  return BGPU_OK;
}

// Float sum of the values in order, starting from init (host; the
// reference's sequential loops).
float seq_sum(float init, const std::vector<float>& v) {
  float t = init;
  for (float x : v) t += x;
  return t;
}

}  // namespace
}  // namespace bgpu

extern "C" int bgpu_kmeans(const float* X, uint32_t* cluster_labels, float* centroids,
                           float* centroids_new, uint32_t* num_cells_per_cluster,
                           float* min_distances, float* cell_norms, int kmeans_barbar,
                           uint32_t num_kmeans_iterations, float tolerance,
                           uint32_t chunk_size, uint64_t seed, uint64_t num_cells,
                           uint32_t num_dimensions, uint32_t num_clusters,
                           uint32_t* iterations, void* stream) {
  BGPU_REQUIRE(X && cluster_labels && centroids && centroids_new && num_cells_per_cluster &&
                   min_distances && iterations,
               BGPU_ERR_INVALID, "kmeans: NULL argument");
  BGPU_REQUIRE(!kmeans_barbar, BGPU_ERR_UNSUPPORTED,
               "kmeans: only the random initialisation (kmeans_barbar=False, the "
               "reference's default) runs on the GPU");
  const uint64_t n = num_cells;
  const uint32_t d = num_dimensions, nc = num_clusters;
  BGPU_REQUIRE(n >= 1 && d >= 1 && nc >= 1 && nc <= n, BGPU_ERR_INVALID,
               "kmeans: needs 1 <= num_clusters <= num_cells and >= 1 dimension");
  BGPU_REQUIRE(d <= kMaxDims, BGPU_ERR_UNSUPPORTED, "kmeans: at most 128 dimensions");
  BGPU_REQUIRE(nc <= kMaxClusters, BGPU_ERR_UNSUPPORTED, "kmeans: at most 32768 clusters");
  BGPU_REQUIRE(chunk_size >= 1 && num_kmeans_iterations >= 1, BGPU_ERR_INVALID,
               "kmeans: chunk_size and num_kmeans_iterations must be >= 1");
  BGPU_REQUIRE(n <= 0xFFFFFFFFull, BGPU_ERR_UNSUPPORTED, "kmeans: at most 2^32 - 1 cells");
  cudaStream_t s = (cudaStream_t)stream;
  const uint32_t nchunks = (uint32_t)ceil_div(n, chunk_size);
  const uint64_t per = (uint64_t)nc * d;
  const uint64_t sums_bytes = (uint64_t)nchunks * per * 4;
  BGPU_REQUIRE(sums_bytes <= (64ull << 30), BGPU_ERR_UNSUPPORTED,
               "kmeans: the per-chunk sums would exceed 64 GB; raise chunk_size");

  // random initialisation (kmeans.pyx:13-38)
  std::vector<uint32_t> init(nc);
  {
    std::vector<uint64_t> bits((n + 63) / 64, 0);
    uint64_t state = pcg_srand(seed);
    for (uint32_t i = 0; i < nc; ++i) {
      while (true) {
        const uint32_t j = pcg_randint((uint32_t)n, &state);
        if (!(bits[j >> 6] & (1ull << (j & 63)))) {
          bits[j >> 6] |= 1ull << (j & 63);
          init[i] = j;
          break;
        }
      }
    }
  }
  uint32_t* didx = nullptr;
  const size_t xb = round_up(knn_operand_bytes(n, d), 256);
  const size_t cb = round_up(knn_operand_bytes(nc, d), 256);
  unsigned char* mem = nullptr;  // operands of the cells and the centroids, replays, error word
  float *cn = nullptr, *sums = nullptr, *norms = cell_norms, *own_norms = nullptr;
  BGPU_CUDA(scratch_alloc((void**)&didx, (size_t)nc * 4, s));
  BGPU_CUDA(scratch_alloc((void**)&cn, (size_t)nc * 4, s));
  BGPU_CUDA(scratch_alloc((void**)&sums, sums_bytes, s));
  const size_t rb = round_up(knn_replay_bytes(n), 256);
  BGPU_CUDA(scratch_alloc((void**)&mem, xb + cb + rb + 256, s));
  uint32_t* replay = (uint32_t*)(mem + xb + cb);
  int* err = (int*)(mem + xb + cb + rb);
  if (!norms) {
    BGPU_CUDA(scratch_alloc((void**)&own_norms, n * 4, s));
    norms = own_norms;
  }
  auto cleanup = [&]() {
    cudaFreeAsync(didx, s);
    cudaFreeAsync(cn, s);
    cudaFreeAsync(sums, s);
    cudaFreeAsync(mem, s);
    if (own_norms) cudaFreeAsync(own_norms, s);
  };
  auto run = [&]() -> int {
    BGPU_CUDA(cudaMemcpyAsync(didx, init.data(), (size_t)nc * 4, cudaMemcpyHostToDevice, s));
    float* Cc = centroids;
    float* Cn = centroids_new;
    k_km_gather<<<(unsigned)ceil_div(per, 256), 256, 0, s>>>(X, didx, nc, d, Cc);
    BGPU_CHECK_LAUNCH();
    k_km_cell_norms<<<(unsigned)ceil_div(n, 256), 256, 0, s>>>(X, n, d, norms);
    BGPU_CHECK_LAUNCH();
    std::vector<float> hnorm(n), hmin;
    BGPU_CUDA(cudaMemcpyAsync(hnorm.data(), norms, n * 4, cudaMemcpyDeviceToHost, s));
    BGPU_CUDA(cudaStreamSynchronize(s));
    const float sum_sq = seq_sum(0.f, hnorm);  // kmeans.pyx:954-965
    BGPU_CUDA(cudaMemsetAsync(err, 0, sizeof(int), s));
    KnnOperand x;
    BGPU_TRY(knn_prepare(&x, X, nullptr, n, d, mem, s));
    float old_total = 0.f;
    uint32_t it = 0;
    std::vector<uint32_t> hcount(nc);
    while (true) {
      BGPU_TRY(km_estep(x, d, Cc, cn, nc, mem + xb, replay, cluster_labels, min_distances,
                        num_cells_per_cluster, err, s));
      if (const uint32_t warps = sum_warps(chunk_size, nc)) {
        BGPU_CUDA(allow_max_smem(k_km_chunk_sums));
        k_km_chunk_sums<<<nchunks, kSumThreads,
                          ((size_t)warps * nc + nc + 1 + chunk_size) * 4, s>>>(
            X, n, d, cluster_labels, chunk_size, nc, warps, sums);
      } else {
        BGPU_CUDA(cudaMemsetAsync(sums, 0, sums_bytes, s));
        k_km_chunk_walk<<<nchunks, std::min<uint32_t>(128, (d + 31) & ~31u), 0, s>>>(
            X, n, d, cluster_labels, chunk_size, nc, sums);
      }
      BGPU_CHECK_LAUNCH();
      k_km_reduce<<<(unsigned)ceil_div(per, 256), 256, 0, s>>>(sums, nchunks, nc, d, Cn);
      BGPU_CHECK_LAUNCH();
      BGPU_CUDA(cudaMemcpyAsync(hcount.data(), num_cells_per_cluster, (size_t)nc * 4,
                                cudaMemcpyDeviceToHost, s));
      BGPU_CUDA(cudaStreamSynchronize(s));
      std::vector<uint32_t> empty;
      for (uint32_t c = 0; c < nc; ++c)
        if (hcount[c] == 0) empty.push_back(c);
      if (!empty.empty()) {  // relocate_empty_clusters (kmeans.pyx:747-820)
        float* dist = nullptr;
        BGPU_CUDA(scratch_alloc((void**)&dist, n * 4, s));
        k_km_assigned<<<(unsigned)ceil_div(n, 256), 256, 0, s>>>(X, cluster_labels, Cc,
                                                                  n, d, nc, dist);
        std::vector<float> hd(n), hx, hcn(per);
        std::vector<uint32_t> hl(n);
        cudaMemcpyAsync(hd.data(), dist, n * 4, cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(hl.data(), cluster_labels, n * 4, cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(hcn.data(), Cn, per * 4, cudaMemcpyDeviceToHost, s);
        cudaFreeAsync(dist, s);
        BGPU_CUDA(cudaStreamSynchronize(s));
        // the num_empty largest distances, an earlier cell winning ties, in
        // descending order; cells without a label or a distance come last
        // and are never taken
        const size_t ne = empty.size();
        for (float& x : hd)
          if (!(x >= 0.f)) x = -1.f;
        std::vector<uint64_t> order(n);
        for (uint64_t i = 0; i < n; ++i) order[i] = i;
        std::stable_sort(order.begin(), order.end(),
                         [&](uint64_t a, uint64_t b) { return hd[a] > hd[b]; });
        BGPU_REQUIRE(hd[order[0]] > 0.f, BGPU_ERR_INVALID,
                     "kmeans: num_clusters is greater than the number of cells with "
                     "distinct principal component loadings; decrease num_clusters");
        BGPU_REQUIRE(hd[order[ne - 1]] >= 0.f, BGPU_ERR_INVALID,
                     "kmeans: more empty clusters than cells whose distances are numbers; "
                     "decrease num_clusters");
        std::vector<float> row(d);
        for (size_t e = 0; e < ne; ++e) {
          const uint64_t j = order[e];
          const uint32_t oldc = hl[j], newc = empty[e];
          BGPU_CUDA(cudaMemcpy(row.data(), X + j * d, (size_t)d * 4, cudaMemcpyDeviceToHost));
          for (uint32_t k = 0; k < d; ++k) {
            hcn[(uint64_t)oldc * d + k] -= row[k];
            hcn[(uint64_t)newc * d + k] = row[k];
          }
          hcount[oldc] -= 1;
          hcount[newc] += 1;
        }
        BGPU_CUDA(cudaMemcpyAsync(Cn, hcn.data(), per * 4, cudaMemcpyHostToDevice, s));
        BGPU_CUDA(cudaMemcpyAsync(num_cells_per_cluster, hcount.data(), (size_t)nc * 4,
                                  cudaMemcpyHostToDevice, s));
      }
      k_km_normalize<<<(unsigned)ceil_div(per, 256), 256, 0, s>>>(Cn, num_cells_per_cluster,
                                                                  nc, d);
      BGPU_CHECK_LAUNCH();
      std::swap(Cc, Cn);
      ++it;
      if (it == num_kmeans_iterations) break;
      hmin.resize(n);
      BGPU_CUDA(cudaMemcpyAsync(hmin.data(), min_distances, n * 4, cudaMemcpyDeviceToHost, s));
      BGPU_CUDA(cudaStreamSynchronize(s));
      const float total = seq_sum(sum_sq, hmin);  // kmeans.pyx:1088-1098
      if (it > 1 && old_total - total < tolerance * old_total) break;
      old_total = total;
    }
    // the final E step (kmeans.pyx:1100-1153)
    BGPU_TRY(km_estep(x, d, Cc, cn, nc, mem + xb, replay, cluster_labels, min_distances,
                      num_cells_per_cluster, err, s));
    *iterations = it;
    return knn_status(err, s);
  };
  const int rc = run();
  cleanup();
  return rc;
}
