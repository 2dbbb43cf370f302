// Nearest rows by exact FP32 distances, with the tensor cores as a filter: the
// inner loops of the k-means E step, of knn_self's nearest clusters and of
// knn_self's neighbour search (knn.cu).
//
// What is computed: every query keeps its best list as candidates are offered
// to it in a fixed order (ascending row; for the search, the rows of its
// clusters in ascending cluster label), each kept when strictly closer than
// the list's current worst, which it replaces (ties among the worst: the
// lowest entry). The distance is an FP32 fused-multiply-add chain over the
// dimensions in order. All of that is evaluated here as written, but only for
// the candidates that can be in the final list:
//  - the tensor cores form s = x.c - |c|^2 / 2 for a tile of queries times a
//    tile of candidates, from BF16 high and low parts (high.high + high.low +
//    low.high, |c|^2 / 2 as three BF16 columns of its own against ones);
//  - a candidate can be strictly closer than the worst w only if
//    s > (|x|^2 - w) / 2 - margin, where the margin bounds what the split,
//    the accumulation and the FP32 chain can differ by; w is the worst of an
//    earlier moment, which is never smaller, so nothing is lost;
//  - the few that pass queue per query, and 32 at a time are evaluated exactly,
//    one per lane, and offered.
// Order. The reference's order approaches a cell's own cluster from one side
// (clusters are sorted by their first dimension), and nearly every cluster on
// the way improves the list: ~20 % of the candidates pass. Here the tiles start
// at the queries' own cluster and wrap around, so the worst is tight after a
// tile or two. The k smallest distances are the same in any order; which rows
// hold them is too, unless the k-th and the (k+1)-th distance are equal.
// So each query also keeps the smallest value that its list turned away or
// gave up, and where that equals the list's worst, the query is listed and
// computed again, every candidate in the reference's order: by k_knn_replay, or
// by k_knn_all where many of 32 neighbouring queries are. So are queries on which
// the filter decides nothing.
//
// Error of s against the exact x.c - |c|^2/2, with X = the query's length and
// G = the largest length or sqrt |norm| of the tile: the dropped low.low and
// residual products 3 2^-18 X G; the tensor core's accumulation, at most 27
// steps of 17 terms that each lose under 2^-23 of the largest magnitude, under
// 2^-14 (X G + G^2 / 2); the FP32 chain over at most 128 dimensions 2^-17 X G
// and its last roundings 2^-22 (X + G)^2. kMargin = 2^-13 of G (X + G) covers
// their sum, and 1e-35 what underflows. Values that are not finite fail every
// comparison with <= and so pass to the exact evaluation.
//
// Why: the exhaustive FP32 loop is bound by the SIMT pipes (two candidates x
// four queries per lane, six shared loads per eight multiply-adds: 7.7
// TFLOP/s). Here the products cost tensor time, the filter two instructions
// per pair of a TMEM load, and the exact work is proportional to what passes.
// 300k x 50 dims, 2,191 clusters, 64 searched, 20 neighbours: search 36.7 ->
// 6.9 ms, nearest clusters 20.9 -> 2.5 ms, the E step against 2,191 centroids
// 6.07 -> 0.57 ms. Lists of up to 64 entries take k_knn_two; longer ones
// k_knn_tc, which keeps its lists while it goes (the same lists 15.1 and 10.6 ms;
// a tile waits for the exact evaluations of its slowest warp).
//
// Shape of k_knn_tc: 512 threads, one CTA per SM, kQT queries (rows of the MMA), tiles of
// NT candidates. Warp w reads the TMEM lanes (queries) of quarter w % 4 and
// the columns of quarter w / 4: a thread tests NT / 4 candidates of one query
// into one mask word. The queries' queues and lists belong to warps (query q
// to warp q % 16), so their updates need no synchronisation. The MMAs of tile
// t + 1 run while tile t is filtered and evaluated; its operand arrives by
// bulk copies (one per 8-row group, the operand's storage is the shared
// layout) two tiles ahead. One block barrier per tile: masks alternate between
// two buffers, tile descriptions over four.
// Queries per CTA: 128, fewer when that leaves SMs without a CTA or the lists
// do not fit; a shorter tile's MMA rows past the queries read the bytes that
// follow in shared memory and their results are never looked at.
#include <algorithm>
#include <cfloat>

#include <cuda_bf16.h>

#include "knn_tc.cuh"
#include "tcgen05.cuh"

namespace bgpu {
namespace {

constexpr int kTcKnnThreads = 512;
constexpr int kTcKnnWarps = kTcKnnThreads / 32;
constexpr uint32_t kQueue = 64;       // queued candidates per query (31 + 32 at most)
constexpr uint32_t kUnionCap = 512;   // searched clusters taken at once
constexpr uint32_t kNormCols = 3;
constexpr float kMargin = 1.f / 8192.f;
constexpr uint32_t kNoRun = 0xFFFFFFFFu;
// Queries of a group of 32 from which on k_knn_all takes them: 300k x 50 dims, a
// group costs 2.9 us of the GPU's time, a query by itself 0.33.
constexpr int kGroupReplays = 8;
// Exact evaluations per list entry past which k_knn_tc gives its queries up.
// Ordinary data stay below 16. 300k x 50 dims, against the exhaustive search
// alone: search of 100 neighbours, rows 10 spreads from the origin, 109 ms with
// 16, 89 with 24 (112); 100 nearest clusters, 100 spreads, 95 with 16, 109 with 24
// (97).
constexpr uint32_t kSearchEvals = 24, kNearestEvals = 16;

struct KnnArgs {
  KnnOperand q, c;
  uint32_t d, kp, qt, size;
  uint32_t stages;  // two passes: operand tiles in flight
  // the cells' clusters: the search, and nearest for cells sorted by cluster
  // (nullptr: lists of one entry only, the k-means E step)
  const uint64_t* coff;
  uint32_t nc, cs;
  const uint32_t* nearest;
  const uint32_t* id_map;
  uint32_t* out_id;
  float* out_d;
  uint32_t* counts;  // [0]: queries in replay, [1]: groups
  uint32_t* replay;  // queries for k_knn_replay
  uint32_t* groups;  // (group of 32 queries, mask of those) for k_knn_all, or nullptr
  uint32_t* wide;    // with groups: per group, whether many of its margins were too wide
  int* err;
};

// Set by an earlier kernel only, so every thread of a launch reads the same. Asked
// before the results are written: a return ahead of the tiles cost 2 % of them.
__device__ __forceinline__ bool refused(const KnnArgs& a) {
  return (__ldcg(a.err) & kKnnErrSizes) != 0;
}

struct KnnSmem {  // byte offsets
  uint32_t a, b, list, queue, masks, thr, qlen, qnorm, qcnt, qfill, qnext, runs, qmask, bitmap, total;
};

__host__ __device__ inline uint32_t group_bytes(uint32_t kp) { return kp * 32u; }

__host__ __device__ inline KnnSmem knn_smem(uint32_t kp, uint32_t qt, uint32_t nt, uint32_t R,
                                            bool search, uint32_t nc) {
  KnnSmem L;
  uint32_t o = 1024;
  auto take = [&](uint32_t bytes) {
    const uint32_t at = o;
    o += (bytes + 127u) & ~127u;
    return at;
  };
  L.a = take(qt / 8 * group_bytes(kp));
  L.b = take(2 * nt / 8 * group_bytes(kp));
  // the MMA reads 128 rows of A: the bytes past the queries' are B's
  if (o < L.a + 16 * group_bytes(kp)) o = L.a + 16 * group_bytes(kp);
  L.list = take(qt * R * 32 * 8);
  L.queue = take(qt * kQueue * 4);
  L.masks = take(2 * 4 * 128 * 4);
  L.thr = take(qt * 4);
  L.qlen = take(qt * 4);
  L.qnorm = take(qt * 4);
  L.qcnt = take(qt * 4);
  L.qfill = take(qt * 4);
  L.qnext = take(qt * 4);
  L.runs = take(search ? kUnionCap * 12 + 4 : 16);
  L.qmask = take(search ? kUnionCap * 16 : 16);
  L.bitmap = take(search ? (nc + 31) / 32 * 8 : 16);  // words and their ranks
  L.total = o;
  return L;
}

__device__ __forceinline__ float warp_max_f32(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

__device__ __forceinline__ float warp_min_f32(float v) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
// The larger of three, NaN when one is.
__device__ __forceinline__ float max3_nan(float a, float b, float c) {
  float r;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// A best list of up to 32 * R entries spread over the lanes of a warp: entry
// e lives in lane e % 32, slot e / 32. Entries past the list size hold -inf
// and are never the worst.
template <int R>
struct WarpList {
  float d[R];
  uint32_t id[R];
  float worst;  // warp-uniform
  int worst_lane, worst_slot;

  __device__ __forceinline__ void load(const float* sd, const uint32_t* si, int lane) {
#pragma unroll
    for (int s = 0; s < R; ++s) {
      d[s] = sd[s * 32 + lane];
      id[s] = si[s * 32 + lane];
    }
    find_worst();
  }
  __device__ __forceinline__ void store(float* sd, uint32_t* si, int lane) const {
#pragma unroll
    for (int s = 0; s < R; ++s) {
      sd[s * 32 + lane] = d[s];
      si[s * 32 + lane] = id[s];
    }
  }
  // the largest entry; ties go to the lowest entry index
  __device__ __forceinline__ void find_worst() {
    float m = d[0];
#pragma unroll
    for (int s = 1; s < R; ++s) m = fmaxf(m, d[s]);
    worst = warp_max_f32(m);
    worst_slot = R - 1;
    unsigned at = __ballot_sync(0xffffffffu, d[R - 1] == worst);
#pragma unroll
    for (int s = R - 2; s >= 0; --s) {
      const unsigned b = __ballot_sync(0xffffffffu, d[s] == worst);
      if (b) {
        at = b;
        worst_slot = s;
      }
    }
    worst_lane = __ffs(at) - 1;
  }
  // Offers the candidates of the lanes in `mask`, all strictly closer than the
  // worst, in ascending lane order.
  __device__ __forceinline__ void keep(float cand, uint32_t cid, unsigned mask, int lane) {
    while (mask) {  // its lowest lane is strictly closer than the worst
      replace(cand, cid, __ffs(mask) - 1, lane);
      mask &= mask - 1u;
      mask &= __ballot_sync(0xffffffffu, cand < worst);
    }
  }
  // The worst entry becomes lane src's candidate.
  __device__ __forceinline__ void replace(float cand, uint32_t cid, int src, int lane) {
    const float cd = __shfl_sync(0xffffffffu, cand, src);
    const uint32_t ci = __shfl_sync(0xffffffffu, cid, src);
    if (lane == worst_lane) {
#pragma unroll
      for (int s = 0; s < R; ++s)
        if (s == worst_slot) {
          d[s] = cd;
          id[s] = ci;
        }
    }
    find_worst();
  }
  // Offers the candidates of the lanes in `mask` in ascending lane order;
  // returns the smaller of `next` and the values turned away or given up.
  __device__ __forceinline__ float offer(float cand, uint32_t cid, unsigned mask, int lane,
                                         float next) {
    unsigned away = mask;
    mask &= __ballot_sync(0xffffffffu, cand < worst);
    while (mask) {  // its lowest lane is strictly closer than the worst
      const int src = __ffs(mask) - 1;
      away &= ~(1u << src);
      next = fminf(next, worst);
      replace(cand, cid, src, lane);
      mask &= mask - 1u;
      mask &= __ballot_sync(0xffffffffu, cand < worst);
    }
    return fminf(next, warp_min_f32((away >> lane) & 1u ? cand : INFINITY));
  }
};

// Writes a list of `size` entries sorted by (distance, id) ascending.
__device__ __forceinline__ void write_sorted(const float* sd, const uint32_t* si, uint32_t size,
                                             const uint32_t* id_map, float* od, uint32_t* oi,
                                             int lane) {
  for (uint32_t e = lane; e < size; e += 32) {
    const float de = sd[e];
    const uint32_t ie = si[e];
    uint32_t rank = 0;
    for (uint32_t f = 0; f < size; ++f) {
      const float df = sd[f];
      const uint32_t idf = si[f];
      rank += (df < de || (df == de && (idf < ie || (idf == ie && f < e)))) ? 1u : 0u;
    }
    od[rank] = de;
    oi[rank] = id_map && ie != 0xFFFFFFFFu ? id_map[ie] : ie;
  }
}

// x.c as a chain of fused multiply-adds in dimension order (VEC floats per
// load: both rows aligned to it, d a multiple of it).
template <int VEC>
__device__ __forceinline__ float row_dot(const float* __restrict__ x, const float* __restrict__ c,
                                         uint32_t d) {
  float acc = 0.f;
  if constexpr (VEC == 4) {
#pragma unroll 8
    for (uint32_t j = 0; j < d; j += 4) {
      const float4 a = *(const float4*)(x + j), b = *(const float4*)(c + j);
      acc = fmaf(a.x, b.x, acc);
      acc = fmaf(a.y, b.y, acc);
      acc = fmaf(a.z, b.z, acc);
      acc = fmaf(a.w, b.w, acc);
    }
  } else if constexpr (VEC == 2) {
#pragma unroll 13
    for (uint32_t j = 0; j < d; j += 2) {
      const float2 a = *(const float2*)(x + j), b = *(const float2*)(c + j);
      acc = fmaf(a.x, b.x, acc);
      acc = fmaf(a.y, b.y, acc);
    }
  } else {
#pragma unroll 8
    for (uint32_t j = 0; j < d; ++j) acc = fmaf(x[j], c[j], acc);
  }
  return acc;
}

template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, float (&v)[N]);
template <>
__device__ __forceinline__ void tmem_ld<16>(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,"
      "%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
template <>
__device__ __forceinline__ void tmem_ld<32>(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,"
      "%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// The same in two steps, for loads that overlap other work: the values may be
// used behind tmem_loaded() only, which takes them as operands so that
// nothing that reads them moves ahead of it.
template <int N>
__device__ __forceinline__ void tmem_load(uint32_t taddr, float (&v)[N]);
template <int N>
__device__ __forceinline__ void tmem_loaded(float (&v)[N]);
template <>
__device__ __forceinline__ void tmem_load<8>(uint32_t taddr, float (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]),
                 "=f"(v[6]), "=f"(v[7])
               : "r"(taddr)
               : "memory");
}
template <>
__device__ __forceinline__ void tmem_loaded<8>(float (&v)[8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]),
                 "+f"(v[6]), "+f"(v[7])::"memory");
}
template <>
__device__ __forceinline__ void tmem_load<16>(uint32_t taddr, float (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,"
      "%12,%13,%14,%15}, [%16];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]),
        "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]),
        "=f"(v[14]), "=f"(v[15])
      : "r"(taddr)
      : "memory");
}
template <>
__device__ __forceinline__ void tmem_loaded<16>(float (&v)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]),
                 "+f"(v[6]), "+f"(v[7]), "+f"(v[8]), "+f"(v[9]), "+f"(v[10]), "+f"(v[11]),
                 "+f"(v[12]), "+f"(v[13]), "+f"(v[14]), "+f"(v[15])::"memory");
}

// The clusters that a CTA's queries search, in label order, as a bit per cluster
// and, behind those words, the clusters before each word. uses(q): whether the
// CTA's query q counts. Returns their number; wsum: a word per warp and one more.
template <int THREADS, typename F>
__device__ __forceinline__ uint32_t searched_clusters(const KnnArgs& a, uint64_t q0, uint32_t nq,
                                                      uint32_t* bitmap, uint32_t* wsum, F uses) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const uint32_t words = (a.nc + 31) / 32;
  uint32_t* rank = bitmap + words;
  for (uint32_t w = tid; w < words; w += THREADS) bitmap[w] = 0u;
  __syncthreads();
  for (uint32_t t = tid; t < nq * a.cs; t += THREADS) {
    const uint32_t lab = a.nearest[q0 * a.cs + t];
    if (lab < a.nc && uses(t / a.cs)) atomicOr(&bitmap[lab >> 5], 1u << (lab & 31));  // order-free
  }
  __syncthreads();
  const uint32_t per = (words + THREADS - 1) / THREADS;
  const uint32_t w0 = min(words, tid * per), w1 = min(words, w0 + per);
  uint32_t cnt = 0;
  for (uint32_t w = w0; w < w1; ++w) cnt += __popc(bitmap[w]);
  uint32_t incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) wsum[wid] = incl;
  __syncthreads();
  uint32_t pre = incl - cnt;
  for (int w = 0; w < wid; ++w) pre += wsum[w];
  for (uint32_t w = w0; w < w1; ++w) {
    rank[w] = pre;
    pre += __popc(bitmap[w]);
  }
  if (tid == THREADS - 1) wsum[THREADS / 32] = pre;
  __syncthreads();
  return wsum[THREADS / 32];
}

// The rank of a label among the searched clusters (of the next one, if it is
// not one).
__device__ __forceinline__ uint32_t cluster_rank(const uint32_t* bitmap, uint32_t nc,
                                                 uint32_t lab) {
  return bitmap[(nc + 31) / 32 + (lab >> 5)] +
         __popc(bitmap[lab >> 5] & ((1u << (lab & 31)) - 1u));
}

// Searched clusters [ubase, ubase + nruns) of them: their rows [run_b, run_e),
// and which of the CTA's queries search each (W words of bits). To be read
// behind a barrier.
template <int THREADS, int W, typename F>
__device__ __forceinline__ void searched_runs(const KnnArgs& a, uint64_t q0, uint32_t nq,
                                              const uint32_t* bitmap, uint32_t ubase,
                                              uint32_t nruns, uint32_t* run_b, uint32_t* run_e,
                                              uint32_t* qmask, F uses) {
  if (nruns == 0) return;
  const int tid = threadIdx.x;
  const uint32_t words = (a.nc + 31) / 32;
  for (uint32_t t = tid; t < nruns * W; t += THREADS) qmask[t] = 0u;
  __syncthreads();
  for (uint32_t w = tid; w < words; w += THREADS) {
    uint32_t bits = bitmap[w], pos = bitmap[words + w];
    while (bits) {
      const uint32_t lab = w * 32 + __ffs(bits) - 1;
      bits &= bits - 1u;
      if (pos >= ubase && pos - ubase < nruns) {
        run_b[pos - ubase] = (uint32_t)a.coff[lab];
        run_e[pos - ubase] = (uint32_t)a.coff[lab + 1];
      }
      ++pos;
    }
  }
  for (uint32_t t = tid; t < nq * a.cs; t += THREADS) {
    const uint32_t lab = a.nearest[q0 * a.cs + t], q = t / a.cs;
    if (lab >= a.nc || !uses(q)) continue;
    const uint32_t pos = cluster_rank(bitmap, a.nc, lab);
    if (pos >= ubase && pos - ubase < nruns)
      atomicOr(&qmask[(pos - ubase) * W + (q >> 5)], 1u << (q & 31));
  }
}

// One warp: run_s[u] = size(0) + .. + size(u - 1) for u in [0, nruns].
template <typename F>
__device__ __forceinline__ void run_starts(uint32_t* run_s, uint32_t nruns, F size) {
  const int lane = threadIdx.x & 31;
  uint32_t total = 0;
  for (uint32_t u0 = 0; u0 < nruns; u0 += 32) {
    const uint32_t u = u0 + lane, g = u < nruns ? size(u) : 0u;
    uint32_t incl = g;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (u < nruns) run_s[u] = total + incl - g;
    total += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) run_s[nruns] = total;
}

// The queries of a CTA (bits of bad, a word per 32) that are computed again:
// groups of 32 with many go to k_knn_all, the others' queries to k_knn_replay.
// over: queries whose margins are wider than the distances they are to tell
// apart. Where that holds for a group's nearest clusters, it does for its cells:
// their search does not try the filter (knows_wide).
template <bool SEARCH>
__device__ __forceinline__ void list_replays(const KnnArgs& a, uint64_t q0, const uint32_t* bad,
                                             const uint32_t* over, uint32_t words) {
  const uint32_t first = (uint32_t)q0 + 32 * threadIdx.x;
  if (threadIdx.x >= words || first >= a.q.n) return;
  uint32_t m = bad[threadIdx.x];
  if (!SEARCH && a.groups)
    a.wide[first / 32] = __popc(over[threadIdx.x]) >= kGroupReplays ? 1u : 0u;
  if (a.groups && __popc(m) >= kGroupReplays) {
    const uint32_t i = atomicAdd(a.counts + 1, 1u);
    a.groups[2 * i] = first / 32;
    a.groups[2 * i + 1] = m;
  } else if (m) {
    for (uint32_t i = atomicAdd(a.counts, (uint32_t)__popc(m)); m; m &= m - 1u)
      a.replay[i++] = first + __ffs(m) - 1;
  }
}

// Whether every group of the CTA's queries is known to be too wide for the
// filter; they are listed for k_knn_all then.
__device__ __forceinline__ bool knows_wide(const KnnArgs& a) {
  if (!a.groups || refused(a)) return false;
  const uint64_t q0 = blockIdx.x * (uint64_t)a.qt;
  const uint32_t groups = (uint32_t)((min_u64(a.qt, a.q.n - q0) + 31) / 32);
  bool all = true;
  for (uint32_t g = 0; g < groups; ++g) all = all && a.wide[q0 / 32 + g] != 0u;
  if (all && threadIdx.x < groups) {
    const uint64_t first = q0 + 32 * threadIdx.x, left = a.q.n - first;
    const uint32_t i = atomicAdd(a.counts + 1, 1u);
    a.groups[2 * i] = (uint32_t)(first / 32);
    a.groups[2 * i + 1] = left >= 32 ? 0xFFFFFFFFu : (1u << left) - 1u;
  }
  return all;
}

// Rows to a tensor-core operand. A block takes 4 groups (32 rows); group
// storage: [part high, low][8-column group][row 0..7][8 BF16]. Columns d..d+2
// of the high part hold -norm / 2 as three BF16 numbers; rows past n hold a
// value there that no list takes.
__global__ void __launch_bounds__(256)
k_knn_split(const float* __restrict__ X, const float* __restrict__ norms, uint64_t n, uint32_t d,
            uint32_t kp, unsigned char* __restrict__ tiles, float* __restrict__ length,
            float* __restrict__ gmax) {
  extern __shared__ float xs[];  // [32][d + 1]
  __shared__ float hn[32];
  const uint32_t st = d + 1;
  const uint64_t r0 = blockIdx.x * 32ull;
  const uint32_t rows = (uint32_t)min_u64(32, n - r0);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (uint32_t t = threadIdx.x; t < 32 * d; t += 256) {
    const uint32_t r = t / d, j = t % d;
    xs[r * st + j] = r < rows ? X[(r0 + r) * d + j] : 0.f;
  }
  __syncthreads();
  if (wid == 0) {  // a lane per row
    float s = 0.f;
    for (uint32_t j = 0; j < d; ++j) s = fmaf(xs[lane * st + j], xs[lane * st + j], s);
    const bool in = (uint32_t)lane < rows;
    const float nm = in && norms ? norms[r0 + lane] : 0.f;
    const float len = sqrtf(s) * 1.0001f + 1e-30f;
    if (in) length[r0 + lane] = len;
    hn[lane] = in ? -0.5f * nm : -1e38f;
    float g = in ? fmaxf(len, sqrtf(fabsf(nm)) * 1.0001f) : 0.f;
    g = in && nm != nm ? nm : g;  // a NaN norm must reach the exact evaluation
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      const float h = __shfl_xor_sync(0xffffffffu, g, o);
      g = h != h ? h : (g != g ? g : fmaxf(g, h));
    }
    if ((lane & 7) == 0) gmax[blockIdx.x * 4ull + (lane >> 3)] = g;
  }
  __syncthreads();
  const uint32_t kq = kp / 8;
  const uint64_t ngroups = (n + 7) / 8;
  for (uint32_t t = threadIdx.x; t < 4 * kq * 8; t += 256) {
    const uint32_t r = t & 7u, kg = (t >> 3) % kq, g = (t >> 3) / kq;
    if (blockIdx.x * 4ull + g >= ngroups) continue;
    const uint32_t row = g * 8 + r;
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float h[2], l[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const uint32_t j = kg * 8 + 2 * i + u;
        float v = 0.f, low = 0.f;
        if (j < d) {
          v = xs[row * st + j];
          low = v - __bfloat162float(__float2bfloat16_rn(v));
        } else if (j < d + kNormCols) {
          v = hn[row];
          for (uint32_t k = d; k < j; ++k) v -= __bfloat162float(__float2bfloat16_rn(v));
        }
        h[u] = v;
        l[u] = low;
      }
      const __nv_bfloat162 ph = __floats2bfloat162_rn(h[0], h[1]);
      const __nv_bfloat162 pl = __floats2bfloat162_rn(l[0], l[1]);
      hi[i] = *reinterpret_cast<const uint32_t*>(&ph);
      lo[i] = *reinterpret_cast<const uint32_t*>(&pl);
    }
    unsigned char* base = tiles + (blockIdx.x * 4ull + g) * group_bytes(kp) + kg * 128u + r * 16u;
    *reinterpret_cast<uint4*>(base) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(base + kq * 128u) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
}

template <int R, bool SEARCH, int NT, int VEC>
__global__ void __launch_bounds__(kTcKnnThreads, 1) k_knn_tc(const KnnArgs a) {
  constexpr int CW = NT / 4;             // candidates a thread tests per tile
  constexpr uint32_t SLOTS = NT / 8;     // 8-row groups per tile
  extern __shared__ __align__(1024) unsigned char smem[];
  uint64_t* bfull = reinterpret_cast<uint64_t*>(smem);     // [2] operand of a tile landed
  uint64_t* mfull = reinterpret_cast<uint64_t*>(smem) + 2;  // [2] MMAs of a tile done
  uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + 64);
  __shared__ uint32_t meta_row[4][16], meta_run[4][16];  // per slot: first row, run
  __shared__ float meta_g[4];
  __shared__ uint32_t wsum[kTcKnnWarps + 1], bad[4], over[4], evals, given;
  __shared__ volatile int stop;
  const uint32_t d = a.d, kp = a.kp, QT = a.qt;
  const KnnSmem L = knn_smem(kp, QT, NT, R, SEARCH, a.nc);
  float* ld = reinterpret_cast<float*>(smem + L.list);
  uint32_t* li = reinterpret_cast<uint32_t*>(ld + QT * R * 32);
  uint32_t* queue = reinterpret_cast<uint32_t*>(smem + L.queue);
  uint32_t* masks = reinterpret_cast<uint32_t*>(smem + L.masks);  // [2][4][128]
  volatile float* thr = reinterpret_cast<volatile float*>(smem + L.thr);
  float* qlen = reinterpret_cast<float*>(smem + L.qlen);
  float* qnorm = reinterpret_cast<float*>(smem + L.qnorm);
  uint32_t* qcnt = reinterpret_cast<uint32_t*>(smem + L.qcnt);
  uint32_t* qfill = reinterpret_cast<uint32_t*>(smem + L.qfill);  // entries in use
  float* qnext = reinterpret_cast<float*>(smem + L.qnext);  // least value turned away
  uint32_t* run_b = reinterpret_cast<uint32_t*>(smem + L.runs);  // run: rows [b, e)
  uint32_t* run_e = run_b + (SEARCH ? kUnionCap : 1);
  uint32_t* run_s = run_e + (SEARCH ? kUnionCap : 1);  // first slot; run_s[runs] = slots
  uint32_t* qmask = reinterpret_cast<uint32_t*>(smem + L.qmask);  // [run][4]
  uint32_t* bitmap = reinterpret_cast<uint32_t*>(smem + L.bitmap);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const uint64_t q0 = blockIdx.x * (uint64_t)QT;
  const uint32_t nq = (uint32_t)min_u64(QT, a.q.n - q0);
  const uint32_t gb = group_bytes(kp), kq = kp / 8;
  const uint32_t base = smem_u32(smem);

  if (wid == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(tslot)), "n"(2 * NT)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(bfull + i, 1);
      mbar_init(mfull + i, 1);
    }
    fence_mbar_init();
    stop = 0;
    evals = 0;
  }
  if (tid < 4) bad[tid] = over[tid] = 0u;
  // the queries' operand, with ones against the candidates' norm columns
  const uint64_t qgroups = (a.q.n + 7) / 8;
  for (uint32_t t = tid; t < QT / 8 * (gb / 16); t += kTcKnnThreads) {
    const uint32_t g = t / (gb / 16), o = t % (gb / 16);
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (q0 / 8 + g < qgroups)
      v = *reinterpret_cast<const uint4*>(a.q.tiles + (q0 / 8 + g) * gb + o * 16u);
    *reinterpret_cast<uint4*>(smem + L.a + g * gb + o * 16u) = v;
  }
  __syncthreads();
  for (uint32_t t = tid; t < QT * kNormCols; t += kTcKnnThreads) {
    const uint32_t r = t / kNormCols, j = d + t % kNormCols;
    *reinterpret_cast<uint16_t*>(smem + L.a + (r >> 3) * gb + (j >> 3) * 128u + (r & 7u) * 16u +
                                 (j & 7u) * 2u) = 0x3F80u;  // BF16 1.0
  }
  for (uint32_t q = tid; q < QT; q += kTcKnnThreads) {
    const bool in = q < nq;
    const float nm = SEARCH && in ? a.q.norms[q0 + q] : 0.f;
    qlen[q] = in ? a.q.length[q0 + q] : 0.f;
    qnorm[q] = nm;
    qcnt[q] = 0u;
    qfill[q] = 0u;
    qnext[q] = INFINITY;
    thr[q] = 0.5f * (nm - FLT_MAX) - 4e32f;
  }
  for (uint32_t t = tid; t < QT * R * 32; t += kTcKnnThreads) {
    ld[t] = (t % (R * 32)) < a.size ? FLT_MAX : -INFINITY;
    li[t] = 0xFFFFFFFFu;
  }
  uint32_t nbits = 0;  // searched clusters of the CTA's queries
  uint32_t own = 0;    // the cluster of the middle query
  if (a.coff) {
    const uint64_t mid_row = q0 + nq / 2;
    uint32_t lo = 0, hi = a.nc;
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) / 2;
      if (a.coff[mid] <= mid_row) lo = mid;
      else hi = mid;
    }
    own = lo;
  }
  auto all = [](uint32_t) { return true; };
  if constexpr (SEARCH) {
    const bool wide = knows_wide(a);  // then there is nothing to do here
    if (tid == 0) given = wide;
    if (!wide) nbits = searched_clusters<kTcKnnThreads>(a, q0, nq, bitmap, wsum, all);
  }
  fence_proxy_async_smem();  // A's generic writes -> tensor-core reads
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  const uint32_t idesc = idesc_bf16(128, NT);
  const uint32_t qi = (uint32_t)(wid & 3) * 32u + lane;  // the query this thread filters
  const uint32_t cq = (uint32_t)wid >> 2;                // and its column quarter
  const bool filters = qi < nq;

  // Evaluates the first `cnt` queued candidates of query q and offers them.
  auto evaluate = [&](uint32_t q, uint32_t cnt) {
    const bool use = (uint32_t)lane < cnt;
    const uint32_t row = use ? queue[q * kQueue + lane] : 0u;
    const float nm = qnorm[q];
    float dist = INFINITY;
    if (use) {
      const float* x = a.q.rows + (q0 + q) * d;
      const float* c = a.c.rows + (uint64_t)row * d;
      const float cn = a.c.norms[row];
      const float pd = fmaf(-2.f, row_dot<VEC>(x, c, d), cn);  // |c|^2 - 2 x.c
      dist = SEARCH ? nm + pd : pd;
    }
    float* sd = ld + q * R * 32;
    uint32_t* si = li + q * R * 32;
    const uint32_t fill = qfill[q];
    const unsigned fit = __ballot_sync(0xffffffffu, use && dist < FLT_MAX);
    const uint32_t to = fill + __popc(fit);
    if (to <= a.size) {  // empty entries take them as they come, in order
      if ((fit >> lane) & 1u) {
        const uint32_t e = fill + __popc(fit & ((1u << lane) - 1u));
        sd[e] = dist;
        si[e] = row;
      }
      if (lane == 0) qfill[q] = to;
      __syncwarp();
      if (to < a.size) return;
    }
    WarpList<R> best;
    best.load(sd, si, lane);
    if (to > a.size) {
      const float next = best.offer(dist, row, fit, lane, qnext[q]);
      best.store(sd, si, lane);
      if (lane == 0) {
        qfill[q] = a.size;
        qnext[q] = next;
      }
    }
    if (lane == 0) {
      const float w = best.worst;
      thr[q] = 0.5f * (nm - w) - 1e-6f * (fabsf(nm) + fabsf(w));
    }
    __syncwarp();
  };

  // Past this many exact evaluations the margins are too wide for the data: the
  // CTA's queries go to the replay kernels, what is left of the tiles is not looked at.
  const uint32_t most_evals = nq * a.size * (SEARCH ? kSearchEvals : kNearestEvals);
  bool gave_up = false;  // known to this warp
  uint32_t gt = 0;  // tiles so far: buffers and phases
  uint32_t ubase = 0;
  bool ok = true;
  do {
    uint32_t nruns = 1, nslots;
    if constexpr (SEARCH) {
      // the next kUnionCap searched clusters in label order
      nruns = min(kUnionCap, nbits - ubase);
      searched_runs<kTcKnnThreads, 4>(a, q0, nq, bitmap, ubase, nruns, run_b, run_e, qmask, all);
    } else if (tid == 0) {
      run_b[0] = 0u;
      run_e[0] = (uint32_t)a.c.n;
    }
    __syncthreads();
    if (wid == 0)  // first slot of every run
      run_starts(run_s, nruns, [&](uint32_t u) {
        return run_e[u] > run_b[u] ? (run_e[u] + 7) / 8 - run_b[u] / 8 : 0u;
      });
    __syncthreads();
    nslots = run_s[nruns];
    const uint32_t ntiles = (nslots + SLOTS - 1) / SLOTS;
    // the tile that step t works on: from the own cluster's on, around
    uint32_t t0 = 0;
    if (a.coff && ntiles) {
      uint32_t slot = own / 8;  // nearest: the own centroid's group
      if constexpr (SEARCH) {
        const uint32_t pos = cluster_rank(bitmap, a.nc, own);
        slot = pos >= ubase && pos - ubase < nruns ? run_s[pos - ubase] : 0u;
      }
      t0 = min(slot / SLOTS, ntiles - 1);
    }
    auto tile_of = [&](uint32_t t) { return t0 + t < ntiles ? t0 + t : t0 + t - ntiles; };

    // Warp 0: the description and the operand of tile t (bulk copies, a lane
    // per 8-row group).
    auto fetch = [&](uint32_t t) {
      const uint32_t g = gt + t, m = g & 3u, first = tile_of(t) * SLOTS, slot = first + lane;
      const bool use = (uint32_t)lane < SLOTS && slot < nslots;
      uint32_t group = 0, u = kNoRun;
      float gm = 0.f;
      if (use) {
        uint32_t lo = 0, hi = nruns;  // the last run that starts at or before slot
        while (hi - lo > 1) {
          const uint32_t mid = (lo + hi) / 2;
          if (run_s[mid] <= slot) lo = mid;
          else hi = mid;
        }
        u = lo;
        group = run_b[u] / 8 + (slot - run_s[u]);
        gm = a.c.gmax[group];
      }
      if ((uint32_t)lane < SLOTS) {
        meta_row[m][lane] = group * 8;
        meta_run[m][lane] = u;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {  // a NaN stays a NaN
        const float h = __shfl_xor_sync(0xffffffffu, gm, o);
        gm = h != h ? h : (gm != gm ? gm : fmaxf(gm, h));
      }
      if (lane == 0) {
        meta_g[m] = gm;
        mbar_arrive_expect_tx(bfull + (g & 1u), min(SLOTS, nslots - first) * gb);
      }
      __syncwarp();
      if (use)
        bulk_g2s(smem + L.b + ((g & 1u) * SLOTS + lane) * gb, a.c.tiles + (uint64_t)group * gb,
                 gb, bfull + (g & 1u));
    };
    // One thread: the MMAs of tile t (its operand has landed).
    auto multiply = [&](uint32_t t) {
      const uint32_t g = gt + t, acc = tmem + (g & 1u) * NT;
      if (!tc_wait(bfull + (g & 1u), (g >> 1) & 1u, &stop, a.err)) return;
      tc_fence_after();
      const uint32_t sa = base + L.a, sb = base + L.b + (g & 1u) * SLOTS * gb;
      uint32_t on = 0;
      for (uint32_t ks = 0; ks < kp / 16; ++ks) {
        const uint64_t ah = smem_desc(sa + ks * 256u, 128u, gb);
        const uint64_t al = smem_desc(sa + kq * 128u + ks * 256u, 128u, gb);
        const uint64_t bh = smem_desc(sb + ks * 256u, 128u, gb);
        const uint64_t bl = smem_desc(sb + kq * 128u + ks * 256u, 128u, gb);
        mma_bf16(acc, ah, bl, idesc, on);
        mma_bf16(acc, al, bh, idesc, 1u);
        mma_bf16(acc, ah, bh, idesc, 1u);
        on = 1u;
      }
      mma_commit(mfull + (g & 1u));
    };

    if (wid == 0 && ntiles) {
      fetch(0);
      if (ntiles > 1) fetch(1);
      if (lane == 0) multiply(0);
      __syncwarp();
    }
    __syncthreads();  // the descriptions of tiles 0 and 1
    for (uint32_t t = 0; t < ntiles; ++t) {
      const uint32_t g = gt + t, m = g & 3u;
      if (wid == 0) {
        // accumulator (t + 1) & 1 was read before the last barrier
        if (lane == 0 && t + 1 < ntiles) multiply(t + 1);
        __syncwarp();
      }
      const int done = __shfl_sync(
          0xffffffffu, lane == 0 ? (int)tc_wait(mfull + (g & 1u), (g >> 1) & 1u, &stop, a.err) : 0,
          0);
      if (done) {
        tc_fence_after();
        if (wid == 0 && t + 2 < ntiles) fetch(t + 2);  // tile t's operand is free
        if ((uint32_t)(wid & 3) * 32u < QT) {
          float v[CW];
          tmem_ld<CW>(tmem + (g & 1u) * NT + cq * CW + ((uint32_t)(wid & 3) << 21), v);
          uint32_t mk = 0u;
          const uint32_t valid = (nslots - tile_of(t) * SLOTS) * 8u;  // the last tile may hold fewer
          if (valid < (cq + 1) * CW) {
#pragma unroll
            for (int j = 0; j < CW; ++j)
              if (cq * CW + j >= valid) v[j] = -INFINITY;
          }
          if (filters) {
            const float gm = meta_g[m], mg = kMargin * gm * (qlen[qi] + gm) + 1e-35f;
            const float lim = thr[qi] - mg;
            float top = v[0];  // most threads have nothing above the limit
#pragma unroll
            for (int j = 1; j + 1 < CW; j += 2) top = max3_nan(top, v[j], v[j + 1]);
            top = max3_nan(top, v[CW - 1], top);
            if (!(top <= lim)) {  // NaN passes
#pragma unroll
              for (int j = 0; j < CW; ++j)
                if (!(v[j] <= lim)) mk |= 1u << j;
            }
          }
          masks[((g & 1u) * 4 + cq) * 128 + qi] = mk;
        }
        tc_fence_before();
      }
      ok = !__syncthreads_or(!done);
      if (!ok) break;
      tc_fence_after();
      // this warp's queries (wid, wid + 16, ...; at most 8): lane 4 i + w holds
      // mask word w of query i
      const uint32_t oq = (uint32_t)wid + 16u * ((uint32_t)lane >> 2);
      const uint32_t word =
          oq < nq ? masks[((g & 1u) * 4 + ((uint32_t)lane & 3u)) * 128 + oq] : 0u;
      uint32_t hit = __ballot_sync(0xffffffffu, word != 0u);
      if (gave_up) continue;
      while (hit) {
        const int src = __ffs(hit) - 1;
        hit &= hit - 1u;
        const uint32_t bits = __shfl_sync(0xffffffffu, word, src);
        const uint32_t q = (uint32_t)wid + 16u * ((uint32_t)src >> 2), w = (uint32_t)src & 3u;
        uint32_t row = 0;
        bool use = false;
        if (lane < CW && ((bits >> lane) & 1u)) {
          const uint32_t j = w * CW + lane, u = meta_run[m][j >> 3];
          if (u != kNoRun) {
            row = meta_row[m][j >> 3] + (j & 7u);
            use = row >= run_b[u] && row < run_e[u];
            if (SEARCH)
              use = use && row != q0 + q && ((qmask[u * 4 + (q >> 5)] >> (q & 31)) & 1u);
          }
        }
        const uint32_t vote = __ballot_sync(0xffffffffu, use);
        uint32_t cnt = qcnt[q];
        if (use) queue[q * kQueue + cnt + __popc(vote & ((1u << lane) - 1u))] = row;
        cnt += __popc(vote);
        __syncwarp();
        if (cnt >= 32u) {
          evaluate(q, 32u);
          uint32_t made = 0;
          if (lane == 0) made = atomicAdd(&evals, 32u);
          gave_up = __shfl_sync(0xffffffffu, made, 0) >= most_evals;
          cnt -= 32u;
          const uint32_t rest = (uint32_t)lane < cnt ? queue[q * kQueue + 32 + lane] : 0u;
          __syncwarp();
          if ((uint32_t)lane < cnt) queue[q * kQueue + lane] = rest;
        }
        if (lane == 0) qcnt[q] = cnt;
        __syncwarp();
      }
    }
    gt += ntiles;
    ubase += nruns;
    __syncthreads();  // the runs and tile descriptions are no longer read
  } while (SEARCH && ok && ubase < nbits);

  if (ok && !(SEARCH && given) && !refused(a)) {
    // what is left in the queues, then the sorted lists
    const bool again = evals > most_evals;
    for (uint32_t q = wid; q < nq; q += kTcKnnWarps) {
      if (again) {
        if (lane == 0) {
          atomicOr(&bad[q >> 5], 1u << (q & 31));
          atomicOr(&over[q >> 5], 1u << (q & 31));
        }
        continue;
      }
      const uint32_t cnt = qcnt[q];
      if (cnt) evaluate(q, cnt);
      write_sorted(ld + q * R * 32, li + q * R * 32, a.size, SEARCH ? a.id_map : nullptr,
                   a.out_d + (q0 + q) * a.size, a.out_id + (q0 + q) * a.size, lane);
      if (a.coff && lane == 0) {
        float w = ld[q * R * 32];
        for (uint32_t e = 1; e < a.size; ++e) w = fmaxf(w, ld[q * R * 32 + e]);
        if (qnext[q] == w) atomicOr(&bad[q >> 5], 1u << (q & 31));
      }
    }
  } else if (!ok && tid == 0) {
    // a wait ran out: the copies and MMAs in flight end (waits with a limit)
    // before shared memory and TMEM go back
    for (int i = 0; i < 2; ++i) {
      (void)mbar_wait(bfull + i, 0u, nullptr);
      (void)mbar_wait(bfull + i, 1u, nullptr);
      (void)mbar_wait(mfull + i, 0u, nullptr);
      (void)mbar_wait(mfull + i, 1u, nullptr);
    }
  }
  __syncthreads();
  list_replays<SEARCH>(a, q0, bad, over, QT / 32);
  tc_fence_after();
  if (wid == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                 ::"r"(tmem), "n"(2 * NT)
                 : "memory");
  }
}

// Lists of up to 64 entries in two passes over the candidates, without a list
// that has to be kept up to date:
//  1. each thread (one query, a quarter of every tile's columns) keeps the M
//     largest lower bounds of s (s less the margin) over groups of GS columns:
//     a group's largest. Groups are disjoint, so the size-th largest of a
//     query's 4 M bounds has at least `size` candidates at or above it: tau.
//     Neighbours lie close together in the cells' order, so the search takes
//     every column by itself (groups of 8 left bounds so loose that 5 % of the
//     queues of 2.7k cells overflowed); the nearest clusters, whose longer
//     lists cost more per bound, take 4 at a time.
//  2. the candidates whose s plus the margin reaches tau, a few more than
//     `size`, are queued; at the end they are evaluated exactly and ranked by
//     (distance, row).
// The products are made twice (tensor time), but nothing in the loop waits for
// an exact evaluation and no tile waits for its slowest query. Lists of one
// entry (M == 1) need one pass: the largest lower bound so far, shared by the
// query's four threads once per tile, is tight after a tile or two; what it
// lets through is queued with its upper bound, and the final bound drops most
// of it (E step 0.91 -> 0.57 ms).
// One warp copies operands up to four tiles ahead, one issues the MMAs into
// four accumulators, and the 16 filter warps follow at their own pace (barriers
// per operand and accumulator). Cycles per tile of 128 x 128, of which the 12
// MMAs take ~700: 4,700 with two buffers of each and one warp for both roles;
// 3,100 while the copy warp looked up each tile's runs and norms in turn and
// copied 8 rows at a time (1,250 cycles of issue); ~2,000 now, the filter's
// instructions in the first pass, the MMAs in the second. A thread first takes
// the largest of each slot's 8 values; almost always that ends it.
// Queries with more queued candidates than the queue's room (margins too wide for
// the data), and lists whose last distance is tied, are computed again. Lists of
// one entry need no tie rule: the first of equal distances is the lowest row.
constexpr int kTwoThreads = kTcKnnThreads + 64;  // and the copy and MMA warps
constexpr uint32_t kTwoAcc = 4;                  // accumulators in TMEM
constexpr uint32_t kTwoMeta = 8;                 // tile descriptions in flight
// queries evaluated together: lists of one entry have few rows each to wait for
__host__ __device__ constexpr uint32_t eval_batch(bool one) { return one ? 128u : 64u; }
constexpr uint32_t kRowChunk = 32;               // dimensions of a row staged at once

template <int BYTES>
__device__ __forceinline__ void cp_async(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src),
               "n"(BYTES)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// Exact x.c, in order over the dimensions, for a pair per lane; x lies in
// shared memory. The rows come by asynchronous copies of consecutive
// dimensions, all of a chunk's in flight at once, through the warp's shared
// `buf` (row stride kRowChunk + VEC: no bank conflicts). A lane that walks its
// own row takes 32 sectors per load, reads each of them more than once, and
// waits for L2 once per few loads: 132k cycles for the 9.7k pairs of 128
// queries of the nearest clusters, 93k so.
template <int VEC>
__device__ __forceinline__ float staged_dot(const float* x, const float* __restrict__ rows,
                                            uint32_t row, uint32_t d, float* buf, int lane) {
  constexpr int LPR = kRowChunk / VEC;  // lanes per row, and copies per lane
  constexpr int RPC = 32 / LPR;         // rows per copy
  constexpr int S = kRowChunk + VEC;
  const uint32_t at = (uint32_t)(lane % LPR) * VEC;
  const int r0 = lane / LPR;
  float acc = 0.f;
  for (uint32_t j0 = 0; j0 < d; j0 += kRowChunk) {
    __syncwarp();  // the chunk before has been read
#pragma unroll
    for (int i = 0; i < LPR; ++i) {
      const uint32_t r = __shfl_sync(0xffffffffu, row, i * RPC + r0);
      if (j0 + at < d)
        cp_async<VEC * 4>(buf + (i * RPC + r0) * S + at, rows + (uint64_t)r * d + j0 + at);
    }
    cp_async_wait();
    __syncwarp();
#pragma unroll
    for (int k = 0; k < (int)kRowChunk; k += VEC) {
      if (j0 + k < d) {
        float c[VEC], v[VEC];
        if constexpr (VEC == 4) {
          *(float4*)c = *(const float4*)(buf + lane * S + k);
          *(float4*)v = *(const float4*)(x + j0 + k);
        } else if constexpr (VEC == 2) {
          *(float2*)c = *(const float2*)(buf + lane * S + k);
          *(float2*)v = *(const float2*)(x + j0 + k);
        } else {
          c[0] = buf[lane * S + k];
          v[0] = x[j0 + k];
        }
#pragma unroll
        for (int i = 0; i < VEC; ++i) acc = fmaf(v[i], c[i], acc);
      }
    }
  }
  return acc;
}

struct TwoSmem {  // byte offsets
  uint32_t a, b, x, rows, queue, upper, tau, qlen, qnorm, qcnt, qat, runs, qmask, bitmap, total;
};

__host__ __device__ inline TwoSmem two_smem(uint32_t d, uint32_t kp, uint32_t qt, uint32_t nt,
                                            uint32_t cap, uint32_t stages, uint32_t vec,
                                            bool one, bool search, uint32_t nc) {
  TwoSmem L;
  uint32_t o = 1024;
  auto take = [&](uint32_t bytes) {
    const uint32_t at = o;
    o += (bytes + 127u) & ~127u;
    return at;
  };
  L.a = take(qt / 8 * group_bytes(kp));
  L.b = take(stages * (nt / 8) * group_bytes(kp));
  // the MMA reads 128 rows of A: the bytes past the queries' are B's
  if (o < L.a + 16 * group_bytes(kp)) o = L.a + 16 * group_bytes(kp);
  // at the end these take the operands' place, for a batch of queries: the
  // exact distances of what is queued, the queries, and rows on their way
  const uint32_t batch = qt < eval_batch(one) ? qt : eval_batch(one), end = o;
  o = L.a;
  take(batch * cap * 4);
  L.x = take(batch * d * 4);
  L.rows = take(kTwoThreads * (kRowChunk + vec) * 4);
  if (o < end) o = end;
  L.queue = take(qt * cap * 4);  // pass 1: the bounds, 4 M <= cap per query
  L.upper = take(one ? qt * cap * 4 : 16);
  L.tau = take(qt * 4);
  L.qlen = take(qt * 4);
  L.qnorm = take(qt * 4);
  L.qcnt = take(qt * 4);
  L.qat = take((3 * qt + 1) * 4);
  L.runs = take(search ? kUnionCap * 12 + 4 : 16);
  L.qmask = take(search ? kUnionCap * 16 : 16);
  L.bitmap = take(search ? (nc + 31) / 32 * 8 : 16);  // words and their ranks
  L.total = o;
  return L;
}

// A bound as a number that orders like it does; -inf is the smallest in use.
__device__ __forceinline__ uint32_t order_key(float f) {
  const uint32_t w = __float_as_uint(f);
  return w & 0x80000000u ? ~w : w | 0x80000000u;
}
__device__ __forceinline__ float key_value(uint32_t key) {
  return __uint_as_float(key & 0x80000000u ? key & 0x7FFFFFFFu : ~key);
}

template <int M, int GS, int CAP, bool SEARCH, int NT, int VEC>
__global__ void __launch_bounds__(kTwoThreads, 1) k_knn_two(const KnnArgs a) {
  constexpr int CW = NT / 4;          // candidates a thread tests per tile
  constexpr int CS = CW / 8;          // of its slots
  constexpr uint32_t SLOTS = NT / 8;  // 8-row groups per tile
  static_assert(M == 1 || 4 * M <= CAP, "the bounds of pass 1 lie in the queue's place");
  extern __shared__ __align__(1024) unsigned char smem[];
  uint64_t* bfull = reinterpret_cast<uint64_t*>(smem);       // [4] operand of a tile landed
  uint64_t* bfree = reinterpret_cast<uint64_t*>(smem) + 4;   // [4] operand used
  uint64_t* mfull = reinterpret_cast<uint64_t*>(smem) + 8;   // [4] MMAs of a tile done
  uint64_t* mfree = reinterpret_cast<uint64_t*>(smem) + 12;  // [4] accumulator read
  uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + 256);
  // per slot of a tile: first row, run, rows of the run (bits), norm bound
  __shared__ uint32_t meta_row[kTwoMeta][16], meta_run[kTwoMeta][16], meta_bits[kTwoMeta][16];
  __shared__ __align__(16) float meta_g[kTwoMeta][16];
  __shared__ uint32_t wsum[kTwoThreads / 32 + 1], bad[4], over[4], given;
  __shared__ volatile int stop;
  const uint32_t d = a.d, kp = a.kp, QT = a.qt;
  const uint32_t NB = a.stages;
  constexpr bool ONE = M == 1;
  const TwoSmem L = two_smem(d, kp, QT, NT, CAP, NB, VEC, ONE, SEARCH, a.nc);
  uint32_t* queue = reinterpret_cast<uint32_t*>(smem + L.queue);
  float* upper = reinterpret_cast<float*>(smem + L.upper);  // ONE: upper bounds of the queued
  float* tau = reinterpret_cast<float*>(smem + L.tau);
  uint32_t* best_key = reinterpret_cast<uint32_t*>(tau);  // ONE: largest lower bound so far
  float* qlen = reinterpret_cast<float*>(smem + L.qlen);
  float* qnorm = reinterpret_cast<float*>(smem + L.qnorm);
  uint32_t* qcnt = reinterpret_cast<uint32_t*>(smem + L.qcnt);
  uint32_t* run_b = reinterpret_cast<uint32_t*>(smem + L.runs);  // run: rows [b, e)
  uint32_t* run_e = run_b + (SEARCH ? kUnionCap : 1);
  uint32_t* run_s = run_e + (SEARCH ? kUnionCap : 1);  // first slot; run_s[runs] = slots
  uint32_t* qmask = reinterpret_cast<uint32_t*>(smem + L.qmask);  // [run][4]
  uint32_t* bitmap = reinterpret_cast<uint32_t*>(smem + L.bitmap);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const bool copies = wid == kTcKnnWarps;        // the copy warp
  const bool multiplies = wid == kTcKnnWarps + 1;  // the MMA warp
  const bool service = copies || multiplies;
  const uint64_t q0 = blockIdx.x * (uint64_t)QT;
  const uint32_t nq = (uint32_t)min_u64(QT, a.q.n - q0);
  const uint32_t gb = group_bytes(kp), kq = kp / 8;
  const uint32_t base = smem_u32(smem);
  const uint32_t readers = 4 * (QT / 32);  // warps that read an accumulator

  if (wid == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(tslot)), "n"(kTwoAcc * NT)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < 4; ++i) {
      mbar_init(bfull + i, 1);
      mbar_init(bfree + i, 1);
      mbar_init(mfull + i, 2);  // the commit, and the MMA lane for the description
      mbar_init(mfree + i, readers);
    }
    fence_mbar_init();
    stop = 0;
  }
  if (tid < 4) bad[tid] = over[tid] = 0u;
  // the queries' operand, with ones against the candidates' norm columns
  const uint64_t qgroups = (a.q.n + 7) / 8;
  for (uint32_t t = tid; t < QT / 8 * (gb / 16); t += kTwoThreads) {
    const uint32_t g = t / (gb / 16), o = t % (gb / 16);
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (q0 / 8 + g < qgroups)
      v = *reinterpret_cast<const uint4*>(a.q.tiles + (q0 / 8 + g) * gb + o * 16u);
    *reinterpret_cast<uint4*>(smem + L.a + g * gb + o * 16u) = v;
  }
  __syncthreads();
  for (uint32_t t = tid; t < QT * kNormCols; t += kTwoThreads) {
    const uint32_t r = t / kNormCols, j = d + t % kNormCols;
    *reinterpret_cast<uint16_t*>(smem + L.a + (r >> 3) * gb + (j >> 3) * 128u + (r & 7u) * 16u +
                                 (j & 7u) * 2u) = 0x3F80u;  // BF16 1.0
  }
  for (uint32_t q = tid; q < QT; q += kTwoThreads) {
    const bool in = q < nq;
    qlen[q] = in ? a.q.length[q0 + q] : 0.f;
    qnorm[q] = SEARCH && in ? a.q.norms[q0 + q] : 0.f;
    qcnt[q] = 0u;
    if (ONE) best_key[q] = order_key(-INFINITY);
  }
  uint32_t nbits = 0;  // searched clusters of the CTA's queries
  uint32_t own = 0;    // the cluster of the middle query
  if (a.coff) {
    const uint64_t mid_row = q0 + nq / 2;
    uint32_t lo = 0, hi = a.nc;
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) / 2;
      if (a.coff[mid] <= mid_row) lo = mid;
      else hi = mid;
    }
    own = lo;
  }
  auto all = [](uint32_t) { return true; };
  if constexpr (SEARCH) {
    const bool wide = knows_wide(a);  // then there is nothing to do here
    if (tid == 0) given = wide;
    if (!wide) nbits = searched_clusters<kTwoThreads>(a, q0, nq, bitmap, wsum, all);
  }
  fence_proxy_async_smem();  // A's generic writes -> tensor-core reads
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  const uint32_t idesc = idesc_bf16(128, NT);
  const uint32_t qi = (uint32_t)(wid & 3) * 32u + lane;  // the query this thread filters
  const uint32_t cq = (uint32_t)(wid >> 2) & 3u;         // and its column quarter
  const bool filters = !service && qi < nq;
  const bool reads = !service && (uint32_t)(wid & 3) * 32u < QT;
  const uint32_t qrow = (uint32_t)(q0 + qi);  // the search leaves this row out
  const float ql = filters ? qlen[qi] : 0.f;
  const float aq = filters ? 1e-6f * fabsf(qnorm[qi]) + 1e-35f : 0.f;
  float top[M];
#pragma unroll
  for (int i = 0; i < M; ++i) top[i] = -INFINITY;
  float mytau = -INFINITY;
  bool open = filters;  // pass 2: until the query's queue overflows

  uint32_t gt = 0;              // tiles so far: accumulators and phases
  uint32_t st = 0, phase = 0;   // the operand stage that comes next, its round (parity)
  bool ok = true;
  for (int pass = 0; pass < (ONE ? 1 : 2) && ok; ++pass) {
    uint32_t ubase = 0;
    do {
      uint32_t nruns = 1;
      if constexpr (SEARCH) {
        // the next kUnionCap searched clusters in label order
        nruns = min(kUnionCap, nbits - ubase);
        searched_runs<kTwoThreads, 4>(a, q0, nq, bitmap, ubase, nruns, run_b, run_e, qmask, all);
      } else if (tid == 0) {
        run_b[0] = 0u;
        run_e[0] = (uint32_t)a.c.n;
      }
      __syncthreads();
      if (wid == 0)  // first slot of every run
        run_starts(run_s, nruns, [&](uint32_t u) {
          return run_e[u] > run_b[u] ? (run_e[u] + 7) / 8 - run_b[u] / 8 : 0u;
        });
      __syncthreads();
      const uint32_t nslots = run_s[nruns];
      const uint32_t ntiles = (nslots + SLOTS - 1) / SLOTS;
      // the tile that step t works on: from the own cluster's on, around
      uint32_t t0 = 0;
      if (a.coff && ntiles) {
        uint32_t slot = own / 8;  // nearest: the own centroid's group
        if constexpr (SEARCH) {
          const uint32_t pos = cluster_rank(bitmap, a.nc, own);
          slot = pos >= ubase && pos - ubase < nruns ? run_s[pos - ubase] : 0u;
        }
        t0 = min(slot / SLOTS, ntiles - 1);
      }

      if (copies) {
        // ---- copies: tile t's description, then its operand into stage g % NB,
        // whose MMAs (tile g - NB) have completed. The description is looked up
        // one tile ahead: its chain of shared and global loads is as long as a
        // tile's MMAs.
        uint32_t group = 0, u = kNoRun, bits = 0, walk = 0;
        float gm = 0.f;
        auto look_up = [&](uint32_t t) {
          const uint32_t slot = (t0 + t < ntiles ? t0 + t : t0 + t - ntiles) * SLOTS + lane;
          group = 0, u = kNoRun, bits = 0;
          gm = 0.f;
          if ((uint32_t)lane < SLOTS && slot < nslots) {
            if (t0 + t == ntiles) walk = 0;
            if (t == 0) {
              uint32_t hi = nruns;  // the last run that starts at or before slot
              while (hi - walk > 1) {
                const uint32_t mid = (walk + hi) / 2;
                if (run_s[mid] <= slot) walk = mid;
                else hi = mid;
              }
            } else {
              while (run_s[walk + 1] <= slot) ++walk;  // run_s[nruns] = nslots
            }
            u = walk;
            group = run_b[u] / 8 + (slot - run_s[u]);
            gm = a.c.gmax[group];
            const uint32_t r0 = group * 8, rb = max(run_b[u], r0) - r0;
            const uint32_t re = min(run_e[u] - r0, 8u);
            bits = ((1u << re) - 1u) & ~((1u << rb) - 1u);
          }
        };
        if (ntiles) look_up(0);
        for (uint32_t t = 0; t < ntiles; ++t) {
          const uint32_t g = gt + t, m = g % kTwoMeta;
          int fine = 1;
          if (g >= NB && lane == 0) fine = tc_wait(bfree + st, phase ^ 1u, &stop, a.err);
          fine = __shfl_sync(0xffffffffu, fine, 0);
          if (!fine) break;
          // description slot m: its last tile, g - 8, was read before tile g -
          // NB's MMAs were issued (they follow the readers of tile g - NB - 4)
          const unsigned used = __ballot_sync(0xffffffffu, u != kNoRun);
          if ((uint32_t)lane < SLOTS) {
            meta_row[m][lane] = group * 8;
            meta_run[m][lane] = u;
            meta_bits[m][lane] = bits;
            meta_g[m][lane] = gm;
          }
          __syncwarp();
          if (lane == 0) mbar_arrive_expect_tx(bfull + st, __popc(used) * gb);
          __syncwarp();
          // one copy per stretch of successive groups: a copy's issue costs
          // ~70 cycles, 16 of them more than the tile's MMAs
          const uint32_t before = __shfl_up_sync(0xffffffffu, group, 1);
          const bool starts = lane == 0 || group != before + 1;
          const unsigned heads = __ballot_sync(0xffffffffu, starts) & used;
          if ((heads >> lane) & 1u) {
            const unsigned later = heads & ~((2u << lane) - 1u);
            const uint32_t end = later ? __ffs(later) - 1u : __popc(used);
            bulk_g2s(smem + L.b + (st * SLOTS + lane) * gb, a.c.tiles + (uint64_t)group * gb,
                     (end - lane) * gb, bfull + st);
          }
          if (++st == NB) st = 0, phase ^= 1u;
          if (t + 1 < ntiles) look_up(t + 1);
        }
      } else if (multiplies) {
        // ---- MMAs: tile t into accumulator g % 4, which the readers of tile
        // g - 4 have left
        if (elect_lane()) {
          const uint64_t ah0 = smem_desc(base + L.a, 128u, gb);
          const uint64_t bh0 = smem_desc(base + L.b, 128u, gb);
          const uint32_t low = kq * 128u >> 4;  // from the high parts to the low ones
          for (uint32_t t = 0; t < ntiles; ++t) {
            const uint32_t g = gt + t, b = g % kTwoAcc;
            if (g >= kTwoAcc && !tc_wait(mfree + b, (g / kTwoAcc - 1u) & 1u, &stop, a.err)) break;
            if (!tc_wait(bfull + st, phase, &stop, a.err)) break;
            tc_fence_after();
            const uint32_t acc = tmem + b * NT;
            uint64_t ah = ah0, bh = bh0 + (st * SLOTS * gb >> 4);
            for (uint32_t ks = 0; ks < kp / 16; ++ks) {
              mma_bf16(acc, ah, bh + low, idesc, ks ? 1u : 0u);
              mma_bf16(acc, ah + low, bh, idesc, 1u);
              mma_bf16(acc, ah, bh, idesc, 1u);
              ah += 16;  // 256 bytes
              bh += 16;
            }
            mma_commit(bfree + st);
            mma_commit(mfull + b);
            mbar_arrive(mfull + b);  // passes the tile's description on
            if (++st == NB) st = 0, phase ^= 1u;
          }
        }
        __syncwarp();
      } else if (reads) {
        // ---- filter warps: half of the thread's columns are tested while the
        // load of the next half (or of the next tile's first half) is in flight
        constexpr int HW = CW / 2, HS = CS / 2;
        const uint32_t lanes = tmem + cq * CW + ((uint32_t)(wid & 3) << 21);
        auto ready = [&](uint32_t t) -> bool {
          const uint32_t g = gt + t;
          const int done = __shfl_sync(0xffffffffu,
                                       lane == 0 ? (int)tc_wait(mfull + g % kTwoAcc,
                                                                (g / kTwoAcc) & 1u, &stop, a.err)
                                                 : 0,
                                       0);
          tc_fence_after();
          return done != 0;
        };
        auto test = [&](float* v, uint32_t m, uint32_t slot0) {
          float gs[HS], mx[HS];
#pragma unroll
          for (int i = 0; i < HS; ++i) {
            const float* w = v + 8 * i;
            gs[i] = meta_g[m][slot0 + i];
            mx[i] = max3_nan(max3_nan(w[0], w[1], w[2]), max3_nan(w[3], w[4], w[5]),
                             max3_nan(w[6], w[7], w[7]));
          }
#pragma unroll
          for (int i = 0; i < HS; ++i) {
            const float* w = v + 8 * i;
            const float mg = kMargin * gs[i] * (ql + gs[i]) + aq;
            const float lim = ONE ? mytau - mg : pass == 0 ? top[M - 1] + mg : mytau - mg;
            if (mx[i] <= lim || !open) continue;  // NaN goes on
            const uint32_t slot = slot0 + i, u = meta_run[m][slot], row = meta_row[m][slot];
            uint32_t left = u != kNoRun ? meta_bits[m][slot] : 0u;
            if (SEARCH) {
              if (u == kNoRun || !((qmask[u * 4 + (qi >> 5)] >> (qi & 31)) & 1u)) left = 0u;
              if (qrow - row < 8u) left &= ~(1u << (qrow - row));
            }
            if (!left) continue;
            if constexpr (ONE) {
              float x = -INFINITY;  // NaN and what overflows are no bound
#pragma unroll
              for (int k = 0; k < 8; ++k)
                if (((left >> k) & 1u) && w[k] < 1e37f) x = fmaxf(x, w[k]);
              mytau = fmaxf(mytau, x - mg);
#pragma unroll
              for (int k = 0; k < 8; ++k)
                if (((left >> k) & 1u) && !(w[k] <= mytau - mg)) {
                  const uint32_t pos = atomicAdd(&qcnt[qi], 1u);
                  if (pos < (uint32_t)CAP) {
                    queue[qi * CAP + pos] = row + k;
                    upper[qi * CAP + pos] = w[k] + mg;
                  }
                }
            } else if (pass == 0) {
#pragma unroll
              for (int k = 0; k < 8; k += GS) {
                float x = -INFINITY;  // NaN and what overflows are no bound
#pragma unroll
                for (int j = k; j < k + GS; ++j)
                  if (((left >> j) & 1u) && w[j] < 1e37f) x = fmaxf(x, w[j]);
                x -= mg;
                if (x > top[M - 1]) {
#pragma unroll
                  for (int n = M - 1; n > 0; --n) top[n] = fmaxf(top[n], fminf(top[n - 1], x));
                  top[0] = fmaxf(top[0], x);
                }
              }
            } else {
#pragma unroll
              for (int k = 0; k < 8; ++k)
                if (((left >> k) & 1u) && !(w[k] <= lim)) {
                  const uint32_t pos = atomicAdd(&qcnt[qi], 1u);
                  if (pos < (uint32_t)CAP) queue[qi * CAP + pos] = row + k;
                  else open = false;
                }
            }
          }
        };
        float v0[HW], v1[HW];
        bool go = ntiles > 0 && ready(0);
        if (go) tmem_load<HW>(lanes + (gt % kTwoAcc) * NT, v0);
        for (uint32_t t = 0; t < ntiles && go; ++t) {
          const uint32_t g = gt + t, b = g % kTwoAcc, m = g % kTwoMeta;
          tmem_loaded<HW>(v0);
          tmem_load<HW>(lanes + b * NT + HW, v1);
          float seen = mytau;
          if constexpr (ONE) mytau = seen = filters ? key_value(best_key[qi]) : mytau;
          test(v0, m, cq * CS);
          tmem_loaded<HW>(v1);
          tc_fence_before();
          if (t + 1 < ntiles) {
            go = ready(t + 1);
            if (go) tmem_load<HW>(lanes + ((g + 1) % kTwoAcc) * NT, v0);
          }
          test(v1, m, cq * CS + HS);
          if (ONE && mytau > seen) atomicMax(&best_key[qi], order_key(mytau));
          __syncwarp();
          if (lane == 0) mbar_arrive(mfree + b);  // values and description are read
        }
      }
      gt += ntiles;
      st = gt % NB;
      phase = (gt / NB) & 1u;
      ubase += nruns;
      ok = !__syncthreads_or(stop);  // and the runs are no longer read
    } while (SEARCH && ok && ubase < nbits);
    if (!ONE && pass == 0 && ok) {
      float* bound = reinterpret_cast<float*>(queue);  // [query][4 M]
      if (filters)
#pragma unroll
        for (int i = 0; i < M; ++i) bound[qi * CAP + cq * M + i] = top[i];
      __syncthreads();
      if (!service) {
        // tau: the size-th largest bound, the largest number with 23 leading
        // bits that at least `size` bounds reach, bit by bit (keys: floats in
        // the order of integers), four queries at a time: a bit's votes wait
        // for the bit before
        constexpr int E = (4 * M + 31) / 32, Q = 4;
        for (uint32_t q1 = wid * Q; q1 < nq; q1 += kTcKnnWarps * Q) {
          uint32_t key[Q][E], cut[Q];
#pragma unroll
          for (int i = 0; i < Q; ++i) {
            const uint32_t q = min(q1 + i, nq - 1);
            cut[i] = 0;
#pragma unroll
            for (int e = 0; e < E; ++e) {
              const int n = e * 32 + lane;
              key[i][e] = n < 4 * M ? order_key(bound[q * CAP + n]) : 0u;  // 0: no bound
            }
          }
          for (uint32_t bit = 0x80000000u; bit >= 0x200u; bit >>= 1) {
#pragma unroll
            for (int i = 0; i < Q; ++i) {
              uint32_t have = 0;
#pragma unroll
              for (int e = 0; e < E; ++e)
                have += __popc(__ballot_sync(0xffffffffu, key[i][e] >= (cut[i] | bit)));
              if (have >= a.size) cut[i] |= bit;
            }
          }
#pragma unroll
          for (int i = 0; i < Q; ++i) {
            // back to a float; fewer bounds than entries: no limit
            float t = key_value(cut[i]);
            if (cut[i] <= 0x007FFFFFu) t = -INFINITY;  // -inf's key and below
            if (lane == i && q1 + i < nq) tau[q1 + i] = t;
            if constexpr (!SEARCH) {  // the list's own range is within the margins
              uint32_t most = key[i][0];
#pragma unroll
              for (int e = 1; e < E; ++e) most = max(most, key[i][e]);
              const float range = key_value(__reduce_max_sync(0xffffffffu, most)) - t;
              const float len = qlen[min(q1 + i, nq - 1)];
              if (lane == i && q1 + i < nq && range <= 4.f * kMargin * len * len)
                atomicOr(&over[(q1 + i) >> 5], 1u << ((q1 + i) & 31));
            }
          }
        }
      }
      __syncthreads();
      if (filters) mytau = tau[qi];
    }
  }

  if (ok && !(SEARCH && given) && !refused(a)) {
    // The exact distances of what is queued, a thread per (query, entry) over
    // the whole CTA (a warp per query instead waits for its few rows alone,
    // eight times in turn), where the operands were; then the entries' ranks.
    uint32_t* at = reinterpret_cast<uint32_t*>(smem + L.qat);  // first entry of each query
    uint32_t* qbad = at + QT + 1;                              // entries that no list keeps
    uint32_t* ranks = qbad + QT;                               // sum of the others' ranks
    float* dists = reinterpret_cast<float*>(smem + L.a);       // [query of the batch][CAP]
    float* xs = reinterpret_cast<float*>(smem + L.x);          // [query of the batch][d]
    float* buf = reinterpret_cast<float*>(smem + L.rows) + wid * 32 * (kRowChunk + VEC);
    float *last = tau, *next = qlen;  // distances of entries size - 1 and size
    for (uint32_t q = tid; q < QT; q += kTwoThreads) {
      if constexpr (ONE) {  // only what reaches the final bound
        const uint32_t cnt = qcnt[q];
        const float bound = key_value(best_key[q]);
        uint32_t kept = 0;
        if (cnt <= (uint32_t)CAP) {
          for (uint32_t e = 0; e < cnt; ++e)
            if (!(upper[q * CAP + e] < bound)) queue[q * CAP + kept++] = queue[q * CAP + e];
          qcnt[q] = kept;
        }
      }
      qbad[q] = ranks[q] = 0u;
      last[q] = next[q] = INFINITY;
    }
    if (ONE) __syncthreads();
    if (wid == 0) {
      uint32_t total = 0;
      for (uint32_t p0 = 0; p0 < QT; p0 += 32) {
        const uint32_t q = p0 + lane;
        const uint32_t c = q < nq && qcnt[q] <= (uint32_t)CAP ? qcnt[q] : 0u;
        uint32_t incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += v;
        }
        if (q < QT) at[q] = total + incl - c;
        total += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (lane == 0) at[QT] = total;
    }
    constexpr uint32_t BATCH = eval_batch(ONE);
    for (uint32_t qb = 0; qb < nq; qb += BATCH) {
      const uint32_t qe = min(qb + BATCH, nq);
      const float* src = a.q.rows + (q0 + qb) * d;
      for (uint32_t t = tid * VEC; t < (qe - qb) * d; t += kTwoThreads * VEC) {
        if constexpr (VEC == 4) *(float4*)(xs + t) = *(const float4*)(src + t);
        else if constexpr (VEC == 2) *(float2*)(xs + t) = *(const float2*)(src + t);
        else xs[t] = src[t];
      }
      __syncthreads();
      const uint32_t first = at[qb], entries = at[qe];
      auto owner = [&](uint32_t t) {  // the batch's last query that starts at or before t
        uint32_t q = qb, hi = qe;
        while (hi - q > 1) {
          const uint32_t mid = (q + hi) / 2;
          if (at[mid] <= t) q = mid;
          else hi = mid;
        }
        return q;
      };
      for (uint32_t t0 = first + wid * 32u; t0 < entries; t0 += kTwoThreads) {
        const uint32_t t = min(t0 + lane, entries - 1), q = owner(t), self = t - at[q];
        const uint32_t row = queue[q * CAP + self];
        const float cn = a.c.norms[row];
        const float dot = staged_dot<VEC>(xs + (q - qb) * d, a.c.rows, row, d, buf, lane);
        const float pd = fmaf(-2.f, dot, cn);  // |c|^2 - 2 x.c
        const float ds = SEARCH ? qnorm[q] + pd : pd;
        // what is not finite is never kept, as by the lists
        dists[(q - qb) * CAP + self] = ds < FLT_MAX ? ds : INFINITY;
      }
      __syncthreads();
      auto put = [&](uint32_t q, uint32_t rank, float de, uint32_t id) {
        if (rank < a.size) {
          a.out_d[(q0 + q) * a.size + rank] = de;
          a.out_id[(q0 + q) * a.size + rank] = SEARCH ? a.id_map[id] : id;
        }
        if (rank == a.size - 1) last[q] = de;
        if (rank == a.size) next[q] = de;
      };
      // rank: the closer entries, as if no two were equally close
      for (uint32_t t = first + tid; t < entries; t += kTwoThreads) {
        const uint32_t q = owner(t), cnt = at[q + 1] - at[q], self = t - at[q];
        const float* dist = dists + (q - qb) * CAP;
        const float de = dist[self];
        if (!(de < FLT_MAX)) {
          atomicAdd(&qbad[q], 1u);
          continue;
        }
        uint32_t rank = 0, f = 0;
        for (; f + 4 <= cnt; f += 4) {
          const float4 v = *reinterpret_cast<const float4*>(dist + f);
          rank += (v.x < de) + (v.y < de) + (v.z < de) + (v.w < de);
        }
        for (; f < cnt; ++f) rank += dist[f] < de;
        atomicAdd(&ranks[q], rank);
        put(q, rank, de, queue[q * CAP + self]);
      }
      __syncthreads();
      // the ranks add up to 0 + 1 + .. unless some are equal: then by row too
      for (uint32_t q = qb + wid; q < qe; q += kTwoThreads / 32) {
        const uint32_t cnt = at[q + 1] - at[q], valid = cnt - qbad[q];
        if (ranks[q] != valid * (valid - 1u) / 2u) {
          const float* dist = dists + (q - qb) * CAP;
          const uint32_t* ids = queue + q * CAP;
          for (uint32_t e = lane; e < cnt; e += 32) {
            const float de = dist[e];
            uint32_t rank = 0;
            for (uint32_t f = 0; f < cnt; ++f)
              rank += dist[f] < de || (dist[f] == de && ids[f] < ids[e]);
            if (de < FLT_MAX) put(q, rank, de, ids[e]);
          }
          __syncwarp();
        }
        const bool full = qcnt[q] > (uint32_t)CAP;
        if (lane == 0 && (full || (a.size > 1 && valid > a.size && last[q] == next[q])))
          atomicOr(&bad[q >> 5], 1u << (q & 31));
        if (!full)
          for (uint32_t e = valid + lane; e < a.size; e += 32) {  // empty entries
            a.out_d[(q0 + q) * a.size + e] = FLT_MAX;
            a.out_id[(q0 + q) * a.size + e] = 0xFFFFFFFFu;
          }
      }
      __syncthreads();
    }
  } else if (!ok && tid == 0) {
    // a wait ran out: the copies and MMAs in flight end (waits with a limit)
    // before shared memory and TMEM go back
    const long long until = clock64() + (1LL << 30);
    for (int i = 0; i < 4; ++i)
      for (uint32_t phase = 0; phase < 2; ++phase)
        while (clock64() < until && !(mbar_test(bfull + i, phase) && mbar_test(mfull + i, phase)))
          __nanosleep(64);
  }
  __syncthreads();
  list_replays<SEARCH>(a, q0, bad, over, QT / 32);
  tc_fence_after();
  if (wid == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                 ::"r"(tmem), "n"(kTwoAcc * NT)
                 : "memory");
  }
}

// The queries in replay, a CTA each: every candidate evaluated
// (kReplayBatch at a time, a thread each) and offered by one warp in the
// reference's order. The searched clusters' rows are one sequence: batches that
// ended with each cluster of ~137 rows took 0.69 ms for 38 queries of 8.8k
// candidates (three barriers and a latency per cluster), 0.35 ms so.
constexpr int kReplayThreads = 256;
constexpr uint32_t kReplayBatch = 1024;
template <int R, bool SEARCH, int VEC>
__global__ void __launch_bounds__(kReplayThreads) k_knn_replay(const KnnArgs a) {
  __shared__ float rd[R * 32];
  __shared__ uint32_t ri[R * 32];
  __shared__ float dist[kReplayBatch];
  __shared__ uint32_t ids[kReplayBatch];
  // the searched clusters in label order: first row, rows before them
  __shared__ uint32_t lab[SEARCH ? kReplayThreads : 1], begin[SEARCH ? kReplayThreads : 1];
  __shared__ uint32_t before[SEARCH ? kReplayThreads + 1 : 1], wsum[kReplayThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t count = a.counts[0], d = a.d;
  for (uint32_t i = blockIdx.x; i < count; i += gridDim.x) {
    const uint64_t q = a.replay[i];
    const float* x = a.q.rows + q * d;
    const float nm = SEARCH ? a.q.norms[q] : 0.f;
    for (uint32_t e = threadIdx.x; e < R * 32; e += kReplayThreads) {
      rd[e] = e < a.size ? FLT_MAX : -INFINITY;
      ri[e] = 0xFFFFFFFFu;
    }
    uint32_t total = (uint32_t)a.c.n;
    if constexpr (SEARCH) {
      const uint32_t u = threadIdx.x;
      const uint32_t mine = u < a.cs ? a.nearest[q * a.cs + u] : 0xFFFFFFFFu;
      lab[u] = mine;
      __syncthreads();
      uint32_t rank = 0;  // labels are distinct, except of clusters that do not exist
      for (uint32_t v = 0; v < (uint32_t)kReplayThreads; ++v)
        rank += lab[v] < mine || (lab[v] == mine && v < u);
      __syncthreads();
      lab[rank] = mine;
      __syncthreads();
      const uint32_t l = lab[u];
      const bool has = l < a.nc && (u == 0 || lab[u - 1] != l);
      const uint32_t first = has ? (uint32_t)a.coff[l] : 0u;
      const uint32_t size = has ? (uint32_t)a.coff[l + 1] - first : 0u;
      begin[u] = first;
      uint32_t incl = size;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      if (lane == 31) wsum[wid] = incl;
      __syncthreads();
      for (int w = 0; w < wid; ++w) incl += wsum[w];
      before[u] = incl - size;
      if (u == kReplayThreads - 1) before[kReplayThreads] = incl;
      __syncthreads();
      total = before[kReplayThreads];
    }
    __syncthreads();
    WarpList<R> best;  // warp 0's
    if (wid == 0) best.load(rd, ri, lane);
    for (uint64_t r0 = 0; r0 < total; r0 += kReplayBatch) {
      const uint32_t len = (uint32_t)min_u64(kReplayBatch, total - r0);
      for (uint32_t k = threadIdx.x; k < len; k += kReplayThreads) {
        uint32_t row = (uint32_t)r0 + k;
        if constexpr (SEARCH) {
          uint32_t u = 0, hi = kReplayThreads;  // the last cluster that starts at or before it
          while (hi - u > 1) {
            const uint32_t mid = (u + hi) / 2;
            if (before[mid] <= row) u = mid;
            else hi = mid;
          }
          row = begin[u] + (row - before[u]);
        }
        const float pd =
            fmaf(-2.f, row_dot<VEC>(x, a.c.rows + (uint64_t)row * d, d), a.c.norms[row]);
        dist[k] = SEARCH ? nm + pd : pd;
        ids[k] = row;
      }
      __syncthreads();
      if (wid == 0)
        for (uint32_t k = 0; k < len; k += 32) {
          const bool in = k + lane < len;
          const uint32_t row = in ? ids[k + lane] : 0u;
          const bool use = in && !(SEARCH && row == q);
          const float cand = use ? dist[k + lane] : INFINITY;
          best.keep(cand, row, __ballot_sync(0xffffffffu, cand < best.worst), lane);
        }
      __syncthreads();
    }
    if (wid == 0) {
      best.store(rd, ri, lane);
      __syncwarp();
      write_sorted(rd, ri, a.size, SEARCH ? a.id_map : nullptr, a.out_d + q * a.size,
                   a.out_id + q * a.size, lane);
    }
    __syncthreads();
  }
}

// Row stride (floats) of rows staged whole: a multiple of 4 whose float4 count
// is odd, so that lanes reading float4s of successive rows meet no bank twice.
__host__ __device__ inline uint32_t row_stride(uint32_t d) {
  const uint32_t s = (d + 3u) & ~3u;
  return (s >> 2) & 1u ? s : s + 4u;
}

// The groups of 32 queries in groups, a CTA each: the exhaustive search, for
// data on which the filter decides nothing (margins wider than the distances'
// spread, as PCs far from their origin have, or ties at most lists' ends, as
// repeated cells have). All rows of the group's searched clusters as one
// sequence, 128 staged at a time; a warp takes four of the queries and four rows
// per lane, an FP32 chain each, and offers what is closer than a list's worst in
// the reference's order. Shared loads: 20 wavefronts per 16 warp multiply-adds
// of four dimensions, against 12 per 8 for two rows per lane. 300k x 50 dims, 2,191
// clusters, 64 searched, 20 neighbours, every list: search 27 ms, nearest clusters
// 10.5 ms (two rows per lane, lists in registers: 36.7 and 20.9; a CTA per query:
// 124 both). Three CTAs per SM: with 256 clusters at a time for lists of up to 128
// (100 neighbours 48.6 ms, with two CTAs 70); four leave 64 registers, slower for
// lists past 32 (50 neighbours 33 and 42 ms).
constexpr int kAllThreads = 256;
constexpr uint32_t kAllQueries = 32, kAllRows = 128;
constexpr uint32_t kAllRuns = 256;  // searched clusters taken at once
constexpr int kAllPerWarp = (int)kAllQueries / (kAllThreads / 32), kAllPerLane = (int)kAllRows / 32;

struct AllSmem {  // byte offsets
  uint32_t tile, x, norm, row, mask, list, runs, qmask, bitmap, total;
};

__host__ __device__ inline AllSmem all_smem(uint32_t d, uint32_t R, bool search, uint32_t nc) {
  AllSmem L;
  uint32_t o = 0;
  auto take = [&](uint32_t bytes) {
    const uint32_t at = o;
    o += (bytes + 15u) & ~15u;
    return at;
  };
  L.tile = take(kAllRows * row_stride(d) * 4);
  L.x = take(kAllQueries * row_stride(d) * 4);
  L.norm = take(kAllRows * 4);
  L.row = take(kAllRows * 4);
  L.mask = take(kAllRows * 4);  // the group's queries that search the row's cluster
  L.list = take(kAllQueries * R * 32 * 8);
  L.runs = take(search ? kAllRuns * 12 + 4 : 16);
  L.qmask = take(search ? kAllRuns * 4 : 16);
  L.bitmap = take(search ? (nc + 31) / 32 * 8 : 16);  // words and their ranks
  L.total = o;
  return L;
}

template <int R, bool SEARCH>
__global__ void __launch_bounds__(kAllThreads, R <= 4 ? 3 : 2)
k_knn_all(const KnnArgs a, int vec) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ uint32_t wsum[kAllThreads / 32 + 1];
  const uint32_t d = a.d, st = row_stride(d);
  const AllSmem L = all_smem(d, R, SEARCH, a.nc);
  float* tile = reinterpret_cast<float*>(smem + L.tile);
  float* xs = reinterpret_cast<float*>(smem + L.x);
  float* norm = reinterpret_cast<float*>(smem + L.norm);
  uint32_t* rows = reinterpret_cast<uint32_t*>(smem + L.row);
  uint32_t* mask = reinterpret_cast<uint32_t*>(smem + L.mask);
  float* ld = reinterpret_cast<float*>(smem + L.list);
  uint32_t* li = reinterpret_cast<uint32_t*>(ld + kAllQueries * R * 32);
  uint32_t* run_b = reinterpret_cast<uint32_t*>(smem + L.runs);  // run: rows [b, e)
  uint32_t* run_e = run_b + (SEARCH ? kAllRuns : 1);
  uint32_t* run_s = run_e + (SEARCH ? kAllRuns : 1);  // rows before the run
  uint32_t* qmask = reinterpret_cast<uint32_t*>(smem + L.qmask);
  uint32_t* bitmap = reinterpret_cast<uint32_t*>(smem + L.bitmap);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  // a query's columns past d are zero, so what the rows hold there adds nothing
  // once it is a number
  for (uint32_t t = tid; t < kAllRows * (st - d); t += kAllThreads)
    tile[t / (st - d) * st + d + t % (st - d)] = 0.f;
  const uint32_t count = a.counts[1];
  for (uint32_t gi = blockIdx.x; gi < count; gi += gridDim.x) {
    const uint64_t q0 = (uint64_t)a.groups[2 * gi] * kAllQueries;
    const uint32_t live = a.groups[2 * gi + 1];
    const uint32_t nq = (uint32_t)min_u64(kAllQueries, a.q.n - q0);
    auto uses = [&](uint32_t q) { return ((live >> q) & 1u) != 0u; };
    __syncthreads();  // the group before is done
    for (uint32_t t = tid; t < kAllQueries * st; t += kAllThreads) {
      const uint32_t q = t / st, j = t % st;
      xs[t] = q < nq && j < d ? a.q.rows[(q0 + q) * d + j] : 0.f;
    }
    for (uint32_t t = tid; t < kAllQueries * R * 32; t += kAllThreads) {
      ld[t] = t % (R * 32) < a.size ? FLT_MAX : -INFINITY;
      li[t] = 0xFFFFFFFFu;
    }
    float worst[kAllPerWarp], qn[kAllPerWarp];
#pragma unroll
    for (int i = 0; i < kAllPerWarp; ++i) {
      const uint32_t q = wid * kAllPerWarp + i;
      worst[i] = uses(q) ? FLT_MAX : -INFINITY;  // nothing is closer than -inf
      qn[i] = SEARCH && q < nq ? a.q.norms[q0 + q] : 0.f;
    }
    const uint32_t mine = live & (((1u << kAllPerWarp) - 1u) << (wid * kAllPerWarp));
    uint32_t nbits = 0, ubase = 0;
    if constexpr (SEARCH) nbits = searched_clusters<kAllThreads>(a, q0, nq, bitmap, wsum, uses);
    do {
      uint32_t nruns = 1, total = (uint32_t)a.c.n;
      if constexpr (SEARCH) {
        nruns = min(kAllRuns, nbits - ubase);
        searched_runs<kAllThreads, 1>(a, q0, nq, bitmap, ubase, nruns, run_b, run_e, qmask, uses);
        __syncthreads();
        if (wid == 0) run_starts(run_s, nruns, [&](uint32_t u) { return run_e[u] - run_b[u]; });
        __syncthreads();
        total = run_s[nruns];
      }
      for (uint32_t r0 = 0; r0 < total; r0 += kAllRows) {
        __syncthreads();  // the tile before has been read
        if (tid < (int)kAllRows) {
          const uint32_t at = r0 + tid;
          uint32_t row = 0, who = 0;
          if (at < total) {
            row = at;
            who = live;
            if constexpr (SEARCH) {
              uint32_t u = 0, hi = nruns;  // the last run that starts at or before it
              while (hi - u > 1) {
                const uint32_t mid = (u + hi) / 2;
                if (run_s[mid] <= at) u = mid;
                else hi = mid;
              }
              row = run_b[u] + (at - run_s[u]);
              who = qmask[u];
            }
          }
          rows[tid] = row;
          mask[tid] = who;
          norm[tid] = who ? a.c.norms[row] : 0.f;
        }
        __syncthreads();
        for (uint32_t r = wid; r < kAllRows; r += kAllThreads / 32) {
          if (mask[r] == 0u) continue;  // past the last row
          const float* src = a.c.rows + (uint64_t)rows[r] * d;
          float* dst = tile + r * st;
          if (vec == 4)
            for (uint32_t j = lane * 4; j < d; j += 128) cp_async<16>(dst + j, src + j);
          else if (vec == 2)
            for (uint32_t j = lane * 2; j < d; j += 64) cp_async<8>(dst + j, src + j);
          else
            for (uint32_t j = lane; j < d; j += 32) cp_async<4>(dst + j, src + j);
        }
        cp_async_wait();
        __syncthreads();
        uint32_t who = 0;
#pragma unroll
        for (int c = 0; c < kAllPerLane; ++c) who |= mask[32 * c + lane];
        if (!__any_sync(0xffffffffu, (who & mine) != 0u)) continue;
        float acc[kAllPerWarp][kAllPerLane];
#pragma unroll
        for (int i = 0; i < kAllPerWarp; ++i)
#pragma unroll
          for (int c = 0; c < kAllPerLane; ++c) acc[i][c] = 0.f;
        const float* xp = xs + (size_t)wid * kAllPerWarp * st;
        const float* cp = tile + (size_t)lane * st;
        for (uint32_t j = 0; j < d; j += 4) {
          float4 cv[kAllPerLane];
#pragma unroll
          for (int c = 0; c < kAllPerLane; ++c)
            cv[c] = *reinterpret_cast<const float4*>(cp + 32 * c * st + j);
#pragma unroll
          for (int i = 0; i < kAllPerWarp; ++i) {
            const float4 x = *reinterpret_cast<const float4*>(xp + i * st + j);
#pragma unroll
            for (int c = 0; c < kAllPerLane; ++c) {
              acc[i][c] = fmaf(x.x, cv[c].x, acc[i][c]);
              acc[i][c] = fmaf(x.y, cv[c].y, acc[i][c]);
              acc[i][c] = fmaf(x.z, cv[c].z, acc[i][c]);
              acc[i][c] = fmaf(x.w, cv[c].w, acc[i][c]);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < kAllPerWarp; ++i) {
          const uint32_t q = wid * kAllPerWarp + i;
          WarpList<R> best;
          bool loaded = false;
#pragma unroll
          for (int c = 0; c < kAllPerLane; ++c) {
            const uint32_t r = 32 * c + lane, row = rows[r];
            const float pd = fmaf(-2.f, acc[i][c], norm[r]);  // |c|^2 - 2 x.c
            const float cand = SEARCH ? qn[i] + pd : pd;
            const bool use = ((mask[r] >> q) & 1u) && !(SEARCH && row == q0 + q);
            const unsigned closer = __ballot_sync(0xffffffffu, use && cand < worst[i]);
            if (!closer) continue;
            if (!loaded) best.load(ld + q * R * 32, li + q * R * 32, lane);
            loaded = true;
            // lanes that may not be offered never get closer than the worst
            best.keep(use ? cand : INFINITY, row, closer, lane);
            worst[i] = best.worst;
          }
          if (loaded) best.store(ld + q * R * 32, li + q * R * 32, lane);
        }
      }
      ubase += nruns;
    } while (SEARCH && ubase < nbits);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kAllPerWarp; ++i) {
      const uint32_t q = wid * kAllPerWarp + i;
      if (uses(q))
        write_sorted(ld + q * R * 32, li + q * R * 32, a.size, SEARCH ? a.id_map : nullptr,
                     a.out_d + (q0 + q) * a.size, a.out_id + (q0 + q) * a.size, lane);
    }
  }
}

// Floats per load of both matrices' rows.
int row_vec(const KnnArgs& a) {
  const uintptr_t at = (uintptr_t)a.q.rows | (uintptr_t)a.c.rows;
  return a.d % 4 == 0 && at % 16 == 0 ? 4 : a.d % 2 == 0 && at % 8 == 0 ? 2 : 1;
}

template <int R, bool SEARCH, int VEC>
int launch_replay(const KnnArgs& a, cudaStream_t s) {
  k_knn_replay<R, SEARCH, VEC><<<num_sms() * 4, kReplayThreads, 0, s>>>(a);
  BGPU_CHECK_LAUNCH();
  if (!a.groups) return BGPU_OK;
  const size_t smem = all_smem(a.d, R, SEARCH, a.nc).total;
  BGPU_CUDA((allow_max_smem(k_knn_all<R, SEARCH>)));
  const uint64_t want = ceil_div(a.q.n, kAllQueries);
  k_knn_all<R, SEARCH><<<(unsigned)std::min<uint64_t>(want, (uint64_t)num_sms() * 3),
                         kAllThreads, smem, s>>>(a, VEC);
  BGPU_CHECK_LAUNCH();
  return BGPU_OK;
}

// at least 120 KB of shared memory, so that one CTA (and one TMEM allocation)
// runs per SM
template <int R, bool SEARCH, int NT, int VEC>
int launch_one(const KnnArgs& a, cudaStream_t s) {
  const size_t smem =
      std::max<size_t>(knn_smem(a.kp, a.qt, NT, R, SEARCH, a.nc).total, 120 * 1024);
  BGPU_CUDA((allow_max_smem(k_knn_tc<R, SEARCH, NT, VEC>)));
  k_knn_tc<R, SEARCH, NT, VEC>
      <<<(unsigned)ceil_div(a.q.n, a.qt), kTcKnnThreads, smem, s>>>(a);
  BGPU_CHECK_LAUNCH();
  return launch_replay<R, SEARCH, VEC>(a, s);
}

template <int M, int GS, int CAP, bool SEARCH, int NT, int VEC>
int launch_two(const KnnArgs& a, cudaStream_t s) {
  const size_t smem = std::max<size_t>(
      two_smem(a.d, a.kp, a.qt, NT, CAP, a.stages, VEC, M == 1, SEARCH, a.nc).total, 120 * 1024);
  BGPU_CUDA((allow_max_smem(k_knn_two<M, GS, CAP, SEARCH, NT, VEC>)));
  k_knn_two<M, GS, CAP, SEARCH, NT, VEC>
      <<<(unsigned)ceil_div(a.q.n, a.qt), kTwoThreads, smem, s>>>(a);
  BGPU_CHECK_LAUNCH();
  return launch_replay<CAP <= 96 ? 1 : 2, SEARCH, VEC>(a, s);
}

// Dynamic shared memory beside the kernels' static part.
size_t knn_smem_limit() { return (size_t)device_smem_optin() - 4096; }

// 128-candidate tiles where they fit with 128 queries, else 64; then the most
// queries per CTA (128, 64, 32) that fit and leave no SM idle. bytes(qt, nt):
// the kernel's shared memory. Returns nt, 0 where nothing fits.
template <typename F>
uint32_t choose_shape(KnnArgs* a, F bytes) {
  const size_t limit = knn_smem_limit();
  const uint32_t nt = bytes(128, 128) <= limit ? 128u : 64u;
  for (a->qt = 128; a->qt > 32; a->qt /= 2)
    if (bytes(a->qt, nt) <= limit && ceil_div(a->q.n, a->qt) >= (uint64_t)num_sms()) break;
  return bytes(a->qt, nt) <= limit ? nt : 0u;
}

template <int M, int GS, int CAP, bool SEARCH>
int launch_two_shape(KnnArgs a, cudaStream_t s) {
  const int vec = row_vec(a);
  auto bytes = [&](uint32_t qt, uint32_t n, uint32_t stages) {
    return (size_t)two_smem(a.d, a.kp, qt, n, CAP, stages, vec, M == 1, SEARCH, a.nc).total;
  };
  const uint32_t nt =
      choose_shape(&a, [&](uint32_t qt, uint32_t n) { return bytes(qt, n, 2); });
  BGPU_REQUIRE(nt, BGPU_ERR_UNSUPPORTED,
               "nearest rows: the queues do not fit one CTA's shared memory");
  for (a.stages = 4; a.stages > 2 && bytes(a.qt, nt, a.stages) > knn_smem_limit();) --a.stages;
  if (nt == 128)
    return vec == 4   ? launch_two<M, GS, CAP, SEARCH, 128, 4>(a, s)
           : vec == 2 ? launch_two<M, GS, CAP, SEARCH, 128, 2>(a, s)
                      : launch_two<M, GS, CAP, SEARCH, 128, 1>(a, s);
  return vec == 4   ? launch_two<M, GS, CAP, SEARCH, 64, 4>(a, s)
         : vec == 2 ? launch_two<M, GS, CAP, SEARCH, 64, 2>(a, s)
                    : launch_two<M, GS, CAP, SEARCH, 64, 1>(a, s);
}

template <int R, bool SEARCH>
int launch_one_shape(KnnArgs a, cudaStream_t s) {
  const uint32_t nt = choose_shape(&a, [&](uint32_t qt, uint32_t n) {
    return (size_t)knn_smem(a.kp, qt, n, R, SEARCH, a.nc).total;
  });
  BGPU_REQUIRE(nt, BGPU_ERR_UNSUPPORTED,
               "nearest rows: the lists do not fit one CTA's shared memory");
  const int vec = row_vec(a);
  if (nt == 128)
    return vec == 4   ? launch_one<R, SEARCH, 128, 4>(a, s)
           : vec == 2 ? launch_one<R, SEARCH, 128, 2>(a, s)
                      : launch_one<R, SEARCH, 128, 1>(a, s);
  return vec == 4   ? launch_one<R, SEARCH, 64, 4>(a, s)
         : vec == 2 ? launch_one<R, SEARCH, 64, 2>(a, s)
                    : launch_one<R, SEARCH, 64, 1>(a, s);
}

// Lists of up to 64 entries take the two passes (bounds per thread and queue
// room by the size: the queue holds twice the entries and more); longer ones
// would need bounds past a thread's registers and update their lists.
template <bool SEARCH>
int launch_lists(const KnnArgs& a, cudaStream_t s) {
  constexpr int G = SEARCH ? 1 : 4;
  if (a.size == 1) return launch_two_shape<1, 8, 64, SEARCH>(a, s);
  if (a.size <= 24) return launch_two_shape<8, G, 96, SEARCH>(a, s);
  if (a.size <= 40) return launch_two_shape<12, G, 128, SEARCH>(a, s);
  if (a.size <= 64) return launch_two_shape<20, G, 160, SEARCH>(a, s);
  if constexpr (SEARCH)  // at most 128 neighbours
    return launch_one_shape<4, SEARCH>(a, s);
  else
    return a.size <= 128 ? launch_one_shape<4, SEARCH>(a, s) : launch_one_shape<8, SEARCH>(a, s);
}

// The lists of what is computed again. Groups from one per SM on: where every list
// is computed again they pay from 1,800 cells (2,700 cells: 0.50 ms against 0.65,
// 4,500: 0.69 against 1.31), but k_knn_all's two launches cost every call ~8 us.
int set_replay(KnnArgs* a, uint32_t* mem, cudaStream_t s) {
  a->counts = mem;
  a->replay = mem + 2;
  const uint64_t groups = ceil_div(a->q.n, kAllQueries);
  a->groups = groups >= (uint64_t)num_sms() ? mem + 2 + a->q.n : nullptr;
  a->wide = mem + 2 + a->q.n + 2 * groups;
  BGPU_CUDA(cudaMemsetAsync(mem, 0, 8, s));
  return BGPU_OK;
}

}  // namespace

uint32_t knn_kp(uint32_t d) { return (d + kNormCols + 15u) & ~15u; }

size_t knn_operand_bytes(uint64_t n, uint32_t d) {
  const uint64_t groups = ceil_div(n, 32) * 4;
  return groups * group_bytes(knn_kp(d)) + round_up(n * 4, 256) + groups * 4;
}

int knn_prepare(KnnOperand* op, const float* rows, const float* norms, uint64_t n, uint32_t d,
                void* mem, cudaStream_t s) {
  const uint64_t groups = ceil_div(n, 32) * 4;
  op->rows = rows;
  op->norms = norms;
  op->n = n;
  op->tiles = static_cast<unsigned char*>(mem);
  op->length = reinterpret_cast<float*>(op->tiles + groups * group_bytes(knn_kp(d)));
  op->gmax = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(op->length) +
                                      round_up(n * 4, 256));
  k_knn_split<<<(unsigned)ceil_div(n, 32), 256, 32 * (d + 1) * 4, s>>>(
      rows, norms, n, d, knn_kp(d), op->tiles, op->length, op->gmax);
  BGPU_CHECK_LAUNCH();
  return BGPU_OK;
}

size_t knn_replay_bytes(uint64_t n) { return (2 + n + 3 * ceil_div(n, kAllQueries)) * 4; }

int knn_tc_nearest(const KnnOperand& queries, const KnnOperand& cand, uint32_t d, uint32_t count,
                   const uint64_t* coff, uint32_t* replay, uint32_t* out_id, float* out_d,
                   int* err, cudaStream_t s) {
  KnnArgs a{};
  a.q = queries;
  a.c = cand;
  a.d = d;
  a.kp = knn_kp(d);
  a.size = count;
  a.coff = coff;
  a.nc = (uint32_t)cand.n;
  BGPU_TRY(set_replay(&a, replay, s));
  a.out_id = out_id;
  a.out_d = out_d;
  a.err = err;
  return launch_lists<false>(a, s);
}

int knn_tc_search(const KnnOperand& cells, uint32_t d, const uint64_t* coff, uint32_t nc,
                  const uint32_t* nearest, uint32_t cs, uint32_t k, const uint32_t* id_map,
                  uint32_t* replay, uint32_t* out_id, float* out_d, int* err, cudaStream_t s) {
  KnnArgs a{};
  a.q = cells;
  BGPU_TRY(set_replay(&a, replay, s));
  a.c = cells;
  a.d = d;
  a.kp = knn_kp(d);
  a.size = k;
  a.coff = coff;
  a.nc = nc;
  a.cs = cs;
  a.nearest = nearest;
  a.id_map = id_map;
  a.out_id = out_id;
  a.out_d = out_d;
  a.err = err;
  return launch_lists<true>(a, s);
}

}  // namespace bgpu
