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
// k_knn_replay computes it again, every candidate in the reference's order.
// (The k-means E step keeps the reference's order itself: its cells have no
// clusters yet, and lists of one entry tighten at once.)
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
// per pair of a 32-column TMEM load, and the exact work is proportional to
// the list's replacements. 300k x 50 dims, 2,191 clusters, 64 searched, 20
// neighbours: search 36.7 -> 15.1 ms, nearest clusters 20.9 -> 10.6 ms; the
// E step against 2,191 centroids 6.07 -> 1.52 ms. What bounds it now is the
// latency of the exact evaluations (a tile waits for its slowest warp).
//
// Shape: 512 threads, one CTA per SM, kQT queries (rows of the MMA), tiles of
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

struct KnnArgs {
  KnnOperand q, c;
  uint32_t d, kp, qt, size;
  // the cells' clusters: the search, and nearest for cells sorted by cluster
  // (nullptr: the tiles go in order and ties need no replay)
  const uint64_t* coff;
  uint32_t nc, cs;
  const uint32_t* nearest;
  const uint32_t* id_map;
  uint32_t* out_id;
  float* out_d;
  uint32_t* replay;  // [0]: number of queries to replay, [1..]: the queries
  int* err;
};

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
#pragma unroll 4
    for (uint32_t j = 0; j < d; j += 4) {
      const float4 a = *(const float4*)(x + j), b = *(const float4*)(c + j);
      acc = fmaf(a.x, b.x, acc);
      acc = fmaf(a.y, b.y, acc);
      acc = fmaf(a.z, b.z, acc);
      acc = fmaf(a.w, b.w, acc);
    }
  } else if constexpr (VEC == 2) {
#pragma unroll 5
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
  __shared__ uint32_t wsum[kTcKnnWarps], s_union, s_slots;
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
  }
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
  if constexpr (SEARCH) {
    const uint32_t words = (a.nc + 31) / 32;
    uint32_t* rank = bitmap + words;
    for (uint32_t w = tid; w < words; w += kTcKnnThreads) bitmap[w] = 0u;
    __syncthreads();
    for (uint32_t t = tid; t < nq * a.cs; t += kTcKnnThreads) {
      const uint32_t lab = a.nearest[q0 * a.cs + t];
      if (lab < a.nc) atomicOr(&bitmap[lab >> 5], 1u << (lab & 31));  // order-free
    }
    __syncthreads();
    // rank of each word: the searched clusters before it
    const uint32_t per = (words + kTcKnnThreads - 1) / kTcKnnThreads;
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
    if (tid == kTcKnnThreads - 1) s_union = pre;
    __syncthreads();
    nbits = s_union;
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
  float trun = -INFINITY;  // lists of one entry: the best approximate value, less margins

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

  uint32_t gt = 0;  // tiles so far: buffers and phases
  uint32_t ubase = 0;
  bool ok = true;
  do {
    uint32_t nruns = 1, nslots;
    if constexpr (SEARCH) {
      // the next kUnionCap searched clusters in label order: their rows, and
      // which queries search them
      const uint32_t words = (a.nc + 31) / 32;
      const uint32_t* rank = bitmap + words;
      nruns = min(kUnionCap, nbits - ubase);
      for (uint32_t t = tid; t < nruns * 4; t += kTcKnnThreads) qmask[t] = 0u;
      __syncthreads();
      for (uint32_t w = tid; w < words; w += kTcKnnThreads) {
        uint32_t bits = bitmap[w], pos = rank[w];
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
      for (uint32_t t = tid; t < nq * a.cs; t += kTcKnnThreads) {
        const uint32_t lab = a.nearest[q0 * a.cs + t], q = t / a.cs;
        if (lab >= a.nc) continue;
        const uint32_t pos =
            rank[lab >> 5] + __popc(bitmap[lab >> 5] & ((1u << (lab & 31)) - 1u));
        if (pos >= ubase && pos - ubase < nruns)
          atomicOr(&qmask[(pos - ubase) * 4 + (q >> 5)], 1u << (q & 31));
      }
    } else if (tid == 0) {
      run_b[0] = 0u;
      run_e[0] = (uint32_t)a.c.n;
    }
    __syncthreads();
    if (wid == 0) {  // first slot of every run
      uint32_t total = 0;
      for (uint32_t u0 = 0; u0 < nruns; u0 += 32) {
        const uint32_t u = u0 + lane;
        uint32_t g = 0;
        if (u < nruns && run_e[u] > run_b[u]) g = (run_e[u] + 7) / 8 - run_b[u] / 8;
        uint32_t incl = g;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += v;
        }
        if (u < nruns) run_s[u] = total + incl - g;
        total += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (lane == 0) {
        run_s[nruns] = total;
        s_slots = total;
      }
    }
    __syncthreads();
    nslots = s_slots;
    const uint32_t ntiles = (nslots + SLOTS - 1) / SLOTS;
    // the tile that step t works on: from the own cluster's on, around
    uint32_t t0 = 0;
    if (a.coff && ntiles) {
      uint32_t slot = own / 8;  // nearest: the own centroid's group
      if constexpr (SEARCH) {
        const uint32_t* rank = bitmap + (a.nc + 31) / 32;
        const uint32_t pos =
            rank[own >> 5] + __popc(bitmap[own >> 5] & ((1u << (own & 31)) - 1u));
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
            float lim = thr[qi] - mg;
            float top = v[0];  // most threads have nothing above the limit
#pragma unroll
            for (int j = 1; j + 1 < CW; j += 2) top = max3_nan(top, v[j], v[j + 1]);
            top = max3_nan(top, v[CW - 1], top);
            if (!SEARCH && R == 1 && a.size == 1) {
              // one entry: the best approximate value so far bounds it too
              trun = fmaxf(trun, top - 2.f * mg);
              lim = fmaxf(lim, trun - mg);
            }
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

  if (ok) {
    // what is left in the queues, then the sorted lists
    for (uint32_t q = wid; q < nq; q += kTcKnnWarps) {
      const uint32_t cnt = qcnt[q];
      if (cnt) evaluate(q, cnt);
      write_sorted(ld + q * R * 32, li + q * R * 32, a.size, SEARCH ? a.id_map : nullptr,
                   a.out_d + (q0 + q) * a.size, a.out_id + (q0 + q) * a.size, lane);
      if (a.coff && lane == 0) {
        float w = ld[q * R * 32];
        for (uint32_t e = 1; e < a.size; ++e) w = fmaxf(w, ld[q * R * 32 + e]);
        if (qnext[q] == w) a.replay[1 + atomicAdd(a.replay, 1u)] = (uint32_t)(q0 + q);
      }
    }
  } else if (tid == 0) {
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
  tc_fence_after();
  if (wid == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                 ::"r"(tmem), "n"(2 * NT)
                 : "memory");
  }
}

// The queries in replay[1..replay[0]], a warp each: every candidate evaluated
// and offered in the reference's order.
constexpr int kReplayThreads = 128;
template <int R, bool SEARCH, int VEC>
__global__ void __launch_bounds__(kReplayThreads) k_knn_replay(const KnnArgs a) {
  __shared__ float rd[kReplayThreads / 32][R * 32];
  __shared__ uint32_t ri[kReplayThreads / 32][R * 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t count = a.replay[0], d = a.d;
  for (uint32_t i = blockIdx.x * (kReplayThreads / 32) + wid; i < count;
       i += gridDim.x * (kReplayThreads / 32)) {
    const uint64_t q = a.replay[1 + i];
    const float* x = a.q.rows + q * d;
    const float nm = SEARCH ? a.q.norms[q] : 0.f;
    for (uint32_t e = lane; e < R * 32; e += 32) {
      rd[wid][e] = e < a.size ? FLT_MAX : -INFINITY;
      ri[wid][e] = 0xFFFFFFFFu;
    }
    __syncwarp();
    WarpList<R> best;
    best.load(rd[wid], ri[wid], lane);
    auto offer_rows = [&](uint64_t b, uint64_t e) {
      for (uint64_t r0 = b; r0 < e; r0 += 32) {
        const uint64_t row = r0 + lane;
        const bool use = row < e && !(SEARCH && row == q);
        float dist = INFINITY;
        if (use) {
          const float pd = fmaf(-2.f, row_dot<VEC>(x, a.c.rows + row * d, d), a.c.norms[row]);
          dist = SEARCH ? nm + pd : pd;
        }
        best.offer(dist, (uint32_t)row, __ballot_sync(0xffffffffu, use), lane, 0.f);
      }
    };
    if constexpr (SEARCH) {
      uint32_t lab[8];  // the searched clusters, ascending: the least above the last
#pragma unroll
      for (int u = 0; u < 8; ++u)
        lab[u] = lane + 32u * u < a.cs ? a.nearest[q * a.cs + lane + 32u * u] : 0xFFFFFFFFu;
      uint32_t from = 0;
      while (true) {
        uint32_t m = 0xFFFFFFFFu;
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (lab[u] >= from) m = min(m, lab[u]);
        m = __reduce_min_sync(0xffffffffu, m);
        if (m >= a.nc) break;
        offer_rows(a.coff[m], a.coff[m + 1]);
        from = m + 1;
      }
    } else {
      offer_rows(0, a.c.n);
    }
    best.store(rd[wid], ri[wid], lane);
    __syncwarp();
    write_sorted(rd[wid], ri[wid], a.size, SEARCH ? a.id_map : nullptr, a.out_d + q * a.size,
                 a.out_id + q * a.size, lane);
    __syncwarp();
  }
}

template <int R, bool SEARCH, int NT, int VEC>
int launch_knn(const KnnArgs& a, cudaStream_t s) {
  // at least 120 KB so that one CTA (and one TMEM allocation) runs per SM
  const size_t smem =
      std::max<size_t>(knn_smem(a.kp, a.qt, NT, R, SEARCH, a.nc).total, 120 * 1024);
  BGPU_CUDA((allow_max_smem(k_knn_tc<R, SEARCH, NT, VEC>)));
  k_knn_tc<R, SEARCH, NT, VEC>
      <<<(unsigned)ceil_div(a.q.n, a.qt), kTcKnnThreads, smem, s>>>(a);
  BGPU_CHECK_LAUNCH();
  if (a.coff) {
    k_knn_replay<R, SEARCH, VEC><<<num_sms() * 4, kReplayThreads, 0, s>>>(a);
    BGPU_CHECK_LAUNCH();
  }
  return BGPU_OK;
}

template <int R, bool SEARCH, int NT>
int launch_vec(const KnnArgs& a, cudaStream_t s) {
  const uintptr_t at = (uintptr_t)a.q.rows | (uintptr_t)a.c.rows;
  if (a.d % 4 == 0 && at % 16 == 0) return launch_knn<R, SEARCH, NT, 4>(a, s);
  if (a.d % 2 == 0 && at % 8 == 0) return launch_knn<R, SEARCH, NT, 2>(a, s);
  return launch_knn<R, SEARCH, NT, 1>(a, s);
}

// 128-candidate tiles where they fit with 128 queries' lists, else 64; then
// the most queries per CTA (128, 64, 32) that fit and leave no SM idle.
template <int R, bool SEARCH>
int launch_shape(KnnArgs a, cudaStream_t s) {
  const size_t limit = (size_t)device_smem_optin() - 2048;
  const bool wide = knn_smem(a.kp, 128, 128, R, SEARCH, a.nc).total <= limit;
  const uint32_t nt = wide ? 128u : 64u;
  for (a.qt = 128; a.qt > 32; a.qt /= 2)
    if (knn_smem(a.kp, a.qt, nt, R, SEARCH, a.nc).total <= limit &&
        ceil_div(a.q.n, a.qt) >= (uint64_t)num_sms())
      break;
  BGPU_REQUIRE(knn_smem(a.kp, a.qt, nt, R, SEARCH, a.nc).total <= limit, BGPU_ERR_UNSUPPORTED,
               "nearest rows: the lists do not fit one CTA's shared memory");
  return wide ? launch_vec<R, SEARCH, 128>(a, s) : launch_vec<R, SEARCH, 64>(a, s);
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
  a.replay = replay;
  if (coff) BGPU_CUDA(cudaMemsetAsync(replay, 0, 4, s));
  a.out_id = out_id;
  a.out_d = out_d;
  a.err = err;
  if (count <= 32) return launch_shape<1, false>(a, s);
  if (count <= 64) return launch_shape<2, false>(a, s);
  if (count <= 128) return launch_shape<4, false>(a, s);
  return launch_shape<8, false>(a, s);
}

int knn_tc_search(const KnnOperand& cells, uint32_t d, const uint64_t* coff, uint32_t nc,
                  const uint32_t* nearest, uint32_t cs, uint32_t k, const uint32_t* id_map,
                  uint32_t* replay, uint32_t* out_id, float* out_d, int* err, cudaStream_t s) {
  KnnArgs a{};
  BGPU_CUDA(cudaMemsetAsync(replay, 0, 4, s));
  a.replay = replay;
  a.q = cells;
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
  if (k <= 32) return launch_shape<1, true>(a, s);
  if (k <= 64) return launch_shape<2, true>(a, s);
  return launch_shape<4, true>(a, s);
}

}  // namespace bgpu
