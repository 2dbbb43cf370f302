// Per-gene statistics for highly-variable-gene selection, the inputs of
// brisc's HVG step (brisc/hvg.pyx): gene means, variances and nonzero counts
// of the raw counts (gene_mean_and_variance_csr/_csc, hvg.pyx:9-252), and the
// per-gene sums and squared sums of counts clipped at a per-gene value
// (clipped_sum_csr/_csc, hvg.pyx:255-530).
//
// Exactness: every count is cast to uint64 as the reference casts it
// (`<unsigned long long> data[i]`), and the sums, squared sums and counts are
// integer sums, so their totals do not depend on the order of accumulation:
// shared-memory and global 64-bit atomics give the reference's integers
// exactly. The float outputs then follow the reference's expressions with
// every rounding written out (no contraction left to the compiler):
//   mean = float(sum) * inv_num_cells
//   var  = float(double(inv_num_pairs) * (double(n) * double(sumsq) -
//                                         double(sum) * double(sum)))
//   batch_counts_sum         = fma(float(out), clip, float(sum))
//   squared_batch_counts_sum = fma(float(out), clip * clip, float(sumsq))
// The last two are the forms the reference's -Ofast build computes (an FMA,
// and clip * clip associated first); the oracle's tests pin them against the
// compiled reference.
//
// Indices are checked: a gene or cell index outside its range, or an indptr
// that is not a valid range, sets an error word and the entry is skipped
// (the reference does not check; here the call returns BGPU_ERR_INVALID).
#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace bgpu {
namespace {

enum : int { kMeanVar = 0, kClipped = 1 };

constexpr int kHvgThreads = 512;
// CSR: threads of a CTA, the values that take its shared 32-bit accumulators
// (larger ones add to the 64-bit totals in global memory), the shared bytes a
// gene needs (three words), and the loads a lane keeps in flight.
constexpr int kCsrThreads = 1024;
constexpr uint32_t kCsrSmall = 15;
constexpr uint32_t kCsrGeneBytes = 12;
constexpr int kCsrUnroll = 8;
constexpr int kCsrRows = 4;        // listed rows a warp reads at once
constexpr uint32_t kCsrMaxSlices = 8;
// Most contributions a CTA may add to one gene: each adds at most 15^2 to a
// 32-bit sum of squares.
constexpr uint64_t kCsrMaxPerGene = 0xFFFFFFFFull / (kCsrSmall * kCsrSmall);
// Sampled values, of one per thread, above kCsrSmall from which on a CTA counts
// carries instead. 12M entries of 2,000 genes, both statistics, us without and with
// carries: 0.3 % large 258, 249; 2.3 % 262, 228; 5.3 % 311, 233; 23 % 448, 231; all
// 1,078, 227. 45M entries of 20,000 genes: 0.1 % 489, 507; 1.6 % 499, 504; 4.1 % 517,
// 506; all 1,502, 472.
constexpr int kCsrManyLarge = kCsrThreads / 64;

// `<unsigned long long> x` of the reference, per stored value type. Signed
// integers wrap modulo 2^64; floating values are truncated toward zero
// (counts are non-negative).
__device__ __forceinline__ unsigned long long as_u64(uint16_t x) { return x; }
__device__ __forceinline__ unsigned long long as_u64(uint32_t x) { return x; }
__device__ __forceinline__ unsigned long long as_u64(int32_t x) {
  return (unsigned long long)(long long)x;
}
__device__ __forceinline__ unsigned long long as_u64(int64_t x) {
  return (unsigned long long)x;
}
__device__ __forceinline__ unsigned long long as_u64(uint64_t x) { return x; }
__device__ __forceinline__ unsigned long long as_u64(float x) {
  return __float2ull_rz(x);
}
__device__ __forceinline__ unsigned long long as_u64(double x) {
  return __double2ull_rz(x);
}

// The count as 32 bits when it is below 65536 (every real count); false for
// anything else, which goes through as_u64.
template <typename V>
__device__ __forceinline__ bool small_count(V x, uint32_t& w) {
  w = (uint32_t)x;
  if constexpr (std::is_floating_point<V>::value)
    return x >= V(0) && x < V(65536);
  else
    return (unsigned long long)(long long)x < 65536ull;
}

// acc = [sum | sumsq | count] x g, 64-bit. kMeanVar: count = stored entries.
// kClipped: values above the clip value only count (hvg.pyx:298-303); the
// comparison converts the integer to float, as C's `value > clip_val[gene]`.
template <int MODE>
__device__ __forceinline__ void add_total(unsigned long long* acc, uint32_t g, uint32_t gene,
                                          unsigned long long v, float clip) {
  if (MODE == kClipped && __ull2float_rn(v) > clip) {
    atomicAdd(acc + 2ull * g + gene, 1ull);
    return;
  }
  atomicAdd(acc + gene, v);
  atomicAdd(acc + (uint64_t)g + gene, v * v);
  if (MODE == kMeanVar) atomicAdd(acc + 2ull * g + gene, 1ull);
}

// The totals that a CSR CTA's three words of a gene stand for.
struct WordTotals {
  unsigned long long s, s2, c;
};
template <int MODE>
__device__ __forceinline__ WordTotals word_totals(uint32_t w0, uint32_t w1, uint32_t w2) {
  if (MODE == kMeanVar) return {w0 + w1, w0 + w1 + 2u * w2, w0};  // modulo 2^32
  return {w0, w1, w2};
}

// CSR input: one entry, a count of gene `gene`, whose shared words are
// sw[0..2][j] when the CTA owns the gene. Three 32-bit integer additions at
// most: kMeanVar keeps the entries, sum (v - 1) and sum v (v - 1) / 2 (all
// modulo 2^32; a count of 1, most of them, adds to the first word only),
// kClipped the sums, the sums of squares and the number of clipped entries.
template <typename V, int MODE>
__device__ __forceinline__ void csr_entry(uint32_t* sw, uint32_t gs, uint32_t j, V x, float clip,
                                          unsigned long long* acc, uint32_t g, uint32_t gene) {
  uint32_t w;
  const bool small = small_count(x, w);
  if (small && w <= kCsrSmall) {
    if (MODE == kClipped) {
      if ((float)w > clip) {
        atomicAdd(sw + 2 * gs + j, 1u);
      } else {
        atomicAdd(sw + j, w);
        atomicAdd(sw + gs + j, w * w);
      }
    } else {
      atomicAdd(sw + j, 1u);
      if (w != 1u) {
        atomicAdd(sw + gs + j, w - 1u);
        atomicAdd(sw + 2 * gs + j, w * (w - 1u) / 2u);
      }
    }
    return;
  }
  add_total<MODE>(acc, g, gene, small ? (unsigned long long)w : as_u64(x), clip);
}

// The same for counts that are mostly larger (reads rather than molecules): the
// words keep the low halves of the sums (kMeanVar: entries, sum, sum of squares),
// whatever the counts below 65536, and an addition that wraps its word puts the
// carry into the 64-bit total. An addition whose old value is wanted takes longer
// than one without, so this is not the rule.
__device__ __forceinline__ void add_carry(uint32_t* word, uint32_t v, unsigned long long* total) {
  if (atomicAdd(word, v) + v < v) atomicAdd(total, 1ull << 32);
}
template <typename V, int MODE>
__device__ __forceinline__ void csr_entry_carry(uint32_t* sw, uint32_t gs, uint32_t j, V x,
                                                float clip, unsigned long long* acc, uint32_t g,
                                                uint32_t gene) {
  uint32_t w;
  if (!small_count(x, w)) {
    add_total<MODE>(acc, g, gene, as_u64(x), clip);
    return;
  }
  uint32_t* sums = MODE == kMeanVar ? sw + gs : sw;
  if (MODE == kClipped && (float)w > clip) {
    atomicAdd(sw + 2 * gs + j, 1u);
    return;
  }
  if (MODE == kMeanVar) atomicAdd(sw + j, 1u);
  add_carry(sums + j, w, acc + gene);
  add_carry(sums + gs + j, w * w, acc + (uint64_t)g + gene);
}

// CSR input. A CTA owns the genes [slice * gs, ...) of one of `slices` equal
// runs of genes and one of the launch's chunks of the entries (cells ==
// nullptr: a contiguous share of [range[0], range[1])) or of the listed cells
// (a warp per cell, lanes over its row). It sums them in shared 32-bit words,
// whose additions the hardware does in shared memory; a 64-bit addition there
// is a compare-and-swap loop, and one in global memory costs a trip to L2 per
// entry: 40k x 20,000, 38M float32 entries, 0.98 ms with 64-bit additions in
// global memory, 0.12 ms. A CTA that samples many counts above kCsrSmall keeps
// carries (csr_entry_carry). The words go to part[chunk][3][g] and
// k_hvg_finish adds the chunks. Slices of one chunk are neighbouring CTAs,
// so that all but the first find the entries in L2.
// No word overflows: at most kCsrMaxPerGene entries of a gene are added before
// the words are taken out. The launch bounds a chunk of entries; listed rows
// go in epochs of `epoch` rows, after each of which but the last the words are
// added to the 64-bit totals, and a row longer than g, which repeats genes,
// goes straight to those.
// gs == 0: no shared words, every entry goes to the 64-bit totals (more genes
// than kCsrMaxSlices CTAs hold, where re-reading the entries costs more).
template <typename V, typename I, int MODE>
__global__ void __launch_bounds__(kCsrThreads)
k_hvg_csr(const V* __restrict__ data, const I* __restrict__ indices,
          const I* __restrict__ indptr, uint64_t nnz, uint64_t num_rows,
          const int64_t* __restrict__ range, const int64_t* __restrict__ cells,
          uint64_t num_listed, uint64_t epoch, uint32_t g, uint32_t gs, uint32_t slices,
          const float* __restrict__ clip, unsigned long long* __restrict__ acc,
          uint32_t* __restrict__ part, int* __restrict__ err) {
  extern __shared__ uint32_t sw[];  // [3][gs]
  const uint32_t chunk = blockIdx.x / slices, slice = blockIdx.x % slices;
  const uint32_t nchunks = gridDim.x / slices;
  const uint32_t g0 = slice * gs, gn = gs ? min(g, g0 + gs) - g0 : g;
  // the CTA's entries, or its listed cells
  const uint64_t first = range ? (uint64_t)range[0] : 0ull;
  const uint64_t len = cells ? num_listed : (range ? (uint64_t)range[1] : nnz) - first;
  const uint64_t per = (len + nchunks - 1) / nchunks;
  const uint64_t c0 = first + min_u64(len, per * chunk);
  const uint64_t c1 = first + min_u64(len, per * (chunk + 1));
  // a value per thread, to see whether many are large
  V one = V(0);
  if (gs && c0 < c1) {
    if (cells == nullptr) {
      if (c0 + threadIdx.x < c1) one = data[c0 + threadIdx.x];  // read again soon
    } else {
      const long long cell = cells[c0 + (c1 - c0) * threadIdx.x / kCsrThreads];
      if (cell >= 0 && (uint64_t)cell < num_rows) {
        const long long b = (long long)indptr[cell], e = (long long)indptr[cell + 1];
        if (b >= 0 && e > b && (uint64_t)e <= nnz) one = data[b + (e - b) * (threadIdx.x & 31) / 32];
      }
    }
  }
  for (uint32_t i = threadIdx.x; i < 3 * gs; i += kCsrThreads) sw[i] = 0u;
  uint32_t w = 0;
  const bool carry =  // the same in every thread of the CTA
      __syncthreads_count(!(small_count(one, w) && w <= kCsrSmall)) >= kCsrManyLarge;
  auto entry = [&](I gi, V x) {
    const long long gene = (long long)gi;
    if (gene < 0 || gene >= (long long)g) {
      *err = 1;
      return;
    }
    const uint32_t j = (uint32_t)gene - g0;
    if (j >= gn) return;
    const float cv = MODE == kClipped ? clip[gene] : 0.f;
    if (!gs)
      add_total<MODE>(acc, g, (uint32_t)gene, as_u64(x), cv);
    else if (carry)
      csr_entry_carry<V, MODE>(sw, gs, j, x, cv, acc, g, (uint32_t)gene);
    else
      csr_entry<V, MODE>(sw, gs, j, x, cv, acc, g, (uint32_t)gene);
  };
  auto totals = [&](uint32_t w0, uint32_t w1, uint32_t w2) -> WordTotals {
    if (carry && MODE == kMeanVar) return {w1, w2, w0};
    return word_totals<MODE>(w0, w1, w2);
  };
  if (cells == nullptr) {
    for (uint64_t i0 = c0 + threadIdx.x; i0 < c1; i0 += (uint64_t)kCsrThreads * kCsrUnroll) {
      I gi[kCsrUnroll];
      V x[kCsrUnroll];
#pragma unroll
      for (int u = 0; u < kCsrUnroll; ++u) {
        const uint64_t i = i0 + (uint64_t)u * kCsrThreads;
        gi[u] = i < c1 ? indices[i] : I(0);
        x[u] = i < c1 ? data[i] : V(0);
      }
#pragma unroll
      for (int u = 0; u < kCsrUnroll; ++u)
        if (i0 + (uint64_t)u * kCsrThreads < c1) entry(gi[u], x[u]);
    }
  } else {
    const int lane = threadIdx.x & 31;
    for (uint64_t s0 = c0; s0 < c1; s0 += epoch) {
      const uint64_t s1 = min_u64(c1, s0 + epoch);
      // kCsrRows cells per round of a warp: a lane reads each cell's range,
      // then the warp walks the rows
      for (uint64_t r0 = s0 + (threadIdx.x >> 5) * kCsrRows; r0 < s1;
           r0 += (kCsrThreads / 32) * kCsrRows) {
        long long b = 0, e = 0;
        if (lane < kCsrRows && r0 + lane < s1) {
          const long long cell = cells[r0 + lane];
          if (cell < 0 || (uint64_t)cell >= num_rows) {
            *err = 1;
          } else {
            b = (long long)indptr[cell];
            e = (long long)indptr[cell + 1];
            if (b < 0 || e < b || (uint64_t)e > nnz) {
              *err = 1;
              b = e = 0;
            }
          }
        }
        for (int r = 0; r < kCsrRows; ++r) {
          const uint64_t rb = (uint64_t)__shfl_sync(0xffffffffu, b, r);
          const uint64_t re = (uint64_t)__shfl_sync(0xffffffffu, e, r);
          if (re - rb > min_u64(g, kCsrMaxPerGene)) {  // repeats genes
            for (uint64_t i = rb + lane; i < re; i += 32) {
              const long long gene = (long long)indices[i];
              if (gene < 0 || gene >= (long long)g)
                *err = 1;
              else if ((uint32_t)gene - g0 < gn)
                add_total<MODE>(acc, g, (uint32_t)gene, as_u64(data[i]),
                                MODE == kClipped ? clip[gene] : 0.f);
            }
            continue;
          }
          for (uint64_t i0 = rb + lane; i0 < re; i0 += 32 * kCsrRows) {
            I gi[kCsrRows];
            V x[kCsrRows];
#pragma unroll
            for (int u = 0; u < kCsrRows; ++u) {
              gi[u] = i0 + 32 * u < re ? indices[i0 + 32 * u] : I(0);
              x[u] = i0 + 32 * u < re ? data[i0 + 32 * u] : V(0);
            }
#pragma unroll
            for (int u = 0; u < kCsrRows; ++u)
              if (i0 + 32 * u < re) entry(gi[u], x[u]);
          }
        }
      }
      if (s1 < c1 && gs) {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < gn; i += kCsrThreads) {
          const uint32_t w0 = sw[i], w1 = sw[gs + i], w2 = sw[2 * gs + i];
          sw[i] = sw[gs + i] = sw[2 * gs + i] = 0u;
          if ((w0 | w1 | w2) == 0u) continue;
          const WordTotals t = totals(w0, w1, w2);
          atomicAdd(acc + g0 + i, t.s);
          atomicAdd(acc + (uint64_t)g + g0 + i, t.s2);
          atomicAdd(acc + 2ull * g + g0 + i, t.c);
        }
        __syncthreads();
      }
    }
  }
  if (!gs) return;
  __syncthreads();
  if (carry && MODE == kMeanVar)  // as the other form's words (the low halves)
    for (uint32_t i = threadIdx.x; i < gn; i += kCsrThreads) {
      const uint32_t c = sw[i], s = sw[gs + i], s2 = sw[2 * gs + i];
      sw[gs + i] = s - c;
      sw[2 * gs + i] = (s2 - s) / 2u;  // sum v (v - 1) is even
    }
  for (uint32_t w = 0; w < 3; ++w)
    for (uint32_t i = threadIdx.x; i < gn; i += kCsrThreads)
      part[((uint64_t)chunk * 3 + w) * g + g0 + i] = sw[w * gs + i];
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// CSC input. The stored entries are split evenly over the warps, whatever
// gene they belong to: a warp takes chunks of kCscChunk entries, finds the
// gene of the first by a binary search in indptr, and walks the genes that
// meet the chunk, lanes over each gene's part of it. The warp's integer sums
// of a gene are added to acc by 64-bit atomics (their totals do not depend on
// the order). A warp per gene instead leaves the chip to the few genes that
// hold most of the entries (the means of genes span orders of magnitude):
// 400k x 2000, 36M uint16 entries with a mask, 9.3 ms, the longest gene's
// serial loads; split by entries, kCscUnroll independent loads in flight per
// lane, 0.12 ms.
// The kernel first checks the ranges it reads: a gene whose range is not
// within [0, nnz] or decreases sets err, and the call fails.
constexpr uint32_t kCscChunk = 4096;
constexpr int kCscUnroll = 8;

template <typename I>
__global__ void __launch_bounds__(kHvgThreads)
k_hvg_check_ranges(const I* __restrict__ indptr, uint64_t nnz, uint32_t g,
                   int* __restrict__ err) {
  const uint64_t gene = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (gene >= g) return;
  const long long b = (long long)indptr[gene], e = (long long)indptr[gene + 1];
  if (b < 0 || e < b || (uint64_t)e > nnz) *err = 1;
}

template <typename V, typename I, int MODE>
__global__ void __launch_bounds__(kHvgThreads)
k_hvg_csc(const V* __restrict__ data, const I* __restrict__ indices,
          const I* __restrict__ indptr, uint32_t g, const int8_t* __restrict__ mask,
          uint64_t mask_len, const float* __restrict__ clip,
          unsigned long long* __restrict__ acc, int* __restrict__ err) {
  if (*err) return;  // k_hvg_check_ranges: the ranges are not increasing
  const int lane = threadIdx.x & 31;
  const uint64_t first = (uint64_t)indptr[0], last = (uint64_t)indptr[g];
  bool bad = false;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t c0 = first + kCscChunk *
                                 ((blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5);
       c0 < last; c0 += kCscChunk * nwarps) {
    const uint64_t c1 = c0 + kCscChunk < last ? c0 + kCscChunk : last;
    // the gene of entry c0: the largest one that starts at or before it
    uint32_t lo = 0, hi = g;
    while (hi - lo > 1) {
      const uint32_t mid = lo + (hi - lo) / 2;
      if ((uint64_t)indptr[mid] <= c0) lo = mid;
      else hi = mid;
    }
    for (uint64_t b = c0; b < c1; ++lo) {
      const uint64_t ge = (uint64_t)indptr[lo + 1];
      const uint64_t e = ge < c1 ? ge : c1;
      if (e <= b) continue;  // an empty gene
      const float cv = MODE == kClipped ? clip[lo] : 0.f;
      unsigned long long s = 0, s2 = 0;
      uint32_t c = 0;
      for (uint64_t i0 = b + lane; i0 < e; i0 += 32 * kCscUnroll) {
        V x[kCscUnroll];
        bool use[kCscUnroll];
        I cell[kCscUnroll];
#pragma unroll
        for (int u = 0; u < kCscUnroll; ++u) {  // every load before the first use
          use[u] = i0 + 32 * u < e;
          x[u] = use[u] ? data[i0 + 32 * u] : V(0);
          cell[u] = mask && use[u] ? indices[i0 + 32 * u] : I(0);
        }
        if (mask) {
          int8_t keep[kCscUnroll];
#pragma unroll
          for (int u = 0; u < kCscUnroll; ++u) {
            const bool in = cell[u] >= 0 && (uint64_t)cell[u] < mask_len;
            bad = bad || (use[u] && !in);
            keep[u] = in ? mask[cell[u]] : (int8_t)0;
          }
#pragma unroll
          for (int u = 0; u < kCscUnroll; ++u) use[u] = use[u] && keep[u] != 0;
        }
#pragma unroll
        for (int u = 0; u < kCscUnroll; ++u) {
          if (!use[u]) continue;
          uint32_t w;
          bool over;
          if (small_count(x[u], w)) {
            over = MODE == kClipped && (float)w > cv;
            if (!over) {
              s += w;
              s2 += (unsigned long long)w * w;
            }
          } else {
            const unsigned long long v = as_u64(x[u]);
            over = MODE == kClipped && __ull2float_rn(v) > cv;
            if (!over) {
              s += v;
              s2 += v * v;
            }
          }
          c += MODE == kMeanVar || over ? 1u : 0u;
        }
      }
      s = warp_sum_u64(s);
      s2 = warp_sum_u64(s2);
      c = __reduce_add_sync(0xffffffffu, c);
      if (lane == 0) {
        if (s) atomicAdd(acc + lo, s);
        if (s2) atomicAdd(acc + (uint64_t)g + lo, s2);
        if (c) atomicAdd(acc + 2ull * g + lo, (unsigned long long)c);
      }
      b = e;
    }
  }
  if (bad) *err = 1;
}

// Totals of the genes: acc (the 64-bit additions) plus, for CSR, the 32-bit
// words of the nchunks chunks, then the statistics. A block takes 32 genes, 8
// threads per gene over the chunks. Nothing is written when err is set.
//   mean and variance: hvg.pyx:66-70 / :246-250, every rounding explicit;
//   clipped sums: hvg.pyx:320-325 / :393-399, which the reference's -Ofast
//   build computes as fused multiply-adds, clip * clip rounded first.
template <int MODE>
__global__ void __launch_bounds__(256)
k_hvg_finish(const unsigned long long* __restrict__ acc, const uint32_t* __restrict__ part,
             uint32_t nchunks, uint32_t g, uint64_t num_cells, float inv_num_cells,
             float inv_num_pairs, const float* __restrict__ clip, float* __restrict__ out_a,
             float* __restrict__ out_b, uint32_t* __restrict__ nonzero_count,
             const int* __restrict__ err) {
  __shared__ unsigned long long sh[3][8][33];
  if (*err) return;
  const uint32_t lane = threadIdx.x & 31, row = threadIdx.x >> 5;
  const uint32_t gene = blockIdx.x * 32 + lane;
  unsigned long long s = 0, s2 = 0, c = 0;
  if (gene < g) {
#pragma unroll 4
    for (uint32_t r = row; r < nchunks; r += 8) {
      const uint32_t* p = part + (uint64_t)r * 3 * g + gene;
      const uint32_t w0 = p[0], w1 = p[g], w2 = p[2ull * g];
      const WordTotals t = word_totals<MODE>(w0, w1, w2);
      s += t.s;
      s2 += t.s2;
      c += t.c;
    }
  }
  sh[0][row][lane] = s;
  sh[1][row][lane] = s2;
  sh[2][row][lane] = c;
  __syncthreads();
  if (row != 0 || gene >= g) return;
  for (int r = 1; r < 8; ++r) {
    s += sh[0][r][lane];
    s2 += sh[1][r][lane];
    c += sh[2][r][lane];
  }
  s += acc[gene];
  s2 += acc[(uint64_t)g + gene];
  c += acc[2ull * g + gene];
  if (MODE == kMeanVar) {
    out_a[gene] = __fmul_rn(__ull2float_rn(s), inv_num_cells);
    const double sd = __ull2double_rn(s);
    const double d = __dsub_rn(__dmul_rn(__ull2double_rn(num_cells), __ull2double_rn(s2)),
                               __dmul_rn(sd, sd));
    out_b[gene] = __double2float_rn(__dmul_rn((double)inv_num_pairs, d));
    nonzero_count[gene] = (uint32_t)c;
  } else {
    const float out = __ull2float_rn(c), cv = clip[gene];
    out_a[gene] = __fmaf_rn(out, cv, __ull2float_rn(s));
    out_b[gene] = __fmaf_rn(out, __fmul_rn(cv, cv), __ull2float_rn(s2));
  }
}

// The entries a CSR call without a cell list sums: rows [0, rows) of indptr.
// A range outside [0, nnz] sets err to 2.
template <typename I>
__global__ void k_hvg_range(const I* __restrict__ indptr, uint64_t rows, uint64_t nnz,
                            int64_t* __restrict__ range, int* __restrict__ err) {
  const int64_t b = (int64_t)indptr[0], e = (int64_t)indptr[rows];
  const bool ok = b >= 0 && e >= b && (uint64_t)e <= nnz;
  range[0] = ok ? b : 0;
  range[1] = ok ? e : 0;
  if (!ok) *err = 2;
}

}  // namespace
}  // namespace bgpu

namespace bgpu {
namespace {

struct Scratch {  // stream-ordered device buffer, freed on the same stream
  void* p = nullptr;
  cudaStream_t s = nullptr;
  ~Scratch() { if (p) cudaFreeAsync(p, s); }
  int alloc(size_t bytes, cudaStream_t stream) {
    s = stream;
    cudaError_t e = scratch_alloc(&p, std::max<size_t>(bytes, 16), stream);
    if (e != cudaSuccess) {
      p = nullptr;
      set_error(std::string("cudaMalloc(") + std::to_string(bytes) +
                ") failed: " + cudaGetErrorString(e));
      return BGPU_ERR_ALLOC;
    }
    return BGPU_OK;
  }
};

size_t hvg_value_size(int t) {
  switch (t) {
    case BGPU_VALUE_U16: return 2;
    case BGPU_VALUE_U32: case BGPU_VALUE_I32: case BGPU_VALUE_F32: return 4;
    case BGPU_VALUE_I64: case BGPU_VALUE_U64: case BGPU_VALUE_F64: return 8;
    default: return 0;
  }
}

// `p` on the device: the caller's pointer, or a stream-ordered copy of the
// host array.
int stage(const void* src, size_t bytes, bool on_device, Scratch& buf,
          const void** out, cudaStream_t s) {
  if (on_device || src == nullptr) {
    *out = src;
    return BGPU_OK;
  }
  BGPU_TRY(buf.alloc(bytes, s));
  BGPU_CUDA(cudaMemcpyAsync(buf.p, src, bytes, cudaMemcpyHostToDevice, s));
  *out = buf.p;
  return BGPU_OK;
}

struct HvgArgs {
  const void* data;
  const void* indices;
  const void* indptr;
  const int64_t* cells;
  uint64_t num_listed;
  const int8_t* mask;
  uint64_t mask_len;
  const int64_t* range;  // CSR without a cell list: the entries (nullptr: all)
  uint32_t g;            // genes accumulated
  const float* clip;
  unsigned long long* acc;
  Scratch* part;       // CSR: the chunks' words
  uint32_t num_parts;  // chunks
  int* err;
};

template <typename V, typename I, int MODE>
int launch_hvg_typed(const bgpu_hvg_input& in, HvgArgs& a, cudaStream_t s) {
  const V* data = static_cast<const V*>(a.data);
  const I* idx = static_cast<const I*>(a.indices);
  const I* ptr = static_cast<const I*>(a.indptr);
  if (in.is_csr) {
    // Genes per CTA: the fewest equal runs that fit the shared memory. Two
    // CTAs per SM where their words fit it twice, else one; chunks for one
    // wave, fewer when there is too little to read.
    const uint32_t fit = (uint32_t)((device_smem_optin() - 256) / kCsrGeneBytes);
    uint32_t slices = (uint32_t)ceil_div(a.g, fit);
    uint32_t gs = (uint32_t)ceil_div(a.g, slices);
    if (slices > kCsrMaxSlices) {
      slices = 1;
      gs = 0;
    }
    const size_t sm = (size_t)gs * kCsrGeneBytes;
    const uint32_t per_sm = sm <= 112 * 1024 ? 2 : 1;
    uint64_t chunks = std::max<uint64_t>(1, (uint64_t)num_sms() * per_sm / slices);
    const uint64_t epoch = std::max<uint64_t>(1, kCsrMaxPerGene / a.g);
    if (a.cells)
      chunks = std::min(chunks, ceil_div(a.num_listed, kCsrRows * (kCsrThreads / 32)));
    else
      chunks = std::max(std::min(chunks, ceil_div(in.nnz, kCsrThreads * kCsrUnroll)),
                        ceil_div(in.nnz, kCsrMaxPerGene));
    chunks = std::max<uint64_t>(chunks, 1);
    if (gs) {
      BGPU_TRY(a.part->alloc(chunks * 3 * a.g * 4, s));
      a.num_parts = (uint32_t)chunks;
    }
    BGPU_CUDA((allow_max_smem(k_hvg_csr<V, I, MODE>)));
    k_hvg_csr<V, I, MODE><<<(unsigned)(chunks * slices), kCsrThreads, sm, s>>>(
        data, idx, ptr, in.nnz, in.num_major, a.range, a.cells, a.num_listed, epoch, a.g, gs,
        slices, a.clip, a.acc, (uint32_t*)a.part->p, a.err);
  } else {
    k_hvg_check_ranges<I><<<(a.g + kHvgThreads - 1) / kHvgThreads, kHvgThreads, 0, s>>>(
        ptr, in.nnz, a.g, a.err);
    const uint64_t want = std::max<uint64_t>(1, ceil_div(in.nnz, kCscChunk * (kHvgThreads / 32)));
    const unsigned grid = (unsigned)std::min<uint64_t>(want, (uint64_t)num_sms() * 4);
    k_hvg_csc<V, I, MODE><<<grid, kHvgThreads, 0, s>>>(data, idx, ptr, a.g, a.mask, a.mask_len,
                                                       a.clip, a.acc, a.err);
  }
  BGPU_CHECK_LAUNCH();
  return BGPU_OK;
}

template <typename I, int MODE>
int launch_hvg_index(const bgpu_hvg_input& in, HvgArgs& a, cudaStream_t s) {
  switch (in.value_type) {
    case BGPU_VALUE_U16: return launch_hvg_typed<uint16_t, I, MODE>(in, a, s);
    case BGPU_VALUE_U32: return launch_hvg_typed<uint32_t, I, MODE>(in, a, s);
    case BGPU_VALUE_I32: return launch_hvg_typed<int32_t, I, MODE>(in, a, s);
    case BGPU_VALUE_F32: return launch_hvg_typed<float, I, MODE>(in, a, s);
    case BGPU_VALUE_I64: return launch_hvg_typed<int64_t, I, MODE>(in, a, s);
    case BGPU_VALUE_U64: return launch_hvg_typed<uint64_t, I, MODE>(in, a, s);
    case BGPU_VALUE_F64: return launch_hvg_typed<double, I, MODE>(in, a, s);
  }
  set_error("unknown value_type");
  return BGPU_ERR_INVALID;
}

// Device buffers of one call.
struct HvgWork {
  Scratch data, idx, ptr, cells, mask, err, acc, part, range;
};

// Stages the inputs and launches the accumulation of the integer sums into
// a.acc (3 x g) and, for CSR, a.part. num_cells: as the reference's argument. For CSR
// without a cell list, mean/variance sums every stored entry
// (hvg.pyx:43-52) and the clipped sums every entry of rows [0, num_cells)
// (hvg.pyx:292-303); with a list, mean/variance takes its first num_cells
// cells (hvg.pyx:56-63) and the clipped sums all of them (hvg.pyx:305-314).
template <int MODE>
int hvg_accumulate(const bgpu_hvg_input* in, uint64_t num_cells, uint32_t g,
                   const float* clip_dev, HvgWork& w, HvgArgs& a, cudaStream_t s) {
  const size_t vsz = hvg_value_size(in->value_type);
  BGPU_REQUIRE(vsz != 0, BGPU_ERR_INVALID, "unknown value_type");
  BGPU_REQUIRE(in->index_type == BGPU_INDEX_I32 || in->index_type == BGPU_INDEX_I64,
               BGPU_ERR_INVALID, "unknown index_type");
  BGPU_REQUIRE(in->nnz == 0 || (in->data && in->indices), BGPU_ERR_INVALID,
               "data and indices are required");
  const size_t isz = in->index_type == BGPU_INDEX_I64 ? 8 : 4;
  const bool dev = in->on_device != 0;
  BGPU_REQUIRE(in->indptr, BGPU_ERR_INVALID, "indptr is required");
  BGPU_REQUIRE(!in->is_csr || in->cell_mask == nullptr, BGPU_ERR_INVALID,
               "a CSR input takes cell_indices, not cell_mask");
  BGPU_REQUIRE(in->is_csr || in->cell_indices == nullptr, BGPU_ERR_INVALID,
               "a CSC input takes cell_mask, not cell_indices");
  if (!in->is_csr)
    BGPU_REQUIRE(g <= in->num_major, BGPU_ERR_INVALID,
                 "indptr has fewer genes than num_genes");

  a.g = g;
  a.clip = clip_dev;
  uint64_t listed = 0;
  if (in->is_csr && in->cell_indices) {
    listed = MODE == kMeanVar ? num_cells : in->num_cell_indices;
    BGPU_REQUIRE(listed <= in->num_cell_indices, BGPU_ERR_INVALID,
                 "cell_indices holds fewer than num_cells cells");
  } else if (in->is_csr && MODE == kClipped) {
    BGPU_REQUIRE(num_cells <= in->num_major, BGPU_ERR_INVALID,
                 "num_cells exceeds the rows of indptr");
  }

  BGPU_TRY(stage(in->data, in->nnz * vsz, dev, w.data, &a.data, s));
  BGPU_TRY(stage(in->indices, in->nnz * isz, dev, w.idx, &a.indices, s));
  BGPU_TRY(stage(in->indptr, (in->num_major + 1) * isz, dev, w.ptr, &a.indptr, s));
  const void* cells = nullptr;
  if (in->is_csr && in->cell_indices)
    BGPU_TRY(stage(in->cell_indices, listed * sizeof(int64_t), dev, w.cells, &cells, s));
  a.cells = static_cast<const int64_t*>(cells);
  a.num_listed = listed;
  const void* mask = nullptr;
  if (!in->is_csr && in->cell_mask)
    BGPU_TRY(stage(in->cell_mask, in->cell_mask_len, dev, w.mask, &mask, s));
  a.mask = static_cast<const int8_t*>(mask);
  a.mask_len = in->cell_mask_len;

  BGPU_TRY(w.acc.alloc(3ull * std::max<uint32_t>(g, 1) * sizeof(unsigned long long), s));
  BGPU_TRY(w.err.alloc(sizeof(int), s));
  a.acc = static_cast<unsigned long long*>(w.acc.p);
  a.err = static_cast<int*>(w.err.p);
  a.part = &w.part;
  BGPU_CUDA(cudaMemsetAsync(w.acc.p, 0, 3ull * std::max<uint32_t>(g, 1) * 8, s));
  BGPU_CUDA(cudaMemsetAsync(w.err.p, 0, sizeof(int), s));
  if (in->is_csr && !a.cells && MODE == kClipped) {
    BGPU_TRY(w.range.alloc(2 * sizeof(int64_t), s));
    a.range = static_cast<const int64_t*>(w.range.p);
    if (in->index_type == BGPU_INDEX_I64)
      k_hvg_range<int64_t><<<1, 1, 0, s>>>(static_cast<const int64_t*>(a.indptr), num_cells,
                                           in->nnz, static_cast<int64_t*>(w.range.p), a.err);
    else
      k_hvg_range<int32_t><<<1, 1, 0, s>>>(static_cast<const int32_t*>(a.indptr), num_cells,
                                           in->nnz, static_cast<int64_t*>(w.range.p), a.err);
    BGPU_CHECK_LAUNCH();
  }
  if (g > 0 && (in->is_csr ? (a.cells ? listed > 0 : in->nnz > 0) : true)) {
    if (in->index_type == BGPU_INDEX_I64)
      BGPU_TRY((launch_hvg_index<int64_t, MODE>(*in, a, s)));
    else
      BGPU_TRY((launch_hvg_index<int32_t, MODE>(*in, a, s)));
  }
  return BGPU_OK;
}

// Waits for the stream and reports what the kernels found wrong.
int hvg_check(const HvgArgs& a, cudaStream_t s) {
  int herr = 0;
  BGPU_CUDA(cudaMemcpyAsync(&herr, a.err, sizeof(int), cudaMemcpyDeviceToHost, s));
  BGPU_CUDA(cudaStreamSynchronize(s));
  BGPU_REQUIRE(herr != 2, BGPU_ERR_INVALID, "indptr is not a valid range");
  BGPU_REQUIRE(herr == 0, BGPU_ERR_INVALID,
               "a gene or cell index, or an indptr range, is out of bounds");
  return BGPU_OK;
}

}  // namespace
}  // namespace bgpu

using namespace bgpu;

extern "C" int bgpu_gene_mean_var(const bgpu_hvg_input* in, uint64_t num_cells,
                                  float* mean, float* var, uint32_t* nonzero_count,
                                  void* stream) {
  BGPU_REQUIRE(in && mean && var && nonzero_count, BGPU_ERR_INVALID,
               "bad gene mean/variance arguments");
  cudaStream_t s = (cudaStream_t)stream;
  const uint32_t g = in->num_genes;
  HvgWork w;
  HvgArgs a{};
  BGPU_TRY(hvg_accumulate<kMeanVar>(in, num_cells, g, nullptr, w, a, s));
  // float inv_num_cells = 1.0 / num_cells; inv_num_pairs_of_cells =
  // 1.0 / (num_cells * (num_cells - 1)), an integer product (hvg.pyx:24-25)
  const float inv_n = (float)(1.0 / (double)num_cells);
  const float inv_p = (float)(1.0 / (double)(num_cells * (num_cells - 1)));
  const bool dev = in->on_device != 0;
  Scratch o_mean, o_var, o_nz;
  float* dm = mean;
  float* dv = var;
  uint32_t* dn = nonzero_count;
  if (!dev) {
    BGPU_TRY(o_mean.alloc(g * 4ull, s));
    BGPU_TRY(o_var.alloc(g * 4ull, s));
    BGPU_TRY(o_nz.alloc(g * 4ull, s));
    dm = static_cast<float*>(o_mean.p);
    dv = static_cast<float*>(o_var.p);
    dn = static_cast<uint32_t*>(o_nz.p);
  }
  if (g > 0) {
    k_hvg_finish<kMeanVar><<<(unsigned)ceil_div(g, 32), 256, 0, s>>>(
        a.acc, (const uint32_t*)w.part.p, a.num_parts, g, num_cells, inv_n, inv_p, nullptr, dm,
        dv, dn, a.err);
    BGPU_CHECK_LAUNCH();
  }
  BGPU_TRY(hvg_check(a, s));
  if (!dev && g > 0) {
    BGPU_CUDA(cudaMemcpyAsync(mean, dm, g * 4ull, cudaMemcpyDeviceToHost, s));
    BGPU_CUDA(cudaMemcpyAsync(var, dv, g * 4ull, cudaMemcpyDeviceToHost, s));
    BGPU_CUDA(cudaMemcpyAsync(nonzero_count, dn, g * 4ull, cudaMemcpyDeviceToHost, s));
    BGPU_CUDA(cudaStreamSynchronize(s));
  }
  return BGPU_OK;
}

extern "C" int bgpu_clipped_sum(const bgpu_hvg_input* in, uint64_t num_cells,
                                const float* clip_val, float* batch_counts_sum,
                                float* squared_batch_counts_sum, void* stream) {
  BGPU_REQUIRE(in && clip_val && batch_counts_sum && squared_batch_counts_sum,
               BGPU_ERR_INVALID, "bad clipped-sum arguments");
  cudaStream_t s = (cudaStream_t)stream;
  // genes: num_genes (CSR, num_dataset_genes) or the columns of indptr (CSC,
  // hvg.pyx:414)
  BGPU_REQUIRE(in->is_csr || in->num_major <= 0xFFFFFFFFull, BGPU_ERR_INVALID,
               "too many genes");
  const uint32_t g = in->is_csr ? in->num_genes : (uint32_t)in->num_major;
  const bool dev = in->on_device != 0;
  Scratch d_clip, o_b, o_s;
  const void* clip = nullptr;
  BGPU_TRY(stage(clip_val, g * 4ull, dev, d_clip, &clip, s));
  HvgWork w;
  HvgArgs a{};
  BGPU_TRY(hvg_accumulate<kClipped>(in, num_cells, g, static_cast<const float*>(clip), w, a, s));
  float* db = batch_counts_sum;
  float* ds = squared_batch_counts_sum;
  if (!dev) {
    BGPU_TRY(o_b.alloc(g * 4ull, s));
    BGPU_TRY(o_s.alloc(g * 4ull, s));
    db = static_cast<float*>(o_b.p);
    ds = static_cast<float*>(o_s.p);
  }
  if (g > 0) {
    k_hvg_finish<kClipped><<<(unsigned)ceil_div(g, 32), 256, 0, s>>>(
        a.acc, (const uint32_t*)w.part.p, a.num_parts, g, 0, 0.f, 0.f,
        static_cast<const float*>(clip), db, ds, nullptr, a.err);
    BGPU_CHECK_LAUNCH();
  }
  BGPU_TRY(hvg_check(a, s));
  if (!dev && g > 0) {
    BGPU_CUDA(cudaMemcpyAsync(batch_counts_sum, db, g * 4ull, cudaMemcpyDeviceToHost, s));
    BGPU_CUDA(cudaMemcpyAsync(squared_batch_counts_sum, ds, g * 4ull,
                              cudaMemcpyDeviceToHost, s));
    BGPU_CUDA(cudaStreamSynchronize(s));
  }
  return BGPU_OK;
}
