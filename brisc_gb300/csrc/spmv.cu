// Sparse products on the device layout (matrix.cuh).
//
//  X.v     (brisc/pca.pyx:440-475 matvec_csr_parallel_raw): one group of G lanes
//          per cell row, 128-bit loads of four packed entries starting on a
//          4-entry boundary (the row head and tail are masked), the normalised
//          value log1pf(count * isf[cell]) computed in registers, the gene
//          weight v[gene] / sd[gene] read from shared memory.
//  X^T.u   (brisc/pca.pyx:478-511 rmatvec_csc_parallel_raw): one CTA per
//          (row panel, gene group). The panel's u and size factors are staged
//          in shared memory, so the per-entry gathers hit shared memory instead
//          of L2; a group of lanes reduces one gene's segment (a fixed shuffle
//          tree, no atomics) into a per-panel partial (gene-major
//          layout); a second pass adds the partials of all panels in panel
//          order. These register-vector kernels serve layouts outside the
//          streaming kernels' limits (stream.cu).
//  gene sd (brisc/pca.pyx:51-103 clipped_stddev_csc): same panel traversal,
//          FP64 sums.
#include <algorithm>

#include "matrix.cuh"
#include "moments.cuh"

namespace bgpu {

namespace {

template <int G, int MODE>
__global__ void __launch_bounds__(256)
k_spmv(CsrView X, const float* __restrict__ v, const float* __restrict__ sd,
       float* __restrict__ y) {
  extern __shared__ float w[];
  for (uint32_t c = threadIdx.x; c < X.g; c += blockDim.x)
    w[c] = sd ? v[c] / sd[c] : v[c];  // pca.pyx:461-462
  __syncthreads();

  constexpr int kRowsPerWarp = 32 / G;
  const int lane = threadIdx.x & (G - 1);
  const int grp = (threadIdx.x & 31) / G;
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = (gridDim.x * (uint64_t)blockDim.x) >> 5;
  // bit 31 of a stored word flags a row head when genes fit in 15 bits
  const uint32_t gm = X.g > 32768u ? 0xffffu : 0x7fffu;
  const uint64_t nbatches = ceil_div_dev(X.n, kRowsPerWarp);
  for (uint64_t bt = warp; bt < nbatches; bt += nwarps) {
    const uint64_t r = bt * kRowsPerWarp + grp;
    const bool valid = r < X.n;
    int64_t e0 = 0, e1 = 0;
    if (valid) { e0 = X.rowptr[r]; e1 = X.rowptr[r + 1]; }
    float acc = 0.f;
    if constexpr (MODE == kCounts) {
      const float f = valid ? X.isf[r] : 0.f;
#pragma unroll 4
      for (int64_t b = (e0 & ~3LL) + 4 * lane; b < e1; b += 4 * G) {
        const uint4 q = ld_stream_u4(X.packed + b);
        const uint32_t qq[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int64_t e = b + k;
          if (e >= e0 && e < e1)
            acc += norm_count(qq[k] & 0xffffu, f) * w[(qq[k] >> 16) & gm];
        }
      }
    } else {
#pragma unroll 4
      for (int64_t b = (e0 & ~3LL) + 4 * lane; b < e1; b += 4 * G) {
        const uint4 qv = ld_stream_u4(X.val + b);
        const uint2 qc = ld_stream_u2(X.col + b);
        const float vv[4] = {__uint_as_float(qv.x), __uint_as_float(qv.y),
                             __uint_as_float(qv.z), __uint_as_float(qv.w)};
        const uint32_t cc[4] = {qc.x & 0xffffu, qc.x >> 16, qc.y & 0xffffu,
                                qc.y >> 16};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int64_t e = b + k;
          if (e >= e0 && e < e1) acc += vv[k] * w[cc[k]];
        }
      }
    }
    acc = group_sum<G>(acc);
    if (valid && lane == 0) y[r] = X.post ? acc * X.post[r] : acc;
  }
}

// Lanes per (panel, gene) segment: G lanes take 4 G entries per step, 32 / G
// segments per warp. A whole warp per segment leaves most lanes without an
// entry where segments are short (1024 rows x 8 %: 80 entries) and pays its
// shuffles per segment: 50k x 2000 float values, 7.8M entries: X^T.u 47 us,
// moments 212 us with 32 lanes and one load at a time, 39 us and 37 us with 8 lanes
// and kSegLoads loads in flight.
constexpr int kSegLoads = 3;
template <int G>
struct Segments {
  const uint32_t lane = threadIdx.x & (G - 1);
  const uint32_t first = threadIdx.x / G, step = 256 / G;
};

template <int MODE, int G>
__global__ void __launch_bounds__(256)
k_rmat_partials(CscView X, const float* __restrict__ u,
                const float* __restrict__ u_scale, float* __restrict__ u_out,
                float* __restrict__ partials, uint32_t colgroup) {
  extern __shared__ float sm[];
  const uint32_t P = 1u << X.pshift;
  const uint32_t p = blockIdx.x;
  const uint64_t r0 = (uint64_t)p << X.pshift;
  const uint32_t rows = (uint32_t)min_u64(P, X.n - r0);
  float* us = sm;
  float* fs = sm + P;
  const float scale = u_scale ? *u_scale : 1.f;
  const bool write_u = u_out && blockIdx.y == 0;
  for (uint32_t i = threadIdx.x; i < rows; i += blockDim.x) {
    const float uu = u_scale ? u[r0 + i] * scale : u[r0 + i];
    if (write_u) u_out[r0 + i] = uu;
    if constexpr (MODE == kCounts) {
      fs[i] = X.isf[r0 + i];
      us[i] = X.post ? uu * X.post[r0 + i] : uu;
    } else {
      us[i] = uu;
    }
  }
  __syncthreads();
  const Segments<G> seg;
  const int64_t pbase = X.rowptr[r0];
  const int32_t* cp = X.colptr + (uint64_t)p * (X.g + 1);
  const uint32_t c0 = blockIdx.y * colgroup;
  const uint32_t c1 = min(X.g, c0 + colgroup);
  // every lane of a warp takes the same number of turns (group_sum shuffles);
  // the next segment's bounds load while this one is summed
  uint32_t c = c0 + seg.first;
  int64_t n0 = c < c1 ? cp[c] : 0, n1 = c < c1 ? cp[c + 1] : 0;
  for (uint32_t cb = c0; cb < c1; cb += seg.step, c += seg.step) {
    const int64_t e0 = pbase + n0, e1 = pbase + n1;
    const uint32_t cn = c + seg.step;
    n0 = cn < c1 ? cp[cn] : 0;
    n1 = cn < c1 ? cp[cn + 1] : 0;
    float acc = 0.f;
    for (int64_t b = (e0 & ~3LL) + 4 * seg.lane; b < e1; b += 4 * G * kSegLoads) {
      if constexpr (MODE == kCounts) {
        uint4 q[kSegLoads];
#pragma unroll
        for (int i = 0; i < kSegLoads; ++i)
          q[i] = b + 4 * G * i < e1 ? ld_stream_u4(X.packed + b + 4 * G * i)
                                    : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int i = 0; i < kSegLoads; ++i) {
          const uint32_t qq[4] = {q[i].x, q[i].y, q[i].z, q[i].w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int64_t e = b + 4 * G * i + k;
            if (e >= e0 && e < e1) {
              const uint32_t lr = (qq[k] >> 16) & (P - 1);  // bit 31 may flag a segment head
              acc += norm_count(qq[k] & 0xffffu, fs[lr]) * us[lr];
            }
          }
        }
      } else {
        uint4 qv[kSegLoads];
        uint2 qr[kSegLoads];
#pragma unroll
        for (int i = 0; i < kSegLoads; ++i) {
          const bool in = b + 4 * G * i < e1;
          qv[i] = in ? ld_stream_u4(X.val + b + 4 * G * i) : make_uint4(0u, 0u, 0u, 0u);
          qr[i] = in ? ld_stream_u2(X.row + b + 4 * G * i) : make_uint2(0u, 0u);
        }
#pragma unroll
        for (int i = 0; i < kSegLoads; ++i) {
          const float vv[4] = {__uint_as_float(qv[i].x), __uint_as_float(qv[i].y),
                               __uint_as_float(qv[i].z), __uint_as_float(qv[i].w)};
          const uint32_t rr[4] = {qr[i].x & 0xffffu, qr[i].x >> 16, qr[i].y & 0xffffu,
                                  qr[i].y >> 16};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int64_t e = b + 4 * G * i + k;
            if (e >= e0 && e < e1) acc += vv[k] * us[rr[k]];
          }
        }
      }
    }
    acc = group_sum<G>(acc);
    if (seg.lane == 0 && c < c1) partials[(uint64_t)c * X.num_panels + p] = acc;
  }
}

// Per (panel, gene): sum and sum of squares of the values, in runs of up to
// kMomentTerms entries as floats (moments.cuh), the lanes' together, and the runs
// in FP64: that unit is what short segments wait for (the lanes' sums in FP64, and
// every lane's: segments of 10 entries, 6M of them, 411 us a call against 230; 7.8M
// entries of 80: 40 and 37 us). 62 registers, four blocks per SM: held to 40 it
// spills (53 us).
template <int MODE, int G>
__global__ void __launch_bounds__(256, 4)
k_gene_moments(CscView X, double2* __restrict__ partials, uint32_t colgroup) {
  extern __shared__ float sm[];
  const uint32_t P = 1u << X.pshift;
  const uint32_t p = blockIdx.x;
  const uint64_t r0 = (uint64_t)p << X.pshift;
  const uint32_t rows = (uint32_t)min_u64(P, X.n - r0);
  float* fs = sm;
  float* qs = sm + P;
  if constexpr (MODE == kCounts) {
    for (uint32_t i = threadIdx.x; i < rows; i += blockDim.x) {
      fs[i] = X.isf[r0 + i];
      qs[i] = X.post ? X.post[r0 + i] : 1.f;
    }
  }
  __syncthreads();
  const Segments<G> seg;
  const unsigned group = 0xFFFFFFFFu >> (32 - G) << (threadIdx.x & 31 & ~(G - 1));
  const int64_t pbase = X.rowptr[r0];
  const int32_t* cp = X.colptr + (uint64_t)p * (X.g + 1);
  const uint32_t c0 = blockIdx.y * colgroup;
  const uint32_t c1 = min(X.g, c0 + colgroup);
  uint32_t c = c0 + seg.first;
  int32_t n0 = c < c1 ? cp[c] : 0, n1 = c < c1 ? cp[c + 1] : 0;
  for (uint32_t cb = c0; cb < c1; cb += seg.step, c += seg.step) {
    // the segment from the 4-entry boundary at or before it, in 32 bits
    const int64_t e0 = pbase + n0, at = e0 & ~3LL;
    const uint32_t skip = (uint32_t)(e0 - at), len = (uint32_t)(n1 - n0), span = skip + len;
    const uint32_t cn = c + seg.step;
    n0 = cn < c1 ? cp[cn] : 0;
    n1 = cn < c1 ? cp[cn + 1] : 0;
    auto values = [&](uint32_t b, float (&vals)[4]) {  // b < span
      if constexpr (MODE == kCounts) {
        const uint4 q = ld_stream_u4(X.packed + at + b);
        const uint32_t qq[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t lr = (qq[k] >> 16) & (P - 1);  // bit 31 may flag a segment head
          vals[k] = b + k - skip < len
                        ? (X.post ? norm_count(qq[k] & 0xffffu, fs[lr]) * qs[lr]
                                  : norm_count(qq[k] & 0xffffu, fs[lr]))
                        : 0.f;
        }
      } else {
        const uint4 qv = ld_stream_u4(X.val + at + b);
        const float vv[4] = {__uint_as_float(qv.x), __uint_as_float(qv.y),
                             __uint_as_float(qv.z), __uint_as_float(qv.w)};
#pragma unroll
        for (int k = 0; k < 4; ++k) vals[k] = b + k - skip < len ? vv[k] : 0.f;
      }
    };
    constexpr uint32_t kStep = 4 * G * kSegLoads, kRun = kMomentTerms / kStep * kStep;
    double s1 = 0.0, s2 = 0.0;
    for (uint32_t run = 0; run < span && len != 0u; run += kRun) {
      const uint32_t end = min(span, run + kRun);
      FloatMoments m;
      for (uint32_t b = run + 4 * seg.lane; b < end; b += kStep) {
        float vals[kSegLoads][4];
#pragma unroll
        for (int i = 0; i < kSegLoads; ++i)
          if (b + 4 * G * i < span) values(b + 4 * G * i, vals[i]);
#pragma unroll
        for (int i = 0; i < kSegLoads; ++i)
          if (b + 4 * G * i < span) m.add(vals[i][0], vals[i][1], vals[i][2], vals[i][3]);
      }
      m.merge<G>(group);
      if (m.good()) {
        if (seg.lane == 0) {  // the others' have no reader
          s1 += m.sum();
          s2 += m.squares();
        }
        continue;
      }
      double t1 = 0.0, t2 = 0.0;  // out of the floats' range: again, in FP64
      for (uint32_t b = run + 4 * seg.lane; b < end; b += 4 * G) {
        float vals[4];
        values(b, vals);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          t1 += (double)vals[k];
          t2 += (double)vals[k] * (double)vals[k];
        }
      }
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) {
        t1 += __shfl_xor_sync(group, t1, o);
        t2 += __shfl_xor_sync(group, t2, o);
      }
      s1 += t1;
      s2 += t2;
    }
    if (seg.lane == 0 && c < c1) partials[(uint64_t)p * X.g + c] = make_double2(s1, s2);
  }
}

// The standard deviations from the panels' (or CTAs') moments: a block takes
// 32 genes (lane = gene, so the loads are runs of the gene-major row), its
// warps take every 32nd panel and are added in warp order. A thread per gene
// instead is a serial chain of loads: 114 us for 608 panels x 2000 genes, 17 us.
constexpr int kSdWarps = 32;
__global__ void __launch_bounds__(32 * kSdWarps)
k_gene_sd(const double2* __restrict__ partials, uint32_t num_panels, uint32_t g, uint64_t n,
          float* __restrict__ sd) {
  __shared__ double2 sh[kSdWarps][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t c = blockIdx.x * 32 + lane;
  double s1 = 0.0, s2 = 0.0;
  if (c < g) {
#pragma unroll 4
    for (uint32_t p = wid; p < num_panels; p += kSdWarps) {
      const double2 t = partials[(uint64_t)p * g + c];
      s1 += t.x;
      s2 += t.y;
    }
  }
  sh[wid][lane] = make_double2(s1, s2);
  __syncthreads();
  if (wid != 0 || c >= g) return;
  for (int w = 1; w < kSdWarps; ++w) {
    s1 += sh[w][lane].x;
    s2 += sh[w][lane].y;
  }
  const double dn = (double)n;
  // pca.pyx:83-86: sqrt((n * sum_sq - sum^2) / (n (n - 1))), clipped at 1e-8
  double var = (dn * s2 - s1 * s1) / (dn * (dn - 1.0));
  float s = (float)sqrt(var > 0.0 ? var : 0.0);
  sd[c] = s < 1e-8f ? 1e-8f : s;
}

}  // namespace

double matvec_bytes(const Matrix& m) {
  if (m.sell) {  // stream, per-position factors and descriptors, v, sd, y
    const double npos = (double)m.xv.groups * 32.0;
    return (double)m.xv.total_units * 8.0 + npos * (4.0 + 4.0 + 2.0) +
           (m.post ? npos * 4.0 : 0.0) + m.xv.groups * 6.0 + m.g * 8.0 + m.n * 4.0;
  }
  double per = m.mode == kCounts ? 4.0 : 6.0;
  double b = m.nnz * per + (m.n + 1) * 8.0 + m.n * 4.0 + m.g * 8.0;
  if (m.mode == kCounts) b += m.n * 4.0 * (m.post ? 2 : 1);
  return b;
}

double rmatvec_bytes(const Matrix& m) {
  if (m.sell) {  // stream, descriptors, u (read and written scaled), isf, partials
    const double groups = (double)m.xt.groups;
    return (double)m.xt.total_units * 8.0 + m.n * 12.0 + (m.post ? m.n * 4.0 : 0.0) +
           (double)m.xt.ctas * m.g * 4.0 + groups * 70.0 + m.xt.panels * 8.0;
  }
  double per = m.mode == kCounts ? 4.0 : 6.0;
  double b = m.nnz * per + (double)m.num_panels * (m.g + 1) * 4.0 + m.n * 4.0 +
             (double)m.num_panels * m.g * 4.0;
  if (m.mode == kCounts) b += m.n * 4.0 * (m.post ? 2 : 1);
  return b;
}

int launch_matvec(const Matrix& m, const float* v, const float* sd, float* y,
                  cudaStream_t s) {
  const CsrView X = csr_view(m);
  const int blocks = m.spmv_blocks > 0 ? m.spmv_blocks : num_sms() * 8;
  const size_t smem = (size_t)m.g * sizeof(float);
#define BGPU_SPMV_CASE(GG)                                                    \
  case GG:                                                                      \
    if (m.mode == kCounts) {                                                    \
      if (smem > 48 * 1024)                                                     \
        BGPU_CUDA(allow_max_smem(k_spmv<GG, kCounts>));                          \
      k_spmv<GG, kCounts><<<blocks, 256, smem, s>>>(X, v, sd, y);               \
    } else {                                                                    \
      if (smem > 48 * 1024)                                                     \
        BGPU_CUDA(allow_max_smem(k_spmv<GG, kFloat>));                           \
      k_spmv<GG, kFloat><<<blocks, 256, smem, s>>>(X, v, sd, y);                \
    }                                                                           \
    break;
  switch (m.spmv_group) {
    BGPU_SPMV_CASE(2)
    BGPU_SPMV_CASE(4)
    BGPU_SPMV_CASE(8)
    BGPU_SPMV_CASE(16)
    BGPU_SPMV_CASE(32)
    default:
      set_error("unsupported SpMV group size");
      return BGPU_ERR_INVALID;
  }
#undef BGPU_SPMV_CASE
  BGPU_CHECK_LAUNCH();
  return BGPU_OK;
}

// X^T.u: segments of more than 128 entries on average keep a whole warp's lanes
// at work; below that 8 lanes per segment (see Segments). 6 to 12M floats, us per
// call with 8 and 32 lanes: 43 entries per segment 78, 118; 81: 78, 91; 106: 79, 79;
// 128: 69, 68; 162: 75, 66; 221: 79, 68. The moments take 8 lanes at every length:
// their chains of additions are long, and more lanes have more sums to join (128:
// 81, 127; 162: 86, 122; 221: 75, 108 when each lane's ended in FP64; now 68, 65 and
// 63 with 8).
static bool wide_segments(const Matrix& m) {
  return (double)m.nnz > 128.0 * (double)m.num_panels * (double)m.g;
}

template <int MODE, int G>
static int launch_partials_typed(const Matrix& m, const float* u, const float* u_scale_dev,
                                 float* u_out, float* partials, cudaStream_t s) {
  const uint32_t cg = m.rmat_colgroup;
  const dim3 grid(m.num_panels, (unsigned)ceil_div(m.g, cg));
  const size_t smem = (size_t)m.P * 2 * sizeof(float);
  if (smem > 48 * 1024) BGPU_CUDA((allow_max_smem(k_rmat_partials<MODE, G>)));
  k_rmat_partials<MODE, G><<<grid, 256, smem, s>>>(csc_view(m), u, u_scale_dev, u_out, partials,
                                                   cg);
  BGPU_CHECK_LAUNCH();
  return BGPU_OK;
}

template <int MODE>
static int launch_moments_typed(const Matrix& m, double* partials, cudaStream_t s) {
  const uint32_t cg = m.rmat_colgroup;
  const dim3 grid(m.num_panels, (unsigned)ceil_div(m.g, cg));
  const size_t smem = (size_t)m.P * 2 * sizeof(float);
  if (smem > 48 * 1024) BGPU_CUDA((allow_max_smem(k_gene_moments<MODE, 8>)));
  k_gene_moments<MODE, 8><<<grid, 256, smem, s>>>(csc_view(m), (double2*)partials, cg);
  BGPU_CHECK_LAUNCH();
  return BGPU_OK;
}

int launch_rmatvec_partials(const Matrix& m, const float* u,
                            const float* u_scale_dev, float* u_out,
                            float* partials, cudaStream_t s) {
  const bool wide = wide_segments(m);
  if (m.mode == kCounts)
    return wide ? launch_partials_typed<kCounts, 32>(m, u, u_scale_dev, u_out, partials, s)
                : launch_partials_typed<kCounts, 8>(m, u, u_scale_dev, u_out, partials, s);
  return wide ? launch_partials_typed<kFloat, 32>(m, u, u_scale_dev, u_out, partials, s)
              : launch_partials_typed<kFloat, 8>(m, u, u_scale_dev, u_out, partials, s);
}

int launch_gene_stddev(const Matrix& m, double* partials, float* sd,
                       cudaStream_t s) {
  if (m.sell) {  // per-CTA moments over the sliced-ELL panels, CTA order
    BGPU_TRY(launch_xt_moments(m, partials, s));
    k_gene_sd<<<(unsigned)ceil_div(m.g, 32), 32 * kSdWarps, 0, s>>>(
        (const double2*)partials, m.num_panels, m.g, m.n, sd);
    BGPU_CHECK_LAUNCH();
    return BGPU_OK;
  }
  BGPU_TRY(m.mode == kCounts ? launch_moments_typed<kCounts>(m, partials, s)
                             : launch_moments_typed<kFloat>(m, partials, s));
  k_gene_sd<<<(unsigned)ceil_div(m.g, 32), 32 * kSdWarps, 0, s>>>(
      (const double2*)partials, m.num_panels, m.g, m.n, sd);
  BGPU_CHECK_LAUNCH();
  return BGPU_OK;
}

}  // namespace bgpu
