// Tensor-core candidate filter with exact FP32 evaluation: the nearest rows
// of one matrix for every row of another (knn_tc.cu).
#pragma once

#include "common.cuh"

namespace bgpu {

// Error word of a call, beside kDevErrTimeout of the waits: the cluster sizes do
// not sum to the number of cells. The kernels below write no result where it is
// set, so a refused call leaves its outputs as they were.
enum KnnErr : int { kKnnErrSizes = 2 };

// A matrix of row vectors prepared as a tensor-core operand (knn_tc.cu): BF16
// high and low parts in core-matrix order, 8 rows at a time, with the row's
// norm in extra columns.
struct KnnOperand {
  const float* rows = nullptr;   // the caller's rows, n x d
  const float* norms = nullptr;  // the norms of the distances, n
  uint64_t n = 0;
  unsigned char* tiles = nullptr;  // ceil(n / 8) groups of group_bytes
  float* length = nullptr;         // per row: at least its Euclidean length
  float* gmax = nullptr;           // per group: at least the lengths and
                                   // sqrt |norm| of its rows
};

uint32_t knn_kp(uint32_t d);                       // padded columns of an operand
size_t knn_operand_bytes(uint64_t n, uint32_t d);  // device bytes of one
size_t knn_replay_bytes(uint64_t n);               // scratch of a search by n queries
// Lays `op` out in `mem` (knn_operand_bytes) and fills it. norms may be
// nullptr for an operand used for queries only (zeros take their place).
int knn_prepare(KnnOperand* op, const float* rows, const float* norms, uint64_t n, uint32_t d,
                void* mem, cudaStream_t s);

// For every query row, the `count` candidate rows with the smallest
// |c|^2 - 2 x.c, sorted; ids are candidate rows. coff (may be nullptr): the
// offsets of the queries' clusters where those are sorted by cluster and the
// candidates are the clusters' centroids in order; nullptr with count 1.
// replay: knn_replay_bytes(queries) of scratch. err: device error word.
int knn_tc_nearest(const KnnOperand& queries, const KnnOperand& cand, uint32_t d, uint32_t count,
                   const uint64_t* coff, uint32_t* replay, uint32_t* out_id, float* out_d,
                   int* err, cudaStream_t s);

// For every row of `cells` (grouped by cluster, offsets coff[nc + 1]), the k
// other rows with the smallest distance among the clusters of its row of
// nearest (n x cs); ids through id_map.
int knn_tc_search(const KnnOperand& cells, uint32_t d, const uint64_t* coff, uint32_t nc,
                  const uint32_t* nearest, uint32_t cs, uint32_t k, const uint32_t* id_map,
                  uint32_t* replay, uint32_t* out_id, float* out_d, int* err, cudaStream_t s);

}  // namespace bgpu
