// Locality order of points and tile lists of query blocks (sv_knn_order.cu).
#pragma once
#include "sv_internal.cuh"

constexpr int KNN_MAX_TILES = 16384;   // tiles that a list is sorted for

struct KnnOrder {
  DevBuf<int> perm;                     // place -> point (n entries used)
  DevBuf<unsigned long long> lists;     // per query block: ntiles entries, nearest first
  int ntiles = 0;
};

// the tile that holds query block b's first row (blocks of bq rows, tiles of bp)
__host__ __device__ __forceinline__ int knn_own_tile(int64_t b, int bq, int bp) { return (int)(b * bq / bp); }
// of a list entry: the lower bound of the squared distance, and the tile
__device__ __forceinline__ float knn_list_bound(unsigned long long e) { return __uint_as_float((unsigned)(e >> 32)); }
__device__ __forceinline__ int knn_list_tile(unsigned long long e, int own) {
  const unsigned place = (unsigned)e;
  return (place & 1u) ? own - (int)(place >> 1) : own + (int)(place >> 1);
}

// The dimension of largest variance, and the sum of all dimensions' variances.
struct KnnSpread {
  int dim = 0;
  double sum = 0;
};
KnnSpread sv_knn_spread(sv_context* ctx, const float* X32, int64_t n, int dp, int d);
// Orders the points and lists the tiles (bp points) of every block of bq queries;
// false when the input is too small or too large for it.  halves_of: an order (place
// -> point) whose tiles' halves are kept, for BF16 operands: bounds of the rounded
// coordinates; bp is even; false as well when the points have too little structure
// for the lists to leave out more than the order along the widest dimension does.
bool sv_knn_order(sv_context* ctx, const float* X32, int64_t n, int dp, int d, int bq, int bp,
                  const KnnSpread& spread, KnnOrder& o, const int* halves_of = nullptr);
