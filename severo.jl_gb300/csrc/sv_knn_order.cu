// Locality order of the points and per-block tile lists for the exact kNN
// searches (sv_knn.cu, sv_knn_tc.cu).
//
// The candidate kernels scan tiles of points for blocks of queries and may skip
// a tile whose distance to the block exceeds every query's current threshold.
// How many tiles that leaves depends on the order of the points.  Here every
// point goes to the nearest of P of the points themselves (pivots, spread evenly
// over the input), cells of near pivots next to each other (the pivots in the
// order of a kd-tree), so that a tile is
// a compact piece of the data in all dimensions.  Two lower bounds of the distance
// between a query block and a tile follow: that of their bounding boxes, and the
// gap between their projections on the line through the tiles' means (a box pays
// for its extent in every dimension, a projection once).  Each query block gets
// its tiles sorted by the larger: the nearest first, so that thresholds fall at
// once, and the first tile out of reach ends the scan.
// (Along the widest dimension alone, 300,000 points in 60 clusters x 50
// dimensions left most of the 1,172 tiles to be scanned.)
// The tensor-core search shortlists the points of the two halves of its tiles
// apart, and which points share a half decides which of them the BF16 keys may
// misjudge.  There the halves are those of the tiles along the widest dimension
// (halves_of), as they are for stacked samples; each half is ordered by itself, and
// a tile takes the next part of both.
#include "sv_internal.cuh"
#include "sv_knn_order.cuh"

#include <float.h>

namespace {

constexpr int PV_MAX = 1024;       // most pivots
constexpr int PV_TILE = 64;        // pivots staged at a time
constexpr int PV_THREADS = 128;
constexpr int PV_SAMPLE = 2048;    // points whose nearest pivot's distance is looked at
// The tensor-core search takes the lists while the squared distance to the nearest
// pivot is, on average, below this part of that between two points.  List against
// widest dimension, kernels of the whole search, 300,000 points, k = 20: 0.035 (60
// far clusters) 7.0 and 11.1 ms; 0.094 (30 near ones, 20 dimensions) 10.1 and 13.8;
// 0.138 (uniform, 8 dimensions) 17.5 and 17.5; 0.21 (normal, 10) 22.9 and 22.9; 0.38
// (normal, falling scales, 50) 25.4 and 20.7; 0.55 (normal, 50) 30.9 and 27.5.
constexpr double PV_NEAR = 0.125;

// Per-dimension sums and sums of squares (FP64, atomics: only the choice of the
// widest dimension depends on them).
__global__ void k_dim_moments(const float* __restrict__ X, int64_t n, int dp, double* __restrict__ acc) {
  __shared__ double s1[256], s2[256];
  const int c = threadIdx.x % dp, r0 = threadIdx.x / dp, rstep = blockDim.x / dp;
  double a = 0, b = 0;
  if (r0 < rstep)
    for (int64_t i = blockIdx.x * (int64_t)rstep + r0; i < n; i += (int64_t)gridDim.x * rstep) {
      double v = X[i * dp + c];
      a += v;
      b += v * v;
    }
  s1[threadIdx.x] = a;
  s2[threadIdx.x] = b;
  __syncthreads();
  if (threadIdx.x < dp) {
    double ta = 0, tb = 0;
    for (int r = 0; r < rstep; ++r) {
      ta += s1[r * dp + threadIdx.x];
      tb += s2[r * dp + threadIdx.x];
    }
    atomicAdd(acc + threadIdx.x, ta);
    atomicAdd(acc + dp + threadIdx.x, tb);
  }
}

__device__ __forceinline__ unsigned ordered_bits(float v) {
  const unsigned u = __float_as_uint(v);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// One block: the pivots' order -- halved again and again along the dimension that
// their group is widest in -- and, in that order, their rows and squared norms.
__global__ void __launch_bounds__(PV_MAX) k_pivots(const float* __restrict__ X, int64_t n, int dp, int P,
                                                   float* __restrict__ rows, float* __restrict__ norms) {
  __shared__ int ord[PV_MAX];      // the pivots' points
  __shared__ float co[PV_MAX];
  __shared__ int gdim[PV_MAX / 4];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
  if (tid < P) ord[tid] = (int)((2 * (int64_t)tid + 1) * n / (2 * (int64_t)P));
  __syncthreads();
  for (int G = 1; P / G >= 8 && G <= PV_MAX / 4; G *= 2) {
    for (int g = w; g < G; g += nw) {
      const int a = (int)((int64_t)g * P / G), b = (int)((int64_t)(g + 1) * P / G);
      float wide = -1.f;
      int dim = 0;
      for (int c = lane; c < dp; c += 32) {
        float lo = FLT_MAX, hi = -FLT_MAX;
#pragma unroll 4
        for (int k = a; k < b; ++k) {
          const float v = X[(int64_t)ord[k] * dp + c];
          lo = fminf(lo, v);
          hi = fmaxf(hi, v);
        }
        if (hi - lo > wide) {
          wide = hi - lo;
          dim = c;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float w2 = __shfl_xor_sync(0xffffffffu, wide, o);
        const int d2 = __shfl_xor_sync(0xffffffffu, dim, o);
        if (w2 > wide || (w2 == wide && d2 < dim)) {
          wide = w2;
          dim = d2;
        }
      }
      if (lane == 0) gdim[g] = dim;
    }
    __syncthreads();
    int g = 0, a = 0, b = 0, mine = 0;
    if (tid < P) {
      g = (int)((int64_t)tid * G / P);
      while ((int64_t)(g + 1) * P / G <= tid) ++g;
      a = (int)((int64_t)g * P / G);
      b = (int)((int64_t)(g + 1) * P / G);
      mine = ord[tid];
      const float v = X[(int64_t)mine * dp + gdim[g]];
      co[tid] = v == v ? v : FLT_MAX;
    }
    __syncthreads();
    if (tid < P) {
      const float v = co[tid];
      int r = a;
      for (int k = a; k < b; ++k) r += co[k] < v || (co[k] == v && k < tid);
      ord[r] = mine;
    }
    __syncthreads();
  }
  for (int r = w; r < P; r += nw) {
    const float* src = X + (int64_t)ord[r] * dp;
    float s = 0.f;
    for (int c = lane; c < dp; c += 32) {
      const float v = src[c];
      rows[r * dp + c] = v;
      s = fmaf(v, v, s);
    }
    s = sv_warp_sum(s);
    if (lane == 0) norms[r] = s;
  }
}

// Sort key of every point: its half (if any), its nearest pivot's place, then its
// widest coordinate.  near (optional): instead, of every step-th point the squared
// distance to the nearest pivot.
template <int DP>
__global__ void __launch_bounds__(PV_THREADS) k_pivot_assign(const float* __restrict__ X, int64_t n,
                                                             const float* __restrict__ rows,
                                                             const float* __restrict__ norms, int P, int dim,
                                                             const unsigned char* __restrict__ half,
                                                             unsigned long long* __restrict__ key,
                                                             int* __restrict__ val, int64_t step,
                                                             float* __restrict__ near) {
  __shared__ __align__(16) float tile[PV_TILE * DP];
  __shared__ float tn[PV_TILE];
  const int64_t i = (int64_t)blockIdx.x * PV_THREADS + threadIdx.x;
  float q[DP];
#pragma unroll
  for (int c = 0; c < DP; c += 4) {
    const float4 v = i < n ? *(const float4*)(X + i * step * DP + c) : make_float4(0, 0, 0, 0);
    q[c] = -2.f * v.x;
    q[c + 1] = -2.f * v.y;
    q[c + 2] = -2.f * v.z;
    q[c + 3] = -2.f * v.w;
  }
  float bd = FLT_MAX;
  int best = 0;
  for (int p0 = 0; p0 < P; p0 += PV_TILE) {
    __syncthreads();
    for (int k = threadIdx.x; k < PV_TILE * DP / 4; k += PV_THREADS)
      ((float4*)tile)[k] = p0 + k / (DP / 4) < P ? ((const float4*)(rows + (int64_t)p0 * DP))[k]
                                                  : make_float4(0, 0, 0, 0);
    for (int k = threadIdx.x; k < PV_TILE; k += PV_THREADS) tn[k] = p0 + k < P ? norms[p0 + k] : FLT_MAX;
    __syncthreads();
#pragma unroll 1
    for (int r0 = 0; r0 < PV_TILE; r0 += 8) {
      float acc[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) acc[u] = tn[r0 + u];
#pragma unroll
      for (int c = 0; c < DP; c += 4) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const float4 v = ((const float4*)(tile + (r0 + u) * DP))[c / 4];
          acc[u] = fmaf(q[c], v.x, acc[u]);
          acc[u] = fmaf(q[c + 1], v.y, acc[u]);
          acc[u] = fmaf(q[c + 2], v.z, acc[u]);
          acc[u] = fmaf(q[c + 3], v.w, acc[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (acc[u] < bd) {
          bd = acc[u];
          best = p0 + r0 + u;
        }
    }
  }
  if (i < n && near) {
    float s = 0.f;
#pragma unroll
    for (int c = 0; c < DP; ++c) s = fmaf(0.25f * q[c], q[c], s);
    near[i] = fmaxf(bd + s, 0.f);
  } else if (i < n) {
    const unsigned place = (unsigned)best | (half && half[i] ? 0x80000000u : 0u);
    key[i] = ((unsigned long long)place << 32) | ordered_bits(X[i * DP + dim]);
    val[i] = (int)i;
  }
}

// The half of the tiles (bp points) of an order that every point lies in.
__global__ void k_halves(const int* __restrict__ perm, int64_t n, int bp, unsigned char* __restrict__ half) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    half[perm[i]] = (i % bp) >= bp / 2;
}

// Points sorted by half (n0 of the first) to tiles with a part of each: the i-th
// point of a half is in tile i / (bp / 2).
__global__ void k_join_halves(const int* __restrict__ in, int64_t n, int64_t n0, int bp, int* __restrict__ out) {
  const int h = bp / 2;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = i < n0 ? i : i - n0;
    out[k / h * bp + k % h + (i < n0 ? 0 : h)] = in[i];
  }
}

// Bounding boxes of groups of `rows` consecutive rows (permuted), dimension-major
// (lo[c * ng + g]); BF16: of the rounded coordinates.  mean, meant (optional):
// the groups' means, row-major with zero rows up to a multiple of 64 groups, and
// dimension-major.
template <bool BF16>
__global__ void __launch_bounds__(256) k_boxes(const float* __restrict__ X, const int* __restrict__ perm,
                                               int64_t n, int dp, int rows, int64_t ng, float* __restrict__ lo,
                                               float* __restrict__ hi, float* __restrict__ mean,
                                               float* __restrict__ meant) {
  __shared__ float slo[256], shi[256], sme[256];
  const int c = threadIdx.x % dp, r0 = threadIdx.x / dp, rs = blockDim.x / dp;
  const int64_t g = blockIdx.x;
  float a = FLT_MAX, b = -FLT_MAX, m = 0.f;
  const int64_t e = min(n, (g + 1) * rows);
  for (int64_t i = g * rows + r0; i < e; i += rs) {
    float v = X[(int64_t)perm[i] * dp + c];
    if (BF16) v = __bfloat162float(__float2bfloat16_rn(v));
    a = fminf(a, v);
    b = fmaxf(b, v);
    m += v;
  }
  slo[threadIdx.x] = a;
  shi[threadIdx.x] = b;
  sme[threadIdx.x] = m;
  __syncthreads();
  if (r0 == 0) {
    for (int r = 1; r < rs; ++r) {
      a = fminf(a, slo[r * dp + c]);
      b = fmaxf(b, shi[r * dp + c]);
      m += sme[r * dp + c];
    }
    if (g < ng) {
      lo[c * ng + g] = a;
      hi[c * ng + g] = b;
    }
    if (mean) {
      m = g < ng ? m / (float)(e - g * rows) : 0.f;
      mean[g * dp + c] = m;
      if (g < ng) meant[c * ng + g] = m;
    }
  }
}

// A bound of the points' largest norm from the tiles' boxes.
__global__ void __launch_bounds__(1024) k_far(const float* __restrict__ lo, const float* __restrict__ hi,
                                              int64_t nt, int dp, float* __restrict__ out) {
  __shared__ float red[32];
  float best = 0.f;
  for (int64_t t = threadIdx.x; t < nt; t += blockDim.x) {
    float s = 0.f;
    for (int c = 0; c < dp; ++c) {
      const float m = fmaxf(fabsf(lo[c * nt + t]), fabsf(hi[c * nt + t]));
      s = fmaf(m, m, s);
    }
    best = fmaxf(best, s);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x < 32) {
    best = red[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
    if (threadIdx.x == 0) *out = sqrtf(best);
  }
}

// sep[X * nt + Y] = min over the points x of tile X of x . (m_X - m_Y), m the
// tiles' means: 64 points x 64 means per step, 4 x 4 per thread, the tile's
// points kept in shared memory.  With the same of Y against X the gap of the two
// tiles' projections on the line through their means is (sep_XY + sep_YX) /
// |m_X - m_Y|.
constexpr int SEP_THREADS = 256;
template <int DP, bool BF16>
__global__ void __launch_bounds__(SEP_THREADS) k_sep(const float* __restrict__ X, const int* __restrict__ perm,
                                                     int64_t n, int bp, int64_t nt,
                                                     const float* __restrict__ mean, float* __restrict__ sep) {
  extern __shared__ __align__(16) float sp_dyn[];
  float* Q = sp_dyn;                    // [bp / 64][DP][64] points
  float* M = Q + (size_t)bp * DP;       // [DP][64] means
  float* own = M + DP * 64;             // [bp] x . m_X
  __shared__ float red[SEP_THREADS / 32][64];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, tx = tid & 15, ty = tid >> 4;
  const int64_t t = blockIdx.x, i0 = t * bp;
  for (int k = tid; k < bp * (DP / 4); k += SEP_THREADS) {
    const int r = k % 64 + 64 * (k / (16 * DP)), c4 = k / 64 % (DP / 4);
    float4 v = make_float4(0, 0, 0, 0);
    if (i0 + r < n) v = *(const float4*)(X + (int64_t)perm[i0 + r] * DP + 4 * c4);
    float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (BF16) e[u] = __bfloat162float(__float2bfloat16_rn(e[u]));
      Q[((r >> 6) * DP + 4 * c4 + u) * 64 + (r & 63)] = e[u];
    }
  }
  __syncthreads();
  for (int r = tid; r < bp; r += SEP_THREADS) {
    float s = 0.f;
    for (int c = 0; c < DP; ++c) s = fmaf(Q[((r >> 6) * DP + c) * 64 + (r & 63)], mean[t * DP + c], s);
    own[r] = i0 + r < n ? s : FLT_MAX;
  }
  for (int64_t y0 = (int64_t)blockIdx.y * 64; y0 < nt; y0 += (int64_t)gridDim.y * 64) {
    __syncthreads();
    for (int k = tid; k < 16 * DP; k += SEP_THREADS) {
      const int r = k % 64, c4 = k / 64;
      const float4 v = *(const float4*)(mean + (y0 + r) * DP + 4 * c4);
      M[(4 * c4) * 64 + r] = v.x;
      M[(4 * c4 + 1) * 64 + r] = v.y;
      M[(4 * c4 + 2) * 64 + r] = v.z;
      M[(4 * c4 + 3) * 64 + r] = v.w;
    }
    __syncthreads();
    float least[4] = {FLT_MAX, FLT_MAX, FLT_MAX, FLT_MAX};
    for (int sub = 0; sub < bp / 64; ++sub) {
      float acc[4][4] = {};
#pragma unroll 8
      for (int c = 0; c < DP; ++c) {
        const float4 qv = *(const float4*)(Q + (sub * DP + c) * 64 + 4 * ty);
        const float4 mv = *(const float4*)(M + c * 64 + 4 * tx);
        const float qa[4] = {qv.x, qv.y, qv.z, qv.w}, ma[4] = {mv.x, mv.y, mv.z, mv.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int u = 0; u < 4; ++u) acc[i][u] = fmaf(qa[i], ma[u], acc[i][u]);
      }
      const float4 ov = *(const float4*)(own + sub * 64 + 4 * ty);
      const float oa[4] = {ov.x, ov.y, ov.z, ov.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int u = 0; u < 4; ++u) least[u] = fminf(least[u], oa[i] - acc[i][u]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      least[u] = fminf(least[u], __shfl_xor_sync(0xffffffffu, least[u], 16));
      if (lane < 16) red[w][4 * tx + u] = least[u];
    }
    __syncthreads();
    if (tid < 64 && y0 + tid < nt) {
      float v = red[0][tid];
#pragma unroll
      for (int k = 1; k < SEP_THREADS / 32; ++k) v = fminf(v, red[k][tid]);
      sep[t * nt + y0 + tid] = v;
    }
  }
}

// The tiles of one query block by their lower bound: (squared distance, rounded
// down by more than its FP32 error) << 32 | place, place = twice the distance in
// tiles from the block's own, odd below it (see knn_list_tile).  The error of a
// projection is below 2^-15 (|m_X| + |m_Y|) max |p| (dot products of at most 64
// terms); a bound that is not a number counts as 0.
__global__ void k_tile_lists(const float* __restrict__ qlo, const float* __restrict__ qhi, int64_t nq,
                             const float* __restrict__ plo, const float* __restrict__ phi, int64_t np, int dp,
                             int bq, int bp, int n2, const float* __restrict__ meant,
                             const float* __restrict__ sep, const float* __restrict__ rmax,
                             unsigned long long* __restrict__ lists) {
  extern __shared__ unsigned long long tl_key[];
  __shared__ float lo[64], hi[64], mx[64];
  const int64_t b = blockIdx.x;
  const int own = knn_own_tile(b, bq, bp);
  for (int c = threadIdx.x; c < dp; c += blockDim.x) {
    lo[c] = qlo[c * nq + b];
    hi[c] = qhi[c * nq + b];
    mx[c] = meant[c * np + own];
  }
  __syncthreads();
  float own2 = 0.f;
  for (int c = 0; c < dp; ++c) own2 = fmaf(mx[c], mx[c], own2);
  const float far = *rmax;              // the largest |p|
  for (int t = threadIdx.x; t < n2; t += blockDim.x) {
    unsigned long long key = ~0ull;
    if (t < np) {
      float s = 0.f;
      for (int c = 0; c < dp; ++c) {
        const float g = fmaxf(0.f, fmaxf(plo[c * np + t] - hi[c], lo[c] - phi[c * np + t]));
        s = fmaf(g, g, s);
      }
      if (t != own) {
        float d2 = 0.f, m2 = 0.f;
        for (int c = 0; c < dp; ++c) {
          const float m = meant[c * np + t], d = m - mx[c];
          d2 = fmaf(d, d, d2);
          m2 = fmaf(m, m, m2);
        }
        const float gap = sep[(int64_t)own * np + t] + sep[(int64_t)t * np + own] -
                          0x1p-15f * (sqrtf(own2) + sqrtf(m2)) * far;
        if (gap > 0.f && d2 > 0.f) s = fmaxf(s, gap * gap / d2);
      }
      s *= 1.f - 0x1p-16f;
      if (!(s >= 0.f && s <= FLT_MAX)) s = 0.f;
      const unsigned place = t >= own ? 2u * (unsigned)(t - own) : 2u * (unsigned)(own - t) + 1u;
      key = ((unsigned long long)__float_as_uint(s) << 32) | place;
    }
    tl_key[t] = key;
  }
  __syncthreads();
  for (int k = 2; k <= n2; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int x = threadIdx.x; x < n2 / 2; x += blockDim.x) {
        const int i = 2 * j * (x / j) + x % j, l = i + j;
        const unsigned long long a = tl_key[i], d = tl_key[l];
        if ((a > d) == ((i & k) == 0)) {
          tl_key[i] = d;
          tl_key[l] = a;
        }
      }
      __syncthreads();
    }
  }
  for (int t = threadIdx.x; t < np; t += blockDim.x) lists[b * np + t] = tl_key[t];
}

}  // namespace

KnnSpread sv_knn_spread(sv_context* ctx, const float* X32, int64_t n, int dp, int d) {
  DevBuf<double> mom(2 * dp);
  sv_memset(ctx, mom.get(), 0, 2 * dp * 8);
  sv_launch(ctx, "knn_order", k_dim_moments, dim3(sv_grid_for(ctx, n, 256, 2)), dim3(256 / dp * dp), 0, X32, n, dp,
            mom.get());
  std::vector<double> hm(2 * dp);
  sv_d2h(ctx, hm.data(), mom.get(), 2 * dp * 8);
  KnnSpread s;
  double best = -1;
  for (int c = 0; c < d; ++c) {
    double mean = hm[c] / (double)n, var = hm[dp + c] / (double)n - mean * mean;
    s.sum += var;
    if (var > best) {
      best = var;
      s.dim = c;
    }
  }
  return s;
}

bool sv_knn_order(sv_context* ctx, const float* X32, int64_t n, int dp, int d, int bq, int bp,
                  const KnnSpread& spread, KnnOrder& o, const int* halves_of) {
  const bool bf16 = halves_of != nullptr;
  const int64_t nq = (n + bq - 1) / bq, np = (n + bp - 1) / bp;
  // worth it from a few tiles up; a list has to fit the shared memory that it is
  // sorted in (16,384 tiles: 1,048,576 points of the FP32 search's 64, 4 M of the
  // tensor-core search's 256), and all of them 1/64 of the device's memory (4.4 GB of
  // 284: 4.3 M points of the tensor-core search); beyond that the order stays the
  // caller's
  if (np < 4 || np > KNN_MAX_TILES || (size_t)(nq * np) * 8 > ctx->pool->keep / 4) return false;
  const int64_t npad = (np + 63) / 64 * 64;
  // a cell of about two tiles of 64 points while that takes few pivots (a cluster
  // without one is split among its neighbours' cells), more than 512 only where a
  // cell would hold 2,000 points or more
  const int P = (int)std::max<int64_t>(8, std::min<int64_t>(n >= 1 << 20 ? PV_MAX : PV_MAX / 2, n / 128));
  DevBuf<float> rows((size_t)P * dp), norms(P);
  sv_launch(ctx, "knn_pivots", k_pivots, dim3(1), dim3(PV_MAX), 0, X32, n, dp, P, rows.get(), norms.get());
  auto assign = [&](int64_t m, int64_t step, const unsigned char* half, unsigned long long* key, int* val,
                    float* near) {
    const dim3 g((unsigned)((m + PV_THREADS - 1) / PV_THREADS));
#define PV_CASE(D)                                                                                             \
  case D:                                                                                                      \
    sv_launch(ctx, "knn_assign", k_pivot_assign<D>, g, dim3(PV_THREADS), 0, X32, m, (const float*)rows.get(),   \
              (const float*)norms.get(), P, spread.dim, half, key, val, step, near);                            \
    break;
    switch (dp) {
      PV_CASE(8) PV_CASE(16) PV_CASE(24) PV_CASE(32) PV_CASE(40) PV_CASE(48) PV_CASE(56) PV_CASE(64)
      default: sv_throw(SV_ERR_UNSUPPORTED, "padded dimension %d", dp);
    }
#undef PV_CASE
  };
  if (halves_of) {
    const int64_t m = std::min<int64_t>(n, PV_SAMPLE);
    DevBuf<float> near(m);
    assign(m, n / m, nullptr, nullptr, nullptr, near.get());
    std::vector<float> hn(m);
    sv_d2h(ctx, hn.data(), near.get(), m * 4);
    double sum = 0;
    for (float v : hn) sum += v;
    if (!(sum / (double)m < PV_NEAR * 2 * spread.sum)) return false;
  }
  int64_t n2 = 2048;
  while (n2 < n) n2 <<= 1;
  DevBuf<unsigned long long> key(n2);
  DevBuf<unsigned char> half;
  if (halves_of) {
    half.alloc(n);
    sv_launch(ctx, "knn_halves", k_halves, dim3(sv_grid_for(ctx, n, 256)), dim3(256), 0, halves_of, n, bp, half.get());
  }
  o.perm.alloc(n2);
  assign(n, 1, half.get(), key.get(), o.perm.get(), nullptr);
  sv_sort_pairs(ctx, key.get(), o.perm.get(), n, n2);
  if (halves_of) {
    DevBuf<int> joined(n);
    const int64_t n0 = n / bp * (bp / 2) + std::min<int64_t>(n % bp, bp / 2);
    sv_launch(ctx, "knn_join_halves", k_join_halves, dim3(sv_grid_for(ctx, n, 256)), dim3(256), 0,
              (const int*)o.perm.get(), n, n0, bp, joined.get());
    o.perm = std::move(joined);
  }
  DevBuf<float> ql((size_t)nq * dp), qh((size_t)nq * dp), pl((size_t)np * dp), ph((size_t)np * dp);
  DevBuf<float> mean((size_t)npad * dp), meant((size_t)np * dp), sep((size_t)(np * np)), rmax(1);
  auto boxes = bf16 ? k_boxes<true> : k_boxes<false>;
  const dim3 bt(256 / dp * dp);
  const int* pm = o.perm.get();
  sv_launch(ctx, "knn_boxes", boxes, dim3((unsigned)nq), bt, 0, X32, pm, n, dp, bq, nq, ql.get(), qh.get(),
            (float*)nullptr, (float*)nullptr);
  sv_launch(ctx, "knn_boxes", boxes, dim3((unsigned)npad), bt, 0, X32, pm, n, dp, bp, np, pl.get(), ph.get(),
            mean.get(), meant.get());
  sv_launch(ctx, "knn_far", k_far, dim3(1), dim3(1024), 0, (const float*)pl.get(), (const float*)ph.get(), np, dp,
            rmax.get());
  const size_t ssm = ((size_t)bp * dp + (size_t)dp * 64 + bp) * 4;
  const dim3 gs((unsigned)np, (unsigned)std::max<int64_t>(1, std::min<int64_t>(npad / 64, 1 + 8 * ctx->num_sms / np)));
#define SEP_CASE(D)                                                                                       \
  case D: {                                                                                               \
    auto kern = bf16 ? k_sep<D, true> : k_sep<D, false>;                                                  \
    SV_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ssm));           \
    sv_launch(ctx, "knn_sep", kern, gs, dim3(SEP_THREADS), ssm, X32, pm, n, bp, np, (const float*)mean.get(), \
              sep.get());                                                                                 \
    break;                                                                                                \
  }
  switch (dp) {
    SEP_CASE(8) SEP_CASE(16) SEP_CASE(24) SEP_CASE(32) SEP_CASE(40) SEP_CASE(48) SEP_CASE(56) SEP_CASE(64)
  }
#undef SEP_CASE
  int t2 = 2;
  while (t2 < np) t2 <<= 1;
  o.lists.alloc((size_t)(nq * np));
  o.ntiles = (int)np;
  SV_CUDA(cudaFuncSetAttribute(k_tile_lists, cudaFuncAttributeMaxDynamicSharedMemorySize, KNN_MAX_TILES * 8));
  sv_launch(ctx, "knn_tile_lists", k_tile_lists, dim3((unsigned)nq), dim3(std::max(32, std::min(1024, t2 / 2))),
            (size_t)t2 * 8, (const float*)ql.get(), (const float*)qh.get(), nq, (const float*)pl.get(),
            (const float*)ph.get(), np, dp, bq, bp, t2, (const float*)meant.get(), (const float*)sep.get(),
            (const float*)rmax.get(), o.lists.get());
  return true;
}
