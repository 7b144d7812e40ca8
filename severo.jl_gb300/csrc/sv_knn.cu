// Exact k-nearest neighbours (replaces the approximate native FindNeighbours*
// routines that src/neighbours.jl:19-74 calls).
//
// Stage 1 (candidates): every query scans every point.  The distance key is the
// GEMM form |p|^2 - 2 q.p (|q|^2 is constant per query); each query keeps its
// K2 >= 2k smallest keys.  Two implementations:
//   * FP32 CUDA cores (k_knn_fp32): 64 queries x 64 points per block and tile;
//     from KNN_ORDER_MIN points up in the order of sv_knn_order, tiles out of
//     every query's reach left out;
//   * BF16 tcgen05 tensor cores with FP32 accumulation in TMEM (sv_knn_tc.cu).
// Stage 2 (k_rerank): exact FP32 distances sum (q_c - p_c)^2 of the K2
// candidates, sorted by (distance, index); the point itself first when
// include_self, excluded otherwise.
//
// Layout in HBM: points row-major FP32 [n][dp] (dp = d rounded up to 8, zero
// padded) plus FP32 squared norms; candidates [n][K2]; results [n][k] (0-based).
#include "sv_internal.cuh"
#include "sv_knn_order.cuh"
#include <float.h>
#include <type_traits>

int sv_knn_tc_candidates(sv_context* ctx, const float* X32, const float* sq, int64_t n, int dp, int d,
                         int K2, int include_self, int32_t* cand,
                         const std::vector<int64_t>* segs, bool lists);
sv_context* sv_default_context();

namespace {

constexpr int KNN_THREADS = 256;
constexpr int KNN_TILE = 64;       // points per tile and queries per block
constexpr int KNN_LIST = 64;       // most candidates of a query (the length of its sorted list)
constexpr int KNN_MERGE = 2;       // queries merged at a time
// Points from which the order and the tile lists pay (they take 0.2-0.3 ms up to
// 10,000 points): in 50 dimensions, k = 8, in 60 clusters 4,000 points 0.41 ms
// without and 0.50 with, 10,000 1.01 and 0.69, 30,000 4.8 and 1.3; without clusters
// 1.01 and 1.26, 4.8 and 5.2.
constexpr int64_t KNN_ORDER_MIN = 8192;

// X (n x d, column-major, leading dim ld, FP32 or FP64) -> row-major FP32 [n][dp]
// (optionally unit-normalised rows for the cosine metric) and squared norms.
template <typename T>
__global__ void k_pack_rows(const T* __restrict__ X, int64_t ld, int64_t n, int d, int dp,
                            int normalise, float* __restrict__ out, float* __restrict__ sq) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    double nr = 1.0;
    if (normalise) {
      double s = 0;
      for (int c = 0; c < d; ++c) {
        double v = (double)X[(int64_t)c * ld + i];
        s += v * v;
      }
      nr = s > 0 ? sqrt(s) : 1.0;
    }
    float s2 = 0.f;
    for (int c = 0; c < dp; ++c) {
      float v = c < d ? (float)((double)X[(int64_t)c * ld + i] / nr) : 0.f;
      out[i * dp + c] = v;
      s2 += v * v;
    }
    sq[i] = s2;
  }
}

// ---- FP32 candidates -----------------------------------------------------------
// Points tile by tile, dimension-major within a tile (Xt[tile][c][64], zero rows
// past the end) with their norms (FLT_MAX past the end) and original indices; the
// largest norm (float bits) for the pruning margin.
__global__ void k_tiles_fp32(const float* __restrict__ X, const float* __restrict__ sq, const int* __restrict__ perm,
                             int64_t n, int dp, int64_t npad, float* __restrict__ Xt, float* __restrict__ sqt,
                             int* __restrict__ orig, unsigned* __restrict__ pmax) {
  const int q4 = dp / 4;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < npad * q4;
       e += (int64_t)gridDim.x * blockDim.x) {
    // 64 consecutive threads: the rows of one tile, the same four dimensions
    const int64_t t = e / (KNN_TILE * q4);
    const int r = (int)(e % KNN_TILE), c4 = (int)(e / KNN_TILE % q4);
    const int64_t i = t * KNN_TILE + r, src = i < n ? (perm ? perm[i] : i) : 0;
    const float4 v = i < n ? ((const float4*)X)[src * q4 + c4] : make_float4(0, 0, 0, 0);
    float* o = Xt + t * KNN_TILE * dp + (int64_t)c4 * 4 * KNN_TILE + r;
    o[0] = v.x;
    o[KNN_TILE] = v.y;
    o[2 * KNN_TILE] = v.z;
    o[3 * KNN_TILE] = v.w;
    if (c4 == 0) {
      const float s = i < n ? sq[src] : FLT_MAX;
      sqt[i] = s;
      orig[i] = i < n ? (int)src : -1;
      if (i < n) atomicMax(pmax, __float_as_uint(s));
    }
  }
}

__device__ __forceinline__ unsigned key_bits(float v) {
  const unsigned u = __float_as_uint(v);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_float(unsigned b) {
  return __uint_as_float((b & 0x80000000u) ? (b & 0x7fffffffu) : ~b);
}

// M times 64 values over a warp, element lane + 32 r in v[.][r]: the compare-exchange
// of element e with e ^ stride, ascending where (e & dir) == 0
template <int M>
__device__ __forceinline__ void w64_step(unsigned long long (&v)[M][2], int stride, int dir) {
  const int lane = threadIdx.x & 31;
  if (stride == 32) {
    const bool up = (lane & dir) == 0;
#pragma unroll
    for (int i = 0; i < M; ++i) {
      const unsigned long long x = v[i][0], y = v[i][1];
      const bool keep = (x < y) == up;
      v[i][0] = keep ? x : y;
      v[i][1] = keep ? y : x;
    }
    return;
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const bool least = (((lane + 32 * r) & dir) == 0) == ((lane & stride) == 0);
#pragma unroll
    for (int i = 0; i < M; ++i) {
      const unsigned long long o = __shfl_xor_sync(0xffffffffu, v[i][r], stride);
      v[i][r] = (o < v[i][r]) == least ? o : v[i][r];
    }
  }
}

// The `keep` smallest keys |p|^2 - 2 q.p of every query, equal keys by index, in K2
// places (-1 after them).  Block of
// 64 queries; per tile of 64 points a thread forms a 4 x 4 patch of keys (two
// 16-byte shared loads per 16 FMAs; each key one chain over the dimensions), and
// keys that pass their query's threshold are appended to the query's buffer in
// shared memory.  A buffer above half full is merged into the query's sorted list
// by a warp (bitonic sort and merge of 64 packed (key, index) words), which
// lowers the threshold; keys that found a full buffer try again after that.  With
// a list of the tiles by their lower bound (sv_knn_order) the scan ends at the
// first tile beyond every query's threshold + |q|^2 + a margin for the keys' FP32
// rounding (2^-15 (|q|^2 + max |p|^2), several times its bound).
// A merge is a chain of 27 shuffled compare-exchanges, and with few blocks, or in
// a scan's first tiles, where most keys pass, the warps wait for it: a warp merges
// two queries at a time (500 points in 50 dimensions, 64 candidates: 0.36 -> 0.12
// ms; 30,000 without a list: 8.6 -> 5.1 ms; four at a time are 3% slower).
// 30,000 points in 60 clusters x 50 dimensions, 64 candidates, with lists: 0.8 ms
// for the tiles; a query per thread with 64 candidates in registers over every
// tile, 235 blocks of four warps, took 7.5 ms.
template <int DP>
__global__ void __launch_bounds__(KNN_THREADS, 2) k_knn_fp32(
    const float* __restrict__ Xt, const float* __restrict__ sqt, const int* __restrict__ orig, int64_t n,
    int keep, int K2, int32_t* __restrict__ cand, const unsigned long long* __restrict__ lists,
    const unsigned* __restrict__ pmax) {
  extern __shared__ __align__(16) unsigned char knn_dyn[];
  float* Q = (float*)knn_dyn;                       // [DP][64], times -2
  float* Pt = Q + DP * KNN_TILE;                    // [DP][64]
  unsigned long long* ent = (unsigned long long*)(Pt + DP * KNN_TILE);   // [query][list 64, buffer 64]
  __shared__ __align__(16) float thr[KNN_TILE], psq[KNN_TILE];
  __shared__ unsigned long long thr64[KNN_TILE];
  __shared__ int cnt[KNN_TILE], pid[KNN_TILE];
  __shared__ float bound[KNN_TILE], wm[KNN_THREADS / 32];
  static_assert(KNN_TILE / (KNN_THREADS / 32) == 8, "a warp's queries");
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, tx = tid & 15, ty = tid >> 4;
  const int64_t ntiles = (n + KNN_TILE - 1) / KNN_TILE;
  const int own = blockIdx.x;
  const unsigned long long* list = lists ? lists + (int64_t)blockIdx.x * ntiles : nullptr;
  constexpr int NV = (DP * KNN_TILE / 4 + KNN_THREADS - 1) / KNN_THREADS;   // float4 per thread and tile
  float4 pre[NV];
  auto fetch = [&](int64_t t) {
    const float4* src = (const float4*)(Xt + t * KNN_TILE * DP);
#pragma unroll
    for (int u = 0; u < NV; ++u)
      if (tid + u * KNN_THREADS < DP * KNN_TILE / 4) pre[u] = src[tid + u * KNN_THREADS];
  };
  fetch(own);
#pragma unroll
  for (int u = 0; u < NV; ++u)
    if (tid + u * KNN_THREADS < DP * KNN_TILE / 4)
      ((float4*)Q)[tid + u * KNN_THREADS] =
          make_float4(-2.f * pre[u].x, -2.f * pre[u].y, -2.f * pre[u].z, -2.f * pre[u].w);
  for (int k = tid; k < KNN_TILE * 2 * KNN_LIST; k += KNN_THREADS) ent[k] = ~0ull;
  if (tid < KNN_TILE) {
    thr[tid] = FLT_MAX;
    thr64[tid] = (unsigned long long)key_bits(FLT_MAX) << 32;
    cnt[tid] = 0;
    const bool in = own * (int64_t)KNN_TILE + tid < n;
    bound[tid] = in ? __int_as_float(0x7f800000) : -FLT_MAX;
  }
  if (tid < KNN_THREADS / 32) wm[tid] = __int_as_float(0x7f800000);
  unsigned long long e0 = list ? list[0] : 0;
  int64_t t = list ? knn_list_tile(e0, own) : 0;
  if (t != own) fetch(t);
  // merges the buffers of M queries into their lists (a warp)
  auto merge = [&](auto m_tag, unsigned& need) {
    constexpr int M = decltype(m_tag)::value;
    unsigned long long a[M][2], b[M][2];
    int q[M];
#pragma unroll
    for (int i = 0; i < M; ++i) {
      q[i] = w + 8 * (__ffs(need) - 1);             // the last one again when there are fewer
      if (need & (need - 1)) need &= need - 1;
      else if (i == M - 1) need = 0;
      const unsigned long long* L = ent + (size_t)q[i] * 2 * KNN_LIST;
      const int m = min(cnt[q[i]], KNN_LIST);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        a[i][r] = L[lane + 32 * r];
        b[i][r] = lane + 32 * r < m ? L[KNN_LIST + lane + 32 * r] : ~0ull;
      }
    }
#pragma unroll
    for (int k = 2; k <= 64; k <<= 1)
#pragma unroll
      for (int s = k >> 1; s > 0; s >>= 1) w64_step(b, s, k);
    // the 64 smallest of two ascending sequences: min(a[e], b[63 - e]), bitonic
#pragma unroll
    for (int i = 0; i < M; ++i) {
      const unsigned long long r0 = __shfl_sync(0xffffffffu, b[i][1], 31 - lane);
      const unsigned long long r1 = __shfl_sync(0xffffffffu, b[i][0], 31 - lane);
      a[i][0] = a[i][0] < r0 ? a[i][0] : r0;
      a[i][1] = a[i][1] < r1 ? a[i][1] : r1;
    }
#pragma unroll
    for (int s = 32; s > 0; s >>= 1) w64_step(a, s, 64);
#pragma unroll
    for (int i = 0; i < M; ++i) {
      unsigned long long* L = ent + (size_t)q[i] * 2 * KNN_LIST;
      L[lane] = a[i][0];
      L[lane + 32] = a[i][1];
      const unsigned long long last = keep > 32 ? a[i][1] : a[i][0];
      if (lane == ((keep - 1) & 31)) {
        if (last != ~0ull) {
          thr[q[i]] = key_float((unsigned)(last >> 32));
          thr64[q[i]] = last;
        }
        cnt[q[i]] = 0;
        const int64_t qi = own * (int64_t)KNN_TILE + q[i];
        if (last != ~0ull && qi < n) {
          const float v = thr[q[i]] + sqt[qi] + 0x1p-15f * (sqt[qi] + __uint_as_float(*pmax));
          bound[q[i]] = v != v ? __int_as_float(0x7f800000) : v;   // no bound from a NaN
        }
      }
    }
    __syncwarp();
  };
  // merges the buffers with more than `above` entries; true when there were any
  auto settle = [&](int above) {
    unsigned need = __ballot_sync(0xffffffffu, lane < 8 && cnt[w + 8 * (lane & 7)] > above);
    if (!need) return false;
    while (need) {
      if (need & (need - 1)) merge(std::integral_constant<int, KNN_MERGE>(), need);
      else merge(std::integral_constant<int, 1>(), need);
    }
    return true;
  };
  for (int64_t it = 0; it < ntiles; ++it) {
    __syncthreads();                                // the previous tile is done with Pt
    if (list && it > 0) {
      float T = wm[0];
#pragma unroll
      for (int u = 1; u < KNN_THREADS / 32; ++u) T = fmaxf(T, wm[u]);
      if (knn_list_bound(e0) > T) break;
    }
#pragma unroll
    for (int u = 0; u < NV; ++u)
      if (tid + u * KNN_THREADS < DP * KNN_TILE / 4) ((float4*)Pt)[tid + u * KNN_THREADS] = pre[u];
    if (tid < KNN_TILE) {
      psq[tid] = sqt[t * KNN_TILE + tid];
      pid[tid] = orig[t * KNN_TILE + tid];
    }
    const int64_t tc = t;
    if (it + 1 < ntiles) {
      e0 = list ? list[it + 1] : 0;
      t = list ? knn_list_tile(e0, own) : it + 1;
      fetch(t);
    }
    __syncthreads();
    float acc[4][4];
    {
      const float4 v = *(const float4*)(psq + 4 * tx);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc[i][0] = v.x;
        acc[i][1] = v.y;
        acc[i][2] = v.z;
        acc[i][3] = v.w;
      }
    }
#pragma unroll 8
    for (int c = 0; c < DP; ++c) {
      const float4 qv = *(const float4*)(Q + c * KNN_TILE + 4 * ty);
      const float4 pv = *(const float4*)(Pt + c * KNN_TILE + 4 * tx);
      const float qa[4] = {qv.x, qv.y, qv.z, qv.w}, pa[4] = {pv.x, pv.y, pv.z, pv.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[i][u] = fmaf(qa[i], pa[u], acc[i][u]);
    }
    unsigned todo = 0;
    {
      const float4 tv = *(const float4*)(thr + 4 * ty);
      const float ta[4] = {tv.x, tv.y, tv.z, tv.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (acc[i][u] <= ta[i] && pid[4 * tx + u] >= 0 && !(tc == own && 4 * ty + i == 4 * tx + u))
            todo |= 1u << (4 * i + u);
    }
    while (true) {
      if (todo) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (todo & (1u << (4 * i + u))) {
              const int q = 4 * ty + i;
              const unsigned long long e =
                  ((unsigned long long)key_bits(acc[i][u]) << 32) | (unsigned)pid[4 * tx + u];
              if (e < thr64[q]) {
                const int pos = atomicAdd(&cnt[q], 1);
                if (pos < KNN_LIST) {
                  ent[(size_t)q * 2 * KNN_LIST + KNN_LIST + pos] = e;
                  todo &= ~(1u << (4 * i + u));
                }
              } else {
                todo &= ~(1u << (4 * i + u));
              }
            }
          }
        }
      }
      const int again = __syncthreads_or(todo != 0);
      if (settle(KNN_LIST / 2)) {
        float v = lane < KNN_TILE / (KNN_THREADS / 32) ? bound[w + lane * (KNN_THREADS / 32)] : -FLT_MAX;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0) wm[w] = v;
      }
      if (!again) break;
      __syncthreads();
    }
  }
  __syncthreads();
  settle(0);
  for (int q = w; q < KNN_TILE; q += KNN_THREADS / 32) {
    const int64_t qi = own * (int64_t)KNN_TILE + q;
    if (qi >= n) break;
    const unsigned long long* L = ent + (size_t)q * 2 * KNN_LIST;
    int32_t* o = cand + (int64_t)orig[qi] * K2;
    for (int k = lane; k < K2; k += 32) o[k] = k >= keep || L[k] == ~0ull ? -1 : (int32_t)(unsigned)L[k];
  }
}

// Exact FP32 re-rank: one warp per query; K2 candidates sorted by (d2, index)
// (a bitonic sort over the next power of two, P2, padded with the largest key).
template <int DP>
__global__ void k_rerank(const float* __restrict__ X, int64_t n, const int32_t* __restrict__ cand,
                         int K2, int k, int include_self, int cosine, int32_t* __restrict__ out_idx,
                         float* __restrict__ out_dist) {
  extern __shared__ unsigned long long keys_all[];
  int P2 = 32;
  while (P2 < K2) P2 <<= 1;
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned long long* keys = keys_all + wid * P2;
  int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t qi = warp; qi < n; qi += nwarps) {
    const float* q = X + qi * DP;
    for (int t = lane; t < P2; t += 32) {
      int c = t < K2 ? cand[qi * K2 + t] : -1;
      unsigned long long key = ~0ull;
      if (c >= 0 && c != qi) {
        // one chain over the dimensions; 16-byte loads (300,000 queries of 64
        // candidates in 50 dimensions: 1.1 ms, with 4-byte ones 2.2)
        const float4* p4 = (const float4*)(X + (int64_t)c * DP);
        const float4* q4 = (const float4*)q;
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < DP / 4; ++j) {
          const float4 a = q4[j], b = p4[j];
          float df = a.x - b.x;
          s = fmaf(df, df, s);
          df = a.y - b.y;
          s = fmaf(df, df, s);
          df = a.z - b.z;
          s = fmaf(df, df, s);
          df = a.w - b.w;
          s = fmaf(df, df, s);
        }
        // order-preserving bit pattern of a float (all finite here)
        unsigned int b = __float_as_uint(s);
        b = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
        key = ((unsigned long long)b << 32) | (unsigned int)c;
      }
      keys[t] = key;
    }
    __syncwarp();
    // bitonic sort of the P2 keys by the warp
    for (int kk = 2; kk <= P2; kk <<= 1) {
      for (int j = kk >> 1; j > 0; j >>= 1) {
        for (int i = lane; i < P2; i += 32) {
          int ixj = i ^ j;
          if (ixj > i) {
            unsigned long long a = keys[i], b = keys[ixj];
            bool up = (i & kk) == 0;
            if ((a > b) == up) {
              keys[i] = b;
              keys[ixj] = a;
            }
          }
        }
        __syncwarp();
      }
    }
    // the point itself first when include_self (distance 0), then the others
    int off = include_self ? 1 : 0;
    if (include_self && lane == 0) {
      out_idx[qi * k] = (int32_t)qi;
      out_dist[qi * k] = 0.f;
    }
    for (int t = lane; t + off < k; t += 32) {
      unsigned long long key = keys[t];
      int c = (int)(key & 0xffffffffu);
      unsigned int b = (unsigned int)(key >> 32);
      b = (b & 0x80000000u) ? (b & 0x7fffffffu) : ~b;
      float s = __uint_as_float(b);
      if (s < 0.f) s = 0.f;
      out_idx[qi * k + t + off] = key == ~0ull ? -1 : c;
      out_dist[qi * k + t + off] = cosine ? 0.5f * s : sqrtf(s);
    }
    __syncwarp();
  }
}

template <int DP>
void launch_fp32(sv_context* ctx, const float* X, const float* sq, int64_t n, int d, int keep, int K2, int32_t* cand,
                 bool lists) {
  const int64_t ntiles = (n + KNN_TILE - 1) / KNN_TILE, npad = ntiles * KNN_TILE;
  KnnOrder ord;
  const bool listed = lists && n >= KNN_ORDER_MIN && sv_knn_order(ctx, X, n, DP, d, KNN_TILE, KNN_TILE,
                                                         sv_knn_spread(ctx, X, n, DP, d), ord);
  DevBuf<float> Xt((size_t)npad * DP), sqt(npad);
  DevBuf<int> orig(npad);
  DevBuf<unsigned> pmax(1);
  sv_memset(ctx, pmax.get(), 0, 4);
  sv_launch(ctx, "knn_tiles_layout", k_tiles_fp32, dim3(sv_grid_for(ctx, npad * DP / 4, 256, 8)), dim3(256), 0, X, sq,
            listed ? (const int*)ord.perm.get() : (const int*)nullptr, n, DP, npad, Xt.get(), sqt.get(), orig.get(),
            pmax.get());
  const size_t smem = (size_t)2 * DP * KNN_TILE * 4 + (size_t)KNN_TILE * 2 * KNN_LIST * 8;
  SV_CUDA(cudaFuncSetAttribute(k_knn_fp32<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  sv_launch(ctx, "knn_fp32_tiles", k_knn_fp32<DP>, dim3((unsigned)ntiles), dim3(KNN_THREADS), smem,
            (const float*)Xt.get(), (const float*)sqt.get(), (const int*)orig.get(), n, keep, K2, cand,
            listed ? (const unsigned long long*)ord.lists.get() : (const unsigned long long*)nullptr,
            (const unsigned*)pmax.get());
}

template <int DP>
void launch_rerank(sv_context* ctx, const float* X, int64_t n, const int32_t* cand, int K2, int k,
                   int inc, int cosine, int32_t* idx, float* dist) {
  int P2 = 32;
  while (P2 < K2) P2 <<= 1;
  sv_launch(ctx, "knn_rerank", k_rerank<DP>, dim3(sv_grid_for(ctx, n * 32, 256, 8)), dim3(256),
            (size_t)8 * P2 * 8, X, n, cand, K2, k, inc, cosine, idx, dist);
}

// candidate indices of one sample (local, >= 0) -> stacked rows
__global__ void k_add_offset(int32_t* __restrict__ c, int64_t count, int32_t off) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < count;
       e += (int64_t)gridDim.x * blockDim.x)
    if (c[e] >= 0) c[e] += off;
}

__global__ void k_to_host_layout(const int32_t* __restrict__ idx, const float* __restrict__ dist,
                                 int64_t n, int k, int32_t* __restrict__ oidx, float* __restrict__ of,
                                 double* __restrict__ od) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n * k;
       e += (int64_t)gridDim.x * blockDim.x) {
    int64_t i = e / k;
    int t = (int)(e % k);
    if (oidx) oidx[(int64_t)t * n + i] = idx[e] + 1;   // column-major n x k, 1-based
    if (of) of[(int64_t)t * n + i] = dist[e];
    if (od) od[(int64_t)t * n + i] = (double)dist[e];
  }
}

}  // namespace

// Core: X32 row-major [n][dp] FP32 with norms -> knn handle (row-major, 0-based).
// segs (optional, nseg + 1 row offsets): stacked samples, each point's
// neighbours searched among the points of its own sample only.
static void knn_core(sv_context* ctx, const float* X32, const float* sq, int64_t n, int dp, int d, int k,
                     int include_self, int cosine, int precision, sv_knn* out,
                     const std::vector<int64_t>* segs = nullptr) {
  // candidates per query, at least 2k: 32 (k <= 16) or 64 from the FP32 tiles, the point
  // itself among them where it is its own neighbour; 40 (k <= 20) or 64 from the
  // tensor-core tiles.  More than 2k because the FP32 keys cancel far from the origin:
  // 4,000 points in 50 dimensions 500 times their spread away, k = 8: recall 0.999 with
  // 32, 0.976 with 16
  int K2 = precision == SV_KNN_BF16 ? (2 * k <= 40 ? 40 : 64) : (2 * k <= 32 ? 32 : 64);
  if (2 * k > 64) sv_throw(SV_ERR_UNSUPPORTED, "k = %d exceeds the supported maximum of 32", k);
  DevBuf<int32_t> cand((size_t)n * K2);
  sv_if_memory([&](bool lists) {
    if (precision == SV_KNN_BF16) {
      int st = sv_knn_tc_candidates(ctx, X32, sq, n, dp, d, K2, include_self, cand.get(), segs, lists);
      if (st != SV_OK) sv_throw(st, "tensor-core kNN failed");
      return;
    }
    // FP32 tiles: one launch per sample (each on its own rows)
    const int keep = include_self ? K2 - 1 : K2;   // besides the point itself
    std::vector<int64_t> one = {0, n};
    const std::vector<int64_t>& sg = segs ? *segs : one;
    for (size_t g = 0; g + 1 < sg.size(); ++g) {
      int64_t o = sg[g], ns = sg[g + 1] - sg[g];
      if (ns <= 0) continue;
      const float* Xs = X32 + o * dp;
      const float* qs = sq + o;
      int32_t* cs = cand.get() + o * K2;
      switch (dp) {
        case 8: launch_fp32<8>(ctx, Xs, qs, ns, d, keep, K2, cs, lists); break;
        case 16: launch_fp32<16>(ctx, Xs, qs, ns, d, keep, K2, cs, lists); break;
        case 24: launch_fp32<24>(ctx, Xs, qs, ns, d, keep, K2, cs, lists); break;
        case 32: launch_fp32<32>(ctx, Xs, qs, ns, d, keep, K2, cs, lists); break;
        case 40: launch_fp32<40>(ctx, Xs, qs, ns, d, keep, K2, cs, lists); break;
        case 48: launch_fp32<48>(ctx, Xs, qs, ns, d, keep, K2, cs, lists); break;
        case 56: launch_fp32<56>(ctx, Xs, qs, ns, d, keep, K2, cs, lists); break;
        case 64: launch_fp32<64>(ctx, Xs, qs, ns, d, keep, K2, cs, lists); break;
        default: sv_throw(SV_ERR_UNSUPPORTED, "padded dimension %d", dp);
      }
      if (o > 0)
        sv_launch(ctx, "knn_offset", k_add_offset, dim3(sv_grid_for(ctx, ns * K2, 256, 4)), dim3(256), 0,
                  cs, ns * K2, (int32_t)o);
    }
  });
  out->n = n;
  out->k = k;
  out->idx.alloc((size_t)n * k);
  out->dist.alloc((size_t)n * k);
  switch (dp) {
#define RR(D) case D: launch_rerank<D>(ctx, X32, n, cand.get(), K2, k, include_self, cosine, out->idx.get(), out->dist.get()); break;
    RR(8) RR(16) RR(24) RR(32) RR(40) RR(48) RR(56) RR(64)
#undef RR
  }
  sv_sync(ctx);
}

static void knn_validate(int64_t n, int64_t d, int64_t k, int metric, int include_self, int precision) {
  SV_REQUIRE(n >= 1 && d >= 1, "bad sizes");
  SV_REQUIRE(n < (1ll << 31), "n exceeds Int32 indices");
  SV_REQUIRE(k >= 1 && k <= (include_self ? n : n - 1), "k must be in 1..n (1..n-1 without self)");
  SV_REQUIRE(metric == SV_EUCLIDEAN || metric == SV_COSINE, "unknown metric");
  SV_REQUIRE(precision == SV_KNN_FP32 || precision == SV_KNN_BF16, "unknown precision");
  if (d > 64) sv_throw(SV_ERR_UNSUPPORTED, "d = %lld > 64 dimensions", (long long)d);
}

static void knn_outputs(sv_context* ctx, sv_knn* h, int dtype, int32_t* nn_index, void* distances) {
  int64_t n = h->n;
  int k = (int)h->k;
  if (!nn_index && !distances) return;
  DevBuf<int32_t> oi(nn_index ? (size_t)n * k : 1);
  DevBuf<unsigned char> od(distances ? (size_t)n * k * (dtype == SV_F64 ? 8 : 4) : 1);
  sv_launch(ctx, "knn_layout", k_to_host_layout, dim3(sv_grid_for(ctx, n * k, 256, 8)), dim3(256), 0,
            (const int32_t*)h->idx.get(), (const float*)h->dist.get(), n, k,
            nn_index ? oi.get() : (int32_t*)nullptr,
            distances && dtype == SV_F32 ? (float*)od.get() : (float*)nullptr,
            distances && dtype == SV_F64 ? (double*)od.get() : (double*)nullptr);
  if (nn_index) sv_d2h(ctx, nn_index, oi.get(), (size_t)n * k * 4);
  if (distances) sv_d2h(ctx, distances, od.get(), (size_t)n * k * (dtype == SV_F64 ? 8 : 4));
}

SV_API int sv_knn_host(sv_context* ctx, const void* X, int dtype, int64_t n, int64_t d, int64_t ldX,
                       int64_t k, int metric, int include_self, int precision, int32_t* nn_index,
                       void* distances, sv_knn** out) {
  SV_TRY
  sv_ctx_check(ctx);
  SV_REQUIRE(X, "X is null");
  SV_REQUIRE(dtype == SV_F32 || dtype == SV_F64, "dtype must be F32 or F64");
  knn_validate(n, d, k, metric, include_self, precision);
  SV_REQUIRE(ldX >= n, "ldX < n");
  int dp = (int)((d + 7) / 8 * 8);
  size_t es = dtype == SV_F64 ? 8 : 4;
  DevBuf<unsigned char> dX((size_t)ldX * (d - 1) * es + (size_t)n * es);
  sv_h2d(ctx, dX.get(), X, ((size_t)ldX * (d - 1) + n) * es);
  DevBuf<float> X32((size_t)n * dp), sq(n);
  if (dtype == SV_F64)
    sv_launch(ctx, "knn_pack", k_pack_rows<double>, dim3(sv_grid_for(ctx, n, 256, 8)), dim3(256), 0,
              (const double*)dX.get(), ldX, n, (int)d, dp, metric == SV_COSINE, X32.get(), sq.get());
  else
    sv_launch(ctx, "knn_pack", k_pack_rows<float>, dim3(sv_grid_for(ctx, n, 256, 8)), dim3(256), 0,
              (const float*)dX.get(), ldX, n, (int)d, dp, metric == SV_COSINE, X32.get(), sq.get());
  auto* h = new sv_knn();
  try {
    h->ctx = ctx;
    knn_core(ctx, X32.get(), sq.get(), n, dp, (int)d, (int)k, include_self, metric == SV_COSINE, precision, h);
    knn_outputs(ctx, h, dtype, nn_index, distances);
  } catch (...) {
    delete h;
    throw;
  }
  if (out) *out = h;
  else delete h;
  SV_CATCH
}

SV_API int sv_knn_embed(sv_context* ctx, const sv_embed* e, int64_t ndims, int64_t k, int metric,
                        int include_self, int precision, int32_t* nn_index, double* distances,
                        sv_knn** out) {
  SV_TRY
  sv_ctx_check(ctx);
  SV_REQUIRE(e && e->ctx == ctx, "bad embedding handle");
  if (ndims <= 0) ndims = e->npcs;
  SV_REQUIRE(ndims <= e->npcs, "ndims exceeds the embedding's components");
  int64_t n = e->n_cells;
  knn_validate(n, ndims, k, metric, include_self, precision);
  int dp = (int)((ndims + 7) / 8 * 8);
  DevBuf<float> X32((size_t)n * dp), sq(n);
  sv_launch(ctx, "knn_pack", k_pack_rows<double>, dim3(sv_grid_for(ctx, n, 256, 8)), dim3(256), 0,
            (const double*)e->Z.get(), n, n, (int)ndims, dp, metric == SV_COSINE, X32.get(), sq.get());
  auto* h = new sv_knn();
  try {
    h->ctx = ctx;
    knn_core(ctx, X32.get(), sq.get(), n, dp, (int)ndims, (int)k, include_self, metric == SV_COSINE, precision, h);
    knn_outputs(ctx, h, SV_F64, nn_index, distances);
  } catch (...) {
    delete h;
    throw;
  }
  if (out) *out = h;
  else delete h;
  SV_CATCH
}

// ann over the PCA coordinates of a batch: every cell's neighbours among the
// cells of its own sample, all samples in the same launches (the tensor-core
// candidate kernel takes one sample per CTA).  Indices are stacked rows
// (1-based), as sv_knn_embed returns them.
SV_API int sv_batch_knn(sv_context* ctx, const sv_batch* b, const sv_embed* e, int64_t ndims, int64_t k,
                        int metric, int include_self, int precision, int32_t* nn_index, double* distances,
                        sv_knn** out) {
  SV_TRY
  sv_ctx_check(ctx);
  SV_REQUIRE(b && b->ctx == ctx, "bad batch handle");
  SV_REQUIRE(e && e->ctx == ctx && e->n_cells == b->n_cells, "bad embedding handle");
  if (ndims <= 0) ndims = e->npcs;
  SV_REQUIRE(ndims <= e->npcs, "ndims exceeds the embedding's components");
  int64_t n = e->n_cells;
  int64_t minc = n;
  for (int64_t s = 0; s < b->nseg; ++s) minc = std::min(minc, b->hoff[s + 1] - b->hoff[s]);
  knn_validate(minc, ndims, k, metric, include_self, precision);
  int dp = (int)((ndims + 7) / 8 * 8);
  DevBuf<float> X32((size_t)n * dp), sq(n);
  sv_launch(ctx, "knn_pack", k_pack_rows<double>, dim3(sv_grid_for(ctx, n, 256, 8)), dim3(256), 0,
            (const double*)e->Z.get(), n, n, (int)ndims, dp, metric == SV_COSINE, X32.get(), sq.get());
  auto* h = new sv_knn();
  try {
    h->ctx = ctx;
    knn_core(ctx, X32.get(), sq.get(), n, dp, (int)ndims, (int)k, include_self, metric == SV_COSINE, precision, h,
             &b->hoff);
    knn_outputs(ctx, h, SV_F64, nn_index, distances);
  } catch (...) {
    delete h;
    throw;
  }
  if (out) *out = h;
  else delete h;
  SV_CATCH
}

SV_API int sv_knn_info(const sv_knn* h, int64_t* n, int64_t* k) {
  SV_TRY
  SV_REQUIRE(h, "null handle");
  if (n) *n = h->n;
  if (k) *k = h->k;
  SV_CATCH
}

SV_API int sv_knn_free(sv_knn* h) {
  if (h) {
    delete h;
  }
  return SV_OK;
}

// ---- drop-ins for the native libcell symbols ------------------------------------
static void find_neighbours(const void* X, int dtype, int n, int d, int ldX, int k, int include_self,
                            int metric, int32_t* nn_index, void* distances) {
  int st;
  try {
    sv_context* ctx = sv_default_context();
    st = sv_knn_host(ctx, X, dtype, n, d, ldX, k, metric, include_self, SV_KNN_FP32, nn_index,
                     distances, nullptr);
  } catch (const SvError& e) {
    st = e.code;
  } catch (...) {
    st = SV_ERR_CUDA;
  }
  if (st != SV_OK && nn_index && n > 0 && k > 0) memset(nn_index, 0, (size_t)n * k * sizeof(int32_t));
}

SV_API void FindNeighboursEuclidean32(const float* X, int n, int d, int ldX, int k, int ntables,
                                      int include_self, int seed, int32_t* nn_index, float* distances) {
  (void)ntables;
  (void)seed;
  find_neighbours(X, SV_F32, n, d, ldX, k, include_self, SV_EUCLIDEAN, nn_index, distances);
}

SV_API void FindNeighboursEuclidean64(const double* X, int n, int d, int ldX, int k, int ntables,
                                      int include_self, int seed, int32_t* nn_index, double* distances) {
  (void)ntables;
  (void)seed;
  find_neighbours(X, SV_F64, n, d, ldX, k, include_self, SV_EUCLIDEAN, nn_index, distances);
}

SV_API void FindNeighboursCosine32(const float* X, int n, int d, int ldX, int k, int ntables,
                                   int include_self, int seed, int32_t* nn_index, float* distances) {
  (void)ntables;
  (void)seed;
  find_neighbours(X, SV_F32, n, d, ldX, k, include_self, SV_COSINE, nn_index, distances);
}

SV_API void FindNeighboursCosine64(const double* X, int n, int d, int ldX, int k, int ntables,
                                   int include_self, int seed, int32_t* nn_index, double* distances) {
  (void)ntables;
  (void)seed;
  find_neighbours(X, SV_F64, n, d, ldX, k, include_self, SV_COSINE, nn_index, distances);
}
