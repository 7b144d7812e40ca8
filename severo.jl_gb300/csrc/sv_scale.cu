// scale_features and the CenteredMatrix products (src/scaling.jl:18-44,199-357).
//
// Nothing is densified and no scaled copy is written: the products read the
// normalised values and apply, per element,
//     b = min(a * inv_std_f, clip_f)        clip_f = scale_max + mean_f/std_f
// and the centring as a rank-1 correction:
//     Xs v   = B v  - (mu . v) 1                 (scaling.jl:245-250)
//     Xs^T u = B^T u - (sum u) mu                (scaling.jl:252-257)
//
// Layout in HBM:
//   * the feature (HVF) subset of the CSC copy is a view: per feature its
//     [start, end) range in the full CSC arrays; X^T u walks those ranges in
//     fixed-size chunks (a chunk table built once), one warp per chunk;
//   * X v uses a cell-major copy of the subset (CSR_h): rowptr int64, feature
//     index uint16 (int32 when there are more than 65536 features), value in the
//     data's storage type.  One warp per cell; the per-feature (inv*x, clip*x)
//     pairs are staged in shared memory.
// Algorithmic bytes per product: CSR_h nnz_h*(idx + v) + 8*(n_cells+1) +
// 8*n_cells (y) ; CSC nnz_h*(4 + v) + 4*n_cells (u, FP32) + chunk table.
#include "sv_internal.cuh"

namespace {

constexpr int64_t CHUNK = 4096;   // non-zeros per warp task in the X^T u product

// ---- per-feature moments -----------------------------------------------------
// Mean and unbiased variance of each feature column including its implicit
// zeros (scaling.jl:18-34).  The reference runs Welford over the stored values
// from the state after the n - nnz zeros; here the same two numbers come from
// the sums S1 = sum a and S2 = sum a^2 over the stored values (the zeros add
// nothing): mean = S1 / n, M2 = S2 - S1 * mean, var = M2 / (n - 1).  No
// division per element: the FP64 pipe of this GPU runs at 1/64 of the FP32
// rate, and the former Welford form (one FP64 divide per element) ran at ~1%
// of HBM bandwidth.
//
// FP32 / BF16 values are summed on the FP32 pipe in double-float form (a
// rounded sum and its exact error, Knuth's TwoSum; x^2 exact for BF16, with
// its FMA error term for FP32) over groups of up to 32 elements per thread,
// and each group's (hi, lo) pairs are added into FP64 sums: relative error of
// the sums ~2^-48 per group, of M2 ~2^-47 (1 + mean^2 / var) (3.9e-14 at
// worst on the FP32 test data, 4e-15 for BF16, against FP64 Welford).  FP64
// data are summed in FP64, counts in integers (in FP64 where one has 16 bits or
// more).
//
// Work split: each column is cut into parts of at most MOM_PART entries, one
// warp task each (a device-built task table: per column its range and the
// offset of its first task), so dense features form no tail and short ones
// cost one short task; the per-task sums go to `part` and k_moments_finish
// adds a column's parts in order, so the result does not depend on
// scheduling.  With stacked samples (soff: nseg + 1 cell offsets) every
// (sample, feature) pair is a column of its own (the sample's rows of the
// feature, found by binary search in the sorted CSC rows); outputs at index
// s * nf + f.
__device__ __forceinline__ int64_t lower_bound_rows(const int32_t* __restrict__ r, int64_t lo,
                                                    int64_t hi, int64_t key) {
  while (lo < hi) {
    int64_t mid = (lo + hi) >> 1;
    if ((int64_t)r[mid] < key) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// exact s + e = a + b (TwoSum; explicit roundings so that nothing is contracted)
__device__ __forceinline__ void two_sum_f(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

struct DfAcc {
  float h1 = 0.f, l1 = 0.f, h2 = 0.f, l2 = 0.f;
  template <bool EXACT_SQ>
  __device__ __forceinline__ void add(float x) {
    float s, e;
    two_sum_f(h1, x, s, e);
    h1 = s;
    l1 = __fadd_rn(l1, e);
    float p = __fmul_rn(x, x);
    if (!EXACT_SQ) l2 = __fadd_rn(l2, __fmaf_rn(x, x, -p));
    two_sum_f(h2, p, s, e);
    h2 = s;
    l2 = __fadd_rn(l2, e);
  }
  __device__ __forceinline__ void flush(double& S1, double& S2) {
    S1 += (double)h1;
    S1 += (double)l1;
    S2 += (double)h2;
    S2 += (double)l2;
    h1 = l1 = h2 = l2 = 0.f;
  }
};

// the 16-byte vector of each storage type and how its elements are summed
template <typename ValT> struct MomVec;
template <> struct MomVec<__nv_bfloat16> {
  static constexpr int N = 8;
  static __device__ __forceinline__ void add(const uint4& w, DfAcc& acc, double&, double&) {
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      acc.add<true>(__uint_as_float(u[i] << 16));          // low half: the earlier element
      acc.add<true>(__uint_as_float(u[i] & 0xffff0000u));
    }
  }
  static __device__ __forceinline__ void scalar(const __nv_bfloat16* p, int64_t i, DfAcc& acc,
                                                double&, double&) {
    acc.add<true>(__bfloat162float(p[i]));
  }
  static constexpr bool DF = true;
};
template <> struct MomVec<float> {
  static constexpr int N = 4;
  static __device__ __forceinline__ void add(const uint4& w, DfAcc& acc, double&, double&) {
    acc.add<false>(__uint_as_float(w.x));
    acc.add<false>(__uint_as_float(w.y));
    acc.add<false>(__uint_as_float(w.z));
    acc.add<false>(__uint_as_float(w.w));
  }
  static __device__ __forceinline__ void scalar(const float* p, int64_t i, DfAcc& acc, double&,
                                                double&) {
    acc.add<false>(p[i]);
  }
  static constexpr bool DF = true;
};
template <> struct MomVec<double> {
  static constexpr int N = 2;
  static __device__ __forceinline__ void add(const uint4& w, DfAcc&, double& S1, double& S2) {
    double a = __hiloint2double((int)w.y, (int)w.x), b = __hiloint2double((int)w.w, (int)w.z);
    S1 += a;
    S2 = fma(a, a, S2);
    S1 += b;
    S2 = fma(b, b, S2);
  }
  static __device__ __forceinline__ void scalar(const double* p, int64_t i, DfAcc&, double& S1,
                                                double& S2) {
    double a = p[i];
    S1 += a;
    S2 = fma(a, a, S2);
  }
  static constexpr bool DF = false;
};
template <> struct MomVec<int32_t> {
  static constexpr int N = 4;
  static __device__ __forceinline__ void add(const uint4& w, DfAcc&, double& S1, double& S2) {
    const int32_t u[4] = {(int32_t)w.x, (int32_t)w.y, (int32_t)w.z, (int32_t)w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      double a = (double)u[i];
      S1 += a;
      S2 = fma(a, a, S2);
    }
  }
  static __device__ __forceinline__ void scalar(const int32_t* p, int64_t i, DfAcc&, double& S1,
                                                double& S2) {
    double a = (double)p[i];
    S1 += a;
    S2 = fma(a, a, S2);
  }
  static constexpr bool DF = false;
};

constexpr int MOM_THREADS = 256;
constexpr int MOM_UNROLL = 4;     // 16-byte loads in flight per lane (one group)
constexpr int64_t MOM_PART = 16384;

// per column (s * nf + f): its range and its number of parts
__global__ void k_moments_tasks(const int64_t* __restrict__ fstart, const int64_t* __restrict__ fend,
                                int64_t nf, const int32_t* __restrict__ rowidx,
                                const int64_t* __restrict__ soff, int nseg,
                                int64_t* __restrict__ cs, int64_t* __restrict__ ce,
                                int64_t* __restrict__ nparts) {
  for (int64_t col = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; col < nf * nseg;
       col += (int64_t)gridDim.x * blockDim.x) {
    const int64_t f = col % nf;
    const int sg = (int)(col / nf);
    int64_t s = fstart[f], e = fend[f];
    if (soff) {
      const int64_t lo = lower_bound_rows(rowidx, s, e, soff[sg]);
      e = lower_bound_rows(rowidx, lo, e, soff[sg + 1]);
      s = lo;
    }
    cs[col] = s;
    ce[col] = e;
    nparts[col] = e - s > MOM_PART ? (e - s + MOM_PART - 1) / MOM_PART : 1;
  }
}

// one warp per task: the sums of one part of a column
template <typename ValT>
__global__ void __launch_bounds__(MOM_THREADS)
k_moments_part(const ValT* __restrict__ val, const int64_t* __restrict__ cs,
               const int64_t* __restrict__ ce, const int64_t* __restrict__ toff, int64_t ncol,
               double2* __restrict__ part) {
  using V = MomVec<ValT>;
  constexpr int N = V::N;
  const int lane = threadIdx.x & 31;
  const int64_t ntask = toff[ncol];
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t task = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; task < ntask;
       task += nw) {
    // the column of this task: the last col with toff[col] <= task
    int64_t lo = 0, hi = ncol;
    while (hi - lo > 1) {
      const int64_t mid = (lo + hi) >> 1;
      if (toff[mid] <= task) lo = mid;
      else hi = mid;
    }
    const int64_t col = lo;
    const int64_t P = toff[col + 1] - toff[col], p = task - toff[col];
    const int64_t s = cs[col], L = ce[col] - s;
    const int64_t a = s + L * p / P, b = s + L * (p + 1) / P;
    double S1 = 0.0, S2 = 0.0;
    DfAcc acc;
    const int64_t va = (a + N - 1) / N, vb = b / N;   // whole 16-byte vectors in [a, b)
    if constexpr (sizeof(ValT) == 4 && !V::DF) {
      // Counts below 2^15 (a part's squares then sum to less than 2^45): every FP64
      // partial sum is an exact integer, whatever the order, and integers give the
      // same sums without the FP64 pipe (60 M counts: 0.51 -> 0.14 ms)
      long long i1 = 0, i2 = 0;
      bool small = true;
      auto take = [&](int c) {
        small = small && (unsigned)(c + 32768) < 65536u;
        i1 += c;
        i2 += (long long)c * c;
      };
      for (int64_t i = a + lane; i < min(b, va * N); i += 32) take(val[i]);
      if (va < vb) {
        for (int64_t i = vb * N + lane; i < b; i += 32) take(val[i]);
        const int4* vp = reinterpret_cast<const int4*>(val);
        for (int64_t v0 = va + lane; v0 < vb; v0 += 32 * MOM_UNROLL) {
          int4 w[MOM_UNROLL];
#pragma unroll
          for (int u = 0; u < MOM_UNROLL; ++u) w[u] = v0 + 32 * u < vb ? __ldg(vp + v0 + 32 * u) : make_int4(0, 0, 0, 0);
#pragma unroll
          for (int u = 0; u < MOM_UNROLL; ++u) {
            take(w[u].x);
            take(w[u].y);
            take(w[u].z);
            take(w[u].w);
          }
        }
      } else {
        for (int64_t i = max(a, va * N) + lane; i < b; i += 32) take(val[i]);
      }
      if (__all_sync(0xffffffffu, small)) {
        i1 = sv_warp_sum(i1);
        i2 = sv_warp_sum(i2);
        if (lane == 0) part[task] = make_double2((double)i1, (double)i2);
        continue;
      }
    }
    if (va < vb) {
      // head [a, va*N) and tail [vb*N, b): fewer than N elements each
      if (lane < va * N - a) V::scalar(val, a + lane, acc, S1, S2);
      if (lane < b - vb * N) V::scalar(val, vb * N + lane, acc, S1, S2);
      const uint4* vp = reinterpret_cast<const uint4*>(val);
      for (int64_t v0 = va + lane; v0 < vb; v0 += 32 * MOM_UNROLL) {
        uint4 w[MOM_UNROLL];
#pragma unroll
        for (int u = 0; u < MOM_UNROLL; ++u) {
          const int64_t v = v0 + 32 * u;
          if (v < vb) w[u] = __ldg(vp + v);
        }
#pragma unroll
        for (int u = 0; u < MOM_UNROLL; ++u)
          if (v0 + 32 * u < vb) V::add(w[u], acc, S1, S2);
        if (V::DF) acc.flush(S1, S2);
      }
    } else {
      for (int64_t i = a + lane; i < b; i += 32) V::scalar(val, i, acc, S1, S2);
    }
    if (V::DF) acc.flush(S1, S2);
    S1 = sv_warp_sum(S1);
    S2 = sv_warp_sum(S2);
    if (lane == 0) part[task] = make_double2(S1, S2);
  }
}

__global__ void k_moments_finish(const double2* __restrict__ part, const int64_t* __restrict__ toff,
                                 int64_t nf, int nseg, const int64_t* __restrict__ soff, int64_t n_cells,
                                 double scale_max, double* __restrict__ mean_o,
                                 double* __restrict__ std_o, double* __restrict__ mu_o,
                                 float* __restrict__ inv_f, float* __restrict__ clip_f,
                                 double* __restrict__ inv_d, double* __restrict__ clip_d) {
  for (int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < nf * nseg;
       o += (int64_t)gridDim.x * blockDim.x) {
    double S1 = 0.0, S2 = 0.0;
    for (int64_t t = toff[o]; t < toff[o + 1]; ++t) {
      const double2 q = part[t];
      S1 += q.x;
      S2 += q.y;
    }
    const int sg = (int)(o / nf);
    const double n = soff ? (double)(soff[sg + 1] - soff[sg]) : (double)n_cells;
    const double meanv = S1 / n;
    const double M2 = fmax(fma(-S1, meanv, S2), 0.0);
    const double var = M2 / (n - 1.0);
    const double sd = sqrt(var);
    const double mu = meanv / sd;                   // scaling.jl:207
    mean_o[o] = meanv;
    std_o[o] = sd;
    mu_o[o] = mu;
    inv_d[o] = 1.0 / sd;                            // a * (1/std): within 1 ulp of a/std
    clip_d[o] = scale_max + mu;                     // scaling.jl:209
    inv_f[o] = (float)(1.0 / sd);
    clip_f[o] = (float)(scale_max + mu);
  }
}

// Per-column moments of a feature set (or of every (sample, feature) pair):
// the two launches above with their partial-sum buffer.
template <typename VT>
void launch_moments(sv_context* ctx, const char* name, const VT* val, const int64_t* fs,
                    const int64_t* fe, int64_t nf, int64_t n_cells, double scale_max, double* mean,
                    double* sd, double* mu, float* invf, float* clipf, double* invd, double* clipd,
                    int64_t nnz_bound, const int32_t* rowidx = nullptr, const int64_t* soff = nullptr,
                    int nseg = 1) {
  const int64_t ncol = nf * nseg;
  DevBuf<int64_t> cs(ncol), ce(ncol), np(ncol + 1), toff(ncol + 1);
  sv_launch(ctx, "moments_tasks", k_moments_tasks, dim3(sv_grid_for(ctx, ncol, 256)), dim3(256), 0,
            fs, fe, nf, rowidx, soff, nseg, cs.get(), ce.get(), np.get());
  sv_scan_i64(ctx, np.get(), toff.get(), ncol);
  // tasks: one per column plus one per MOM_PART entries (the columns hold at
  // most nnz_bound entries together)
  const int64_t tasks_max = ncol + nnz_bound / MOM_PART + 1;
  DevBuf<double2> part((size_t)tasks_max);
  int per_sm = 0;
  SV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_moments_part<VT>, MOM_THREADS, 0));
  sv_launch(ctx, name, k_moments_part<VT>,
            dim3(sv_grid_for(ctx, tasks_max * 32, MOM_THREADS, std::max(per_sm, 1))), dim3(MOM_THREADS), 0,
            val, (const int64_t*)cs.get(), (const int64_t*)ce.get(), (const int64_t*)toff.get(), ncol,
            part.get());
  sv_launch(ctx, "moments_finish", k_moments_finish, dim3(sv_grid_for(ctx, ncol, 256)), dim3(256), 0,
            (const double2*)part.get(), (const int64_t*)toff.get(), nf, nseg, soff, n_cells, scale_max,
            mean, sd, mu, invf, clipf, invd, clipd);
  sv_sync(ctx);
}

__global__ void k_feat_ranges(const int32_t* __restrict__ fgene, const int64_t* __restrict__ colptr,
                              int64_t nf, int64_t* __restrict__ fs, int64_t* __restrict__ fe,
                              int32_t* __restrict__ gene_map) {
  for (int64_t f = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; f < nf;
       f += (int64_t)gridDim.x * blockDim.x) {
    int32_t g = fgene[f];
    fs[f] = colptr[g];
    fe[f] = colptr[g + 1];
    gene_map[g] = (int32_t)f;
  }
}

// ---- CSR_h construction ------------------------------------------------------
__global__ void k_hsub_count(const int64_t* __restrict__ rowptr, const int32_t* __restrict__ col,
                             int64_t n_rows, const int32_t* __restrict__ gene_map,
                             int64_t* __restrict__ cnt) {
  int lane = threadIdx.x & 31;
  int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = warp; r < n_rows; r += nwarps) {
    int64_t s = rowptr[r], e = rowptr[r + 1];
    int64_t c = 0;
    for (int64_t i = s + lane; i < e; i += 32) c += __ldg(gene_map + col[i]) >= 0;
    c = sv_warp_sum(c);
    if (lane == 0) cnt[r] = c;
  }
}

template <typename ValT, typename IdxT>
__global__ void k_hsub_write(const int64_t* __restrict__ rowptr, const int32_t* __restrict__ col,
                             const ValT* __restrict__ val, int64_t n_rows,
                             const int32_t* __restrict__ gene_map, const int64_t* __restrict__ hrowptr,
                             IdxT* __restrict__ hcol, ValT* __restrict__ hval) {
  int lane = threadIdx.x & 31;
  int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = warp; r < n_rows; r += nwarps) {
    int64_t s = rowptr[r], e = rowptr[r + 1];
    int64_t pos = hrowptr[r];
    // four groups of 32 entries in flight (one: 1.23 ms for 250 M entries of
    // 100,000 cells, four: 0.66 ms)
    for (int64_t i0 = s; i0 < e; i0 += 128) {
      int32_t f[4];
      ValT v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t i = i0 + 32 * u + lane;
        f[u] = i < e ? col[i] : -1;
        if (i < e) v[u] = val[i];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (f[u] >= 0) f[u] = __ldg(gene_map + f[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const unsigned m = __ballot_sync(0xffffffffu, f[u] >= 0);
        if (f[u] >= 0) {
          const int64_t p = pos + __popc(m & ((1u << lane) - 1));
          hcol[p] = (IdxT)f[u];
          hval[p] = v[u];
        }
        pos += __popc(m);
      }
    }
  }
}

// ---- bank-aware order of the product copies --------------------------------------
// The product kernels read a segment (a CSR_h row, or a (row block, feature)
// run of the row-blocked copy) in groups of 32 EPL entries, lane l taking
// entries EPL l .. EPL l + EPL - 1 of the group (from the segment start rounded
// down to EPL; EPL = 8 for the BF16 X v loop, 4 otherwise); for each t the 32
// lanes then gather from a shared-memory table: 8-byte entries per feature for
// X v (bank pair f mod 16), 4-byte entries per row for X^T u (bank row mod 32).
// With sorted indices the gathers serialise on bank conflicts (ncu: ~4 extra
// wavefronts per gather).  So each segment is permuted such that slot p
// (relative to the rounded start) holds an index of class
// c(p) = ((p / EPL) + (NC / EPL) (p mod EPL)) mod NC where possible (NC = 16 or
// 32 classes): the 32 slots of a gather then hold each class 32/NC times.
// Entries of class c fill the c-slots in order of appearance; the surplus of
// over-full classes fills the slots left empty, in slot order.  The segment's
// sum is then taken in another order (a different, equally valid rounding).
// Applied to the CSR_h rows (X v: 1.61 -> 1.52 ms per product when it was added, at
// the atlas size; once per scale_features, 2.4 ms for 525 M entries); for the row-blocked runs (NC = 32)
// the product gained 1% and the reordering cost more than it saved.
constexpr int BO_EMPTY = 1024;   // most empty slots a segment may have to be reordered
constexpr int BO_WARPS = 4;
constexpr int BO_STAGE = 2048;   // longest segment put together in shared memory
constexpr int XV_DEPTH = 4;      // groups per lane in flight of the double-float X v loop
constexpr int XV_EPL16 = 8;      // entries per lane and group of the BF16 X v loop

template <int NC, int EPL>
__device__ __forceinline__ int bo_class(int64_t p) {
  return (int)(((p / EPL) + (NC / EPL) * (p % EPL)) & (NC - 1));
}
// The slots of class c repeat with period EPL NC: EPL of them per period, at
// the offsets EPL ((c - (NC/EPL) t) mod NC) + t (t < EPL).  The kernel keeps
// per class the sorted offsets (the idx-th slot of the class) and, for every
// position x within a period, the number of the class's offsets below x (the
// slots before a position), so that both are table lookups.
// One warp per segment, three passes (class counts; the empty slots; ranks and
// placement), the result written to a second copy (segments with more than
// BO_EMPTY empty slots are copied unchanged).
// Segments up to BO_STAGE: every lane takes a run of whole groups, counts its
// entries per class in shared memory, the sums over the lanes before it are its
// first ranks, and the segment is put together in shared memory and written whole.
// (32 consecutive entries at a time, with __match_any_sync for the ranks and 2-byte
// scattered stores, 525 M BF16 entries of 500,000 cells took 4.1 ms, this 2.4;
// 125 M FP32 entries of 100,000 cells 1.0, this 0.8.  The shared-memory passes of the
// counters and of the scattered 2-byte stores are what it is bound by.)  Longer ones go that way.
template <int NC, int EPL, typename VT>
struct BoRow {
  __align__(16) uint16_t rank[NC][32];   // class counts per lane, then its next slots' numbers
  int2 cls[NC];                    // the end of the class's slots, what takes a rank past it to its place in the list
  int first[NC];                   // first empty slot of the class, or the segment's end
  __align__(16) uint16_t col[BO_STAGE + EPL];   // the segment in its new order, from its start rounded down
  __align__(16) VT val[BO_STAGE + EPL];
};
// whole groups: EPL entries of 2 or 4 bytes (the copies are padded and 16-byte aligned)
template <int EPL, typename T>
__device__ __forceinline__ void bo_load(const T* p, T (&o)[EPL]) {
  if constexpr (EPL * sizeof(T) == 16) *(uint4*)o = *(const uint4*)p;
  else *(uint2*)o = *(const uint2*)p;
}
template <int EPL, typename T>
__device__ __forceinline__ void bo_copy(const T* p, T* o) {
  if constexpr (EPL * sizeof(T) == 16) *(uint4*)o = *(const uint4*)p;
  else *(uint2*)o = *(const uint2*)p;
}

static_assert(sizeof(BoRow<16, 4, float>) % 16 == 0 && sizeof(BoRow<16, 8, uint16_t>) % 16 == 0, "vector accesses");

template <int NC, int EPL, typename VT>
__global__ void __launch_bounds__(BO_WARPS * 32) k_bankorder(const int64_t* __restrict__ ptr,
                                                             int64_t nseg,
                                                             const uint16_t* __restrict__ icol,
                                                             const VT* __restrict__ ival,
                                                             uint16_t* __restrict__ ocol,
                                                             VT* __restrict__ oval) {
  constexpr int PER = EPL * NC;
  static_assert(NC == 16, "lanes and halves of them per class");
  __shared__ uint16_t sempty[BO_WARPS][BO_EMPTY];
  __shared__ int cnt[BO_WARPS][NC], run[BO_WARPS][NC];
  __shared__ uint8_t soff[NC][EPL], sbelow[NC][PER + 1];
  extern __shared__ __align__(16) unsigned char bo_dyn[];
  BoRow<NC, EPL, VT>& row = ((BoRow<NC, EPL, VT>*)bo_dyn)[threadIdx.x >> 5];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  for (int i = threadIdx.x; i < NC * (PER + 1); i += blockDim.x) {
    const int c = i / (PER + 1), x = i % (PER + 1);
    int k = 0;
#pragma unroll
    for (int t = 0; t < EPL; ++t) k += (EPL * ((c - (NC / EPL) * t) & (NC - 1)) + t) < x;
    sbelow[c][x] = (uint8_t)k;
  }
  for (int c = threadIdx.x; c < NC; c += blockDim.x) {
    int o[EPL];
#pragma unroll
    for (int t = 0; t < EPL; ++t) o[t] = EPL * ((c - (NC / EPL) * t) & (NC - 1)) + t;
    for (int i = 1; i < EPL; ++i)
      for (int j = i; j > 0 && o[j - 1] > o[j]; --j) {
        const int tmp = o[j];
        o[j] = o[j - 1];
        o[j - 1] = tmp;
      }
    for (int t = 0; t < EPL; ++t) soff[c][t] = (uint8_t)o[t];
  }
  __syncthreads();
  // slots of class c before position X; the idx-th slot of class c
  auto bo_count = [&](int c, int64_t X) -> int64_t { return EPL * (X / PER) + sbelow[c][X % PER]; };
  auto bo_slot = [&](int c, int64_t idx) -> int64_t { return (int64_t)PER * (idx / EPL) + soff[c][idx % EPL]; };
  for (int64_t r = (int64_t)blockIdx.x * BO_WARPS + w; r < nseg; r += (int64_t)gridDim.x * BO_WARPS) {
    const int64_t s = ptr[r], e = ptr[r + 1];
    const int64_t L = e - s;
    if (L <= 0) continue;
    const int64_t P0 = s & (EPL - 1), P1 = P0 + L;
    if (L <= BO_STAGE) {
      const int64_t b0 = s - P0;
      const int p0 = (int)P0, p1 = (int)P1;
      const int ng = ((p1 + EPL - 1) / EPL + 31) / 32;        // groups of a lane
      const int g0 = lane * ng * EPL, g1 = min(p1, g0 + ng * EPL);
      const uint16_t* src = icol + b0;
      const VT* vsrc = ival + b0;
      // class counts of the lane's entries
      for (int i = lane; i < NC * 32 / 8; i += 32) ((uint4*)row.rank)[i] = make_uint4(0, 0, 0, 0);
      __syncwarp();
#pragma unroll 2
      for (int g = g0; g < g1; g += EPL) {
        __align__(16) uint16_t f[EPL];
        bo_load<EPL>(src + g, f);
        if (g >= p0 && g + EPL <= p1) {
#pragma unroll
          for (int t = 0; t < EPL; ++t) ++row.rank[f[t] & (NC - 1)][lane];
        } else {
#pragma unroll
          for (int t = 0; t < EPL; ++t)
            if (g + t >= p0 && g + t < p1) ++row.rank[f[t] & (NC - 1)][lane];
        }
      }
      __syncwarp();
      // lane = class: first ranks of the lanes, slots, surplus, first empty slot
      int first = p1, n = 0, slots = 0, base = 0;
      if (lane < NC) {
        base = (int)bo_count(lane, P0);
        slots = (int)bo_count(lane, P1) - base;
        unsigned* rk = (unsigned*)row.rank[lane];
        unsigned v[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = rk[k];
        n = base;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const unsigned lo = v[k] & 0xffffu, hi = v[k] >> 16;
          rk[k] = (unsigned)n | ((unsigned)(n + lo) << 16);
          n += lo + hi;
        }
        n -= base;
        if (n < slots) first = (int)bo_slot(lane, base + n);
        row.first[lane] = first;
      }
      const int sur = max(0, n - slots);
      int incl = sur;
#pragma unroll
      for (int o = 1; o < NC; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane < NC) row.cls[lane] = make_int2(base + slots, incl - sur - (base + slots));
      int least = first;
      const int holes = (int)__reduce_add_sync(0xffffffffu, (unsigned)max(0, slots - n));
      least = __reduce_min_sync(0xffffffffu, least);
      __syncwarp();
      if (holes > BO_EMPTY) {
        for (int64_t i = lane; i < L; i += 32) {
          ocol[s + i] = icol[s + i];
          oval[s + i] = ival[s + i];
        }
        continue;
      }
      // the empty slots, in slot order: from a class's first one on, its slots
      int nempty = 0;
      for (int q0 = least & ~31; q0 < p1; q0 += 32) {
        const int q = q0 + lane;
        const bool emp = q >= p0 && q < p1 && q >= row.first[bo_class<NC, EPL>(q)];
        const unsigned m = __ballot_sync(0xffffffffu, emp);
        if (emp) sempty[w][nempty + __popc(m & lt)] = (uint16_t)q;
        nempty += __popc(m);
      }
      __syncwarp();
      // placement
      auto place = [&](unsigned f, VT v) {
        const int c = (int)(f & (NC - 1));
        const int idx = row.rank[c][lane]++;
        const int2 k = row.cls[c];
        int q = PER * (idx / EPL) + soff[c][idx & (EPL - 1)];
        if (idx >= k.x) q = sempty[w][k.y + idx];
        row.col[q] = (uint16_t)f;
        row.val[q] = v;
      };
#pragma unroll 2
      for (int g = g0; g < g1; g += EPL) {
        __align__(16) uint16_t f[EPL];
        __align__(16) VT v[EPL];
        bo_load<EPL>(src + g, f);
        bo_load<EPL>(vsrc + g, v);
        if (g >= p0 && g + EPL <= p1) {
#pragma unroll
          for (int t = 0; t < EPL; ++t) place(f[t], v[t]);
        } else {
#pragma unroll
          for (int t = 0; t < EPL; ++t)
            if (g + t >= p0 && g + t < p1) place(f[t], v[t]);
        }
      }
      __syncwarp();
      for (int g = EPL * lane; g < p1; g += 32 * EPL) {
        if (g >= p0 && g + EPL <= p1) {
          bo_copy<EPL>(row.col + g, ocol + b0 + g);
          bo_copy<EPL>(row.val + g, oval + b0 + g);
        } else {
          for (int t = 0; t < EPL; ++t)
            if (g + t >= p0 && g + t < p1) {
              ocol[b0 + g + t] = row.col[g + t];
              oval[b0 + g + t] = row.val[g + t];
            }
        }
      }
      __syncwarp();
      continue;
    }
    if (lane < NC) {
      cnt[w][lane] = 0;
      run[w][lane] = 0;
    }
    __syncwarp();
    // pass 1: entries per class
    for (int64_t i0 = 0; i0 < L; i0 += 32) {
      int64_t i = i0 + lane;
      int c = i < L ? (icol[s + i] & (NC - 1)) : NC + lane;
      unsigned same = __match_any_sync(0xffffffffu, c);
      if (i < L && (same & lt) == 0) cnt[w][c] += __popc(same);
      __syncwarp();
    }
    // pass 2: empty slots (classes with fewer entries than slots), in slot order
    int64_t nempty = 0;
    for (int64_t p0 = P0; p0 < P1; p0 += 32) {
      int64_t p = p0 + lane;
      bool emp = false;
      if (p < P1) {
        int c = bo_class<NC, EPL>(p);
        emp = bo_count(c, p) - bo_count(c, P0) >= cnt[w][c];
      }
      unsigned m = __ballot_sync(0xffffffffu, emp);
      int64_t at = nempty + __popc(m & lt);
      if (emp && at < BO_EMPTY) sempty[w][at] = (uint16_t)(p - P0);
      nempty += __popc(m);
    }
    __syncwarp();
    if (nempty > BO_EMPTY || L > 65535) {
      for (int64_t i = lane; i < L; i += 32) {
        ocol[s + i] = icol[s + i];
        oval[s + i] = ival[s + i];
      }
      continue;
    }
    // surplus entries of the classes before c (prefix over the classes)
    int sur = 0;
    if (lane < NC) {
      int64_t slots = bo_count(lane, P1) - bo_count(lane, P0);
      sur = (int)max((int64_t)0, (int64_t)cnt[w][lane] - slots);
    }
    int incl = sur;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    const int excl = incl - sur;
    // pass 3: rank within the class (order of appearance) and placement
    for (int64_t i0 = 0; i0 < L; i0 += 32) {
      int64_t i = i0 + lane;
      bool v = i < L;
      uint16_t f = v ? icol[s + i] : 0;
      int c = v ? (f & (NC - 1)) : NC + lane;
      unsigned same = __match_any_sync(0xffffffffu, c);
      int base_c = v ? run[w][c] : 0;
      int pre = __shfl_sync(0xffffffffu, excl, c & (NC - 1));
      __syncwarp();
      if (v) {
        int rk = base_c + __popc(same & lt);
        if ((same & lt) == 0) run[w][c] = base_c + __popc(same);
        int64_t slots = bo_count(c, P1) - bo_count(c, P0);
        int64_t q = rk < slots ? bo_slot(c, bo_count(c, P0) + rk) - P0
                               : (int64_t)sempty[w][pre + (rk - slots)];
        ocol[s + q] = f;
        oval[s + q] = ival[s + i];
      }
      __syncwarp();
    }
  }
}

// ---- vector loads of 4 consecutive elements (allocation padded) -------------
__device__ __forceinline__ void ld4(const uint16_t* p, int64_t g, int (&o)[4]) {
  uint2 w = __ldg((const uint2*)(p + g));
  o[0] = w.x & 0xffff;
  o[1] = w.x >> 16;
  o[2] = w.y & 0xffff;
  o[3] = w.y >> 16;
}
__device__ __forceinline__ void ld4(const int32_t* p, int64_t g, int (&o)[4]) {
  int4 w = __ldg((const int4*)(p + g));
  o[0] = w.x;
  o[1] = w.y;
  o[2] = w.z;
  o[3] = w.w;
}
__device__ __forceinline__ void ld4v(const __nv_bfloat16* p, int64_t g, float (&o)[4]) {
  uint2 w = __ldg((const uint2*)(p + g));
  o[0] = __uint_as_float(w.x << 16);
  o[1] = __uint_as_float(w.x & 0xffff0000u);
  o[2] = __uint_as_float(w.y << 16);
  o[3] = __uint_as_float(w.y & 0xffff0000u);
}
__device__ __forceinline__ void ld4v(const float* p, int64_t g, float (&o)[4]) {
  float4 w = __ldg((const float4*)(p + g));
  o[0] = w.x;
  o[1] = w.y;
  o[2] = w.z;
  o[3] = w.w;
}
__device__ __forceinline__ void ld4v(const double* p, int64_t g, double (&o)[4]) {
  double2 a = __ldg((const double2*)(p + g));
  double2 b = __ldg((const double2*)(p + g + 2));
  o[0] = a.x;
  o[1] = a.y;
  o[2] = b.x;
  o[3] = b.y;
}

template <typename ValT>
struct AccOf {
  typedef float type;
};
template <>
struct AccOf<double> {
  typedef double type;
};

// v > clip ? clip : v without the FP64 pipe, where a comparison costs as much as a
// product: doubles compare as integers once the negative ones' bits are turned
// round (and the same turns them back).  A clip that is NaN clips nothing, and
// neither is a v that is NaN (a product's: quiet).
__device__ __forceinline__ long long turned(long long b) { return b ^ ((b >> 63) & 0x7fffffffffffffffll); }
__device__ __forceinline__ long long clip_key(double clip) {
  return clip != clip ? 0x7fffffffffffffffll : turned(__double_as_longlong(clip));
}
__device__ __forceinline__ double clip_above(double v, long long key) {
  const bool over = turned(__double_as_longlong(v)) > key &&
                    ((unsigned)__double2hiint(v) & 0x7fffffffu) < 0x7ff80000u;
  return over ? __longlong_as_double(turned(key)) : v;
}

// ---- X v over CSR_h ------------------------------------------------------------
// y = alpha * (B x - (mu . x)) + beta * y - (csub ? *csub : 0) * z
// Per-feature table in shared memory.  FP32 form: (P, Q) = (inv*x, clip*x); the
// product term is min(a*P, Q) for x >= 0 and max(a*P, Q) for x < 0 (= min(a*inv,
// clip)*x).  FP64 form: (1/std, clip, x); a * (1/std) is within one ulp of the
// reference's a/std (FP64 division is slow on this part).
// Every block builds the table and mu.x itself from x (a separate one-block
// kernel preparing the table for all blocks measured no faster).  Blocks have 256
// threads but for FP64 values where 512 make it one block per SM and 256 two on some
// (2,000 features, 256 and 512 threads: 1,000 cells 12.2 and 14.8 us, 1,500 16.6 and
// 14.7, 2,000 16.3 and 15.1, 3,000 20.7 and 23.0, 20,000 64.6 and 64.8; FP32, 3,000
// features, 100,000 cells: 98 and 111).
constexpr int CSR_SUMS = 256;    // threads that sum mu.x: its order
template <typename ValT, typename IdxT, int THREADS>
__global__ void __launch_bounds__(THREADS) k_spmv_csr(
    const int64_t* __restrict__ rowptr, const IdxT* __restrict__ hcol, const ValT* __restrict__ hval,
    int64_t n_rows, int64_t nf, const double* __restrict__ x, const float* __restrict__ inv_f,
    const float* __restrict__ clip_f, const double* __restrict__ inv_d,
    const double* __restrict__ clip_d, const double* __restrict__ mu, double alpha, double beta,
    double* __restrict__ y, const double* __restrict__ csub, const double* __restrict__ z) {
  typedef typename AccOf<ValT>::type AccT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[32];
  double mux = 0;
  {
    // with 512 threads half of them build the table, the other half mu.x; four
    // features per thread in flight
    constexpr int half = CSR_SUMS;
    const int t = threadIdx.x % half;
    const bool sums = threadIdx.x < half, builds = THREADS == half || !sums;
    for (int64_t f0 = t; f0 < nf; f0 += 4 * half) {
      double xs[4], ms[4];
      AccT iv[4], cl[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t f = f0 + u * half;
        if (f >= nf) break;
        xs[u] = x[f];
        if (sums) ms[u] = mu[f];
        if (builds) {
          if constexpr (sizeof(AccT) == 4) {
            iv[u] = inv_f[f];
            cl[u] = clip_f[f];
          } else {
            iv[u] = inv_d[f];
            cl[u] = clip_d[f];
          }
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t f = f0 + u * half;
        if (f >= nf) break;
        if (sums) mux += ms[u] * xs[u];
        if (!builds) continue;
        if constexpr (sizeof(AccT) == 4) {
          const float x1 = (float)xs[u];
          const float P = iv[u] * x1;
          const float Q = x1 == 0.f ? 0.f : cl[u] * x1;
          ((float2*)smem_raw)[f] = make_float2(P, Q);
        } else {
          double* tab = (double*)smem_raw;
          tab[3 * f] = iv[u];
          tab[3 * f + 1] = __longlong_as_double(clip_key(cl[u]));
          tab[3 * f + 2] = xs[u];
        }
      }
    }
    mux = sv_warp_sum(mux);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mux;
    __syncthreads();
    if (threadIdx.x < 32) {
      double v = threadIdx.x < half / 32 ? red[threadIdx.x] : 0.0;
      v = sv_warp_sum(v);
      if (threadIdx.x == 0) red[0] = v;
    }
    __syncthreads();
    mux = red[0];
  }
  double cs = csub ? *csub : 0.0;

  int lane = threadIdx.x & 31;
  int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = warp; r < n_rows; r += nwarps) {
    int64_t s = rowptr[r], e = rowptr[r + 1];
    int64_t a0 = s & ~3ll;
    AccT acc = 0;
    // two 4-element groups per lane in flight; the first load pair is
    // unconditional (a guarded-loop form of the same loads measured 23% slower)
    for (int64_t g = a0 + 4 * lane; g < e; g += 256) {
      int ci[2][4];
      AccT av[2][4];
      bool two = g + 128 < e;
      ld4(hcol, g, ci[0]);
      ld4v(hval, g, av[0]);
      if (two) {
        ld4(hcol, g + 128, ci[1]);
        ld4v(hval, g + 128, av[1]);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (h == 1 && !two) break;
        int64_t gh = g + 128 * h;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          if (gh + t >= s && gh + t < e) {
            if constexpr (sizeof(AccT) == 4) {
              float2 pq = ((const float2*)smem_raw)[ci[h][t]];
              float rr = av[h][t] * pq.x;
              acc += pq.x >= 0.f ? fminf(rr, pq.y) : fmaxf(rr, pq.y);
            } else {
              const double* tab = (const double*)smem_raw;
              double v = av[h][t] * tab[3 * ci[h][t]];          // scaling.jl:211 (times 1/std)
              const long long c = __double_as_longlong(tab[3 * ci[h][t] + 1]);
              acc += clip_above(v, c) * tab[3 * ci[h][t] + 2];   // scaling.jl:212
            }
          }
        }
      }
    }
    acc = sv_warp_sum(acc);
    if (lane == 0) {
      double out = alpha * ((double)acc - mux);
      if (beta != 0.0) out += beta * y[r];
      if (z) out -= cs * z[r];
      y[r] = out;
    }
  }
}

static int csr_threads(sv_context* ctx, int dtype, int64_t n_rows) {
  const int64_t per_sm = (n_rows + ctx->num_sms - 1) / ctx->num_sms;   // a warp per row
  return dtype == SV_F64 && per_sm > 8 && per_sm <= 16 ? 512 : 256;
}
template <typename ValT, typename IdxT>
static auto csr_kernel(int threads) {
  if constexpr (sizeof(ValT) == 8) {
    if (threads == 512) return k_spmv_csr<ValT, IdxT, 512>;
  }
  return k_spmv_csr<ValT, IdxT, 256>;
}

// ---- X v for the Lanczos W side, double-float in and out (FP32 storage) -------
// The rows of k_spmv_csr with every FP64 operation removed: this part
// issues one warp-wide FP64 instruction per ~17 cycles per SM, and the FP64
// prologue and epilogue of k_spmv_csr kept its FP64 pipe 30% busy.  The vector
// arrives as a double-float basis column (its FP32 high part is the FP32 x of
// the table), mu.x is accumulated in double-float, and the result
//   y = (B x - mu.x) - csub * z      (z a double-float basis column)
// is written as a double-float working vector, ready for reorthogonalisation.
// With stacked samples (blk non-null) block b handles the cells of blk[b] of
// sample s = blk[b].seg with that sample's feature parameters (x, 1/std, clip,
// mu at offset s * nf) and csub[s].  Otherwise block b has the rows cut[b] ..
// cut[b + 1] - 1 (k_row_cuts).
// Bound by HBM (525 M BF16 entries of 500,000 cells: 357 us, 5.9 TB/s; 62 M FP32
// entries of 50,000 cells: 77 us).  What it took to get there from 419 us, where
// the issue slots were the limit (22 instructions per entry of a warp): the guards
// at a row's ends only in its first and last round of groups, as a bit mask, and
// for the whole warp (each lane branching by itself ran both forms); the minimum
// without a comparison; rows handed to the warps of a block one at a time, their
// ends loaded one row ahead; XV_DEPTH groups in flight, each reloaded as soon as
// it is added (2, 3, 4, 6 groups: 405, 378, 357, 367 us).  Every lane adds the
// groups it always did in the same order.
__device__ __forceinline__ void dfx_fma(float& sh, float& sl, float ah, float al, float bh, float bl) {
  float p = ah * bh;
  float e = fmaf(ah, bh, -p);
  e = fmaf(ah, bl, e);
  e = fmaf(al, bh, e);
  float t = sh + p;
  float v = t - sh;
  float err = (sh - (t - v)) + (p - v);
  sh = t;
  sl += err + e;
}

// Prologue shared by the double-float X v kernels: with stacked samples (blk
// non-null) selects block b's row range and sample s = blk[b].seg (false: the
// sample is frozen, nothing to do); builds the per-feature (inv*x, clip*|x|)
// table in shared memory and returns mu.x and -csub as double-float pairs.
// Rows are cut into one range per block by their entries: with as many rows each
// the one wave of blocks lasts as long as its deepest range, and samples of
// different depth lie one after the other (300,000 cells, BF16, 30 components: first
// half 1/4 as deep as the second, PCA 654 -> 619 ms; first 95% 1/13 as deep as the
// rest, 1,560 -> 1,188; all alike, 1,131 and 1,132).  A row counts as XV_ROW entries
// besides its own.
constexpr int64_t XV_ROW = 64;
__global__ void k_row_cuts(const int64_t* __restrict__ rowptr, int64_t n_rows, int nblk, int64_t* __restrict__ cut) {
  const int64_t total = rowptr[n_rows] + XV_ROW * n_rows;
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b <= nblk; b += gridDim.x * blockDim.x) {
    const int64_t want = total * b / nblk;
    int64_t lo = 0, hi = n_rows;      // the first row with as many before it
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (rowptr[mid] + XV_ROW * mid >= want) hi = mid;
      else lo = mid + 1;
    }
    cut[b] = lo;
  }
}

struct XvDf {
  int64_t rb0, rb1;
  float muxh, muxl, csh, csl;
};
__device__ __forceinline__ bool xv_df_prologue(
    unsigned char* smem_raw, const int64_t* __restrict__ cut, int64_t nf, const float* __restrict__ xh,
    const float* __restrict__ xl, const float* __restrict__ inv_f, const float* __restrict__ clip_f,
    const float* __restrict__ mu_h, const float* __restrict__ mu_l, const double* __restrict__ csub,
    const BlkRange* __restrict__ blk, const int* __restrict__ active, XvDf& o) {
  __shared__ float redh[32], redl[32];
  __shared__ float sc[4];
  int sg = 0;
  if (!blk) {
    o.rb0 = cut[blockIdx.x];
    o.rb1 = cut[blockIdx.x + 1];
  } else {
    const BlkRange br = blk[blockIdx.x];
    sg = br.seg;
    o.rb0 = br.r0;
    o.rb1 = br.r1;
    if (active && !active[sg]) return false;
    const int64_t po = (int64_t)sg * nf;
    xh += po;
    xl += po;
    inv_f += po;
    clip_f += po;
    mu_h += po;
    mu_l += po;
  }
  float mh = 0.f, ml = 0.f;
  for (int64_t f0 = threadIdx.x; f0 < nf; f0 += 4 * blockDim.x) {
    float in[4][6];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int64_t f = f0 + u * blockDim.x;
      if (f >= nf) break;
      in[u][0] = xh[f];
      in[u][1] = xl[f];
      in[u][2] = inv_f[f];
      in[u][3] = clip_f[f];
      in[u][4] = mu_h[f];
      in[u][5] = mu_l[f];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int64_t f = f0 + u * blockDim.x;
      if (f >= nf) break;
      const float xs = in[u][0];
      const float P = in[u][2] * xs;
      const float Q = xs == 0.f ? 0.f : in[u][3] * fabsf(xs);   // of clip's sign
      ((float2*)smem_raw)[f] = make_float2(P, Q);
      dfx_fma(mh, ml, in[u][4], in[u][5], xs, in[u][1]);
    }
  }
  // mu.x: warp reduction in double-float, then warp 0 over the warps
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    float h2 = __shfl_xor_sync(0xffffffffu, mh, off);
    float l2 = __shfl_xor_sync(0xffffffffu, ml, off);
    float t = mh + h2;
    float v = t - mh;
    float err = (mh - (t - v)) + (h2 - v);
    ml = err + ml + l2;
    mh = t;
  }
  if ((threadIdx.x & 31) == 0) {
    redh[threadIdx.x >> 5] = mh;
    redl[threadIdx.x >> 5] = ml;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float h = 0.f, l = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      float t = h + redh[w];
      float v = t - h;
      float err = (h - (t - v)) + (redh[w] - v);
      l += err + redl[w];
      h = t;
    }
    float t = h + l;
    sc[0] = t;
    sc[1] = l - (t - h);
    if (csub) {
      double c = csub[sg];
      sc[2] = (float)c;
      sc[3] = (float)(c - (double)sc[2]);
    } else {
      sc[2] = sc[3] = 0.f;
    }
  }
  __syncthreads();
  o.muxh = sc[0];
  o.muxl = sc[1];
  o.csh = -sc[2];
  o.csl = -sc[3];
  return true;
}

// (acc - mu.x) - csub * z in double-float, written as (yh, yl)
__device__ __forceinline__ void xv_df_store(float acc, const XvDf& p, bool has_z, float zhr, float zlr,
                                            float* __restrict__ yh, float* __restrict__ yl, int64_t r) {
  float h = acc, l = 0.f;
  float t = h - p.muxh;
  float v = t - h;
  float err = (h - (t - v)) + (-p.muxh - v);
  h = t;
  l = err - p.muxl;
  if (has_z) dfx_fma(h, l, p.csh, p.csl, zhr, zlr);
  t = h + l;
  yl[r] = l - (t - h);
  yh[r] = t;
}

// One lane's group of E consecutive entries of a row, as loaded: 16-byte loads of
// indices and values where both are 16-bit, else 4 entries.
template <typename ValT, typename IdxT>
struct XvGroup {
  static constexpr int E = sizeof(ValT) == 2 && sizeof(IdxT) == 2 ? XV_EPL16 : 4;
  unsigned i[E * sizeof(IdxT) / 4], v[E * sizeof(ValT) / 4];
  template <int N>
  static __device__ __forceinline__ void ld(unsigned (&w)[N], const void* p) {
    if constexpr (N == 4) {
      const uint4 x = __ldg((const uint4*)p);
      w[0] = x.x;
      w[1] = x.y;
      w[2] = x.z;
      w[3] = x.w;
    } else {
      const uint2 x = __ldg((const uint2*)p);
      w[0] = x.x;
      w[1] = x.y;
    }
  }
  __device__ __forceinline__ void load(const IdxT* pi, const ValT* pv, int q) {
    ld(i, pi + q);
    ld(v, pv + q);
  }
  __device__ __forceinline__ unsigned index(int t) const {
    return sizeof(IdxT) == 2 ? ((t & 1) ? i[t >> 1] >> 16 : i[t >> 1] & 0xffffu) : i[t];
  }
  // min(a/std, clip) x with (P, Q) = (x/std, clip |x|): the sign of x, which is P's,
  // on min(a |P|, Q) -- one minimum and no comparison, and clip may be negative
  __device__ __forceinline__ float term(int t, float2 x) const {
    const float a = __uint_as_float(
        sizeof(ValT) == 2 ? ((t & 1) ? v[t >> 1] & 0xffff0000u : v[t >> 1] << 16) : v[t]);
    const float m = fminf(a * fabsf(x.x), x.y);
    return __uint_as_float(__float_as_uint(m) ^ (__float_as_uint(x.x) & 0x80000000u));
  }
};

template <typename ValT, typename IdxT>
__global__ void __launch_bounds__(256, 4) k_spmv_csr_df(
    const int64_t* __restrict__ rowptr, const IdxT* __restrict__ hcol, const ValT* __restrict__ hval,
    const int64_t* __restrict__ cut, int64_t nf, const float* __restrict__ xh, const float* __restrict__ xl,
    const float* __restrict__ inv_f, const float* __restrict__ clip_f, const float* __restrict__ mu_h,
    const float* __restrict__ mu_l, float* __restrict__ yh, float* __restrict__ yl,
    const double* __restrict__ csub, const float* __restrict__ zh, const float* __restrict__ zl,
    const BlkRange* __restrict__ blk, const int* __restrict__ active) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int next_row;
  XvDf pr;
  if (threadIdx.x == 0) next_row = 0;
  if (!xv_df_prologue(smem_raw, cut, nf, xh, xl, inv_f, clip_f, mu_h, mu_l, csub, blk, active, pr))
    return;
  const int64_t rb0 = pr.rb0, rb1 = pr.rb1;
  const float2* pq = (const float2*)smem_raw;

  const int lane = threadIdx.x & 31;
  constexpr int E = XvGroup<ValT, IdxT>::E;
  constexpr int STEP = 32 * E;                 // entries of a warp's group round
  auto take = [&](int64_t& r, int64_t& s, int64_t& e) {
    int k = 0;
    if (lane == 0) k = atomicAdd(&next_row, 1);
    r = rb0 + __shfl_sync(0xffffffffu, k, 0);
    if (r < rb1) {
      s = rowptr[r];
      e = rowptr[r + 1];
    }
  };
  int64_t r, s = 0, e = 0;
  take(r, s, e);
  while (r < rb1) {
    int64_t rn, sn = 0, en = 0;                // the next row's ends arrive meanwhile
    take(rn, sn, en);
    const int64_t b0 = s & ~(int64_t)(E - 1);
    const IdxT* pi = hcol + b0;
    const ValT* pv = hval + b0;
    const int ls = (int)(s - b0), le = (int)(e - b0);
    XvGroup<ValT, IdxT> buf[XV_DEPTH];
#pragma unroll
    for (int h = 0; h < XV_DEPTH; ++h)
      if (STEP * h + E * lane < le) buf[h].load(pi, pv, STEP * h + E * lane);
    float acc = 0.f;
    for (int k0 = 0; k0 < le; k0 += STEP * XV_DEPTH) {
#pragma unroll
      for (int h = 0; h < XV_DEPTH; ++h) {
        const int k = k0 + STEP * h;
        if (k >= le) break;
        const int q = k + E * lane;
        if (k >= ls && k + STEP <= le) {
#pragma unroll
          for (int t = 0; t < E; ++t) acc += buf[h].term(t, pq[buf[h].index(t)]);
        } else if (q < le) {
          unsigned in = 0xffu >> max(0, 8 - (le - q));         // entries q .. of [ls, le)
          if (q < ls) in &= 0xffu << (ls - q);
#pragma unroll
          for (int t = 0; t < E; ++t) {
            const bool on = in & (1u << t);
            const float m = buf[h].term(t, pq[on ? buf[h].index(t) : 0]);
            acc += on ? m : 0.f;
          }
        }
        if (q + STEP * XV_DEPTH < le) buf[h].load(pi, pv, q + STEP * XV_DEPTH);
      }
    }
    acc = sv_warp_sum(acc);
    if (lane == 0) xv_df_store(acc, pr, zh != nullptr, zh ? zh[r] : 0.f, zh ? zl[r] : 0.f, yh, yl, r);
    r = rn;
    s = sn;
    e = en;
  }
}

// ---- X^T u over CSR_h (warp per cell, shared-memory accumulation) -----------
// Each block accumulates sum_i min(a_if * inv_f, clip_f) * u_i for its cells into
// a shared array of nf partial sums (shared atomics), then writes the array to
// its row of `partial` (blocks x nf) together with its sum of u; the finish
// kernel adds the block rows in block order (deterministic result).
template <typename ValT, typename IdxT>
__global__ void __launch_bounds__(256) k_spmv_csr_t(
    const int64_t* __restrict__ rowptr, const IdxT* __restrict__ hcol, const ValT* __restrict__ hval,
    int64_t n_rows, int64_t nf, const double* __restrict__ u, const float* __restrict__ inv_f,
    const float* __restrict__ clip_f, const double* __restrict__ inv_d,
    const double* __restrict__ clip_d, void* __restrict__ partial, double* __restrict__ upart) {
  typedef typename AccOf<ValT>::type AccT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[32];
  AccT* accs;
  if constexpr (sizeof(AccT) == 4) {
    float2* tab = (float2*)smem_raw;
    accs = (AccT*)(tab + nf);
    for (int64_t f = threadIdx.x; f < nf; f += blockDim.x) {
      tab[f] = make_float2(inv_f[f], clip_f[f]);
      accs[f] = 0;
    }
  } else {
    double2* tab = (double2*)smem_raw;
    accs = (AccT*)(tab + nf);
    for (int64_t f = threadIdx.x; f < nf; f += blockDim.x) {
      tab[f] = make_double2(inv_d[f], clip_d[f]);
      accs[f] = 0;
    }
  }
  __syncthreads();
  int lane = threadIdx.x & 31;
  int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  double usum = 0;
  for (int64_t r = warp; r < n_rows; r += nwarps) {
    int64_t s = rowptr[r], e = rowptr[r + 1];
    double ud = u[r];
    usum += ud;
    AccT ur = (AccT)ud;
    int64_t a0 = s & ~3ll;
    for (int64_t g = a0 + 4 * lane; g < e; g += 256) {
      int ci[2][4];
      AccT av[2][4];
      bool two = g + 128 < e;
      ld4(hcol, g, ci[0]);
      ld4v(hval, g, av[0]);
      if (two) {
        ld4(hcol, g + 128, ci[1]);
        ld4v(hval, g + 128, av[1]);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (h == 1 && !two) break;
        int64_t gh = g + 128 * h;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          if (gh + t >= s && gh + t < e) {
            if constexpr (sizeof(AccT) == 4) {
              float2 ic = ((const float2*)smem_raw)[ci[h][t]];
              atomicAdd(&accs[ci[h][t]], fminf(av[h][t] * ic.x, ic.y) * ur);
            } else {
              double2 ic = ((const double2*)smem_raw)[ci[h][t]];
              double v = av[h][t] * ic.x;
              atomicAdd(&accs[ci[h][t]], (v > ic.y ? ic.y : v) * ur);
            }
          }
        }
      }
    }
  }
  // lane 0 of each warp holds the rows' u (all lanes accumulated the same values)
  if (lane != 0) usum = 0;
  usum = sv_warp_sum(usum);
  if (lane == 0) red[threadIdx.x >> 5] = usum;
  __syncthreads();
  AccT* prow = (AccT*)partial + (int64_t)blockIdx.x * nf;
  for (int64_t f = threadIdx.x; f < nf; f += blockDim.x) prow[f] = accs[f];
  if (threadIdx.x == 0) {
    double t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
    upart[blockIdx.x] = t;
  }
}

template <typename AccT>
__global__ void k_spmv_t_finish(const AccT* __restrict__ partial, int nblocks, int64_t nf,
                                const double* __restrict__ mu, const double* __restrict__ upart,
                                double alpha, double beta, double* __restrict__ y,
                                const double* __restrict__ csub, const double* __restrict__ z) {
  __shared__ double su_s;
  if (threadIdx.x < 32) {
    double v = 0;
    for (int i = threadIdx.x; i < nblocks; i += 32) v += upart[i];
    v = sv_warp_sum(v);
    if (threadIdx.x == 0) su_s = v;
  }
  __syncthreads();
  double su = su_s;
  double cs = csub ? *csub : 0.0;
  for (int64_t f = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; f < nf;
       f += (int64_t)gridDim.x * blockDim.x) {
    double acc = 0;
    for (int b = 0; b < nblocks; ++b) acc += (double)partial[(int64_t)b * nf + f];
    double out = alpha * (acc - mu[f] * su);
    if (beta != 0.0) out += beta * y[f];
    if (z) out -= cs * z[f];
    y[f] = out;
  }
}

// ---- X^T u over the row-blocked CSC copy ---------------------------------------
// The feature subset is stored once more, ordered (row block, feature, row): for
// every block of RB consecutive cells and every feature, the entries of that
// feature in those cells, with the row as a 16-bit offset into the block.  A CTA
// (row block b, feature group g) stages u[b*RB : (b+1)*RB] in shared memory as
// FP32 and gathers from there, so the product streams 4 B per entry (uint16 row +
// BF16 value) and no gather reaches L2.
constexpr int64_t RB_ROWS = 16384;
constexpr int RB_THREADS = 512;
constexpr int RB_DEPTH2 = 4, RB_DEPTH4 = 3;   // groups per lane in flight, BF16 and FP32

// first row of row block b: b * RB_ROWS, or row0[b] for blocks aligned to
// sample boundaries
__device__ __forceinline__ int64_t rb_first_row(const int64_t* row0, int64_t b) {
  return row0 ? row0[b] : b * RB_ROWS;
}

// The row-blocked copy codes a segment's rows in groups of 8 entries, one
// 64-bit word per group: bits 0-15 the row (within the block) of the group's
// first entry, bits 16 + 6 (t - 1) .. the 6-bit step from entry t - 1 to entry
// t (t = 1..7).  A step longer than 63 between consecutive entries is bridged
// by padding entries (rows r + 63, r + 126, ... and value -0), and every segment
// is padded with value -0 entries to a whole number of groups, so segments
// start on group boundaries.  Padding adds exactly 0 to the product: where clip
// >= 0 as min(-0 * (1/sigma), clip), and below that, where a stored 0 is clipped
// as well, its sign tells it apart.
constexpr int RB_GROUP = 8;
__device__ __forceinline__ int rb_pads(int64_t step) { return step > 63 ? (int)((step - 1) / 63) : 0; }

// per (row block, feature), one warp: entries + padding (whole groups), first source entry
__global__ void k_rb_count(const int64_t* __restrict__ fstart, const int64_t* __restrict__ fend,
                           const int32_t* __restrict__ rowidx, int64_t nf, int64_t n_rb,
                           int64_t* __restrict__ cnt, int64_t* __restrict__ src,
                           const int64_t* __restrict__ row0) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t p = warp; p < n_rb * nf; p += nwarps) {
    const int64_t b = p / nf, f = p % nf;
    const int64_t s = fstart[f], e = fend[f];
    const int64_t lo = lower_bound_rows(rowidx, s, e, rb_first_row(row0, b));
    const int64_t hi = lower_bound_rows(rowidx, lo, e, rb_first_row(row0, b + 1));
    int pads = 0;
    for (int64_t t = lo + 1 + lane; t < hi; t += 128) {
      int step[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) step[u] = t + 32 * u < hi ? rowidx[t + 32 * u] - rowidx[t + 32 * u - 1] : 0;
#pragma unroll
      for (int u = 0; u < 4; ++u) pads += rb_pads(step[u]);
    }
    pads = sv_warp_sum(pads);
    if (lane == 0) {
      const int64_t n = hi - lo + pads;
      cnt[p] = (n + RB_GROUP - 1) / RB_GROUP * RB_GROUP;
      src[p] = lo;
    }
  }
}

// One warp per (row block, feature): the coded rows and the values, padding
// included.  Entries and padding pass through a ring of RC_RING places per warp in
// shared memory; whenever it holds 256, each lane codes one group of 8 and writes
// its word and values at once (a 64-bit atomic or per entry and scalar value
// stores took 1.77 ms for 117 M FP32 entries of 100,000 cells, this 0.88 ms; one
// group of entries in flight instead of RC_FLIGHT 1.08).
constexpr int RC_RING = 512;
constexpr int RC_WARPS = 8;
constexpr int RC_FLIGHT = 2;   // groups of 32 entries in flight
template <typename ValT>
__global__ void __launch_bounds__(RC_WARPS * 32) k_rb_copy(
    const int64_t* __restrict__ src, const int64_t* __restrict__ dst, const int64_t* __restrict__ fend,
    const int32_t* __restrict__ rowidx, const ValT* __restrict__ val, int64_t npairs, int64_t nf,
    unsigned long long* __restrict__ ocode, ValT* __restrict__ oval, const int64_t* __restrict__ row0) {
  __shared__ __align__(16) uint16_t ring_r[RC_WARPS][RC_RING];
  __shared__ __align__(16) ValT ring_v[RC_WARPS][RC_RING];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint16_t* rr = ring_r[w];
  ValT* rv = ring_v[w];
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t p = warp; p < npairs; p += nwarps) {
    const int64_t b = p / nf;
    const int first = (int)rb_first_row(row0, b);
    const int64_t s = src[p], d = dst[p];
    const int64_t hi = p + nf < npairs ? src[p + nf] : fend[p % nf];   // the next block's first entry
    int64_t word = d / RB_GROUP;   // the next word to write
    int head = 0, cur = 0;         // ring: cur places from head
    // writes the first `words` groups of the ring
    auto flush = [&](int words) {
      __syncwarp();
      if (lane < words) {
        const int at = (head + RB_GROUP * lane) & (RC_RING - 1);
        const uint4 r4 = *(const uint4*)(rr + at);
        const unsigned q[4] = {r4.x, r4.y, r4.z, r4.w};
        int prev = (int)(q[0] & 0xffffu);
        unsigned long long code = (unsigned long long)prev;
#pragma unroll
        for (int t = 1; t < RB_GROUP; ++t) {
          const int r = (int)((t & 1) ? q[t >> 1] >> 16 : q[t >> 1] & 0xffffu);
          code |= (unsigned long long)(r - prev) << (16 + 6 * (t - 1));
          prev = r;
        }
        ocode[word + lane] = code;
        const uint4* v4 = (const uint4*)(rv + at);
        uint4* o4 = (uint4*)(oval + (word + lane) * RB_GROUP);
#pragma unroll
        for (int u = 0; u < (int)sizeof(ValT) * RB_GROUP / 16; ++u) o4[u] = v4[u];
      }
      word += words;
      head = (head + RB_GROUP * words) & (RC_RING - 1);
      cur -= RB_GROUP * words;
      __syncwarp();
    };
    int last = 0;                  // the row before t0
    int nrow[RC_FLIGHT];           // the next groups of 32 entries
    ValT nval[RC_FLIGHT];
#pragma unroll
    for (int h = 0; h < RC_FLIGHT; ++h) {
      const int64_t t = s + 32 * h + lane;
      nrow[h] = t < hi ? rowidx[t] : 0;
      nval[h] = t < hi ? val[t] : ValT(0.f);
    }
    for (int64_t t0 = s; t0 < hi; t0 += 32) {
      const bool on = t0 + lane < hi;
      const int r = nrow[0] - first;
      const ValT v = nval[0];
#pragma unroll
      for (int h = 0; h + 1 < RC_FLIGHT; ++h) {
        nrow[h] = nrow[h + 1];
        nval[h] = nval[h + 1];
      }
      const int64_t tn = t0 + 32 * RC_FLIGHT + lane;
      if (tn < hi) {
        nrow[RC_FLIGHT - 1] = rowidx[tn];
        nval[RC_FLIGHT - 1] = val[tn];
      }
      const int up = __shfl_up_sync(0xffffffffu, r, 1);
      const int rp = lane > 0 ? up : t0 > s ? last : r;
      const int k = on ? rb_pads(r - rp) : 0;
      int incl = lane + 1;                                 // no padding: one place each
      if (__any_sync(0xffffffffu, k > 0)) {
        incl = on ? k + 1 : 0;
#pragma unroll
        for (int sh = 1; sh < 32; sh <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, incl, sh);
          if (lane >= sh) incl += y;
        }
      }
      // the group at once, or as many entries as 256 places take at a time (one entry
      // takes at most 261)
      unsigned todo = __ballot_sync(0xffffffffu, on);
      last = __shfl_sync(0xffffffffu, r, 31 - __clz(todo));
      int before = 0;                // places of the entries done
      while (todo) {
        const bool mine = (todo >> lane & 1) && (incl - before <= 256 || (todo & ((1u << lane) - 1)) == 0);
        const unsigned fit = __ballot_sync(0xffffffffu, mine);
        const int upto = __shfl_sync(0xffffffffu, incl, 31 - __clz(fit));
        if (cur + upto - before > RC_RING) flush(cur / RB_GROUP);   // fewer than 256 places: at most 31 words
        if (mine) {
          int q = head + cur + incl - before - (k + 1);
          for (int u = 1; u <= k; ++u, ++q) {
            rr[q & (RC_RING - 1)] = (uint16_t)(rp + 63 * u);
            rv[q & (RC_RING - 1)] = ValT(-0.f);
          }
          rr[q & (RC_RING - 1)] = (uint16_t)r;
          rv[q & (RC_RING - 1)] = v;
        }
        cur += upto - before;
        before = upto;
        todo &= ~fit;
        if (cur >= 256) flush(32);
      }
    }
    // padding up to the group boundary, at the last row
    const int fill = (RB_GROUP - cur % RB_GROUP) % RB_GROUP;
    if (lane < fill) {
      rr[(head + cur + lane) & (RC_RING - 1)] = (uint16_t)last;
      rv[(head + cur + lane) & (RC_RING - 1)] = ValT(-0.f);
    }
    cur += fill;
    if (cur >= 256) flush(32);
    if (cur > 0) flush(cur / RB_GROUP);
  }
}

// One lane's group of 8 entries of the row-blocked copy, as loaded.
template <typename ValT>
struct RbGroup {
  unsigned long long c;
  uint4 v[sizeof(ValT) == 2 ? 1 : 2];
  __device__ __forceinline__ void load(const unsigned long long* __restrict__ code, const ValT* __restrict__ pv) {
    c = __ldg(code);
    v[0] = __ldg((const uint4*)pv);
    if constexpr (sizeof(ValT) == 4) v[1] = __ldg((const uint4*)pv + 1);
  }
  template <bool BELOW = false>   // BELOW: clip < 0
  __device__ __forceinline__ void add(float& acc, float inv, float clip, const float* us) const {
    // byte offsets into us: a field is shifted to bit 2 and masked
    const unsigned lo = (unsigned)c, hi = (unsigned)(c >> 32);
    unsigned r = (lo & 0xffffu) << 2;
#pragma unroll
    for (int t = 0; t < RB_GROUP; ++t) {
      if (t > 0) {
        const int at = 16 + 6 * (t - 1) - 2;
        r += (at >= 32 ? hi >> (at - 32) : at + 8 > 32 ? __funnelshift_r(lo, hi, at) : lo >> at) & 0xfcu;
      }
      float a;
      if constexpr (sizeof(ValT) == 2) {
        const unsigned w = (&v[0].x)[t >> 1];
        a = __uint_as_float((t & 1) ? (w & 0xffff0000u) : (w << 16));
      } else {
        a = __uint_as_float((&v[t >> 2].x)[t & 3]);
      }
      if (BELOW && __float_as_uint(a) == 0x80000000u) continue;   // padding
      acc += fminf(a * inv, clip) * *(const float*)((const char*)us + r);
    }
  }
};

// sum over a segment of n groups of min(a (1/sigma), clip) u[row]; lane-local
// decoding, a group reloaded as soon as it is added
template <typename ValT>
__device__ __forceinline__ float rb_seg_dot(const unsigned long long* __restrict__ code,
                                           const ValT* __restrict__ pv, int n,
                                           float inv, float clip, const float* us, int lane) {
  constexpr int D = sizeof(ValT) == 2 ? RB_DEPTH2 : RB_DEPTH4;
  float acc = 0.f;
  if (clip < 0.f) {   // scale_max below -mu: rare, one group at a time
    for (int g = lane; g < n; g += 32) {
      RbGroup<ValT> one;
      one.load(code + g, pv + RB_GROUP * g);
      one.template add<true>(acc, inv, clip, us);
    }
    return acc;
  }
  RbGroup<ValT> buf[D];
#pragma unroll
  for (int h = 0; h < D; ++h) {
    const int g = lane + 32 * h;
    if (g < n) buf[h].load(code + g, pv + RB_GROUP * g);
  }
  for (int g0 = lane; g0 < n; g0 += 32 * D) {
#pragma unroll
    for (int h = 0; h < D; ++h) {
      const int g = g0 + 32 * h;
      if (g >= n) break;
      buf[h].add(acc, inv, clip, us);
      if (g + 32 * D < n) buf[h].load(code + g + 32 * D, pv + RB_GROUP * (g + 32 * D));
    }
  }
  return acc;
}

template <typename ValT>
__global__ void __launch_bounds__(RB_THREADS, 2) k_spmv_rb(
    const int64_t* __restrict__ rb_ptr, const unsigned long long* __restrict__ rb_code,
    const ValT* __restrict__ rb_val, int64_t nf, int64_t n_cells, const float* __restrict__ inv_f,
    const float* __restrict__ clip_f, const float* __restrict__ uf, float* __restrict__ partial,
    const int64_t* __restrict__ row0, const int* __restrict__ rb_seg,
    const int* __restrict__ active) {
  extern __shared__ __align__(16) float us[];
  int64_t b = blockIdx.x;
  int64_t r0, nr;
  if (row0) {
    // blocks aligned to samples: that sample's feature parameters
    int sg = rb_seg[b];
    if (active && !active[sg]) return;
    r0 = row0[b];
    nr = row0[b + 1] - r0;
    inv_f += (int64_t)sg * nf;
    clip_f += (int64_t)sg * nf;
  } else {
    r0 = b * RB_ROWS;
    nr = n_cells - r0 < RB_ROWS ? n_cells - r0 : RB_ROWS;
  }
  for (int64_t i = threadIdx.x; i < RB_ROWS; i += blockDim.x) us[i] = i < nr ? uf[r0 + i] : 0.f;
  __syncthreads();
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int fg = gridDim.y, g = blockIdx.y;
  for (int64_t f = g + (int64_t)fg * w; f < nf; f += (int64_t)fg * nw) {
    int64_t s = rb_ptr[b * nf + f], e = rb_ptr[b * nf + f + 1];
    float inv = inv_f[f], clip = clip_f[f];
    float acc = rb_seg_dot<ValT>(rb_code + s / RB_GROUP, rb_val + s, (int)((e - s) / RB_GROUP), inv, clip, us, lane);
    acc = sv_warp_sum(acc);
    if (lane == 0) partial[b * nf + f] = acc;
  }
}

// The same product for one sample, as a single wave of resident blocks: tasks
// (row block b, feature group g) taken round-robin (b-major), the features of
// a task (order[g], order[g + fg], ...: long ones first) handed to the warps one
// at a time through a shared counter, so that dense and sparse features even out
// within the block.  Same sums and partials as k_spmv_rb.  525 M BF16 entries of
// 500,000 cells: 321 us, 4.9 TB/s (368 us with groups of whatever size gave six
// tasks a block -- seven to some -- and features in their own order); 62 M FP32
// entries of 50,000 cells: 74 us.  The gathers are what is left: 32 rows anywhere
// in the vector take 3.4 passes over the shared-memory banks, and the data pipe of
// L1 is busy 0.7 of the time.  48 warps an SM in place of 32 measured the same.
template <typename ValT>
__global__ void __launch_bounds__(RB_THREADS, 2) k_spmv_rb_waves(
    const int64_t* __restrict__ rb_ptr, const unsigned long long* __restrict__ rb_code,
    const ValT* __restrict__ rb_val, int64_t nf, int64_t n_cells, int64_t n_rb, int fg,
    const float* __restrict__ inv_f, const float* __restrict__ clip_f, const float* __restrict__ uf,
    float* __restrict__ partial, const int32_t* __restrict__ order) {
  extern __shared__ __align__(16) float us[];
  __shared__ int next_f;
  const int lane = threadIdx.x & 31;
  const int64_t ntask = n_rb * fg;
  for (int64_t task = blockIdx.x; task < ntask; task += gridDim.x) {
    const int64_t b = task / fg;
    const int g = (int)(task % fg);
    const int64_t r0 = b * RB_ROWS;
    const int64_t nr = n_cells - r0 < RB_ROWS ? n_cells - r0 : RB_ROWS;
    __syncthreads();                        // the previous task is done with us and next_f
    for (int64_t i = threadIdx.x; i < RB_ROWS; i += blockDim.x) us[i] = i < nr ? uf[r0 + i] : 0.f;
    if (threadIdx.x == 0) next_f = 0;
    __syncthreads();
    // a warp's next feature and its segment arrive while it adds this one's
    auto take = [&](int64_t& f, int64_t& s, int64_t& e, float& inv, float& clip) {
      int fi = 0;
      if (lane == 0) fi = atomicAdd(&next_f, 1);
      f = g + (int64_t)__shfl_sync(0xffffffffu, fi, 0) * fg;
      if (f < nf) {
        f = order[f];
        s = rb_ptr[b * nf + f];
        e = rb_ptr[b * nf + f + 1];
        inv = inv_f[f];
        clip = clip_f[f];
      }
    };
    int64_t f, s = 0, e = 0;
    float inv = 0.f, clip = 0.f;
    take(f, s, e, inv, clip);
    while (f < nf) {
      int64_t fn, sn = 0, en = 0;
      float invn = 0.f, clipn = 0.f;
      take(fn, sn, en, invn, clipn);
      float acc = rb_seg_dot<ValT>(rb_code + s / RB_GROUP, rb_val + s, (int)((e - s) / RB_GROUP), inv, clip, us, lane);
      acc = sv_warp_sum(acc);
      if (lane == 0) partial[b * nf + f] = acc;
      f = fn;
      s = sn;
      e = en;
      inv = invn;
      clip = clipn;
    }
  }
}

// order[rank] = f, features by falling number of entries: the warps of a task take
// the long ones first, and what they wait for at its end is a short one.
__global__ void __launch_bounds__(256) k_rb_order(const int64_t* __restrict__ fstart,
                                                  const int64_t* __restrict__ fend, int64_t nf,
                                                  int32_t* __restrict__ order) {
  const int lane = threadIdx.x & 31;
  const int64_t f = blockIdx.x * 8ll + (threadIdx.x >> 5);
  if (f >= nf) return;
  const int64_t n = fend[f] - fstart[f];
  int rank = 0;
  for (int64_t o = lane; o < nf; o += 32) {
    const int64_t m = fend[o] - fstart[o];
    rank += m > n || (m == n && o < f);
  }
  rank = sv_warp_sum(rank);
  if (lane == 0) order[rank] = (int32_t)f;
}

// y_f = alpha * (sum_b partial[b][f] - mu_f * sum(u)) + beta*y_f - csub*z_f
__global__ void k_rb_finish(const float* __restrict__ partial, int64_t n_rb, int64_t nf,
                            const double* __restrict__ mu, const double* __restrict__ upart,
                            int nupart, double alpha, double beta, double* __restrict__ y,
                            const double* __restrict__ csub, const double* __restrict__ z) {
  __shared__ double su_s;
  if (threadIdx.x < 32) {
    double v = 0;
    for (int i = threadIdx.x; i < nupart; i += 32) v += upart[i];
    v = sv_warp_sum(v);
    if (threadIdx.x == 0) su_s = v;
  }
  __syncthreads();
  double su = su_s;
  double cs = csub ? *csub : 0.0;
  for (int64_t f = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; f < nf;
       f += (int64_t)gridDim.x * blockDim.x) {
    double acc = 0;
    for (int64_t bb = 0; bb < n_rb; ++bb) acc += (double)partial[bb * nf + f];
    double out = alpha * (acc - mu[f] * su);
    if (beta != 0.0) out += beta * y[f];
    if (z) out -= cs * z[f];
    y[f] = out;
  }
}

// Stacked samples: y[s*nf + f] = sum over the sample's row blocks of
// partial[b][f] - mu[s*nf + f] * (sum of u over the sample) - csub[s] * z[s*nf + f]
// (blockIdx.y = sample).
__global__ void k_rb_finish_seg(const float* __restrict__ partial, const int64_t* __restrict__ rb_first,
                                int64_t nf, const double* __restrict__ mu,
                                const double* __restrict__ upart, double* __restrict__ y,
                                const double* __restrict__ csub, const double* __restrict__ z,
                                const int* __restrict__ active) {
  const int sg = blockIdx.y;
  if (active && !active[sg]) return;
  const int64_t b0 = rb_first[sg], b1 = rb_first[sg + 1];
  double su = 0;
  for (int64_t b = b0; b < b1; ++b) su += upart[b];
  double cs = csub ? csub[sg] : 0.0;
  for (int64_t f = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; f < nf;
       f += (int64_t)gridDim.x * blockDim.x) {
    double acc = 0;
    for (int64_t b = b0; b < b1; ++b) acc += (double)partial[b * nf + f];
    int64_t o = (int64_t)sg * nf + f;
    double out = acc - mu[o] * su;
    if (z) out -= cs * z[o];
    y[o] = out;
  }
}

// u -> FP32 copy and the FP64 sum of u over each sample-aligned row block
__global__ void k_bu_prep(const double* __restrict__ u, const int64_t* __restrict__ row0,
                          float* __restrict__ uf, double* __restrict__ upart) {
  __shared__ double red[32];
  const int64_t b = blockIdx.x;
  double s = 0;
  for (int64_t i = row0[b] + threadIdx.x; i < row0[b + 1]; i += blockDim.x) {
    double v = u[i];
    uf[i] = (float)v;
    s += v;
  }
  s = sv_warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
    v = sv_warp_sum(v);
    if (threadIdx.x == 0) upart[b] = v;
  }
}

// ---- X^T u over the CSC feature ranges ---------------------------------------
// Prologue: u -> FP32 copy and per-block partial sums of u (FP64).
__global__ void k_split_df(const double* __restrict__ x, int64_t n, float* __restrict__ h,
                           float* __restrict__ l) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    float a = (float)x[i];
    h[i] = a;
    l[i] = (float)(x[i] - (double)a);
  }
}

__global__ void k_u_prep(const double* __restrict__ u, int64_t n, float* __restrict__ uf,
                         double* __restrict__ part) {
  __shared__ double red[32];
  double s = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    double v = u[i];
    if (uf) uf[i] = (float)v;
    s += v;
  }
  s = sv_warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
    v = sv_warp_sum(v);
    if (threadIdx.x == 0) part[blockIdx.x] = v;
  }
}

// A warp per chunk, CHUNK_FLIGHT groups of 4 entries per lane and their gathers in
// flight: with few cells there are few chunks (2,000 of 400 entries at 2,000 cells, 13
// warps an SM), and a chunk is a chain of round trips.  Blocks of two warps share
// the chunks out evenly.  2,000 cells, FP64: 21.0 -> 15.0 us.
constexpr int CHUNK_FLIGHT = 2;
constexpr int CHUNK_THREADS = 64, CHUNK_PER_SM = 16;
template <typename ValT>
__global__ void __launch_bounds__(CHUNK_THREADS) k_spmv_csc_chunks(
    const int32_t* __restrict__ rowidx, const ValT* __restrict__ val,
    const int32_t* __restrict__ chunk_feat, const int64_t* __restrict__ cstart,
    const int64_t* __restrict__ cend, int64_t nchunks, const float* __restrict__ inv_f,
    const float* __restrict__ clip_f, const double* __restrict__ std_d,
    const double* __restrict__ clip_d, const float* __restrict__ uf, const double* __restrict__ ud,
    double* __restrict__ partial) {
  typedef typename AccOf<ValT>::type AccT;
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t c = warp; c < nchunks; c += nwarps) {
    const int32_t f = chunk_feat[c];
    const int64_t s = cstart[c], e = cend[c], a0 = s & ~3ll;
    const int32_t* src = rowidx + a0;
    const ValT* vs = val + a0;
    const int head = (int)(s - a0), len = (int)(e - a0);
    AccT inv, clip;
    const AccT* u;
    if constexpr (sizeof(AccT) == 4) {
      inv = inv_f[f];
      clip = clip_f[f];
      u = uf;
    } else {
      inv = std_d[f];          // 1/std
      clip = clip_d[f];
      u = ud;
    }
    const long long key = clip_key((double)clip);
    AccT acc = 0;
    for (int g0 = 4 * lane; g0 < len; g0 += 128 * CHUNK_FLIGHT) {
      int ri[CHUNK_FLIGHT][4];
      AccT av[CHUNK_FLIGHT][4], x[CHUNK_FLIGHT][4];
#pragma unroll
      for (int h = 0; h < CHUNK_FLIGHT; ++h)
        if (g0 + 128 * h < len) {
          ld4(src, g0 + 128 * h, ri[h]);
          ld4v(vs, g0 + 128 * h, av[h]);
        }
#pragma unroll
      for (int h = 0; h < CHUNK_FLIGHT; ++h)
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int g = g0 + 128 * h + t;
          x[h][t] = g >= head && g < len ? __ldg(u + ri[h][t]) : AccT(0);
        }
#pragma unroll
      for (int h = 0; h < CHUNK_FLIGHT; ++h)
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int g = g0 + 128 * h + t;
          if (g >= head && g < len) {
            if constexpr (sizeof(AccT) == 4) acc += fminf(av[h][t] * inv, clip) * x[h][t];
            else acc += clip_above(av[h][t] * inv, key) * x[h][t];
          }
        }
    }
    acc = sv_warp_sum(acc);
    if (lane == 0) partial[c] = (double)acc;
  }
}

// y_f = alpha * (sum of the feature's chunk partials - mu_f * sum(u)) + beta*y_f - csub*z_f
__global__ void k_spmv_csc_finish(const double* __restrict__ partial,
                                  const int64_t* __restrict__ foff, int64_t nf,
                                  const double* __restrict__ mu, const double* __restrict__ upart,
                                  int nupart, double alpha, double beta, double* __restrict__ y,
                                  const double* __restrict__ csub, const double* __restrict__ z) {
  __shared__ double su_s;
  if (threadIdx.x < 32) {
    double v = 0;
    for (int i = threadIdx.x; i < nupart; i += 32) v += upart[i];
    v = sv_warp_sum(v);
    if (threadIdx.x == 0) su_s = v;
  }
  __syncthreads();
  double su = su_s;
  double cs = csub ? *csub : 0.0;
  for (int64_t f = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; f < nf;
       f += (int64_t)gridDim.x * blockDim.x) {
    double acc = 0;
    for (int64_t c = foff[f]; c < foff[f + 1]; ++c) acc += partial[c];
    double out = alpha * (acc - mu[f] * su);
    if (beta != 0.0) out += beta * y[f];
    if (z) out -= cs * z[f];
    y[f] = out;
  }
}

constexpr int UPREP_BLOCKS = SV_UPREP_BLOCKS;

}  // namespace

// ---------------------------------------------------------------------------
// internal product entry points (device vectors), used by irlba too
// ---------------------------------------------------------------------------
// row-blocked CSC: u (FP32) staged per row block in shared memory
static void launch_rb(sv_context* ctx, const sv_centered* S, const float* uf, bool beside = false) {
  sv_centered* Sm = const_cast<sv_centered*>(S);
  const int64_t resident = (ctx->num_sms - (beside ? 1 : 0)) * (int64_t)S->rb_per_sm;
  const int fg = beside ? S->rb_fg_beside : S->rb_fg;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(resident, S->n_rb * fg));
  size_t smem = RB_ROWS * sizeof(float);
  if (S->dtype == SV_F32)
    sv_launch(ctx, "spmv_rb", k_spmv_rb_waves<float>, dim3(grid), dim3(RB_THREADS), smem,
              (const int64_t*)S->rb_ptr.get(), (const unsigned long long*)S->rb_idx.get(),
              (const float*)S->rb_val.get(), S->nf, S->n_cells, S->n_rb, fg,
              (const float*)S->inv_std_f.get(), (const float*)S->clip_f.get(), uf, Sm->rb_partial.get(),
              (const int32_t*)S->rb_order.get());
  else
    sv_launch(ctx, "spmv_rb", k_spmv_rb_waves<__nv_bfloat16>, dim3(grid), dim3(RB_THREADS), smem,
              (const int64_t*)S->rb_ptr.get(), (const unsigned long long*)S->rb_idx.get(),
              (const __nv_bfloat16*)S->rb_val.get(), S->nf, S->n_cells, S->n_rb, fg,
              (const float*)S->inv_std_f.get(), (const float*)S->clip_f.get(), uf, Sm->rb_partial.get(),
              (const int32_t*)S->rb_order.get());
}

// CSC chunks over the feature ranges: u FP32 (uf) or, for FP64 data, FP64 (ud)
static void launch_chunks(sv_context* ctx, const sv_centered* S, const double* ud, const float* uf,
                          bool beside = false) {
  sv_centered* Sm = const_cast<sv_centered*>(S);
  int grid = sv_grid_for(ctx, S->n_chunks * 32, CHUNK_THREADS, CHUNK_PER_SM);
  if (beside) grid = std::min(grid, CHUNK_PER_SM * (ctx->num_sms - 1));
  const sv_data* D = S->data;
  const int32_t* rowidx = D->counts->csc_rowidx.get();
#define LAUNCH_CSC(VT)                                                                            \
  sv_launch(ctx, "spmv_csc_chunks", k_spmv_csc_chunks<VT>, dim3(grid), dim3(CHUNK_THREADS), 0, rowidx, \
            (const VT*)D->csc_val.get(), (const int32_t*)S->chunk_feat.get(),                     \
            (const int64_t*)S->chunk_start.get(), (const int64_t*)S->chunk_end.get(), S->n_chunks, \
            (const float*)S->inv_std_f.get(), (const float*)S->clip_f.get(),                      \
            (const double*)S->inv_std_d.get(), (const double*)S->clip_d.get(), uf, ud,            \
            Sm->chunk_partial.get())
  switch (S->dtype) {
    case SV_F64: LAUNCH_CSC(double); break;
    case SV_F32: LAUNCH_CSC(float); break;
    default: LAUNCH_CSC(__nv_bfloat16); break;
  }
#undef LAUNCH_CSC
}

// The partial sums of X^T u alone, for a caller that finishes them itself (the
// Lanczos feature side): u as FP64 and as FP32.  Not for the form over CSR_h.
// beside: a block of another kernel runs at the same time; its place is left free.
void sv_centered_apply_t_part(sv_context* ctx, const sv_centered* S, const double* ud, const float* uf,
                              SvTPart* o, bool beside) {
  o->mu = S->mu.get();
  o->nf = S->nf;
  if (S->n_rb > 0) {
    launch_rb(ctx, S, uf, beside);
    o->rb = S->rb_partial.get();
    o->n_rb = S->n_rb;
  } else {
    launch_chunks(ctx, S, ud, uf, beside);
    o->chunk = S->chunk_partial.get();
    o->foff = S->feat_chunk_off.get();
  }
}

void sv_centered_apply(sv_context* ctx, const sv_centered* S, char trans, const double* x, double* y,
                       double alpha, double beta, const double* csub, const double* z) {
  if (trans == 'N') {
    size_t smem = S->dtype == SV_F64 ? (size_t)S->nf * 24 : (size_t)S->nf * 8;
    smem = (smem + 15) & ~(size_t)15;
    const int threads = csr_threads(ctx, S->dtype, S->n_cells);
    int grid = (int)std::max<int64_t>(1, std::min<int64_t>(S->grid_csr, (S->n_cells * 32 + threads - 1) / threads));
#define LAUNCH_CSR(VT, IT, COL)                                                                  \
  sv_launch(ctx, "spmv_csr_h", csr_kernel<VT, IT>(threads), dim3(grid), dim3(threads), smem,     \
            (const int64_t*)S->h_rowptr.get(), (const IT*)COL, (const VT*)S->h_val.get(),         \
            S->n_cells, S->nf, x, (const float*)S->inv_std_f.get(), (const float*)S->clip_f.get(), \
            (const double*)S->inv_std_d.get(), (const double*)S->clip_d.get(),                    \
            (const double*)S->mu.get(), alpha, beta, y, csub, z)
    bool small = S->nf <= 65536;
    switch (S->dtype) {
      case SV_F64:
        if (small) LAUNCH_CSR(double, uint16_t, S->h_col16.get());
        else LAUNCH_CSR(double, int32_t, S->h_col32.get());
        break;
      case SV_F32:
        if (small) LAUNCH_CSR(float, uint16_t, S->h_col16.get());
        else LAUNCH_CSR(float, int32_t, S->h_col32.get());
        break;
      default:
        if (small) LAUNCH_CSR(__nv_bfloat16, uint16_t, S->h_col16.get());
        else LAUNCH_CSR(__nv_bfloat16, int32_t, S->h_col32.get());
        break;
    }
#undef LAUNCH_CSR
  } else if (S->n_rb > 0) {
    sv_centered* Sm = const_cast<sv_centered*>(S);
    sv_launch(ctx, "spmv_csc_uprep", k_u_prep, dim3(UPREP_BLOCKS), dim3(SV_UPREP_THREADS), 0, x, S->n_cells,
              Sm->u_f32.get(), Sm->red_partial.get());
    launch_rb(ctx, S, S->u_f32.get());
    sv_launch(ctx, "spmv_rb_finish", k_rb_finish, dim3(sv_grid_for(ctx, S->nf, 256, 4)), dim3(256), 0,
              (const float*)Sm->rb_partial.get(), S->n_rb, S->nf, (const double*)S->mu.get(),
              (const double*)Sm->red_partial.get(), UPREP_BLOCKS, alpha, beta, y, csub, z);
  } else if (S->t_blocks > 0) {
    // warp per cell over CSR_h, shared-memory accumulation per block
    sv_centered* Sm = const_cast<sv_centered*>(S);
    bool f64 = S->dtype == SV_F64;
    size_t smem = (size_t)S->nf * (f64 ? 24 : 12);
    bool small = S->nf <= 65536;
#define LAUNCH_CT(VT, IT, COL)                                                                     \
  sv_launch(ctx, "spmv_csr_t", k_spmv_csr_t<VT, IT>, dim3(S->t_blocks), dim3(256), smem,            \
            (const int64_t*)S->h_rowptr.get(), (const IT*)COL, (const VT*)S->h_val.get(),            \
            S->n_cells, S->nf, x, (const float*)S->inv_std_f.get(), (const float*)S->clip_f.get(),   \
            (const double*)S->inv_std_d.get(), (const double*)S->clip_d.get(),                       \
            (void*)Sm->t_partial.get(), Sm->red_partial.get())
    switch (S->dtype) {
      case SV_F64:
        if (small) LAUNCH_CT(double, uint16_t, S->h_col16.get());
        else LAUNCH_CT(double, int32_t, S->h_col32.get());
        break;
      case SV_F32:
        if (small) LAUNCH_CT(float, uint16_t, S->h_col16.get());
        else LAUNCH_CT(float, int32_t, S->h_col32.get());
        break;
      default:
        if (small) LAUNCH_CT(__nv_bfloat16, uint16_t, S->h_col16.get());
        else LAUNCH_CT(__nv_bfloat16, int32_t, S->h_col32.get());
        break;
    }
#undef LAUNCH_CT
    if (f64)
      sv_launch(ctx, "spmv_t_finish", k_spmv_t_finish<double>, dim3(sv_grid_for(ctx, S->nf, 256, 4)),
                dim3(256), 0, (const double*)Sm->t_partial.get(), S->t_blocks, S->nf,
                (const double*)S->mu.get(), (const double*)Sm->red_partial.get(), alpha, beta, y, csub,
                z);
    else
      sv_launch(ctx, "spmv_t_finish", k_spmv_t_finish<float>, dim3(sv_grid_for(ctx, S->nf, 256, 4)),
                dim3(256), 0, (const float*)Sm->t_partial.get(), S->t_blocks, S->nf,
                (const double*)S->mu.get(), (const double*)Sm->red_partial.get(), alpha, beta, y, csub,
                z);
  } else {
    sv_centered* Sm = const_cast<sv_centered*>(S);
    bool f64 = S->dtype == SV_F64;
    sv_launch(ctx, "spmv_csc_uprep", k_u_prep, dim3(UPREP_BLOCKS), dim3(256), 0, x, S->n_cells,
              f64 ? (float*)nullptr : Sm->u_f32.get(), Sm->red_partial.get());
    launch_chunks(ctx, S, x, S->u_f32.get());
    sv_launch(ctx, "spmv_csc_finish", k_spmv_csc_finish, dim3(sv_grid_for(ctx, S->nf, 256, 4)),
              dim3(256), 0, (const double*)S->chunk_partial.get(),
              (const int64_t*)S->feat_chunk_off.get(), S->nf, (const double*)S->mu.get(),
              (const double*)Sm->red_partial.get(), UPREP_BLOCKS, alpha, beta, y, csub, z);
  }
}

// Builds the implicit matrix over the features `fg` (0-based genes) of `data`.
// mu_given == nullptr: per-feature moments (scale_features).  Otherwise the
// CenteredMatrix(A, mu) constructor of src/scaling.jl:224-232: std = 1, no clip.
// X v with double-float input and output (the Lanczos W step): false when the
// matrix stores FP64 values (the FP64 product is used then)
bool sv_centered_apply_df(sv_context* ctx, const sv_centered* S, const float* xh, const float* xl,
                          float* yh, float* yl, const double* csub, const float* zh, const float* zl) {
  if (S->dtype == SV_F64) return false;
  size_t smem = ((size_t)S->nf * 8 + 15) & ~(size_t)15;
  const int grid = S->grid_csr_df;
#define LAUNCH_CSRDF(VT, IT, COL)                                                                \
  sv_launch(ctx, "spmv_csr_h", k_spmv_csr_df<VT, IT>, dim3(grid), dim3(256), smem,               \
            (const int64_t*)S->h_rowptr.get(), (const IT*)COL, (const VT*)S->h_val.get(),         \
            (const int64_t*)S->xv_cut.get(), S->nf, xh, xl, (const float*)S->inv_std_f.get(),     \
            (const float*)S->clip_f.get(), (const float*)S->mu_h.get(), (const float*)S->mu_l.get(), \
            yh, yl, csub, zh, zl, (const BlkRange*)nullptr, (const int*)nullptr)
  bool small = S->nf <= 65536;
  if (S->dtype == SV_F32) {
    if (small) LAUNCH_CSRDF(float, uint16_t, S->h_col16.get());
    else LAUNCH_CSRDF(float, int32_t, S->h_col32.get());
  } else {
    if (small) LAUNCH_CSRDF(__nv_bfloat16, uint16_t, S->h_col16.get());
    else LAUNCH_CSRDF(__nv_bfloat16, int32_t, S->h_col32.get());
  }
#undef LAUNCH_CSRDF
  return true;
}

// 1-based feature indices (null: every gene) -> 0-based genes, checked
static std::vector<int32_t> feature_genes(const sv_counts* C, const int64_t* features, int64_t nfeatures) {
  SV_REQUIRE(C->n_cells >= 2, "need at least two cells for a variance");
  int64_t nf = features ? nfeatures : C->n_genes;
  SV_REQUIRE(nf >= 1, "no features");
  std::vector<int32_t> fg(nf);
  std::vector<char> seen(C->n_genes, 0);
  for (int64_t f = 0; f < nf; ++f) {
    int64_t g = features ? features[f] - 1 : f;
    SV_REQUIRE(g >= 0 && g < C->n_genes, "feature %lld out of range 1..%lld", (long long)(g + 1),
               (long long)C->n_genes);
    SV_REQUIRE(!seen[g], "duplicate feature %lld", (long long)(g + 1));
    seen[g] = 1;
    fg[f] = (int32_t)g;
  }
  return fg;
}

// Row-blocked CSC copy of the feature subset (the X^T u layout): for every
// (row block, feature) the block's entries of the feature, their rows within
// the block coded in groups of 8 (see k_rb_count) and their values.  Row blocks of RB_ROWS rows, or with
// first rows row0 (n_rb + 1 entries, device) when aligned to samples.
// Feature groups per row block: the tasks (row block, group) go round robin to
// `resident` blocks, so the time is that of the block with the most; each task also
// loads its row block's vector (~2.5 us, here as bytes of a block's share of the
// bandwidth), and 16 features at least are left to its 16 warps.
static int rb_groups(int64_t resident, int64_t n_cells, int64_t nf, int64_t nnz, size_t es) {
  const int64_t full = n_cells / RB_ROWS, part = n_cells % RB_ROWS;
  const double row_bytes = (double)nnz * (es + 1) / n_cells;       // of a row over all features
  const double load = 2.5e-6 * 6.8e12 / resident;
  int64_t best = 1;
  double least = 0;
  for (int64_t fg = 1; fg <= std::max<int64_t>(1, nf / 16); ++fg) {
    // block 0 has the most full tasks; the partial row block's tasks come last
    const int64_t nt = full * fg + (part ? fg : 0);
    const int64_t most = (full * fg + resident - 1) / resident;
    const bool extra = part && (nt + resident - 1) / resident > most;
    const double t = most * (row_bytes * RB_ROWS / fg + load) + (extra ? row_bytes * part / fg + load : 0);
    if (fg == 1 || t < least) {
      least = t;
      best = fg;
    }
  }
  return (int)best;
}

static void rb_build(sv_context* ctx, const sv_counts* C, const sv_data* data, const int64_t* fstart,
                     const int64_t* fend, int64_t nf, int64_t nnz_h, int64_t n_rb, const int64_t* row0,
                     DevBuf<int64_t>& rb_ptr, DevBuf<unsigned long long>& rb_idx, DevBuf<unsigned char>& rb_val,
                     DevBuf<float>& rb_partial) {
  int64_t np = n_rb * nf;
  DevBuf<int64_t> cnt(np + 1), src(np + 1);
  sv_launch(ctx, "scale_rb_count", k_rb_count, dim3(sv_grid_for(ctx, np * 32, 256, 8)), dim3(256), 0, fstart,
            fend, (const int32_t*)C->csc_rowidx.get(), nf, n_rb, cnt.get(), src.get(), row0);
  rb_ptr.alloc(np + 1);
  sv_scan_i64(ctx, cnt.get(), rb_ptr.get(), np);
  const int64_t tot = sv_read_i64(ctx, rb_ptr.get() + np);   // entries + padding
  if (tot < nnz_h)
    sv_throw(SV_ERR_DEVICE, "row-blocked copy size mismatch (%lld vs %lld)", (long long)tot,
             (long long)nnz_h);
  size_t es2 = sv_elem_size(data->dtype);
  rb_idx.alloc(std::max<int64_t>(1, tot / RB_GROUP));
  rb_val.alloc(std::max<int64_t>(1, tot) * es2);
  rb_partial.alloc(std::max<int64_t>(1, np));
  int gridc = sv_grid_for(ctx, np * 32, 256, 8);
  if (data->dtype == SV_F32)
    sv_launch(ctx, "scale_rb_copy", k_rb_copy<float>, dim3(gridc), dim3(256), 0, (const int64_t*)src.get(),
              (const int64_t*)rb_ptr.get(), fend, (const int32_t*)C->csc_rowidx.get(),
              (const float*)data->csc_val.get(), np, nf, rb_idx.get(), (float*)rb_val.get(), row0);
  else
    sv_launch(ctx, "scale_rb_copy", k_rb_copy<__nv_bfloat16>, dim3(gridc), dim3(256), 0,
              (const int64_t*)src.get(), (const int64_t*)rb_ptr.get(), fend,
              (const int32_t*)C->csc_rowidx.get(), (const __nv_bfloat16*)data->csc_val.get(), np, nf,
              rb_idx.get(), (__nv_bfloat16*)rb_val.get(), row0);
  sv_sync(ctx);
}

static sv_centered* make_centered(sv_context* ctx, const sv_data* data, const std::vector<int32_t>& fg,
                                  double scale_max, const double* mu_given, bool want_rb = true) {
  const sv_counts* C = data->counts;
  int64_t nf = (int64_t)fg.size();
  size_t smem_need = data->dtype == SV_F64 ? (size_t)nf * 24 : (size_t)nf * 8;
  if (smem_need > 200 * 1024)
    sv_throw(SV_ERR_UNSUPPORTED, "%lld features exceed the shared-memory feature table",
             (long long)nf);
  auto* S = new sv_centered();
  try {
    S->ctx = ctx;
    S->data = data;
    S->n_cells = C->n_cells;
    S->nf = nf;
    S->dtype = data->dtype;
    S->scale_max = scale_max;
    S->feat_gene.alloc(nf);
    S->feat_start.alloc(nf);
    S->feat_end.alloc(nf);
    sv_h2d(ctx, S->feat_gene.get(), fg.data(), nf * 4);
    DevBuf<int32_t> gene_map(C->n_genes);
    sv_memset(ctx, gene_map.get(), 0xff, C->n_genes * 4);
    sv_launch(ctx, "scale_feat_ranges", k_feat_ranges, dim3(sv_grid_for(ctx, nf, 256)), dim3(256), 0,
              (const int32_t*)S->feat_gene.get(), (const int64_t*)C->csc_colptr.get(), nf,
              S->feat_start.get(), S->feat_end.get(), gene_map.get());
    // moments
    S->mean.alloc(nf);
    S->std_.alloc(nf);
    S->mu.alloc(nf);
    S->inv_std_f.alloc(nf);
    S->clip_f.alloc(nf);
    S->inv_std_d.alloc(nf);
    S->clip_d.alloc(nf);
#define LAUNCH_MOM(VT)                                                                          \
  launch_moments<VT>(ctx, "scale_moments", (const VT*)data->csc_val.get(),                        \
                     (const int64_t*)S->feat_start.get(), (const int64_t*)S->feat_end.get(), nf,   \
                     C->n_cells, scale_max, S->mean.get(), S->std_.get(), S->mu.get(),             \
                     S->inv_std_f.get(), S->clip_f.get(), S->inv_std_d.get(), S->clip_d.get(),      \
                     C->nnz)
    if (!mu_given) {
      switch (data->dtype) {
        case SV_F64: LAUNCH_MOM(double); break;
        case SV_F32: LAUNCH_MOM(float); break;
        default: LAUNCH_MOM(__nv_bfloat16); break;
      }
    } else {
      std::vector<double> one(nf, 1.0), inf(nf, INFINITY);
      std::vector<float> onef(nf, 1.0f), inff(nf, INFINITY);
      sv_h2d(ctx, S->mu.get(), mu_given, nf * 8);
      sv_h2d(ctx, S->mean.get(), mu_given, nf * 8);
      sv_h2d(ctx, S->std_.get(), one.data(), nf * 8);
      sv_h2d(ctx, S->inv_std_d.get(), one.data(), nf * 8);
      sv_h2d(ctx, S->clip_d.get(), inf.data(), nf * 8);
      sv_h2d(ctx, S->inv_std_f.get(), onef.data(), nf * 4);
      sv_h2d(ctx, S->clip_f.get(), inff.data(), nf * 4);
      sv_sync(ctx);
    }
#undef LAUNCH_MOM
    S->mu_h.alloc(nf);
    S->mu_l.alloc(nf);
    sv_launch(ctx, "scale_mu_split", k_split_df, dim3(sv_grid_for(ctx, nf, 256)), dim3(256), 0,
              (const double*)S->mu.get(), nf, S->mu_h.get(), S->mu_l.get());
    // chunk table of the CSC product (built on the host from the nf ranges)
    std::vector<int64_t> hs(nf), he(nf);
    sv_d2h(ctx, hs.data(), S->feat_start.get(), nf * 8);
    sv_d2h(ctx, he.data(), S->feat_end.get(), nf * 8);
    std::vector<int32_t> cf;
    std::vector<int64_t> cs, ce, foff(nf + 1);
    int64_t nnz_h = 0;
    for (int64_t f = 0; f < nf; ++f) {
      foff[f] = (int64_t)cf.size();
      int64_t s = hs[f], e = he[f];
      nnz_h += e - s;
      if (e == s) continue;
      // chunk boundaries on multiples of 4 elements (16-byte aligned vector loads)
      int64_t b = s;
      while (b < e) {
        int64_t nb = ((b + CHUNK) & ~3ll);
        if (nb > e || e - nb < CHUNK / 4) nb = e;
        cf.push_back((int32_t)f);
        cs.push_back(b);
        ce.push_back(nb);
        b = nb;
      }
    }
    foff[nf] = (int64_t)cf.size();
    S->nnz_h = nnz_h;
    S->n_chunks = (int64_t)cf.size();
    S->chunk_feat.alloc(std::max<int64_t>(1, S->n_chunks));
    S->chunk_start.alloc(std::max<int64_t>(1, S->n_chunks));
    S->chunk_end.alloc(std::max<int64_t>(1, S->n_chunks));
    S->chunk_partial.alloc(std::max<int64_t>(1, S->n_chunks));
    S->feat_chunk_off.alloc(nf + 1);
    sv_h2d(ctx, S->chunk_feat.get(), cf.data(), S->n_chunks * 4);
    sv_h2d(ctx, S->chunk_start.get(), cs.data(), S->n_chunks * 8);
    sv_h2d(ctx, S->chunk_end.get(), ce.data(), S->n_chunks * 8);
    sv_h2d(ctx, S->feat_chunk_off.get(), foff.data(), (nf + 1) * 8);
    // cell-major copy of the subset
    DevBuf<int64_t> rc(C->n_cells + 1);
    sv_launch(ctx, "scale_hsub_count", k_hsub_count, dim3(sv_grid_for(ctx, C->n_cells * 32, 256, 8)),
              dim3(256), 0, (const int64_t*)C->csr_rowptr.get(), (const int32_t*)C->csr_colidx.get(),
              C->n_cells, (const int32_t*)gene_map.get(), rc.get());
    S->h_rowptr.alloc(C->n_cells + 1);
    sv_scan_i64(ctx, rc.get(), S->h_rowptr.get(), C->n_cells);
    int64_t tot = sv_read_i64(ctx, S->h_rowptr.get() + C->n_cells);
    if (tot != nnz_h)
      sv_throw(SV_ERR_DEVICE, "subset sizes disagree between copies (%lld vs %lld)", (long long)tot,
               (long long)nnz_h);
    size_t es = sv_elem_size(data->dtype);
    S->h_val.alloc(std::max<int64_t>(1, nnz_h) * es);
    bool small = nf <= 65536;
    if (small) S->h_col16.alloc(std::max<int64_t>(1, nnz_h));
    else S->h_col32.alloc(std::max<int64_t>(1, nnz_h));
    int gridw = sv_grid_for(ctx, C->n_cells * 32, 256, 8);
#define LAUNCH_HW(VT, IT, COL)                                                                  \
  sv_launch(ctx, "scale_hsub_write", k_hsub_write<VT, IT>, dim3(gridw), dim3(256), 0,           \
            (const int64_t*)C->csr_rowptr.get(), (const int32_t*)C->csr_colidx.get(),            \
            (const VT*)data->csr_val.get(), C->n_cells, (const int32_t*)gene_map.get(),          \
            (const int64_t*)S->h_rowptr.get(), (IT*)COL, (VT*)S->h_val.get())
    switch (data->dtype) {
      case SV_F64:
        if (small) LAUNCH_HW(double, uint16_t, S->h_col16.get());
        else LAUNCH_HW(double, int32_t, S->h_col32.get());
        break;
      case SV_F32:
        if (small) LAUNCH_HW(float, uint16_t, S->h_col16.get());
        else LAUNCH_HW(float, int32_t, S->h_col32.get());
        break;
      default:
        if (small) LAUNCH_HW(uint16_t, uint16_t, S->h_col16.get());
        else LAUNCH_HW(uint16_t, int32_t, S->h_col32.get());
        break;
    }
#undef LAUNCH_HW
    if (small && data->dtype != SV_F64 && !getenv("SV_NO_BANKORDER")) {
      // bank-aware order of the rows (into a second copy, then swapped in)
      DevBuf<uint16_t> col2(std::max<int64_t>(1, nnz_h));
      DevBuf<unsigned char> val2(std::max<int64_t>(1, nnz_h) * es);
      const size_t bsm = BO_WARPS * (data->dtype == SV_F32 ? sizeof(BoRow<16, 4, float>)
                                                           : sizeof(BoRow<16, XV_EPL16, uint16_t>));
      SV_CUDA(cudaFuncSetAttribute(k_bankorder<16, 4, float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)(BO_WARPS * sizeof(BoRow<16, 4, float>))));
      SV_CUDA(cudaFuncSetAttribute(k_bankorder<16, XV_EPL16, uint16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)(BO_WARPS * sizeof(BoRow<16, XV_EPL16, uint16_t>))));
      int bgrid = sv_grid_for(ctx, C->n_cells, BO_WARPS, 16);
      if (data->dtype == SV_F32)
        sv_launch(ctx, "scale_hsub_order", k_bankorder<16, 4, float>, dim3(bgrid), dim3(BO_WARPS * 32), bsm,
                  (const int64_t*)S->h_rowptr.get(), C->n_cells, (const uint16_t*)S->h_col16.get(),
                  (const float*)S->h_val.get(), col2.get(), (float*)val2.get());
      else
        sv_launch(ctx, "scale_hsub_order", k_bankorder<16, XV_EPL16, uint16_t>, dim3(bgrid), dim3(BO_WARPS * 32), bsm,
                  (const int64_t*)S->h_rowptr.get(), C->n_cells, (const uint16_t*)S->h_col16.get(),
                  (const uint16_t*)S->h_val.get(), col2.get(), (uint16_t*)val2.get());
      S->h_col16 = std::move(col2);
      S->h_val = std::move(val2);
    }
    S->u_f32.alloc(C->n_cells);
    S->scal.alloc(64);
    // row-blocked CSC copy for X^T u (FP32 / BF16 storage; SV_TPRODUCT=csc or csr
    // selects the other forms)
    {
      const char* mode = getenv("SV_TPRODUCT");
      bool use_rb = want_rb && data->dtype != SV_F64 &&
                    !(mode && (strcmp(mode, "csc") == 0 || strcmp(mode, "csr") == 0));
      if (use_rb) {
        S->rb_rows = RB_ROWS;
        S->n_rb = (C->n_cells + RB_ROWS - 1) / RB_ROWS;
        rb_build(ctx, C, data, S->feat_start.get(), S->feat_end.get(), nf, nnz_h, S->n_rb, nullptr,
                 S->rb_ptr, S->rb_idx, S->rb_val, S->rb_partial);
        SV_CUDA(cudaFuncSetAttribute(k_spmv_rb<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(RB_ROWS * sizeof(float))));
        SV_CUDA(cudaFuncSetAttribute(k_spmv_rb<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(RB_ROWS * sizeof(float))));
        // three 64 KB blocks per SM: prefer the largest shared-memory carve-out
        SV_CUDA(cudaFuncSetAttribute(k_spmv_rb<float>, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
        SV_CUDA(cudaFuncSetAttribute(k_spmv_rb<__nv_bfloat16>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     100));
        SV_CUDA(cudaFuncSetAttribute(k_spmv_rb_waves<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(RB_ROWS * sizeof(float))));
        SV_CUDA(cudaFuncSetAttribute(k_spmv_rb_waves<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(RB_ROWS * sizeof(float))));
        SV_CUDA(cudaFuncSetAttribute(k_spmv_rb_waves<float>, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
        SV_CUDA(cudaFuncSetAttribute(k_spmv_rb_waves<__nv_bfloat16>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     100));
        int per = 0;
        if (data->dtype == SV_F32)
          SV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_spmv_rb_waves<float>, RB_THREADS,
                                                                RB_ROWS * sizeof(float)));
        else
          SV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_spmv_rb_waves<__nv_bfloat16>, RB_THREADS,
                                                                RB_ROWS * sizeof(float)));
        S->rb_per_sm = std::max(1, per);
        S->rb_fg = rb_groups(ctx->num_sms * S->rb_per_sm, C->n_cells, nf, nnz_h, sv_elem_size(data->dtype));
        S->rb_fg_beside =
            rb_groups((ctx->num_sms - 1) * S->rb_per_sm, C->n_cells, nf, nnz_h, sv_elem_size(data->dtype));
        S->rb_order.alloc(nf);
        sv_launch(ctx, "scale_rb_order", k_rb_order, dim3((unsigned)((nf + 7) / 8)), dim3(256), 0,
                  (const int64_t*)S->feat_start.get(), (const int64_t*)S->feat_end.get(), nf, S->rb_order.get());
        sv_sync(ctx);
      }
    }
    // X^T u: CSC chunks by default (measured faster on GB300: the CSR_h form is
    // bound by shared-memory atomics); SV_TPRODUCT=csr selects the warp-per-cell
    // form over CSR_h when its per-block feature arrays fit in shared memory
    {
      size_t tsmem = (size_t)nf * (data->dtype == SV_F64 ? 24 : 12);
      const char* mode = getenv("SV_TPRODUCT");
      bool want_csr = mode && strcmp(mode, "csr") == 0;
      if (want_csr && tsmem <= 200 * 1024) {
        S->t_blocks = ctx->num_sms * 2;
        S->t_partial.alloc((size_t)S->t_blocks * nf * (data->dtype == SV_F64 ? 8 : 4));
        SV_CUDA(cudaFuncSetAttribute(k_spmv_csr_t<double, uint16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        SV_CUDA(cudaFuncSetAttribute(k_spmv_csr_t<double, int32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        SV_CUDA(cudaFuncSetAttribute(k_spmv_csr_t<float, uint16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        SV_CUDA(cudaFuncSetAttribute(k_spmv_csr_t<float, int32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        SV_CUDA(cudaFuncSetAttribute(k_spmv_csr_t<__nv_bfloat16, uint16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        SV_CUDA(cudaFuncSetAttribute(k_spmv_csr_t<__nv_bfloat16, int32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
      }
      S->red_partial.alloc(std::max<int64_t>(UPREP_BLOCKS, S->t_blocks));
    }
#define SET_SMEM(VT, IT)                                                                         \
  for (int th : {256, 512})                                                                       \
    SV_CUDA(cudaFuncSetAttribute(csr_kernel<VT, IT>(th), cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024))
    SET_SMEM(double, uint16_t);
    SET_SMEM(double, int32_t);
    SET_SMEM(float, uint16_t);
    SET_SMEM(float, int32_t);
    SET_SMEM(__nv_bfloat16, uint16_t);
    SET_SMEM(__nv_bfloat16, int32_t);
#undef SET_SMEM
    SV_CUDA(cudaFuncSetAttribute(k_spmv_csr_df<float, uint16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    SV_CUDA(cudaFuncSetAttribute(k_spmv_csr_df<float, int32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    SV_CUDA(cudaFuncSetAttribute(k_spmv_csr_df<__nv_bfloat16, uint16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    SV_CUDA(cudaFuncSetAttribute(k_spmv_csr_df<__nv_bfloat16, int32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    // the X v kernels loop over rows: one wave of resident blocks (a second,
    // partial wave left SMs idle at the tail)
    {
      size_t tsm = ((size_t)nf * (data->dtype == SV_F64 ? 24 : 8) + 15) & ~(size_t)15;
      size_t tsm_df = ((size_t)nf * 8 + 15) & ~(size_t)15;
      int b1 = 0, b2 = 0;
      bool small16 = nf <= 65536;
      const int th = csr_threads(ctx, data->dtype, C->n_cells);
      switch (data->dtype) {
        case SV_F64:
          SV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
              &b1, small16 ? (const void*)csr_kernel<double, uint16_t>(th) : (const void*)csr_kernel<double, int32_t>(th),
              th, tsm));
          break;
        case SV_F32:
          SV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
              &b1, small16 ? (const void*)csr_kernel<float, uint16_t>(th) : (const void*)csr_kernel<float, int32_t>(th),
              th, tsm));
          SV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
              &b2, small16 ? (const void*)k_spmv_csr_df<float, uint16_t> : (const void*)k_spmv_csr_df<float, int32_t>,
              256, tsm_df));
          break;
        default:
          SV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
              &b1, small16 ? (const void*)csr_kernel<__nv_bfloat16, uint16_t>(th)
                           : (const void*)csr_kernel<__nv_bfloat16, int32_t>(th),
              th, tsm));
          SV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
              &b2, small16 ? (const void*)k_spmv_csr_df<__nv_bfloat16, uint16_t>
                           : (const void*)k_spmv_csr_df<__nv_bfloat16, int32_t>,
              256, tsm_df));
          break;
      }
      S->grid_csr = std::max(1, b1) * ctx->num_sms;
      S->grid_csr_df = (int)std::min<int64_t>(std::max(1, b2) * ctx->num_sms, (C->n_cells + 7) / 8);
      if (data->dtype != SV_F64) {
        S->xv_cut.alloc(S->grid_csr_df + 1);
        sv_launch(ctx, "scale_row_cuts", k_row_cuts, dim3(sv_grid_for(ctx, S->grid_csr_df + 1, 64)), dim3(64), 0,
                  (const int64_t*)S->h_rowptr.get(), C->n_cells, S->grid_csr_df, S->xv_cut.get());
      }
    }
    sv_sync(ctx);
  } catch (...) {
    delete S;
    throw;
  }
  return S;
}

SV_API int sv_scale_features(sv_context* ctx, const sv_data* data, const int64_t* features,
                             int64_t nfeatures, double scale_max, sv_centered** out) {
  SV_TRY
  sv_ctx_check(ctx);
  SV_REQUIRE(out && data, "null argument");
  SV_REQUIRE(data->ctx == ctx, "data handle belongs to another context");
  const sv_counts* C = data->counts;
  SV_REQUIRE(C->n_cells >= 2, "need at least two cells for a variance");
  std::vector<int32_t> fg = feature_genes(C, features, nfeatures);
  *out = make_centered(ctx, data, fg, scale_max, nullptr);
  SV_CATCH
}

// ---- batched samples ----------------------------------------------------------
// Samples stacked by cells in one data matrix, each scaled with its own
// moments (scale_features per sample, src/scaling.jl:335-357): the feature
// subset copies are those of the stacked matrix; the per-(sample, feature)
// moments, the X v block schedule and the sample-aligned row blocks of X^T u
// are the batch's own.  FP32 / BF16 storage.
// cells per X v block: chosen by timing the candidates on the first batch of a
// given shape (device, cells, features, samples), then reused
static const int BATCH_XCELLS_CAND[] = {128, 256, 512, 1024};
static std::mutex g_tune_mu;
static std::map<std::tuple<int, int64_t, int64_t, int64_t>, int> g_tune;

static void batch_xschedule(sv_context* ctx, sv_batch* B, int cells) {
  std::vector<BlkRange> hb;
  for (int64_t s2 = 0; s2 < B->nseg; ++s2)
    for (int64_t r = B->hoff[s2]; r < B->hoff[s2 + 1]; r += cells) {
      BlkRange b;
      b.r0 = r;
      b.r1 = std::min(B->hoff[s2 + 1], r + cells);
      b.seg = (int)s2;
      b.pad = 0;
      hb.push_back(b);
    }
  B->nxblk = (int)hb.size();
  B->xblk.alloc(hb.size());
  sv_h2d(ctx, B->xblk.get(), hb.data(), hb.size() * sizeof(BlkRange));
  B->xcells = cells;
}

void sv_batch_apply_N_df(sv_context* ctx, const sv_batch* b, const float* xh, const float* xl,
                         float* yh, float* yl, const double* csub, const float* zh, const float* zl,
                         const int* active);

// the autotuner: time every candidate block size on this batch (zero vectors)
static int batch_tune_xcells(sv_context* ctx, sv_batch* B) {
  auto key = std::make_tuple(ctx->device, B->n_cells, B->nf, B->nseg);
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    auto it = g_tune.find(key);
    if (it != g_tune.end()) return it->second;
  }
  DevBuf<float> xh((size_t)B->nseg * B->nf), yh(B->n_cells), yl(B->n_cells);
  sv_memset(ctx, xh.get(), 0, (size_t)B->nseg * B->nf * 4);
  cudaEvent_t e0, e1;
  SV_CUDA(cudaEventCreate(&e0));
  SV_CUDA(cudaEventCreate(&e1));
  int best = BATCH_XCELLS_CAND[1];
  float best_ms = 1e30f;
  for (int cand : BATCH_XCELLS_CAND) {
    batch_xschedule(ctx, B, cand);
    sv_batch_apply_N_df(ctx, B, xh.get(), xh.get(), yh.get(), yl.get(), nullptr, nullptr, nullptr, nullptr);
    SV_CUDA(cudaEventRecord(e0, ctx->stream));
    for (int r = 0; r < 3; ++r)
      sv_batch_apply_N_df(ctx, B, xh.get(), xh.get(), yh.get(), yl.get(), nullptr, nullptr, nullptr, nullptr);
    SV_CUDA(cudaEventRecord(e1, ctx->stream));
    SV_CUDA(cudaEventSynchronize(e1));
    float ms = 0;
    SV_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    if (ms < best_ms) {
      best_ms = ms;
      best = cand;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  std::lock_guard<std::mutex> lk(g_tune_mu);
  g_tune[key] = best;
  return best;
}

SV_API int sv_batch_create(sv_context* ctx, const sv_data* data, const int64_t* cell_offsets,
                           int64_t nseg, const int64_t* features, int64_t nfeatures, double scale_max,
                           sv_batch** out) {
  SV_TRY
  sv_ctx_check(ctx);
  SV_REQUIRE(out && data && cell_offsets, "null argument");
  SV_REQUIRE(data->ctx == ctx, "data handle belongs to another context");
  SV_REQUIRE(data->dtype != SV_F64, "batched samples take FP32 or BF16 values");
  const sv_counts* C = data->counts;
  SV_REQUIRE(nseg >= 1, "no samples");
  SV_REQUIRE(cell_offsets[0] == 0 && cell_offsets[nseg] == C->n_cells,
             "cell offsets must run from 0 to the number of cells");
  for (int64_t s = 0; s < nseg; ++s)
    SV_REQUIRE(cell_offsets[s + 1] - cell_offsets[s] >= 2, "sample %lld has fewer than two cells",
               (long long)(s + 1));
  std::vector<int32_t> fg = feature_genes(C, features, nfeatures);
  const int64_t nf = (int64_t)fg.size();
  auto* B = new sv_batch();
  try {
    B->ctx = ctx;
    B->data = data;
    B->nseg = nseg;
    B->n_cells = C->n_cells;
    B->nf = nf;
    B->scale_max = scale_max;
    B->hoff.assign(cell_offsets, cell_offsets + nseg + 1);
    B->off.alloc(nseg + 1);
    sv_h2d(ctx, B->off.get(), cell_offsets, (nseg + 1) * 8);
    B->base = make_centered(ctx, data, fg, scale_max, nullptr, false);
    sv_centered* S = B->base;
    // per-(sample, feature) moments
    size_t sf = (size_t)nseg * nf;
    B->mean.alloc(sf);
    B->std_.alloc(sf);
    B->mu.alloc(sf);
    B->inv_d.alloc(sf);
    B->clip_d.alloc(sf);
    B->inv_f.alloc(sf);
    B->clip_f.alloc(sf);
    B->mu_h.alloc(sf);
    B->mu_l.alloc(sf);
#define LAUNCH_BMOM(VT)                                                                           \
  launch_moments<VT>(ctx, "scale_moments", (const VT*)data->csc_val.get(),                          \
                     (const int64_t*)S->feat_start.get(), (const int64_t*)S->feat_end.get(), nf,     \
                     C->n_cells, scale_max, B->mean.get(), B->std_.get(), B->mu.get(),               \
                     B->inv_f.get(), B->clip_f.get(), B->inv_d.get(), B->clip_d.get(), C->nnz,       \
                     (const int32_t*)C->csc_rowidx.get(), (const int64_t*)B->off.get(), (int)nseg)
    if (data->dtype == SV_F32) LAUNCH_BMOM(float);
    else LAUNCH_BMOM(__nv_bfloat16);
#undef LAUNCH_BMOM
    sv_launch(ctx, "scale_mu_split", k_split_df, dim3(sv_grid_for(ctx, (int64_t)sf, 256)), dim3(256), 0,
              (const double*)B->mu.get(), (int64_t)sf, B->mu_h.get(), B->mu_l.get());
    // X^T u: row blocks of at most RB_ROWS cells, aligned to the samples
    {
      std::vector<int64_t> row0;
      std::vector<int> seg;
      B->h_rb_first.assign(nseg + 1, 0);
      for (int64_t s2 = 0; s2 < nseg; ++s2) {
        B->h_rb_first[s2] = (int64_t)row0.size();
        for (int64_t r = B->hoff[s2]; r < B->hoff[s2 + 1]; r += RB_ROWS) {
          row0.push_back(r);
          seg.push_back((int)s2);
        }
      }
      B->h_rb_first[nseg] = (int64_t)row0.size();
      B->n_rb = (int64_t)row0.size();
      row0.push_back(C->n_cells);
      B->rb_row0.alloc(row0.size());
      B->rb_seg.alloc(seg.size());
      B->rb_first.alloc(nseg + 1);
      sv_h2d(ctx, B->rb_row0.get(), row0.data(), row0.size() * 8);
      sv_h2d(ctx, B->rb_seg.get(), seg.data(), seg.size() * 4);
      sv_h2d(ctx, B->rb_first.get(), B->h_rb_first.data(), (nseg + 1) * 8);
      rb_build(ctx, C, data, S->feat_start.get(), S->feat_end.get(), nf, S->nnz_h, B->n_rb,
               B->rb_row0.get(), B->rb_ptr, B->rb_idx, B->rb_val, B->rb_partial);
      B->upart.alloc(B->n_rb);
      SV_CUDA(cudaFuncSetAttribute(k_spmv_rb<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)(RB_ROWS * sizeof(float))));
      SV_CUDA(cudaFuncSetAttribute(k_spmv_rb<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)(RB_ROWS * sizeof(float))));
    }
    // X v schedule: cells of one sample per block, the block size tuned once per shape
    batch_xschedule(ctx, B, batch_tune_xcells(ctx, B));
    sv_sync(ctx);
  } catch (...) {
    if (B->base) sv_centered_free(B->base);
    delete B;
    throw;
  }
  *out = B;
  SV_CATCH
}

SV_API int sv_batch_info(const sv_batch* b, int64_t* nseg, int64_t* n_cells, int64_t* nf) {
  SV_TRY
  SV_REQUIRE(b, "null handle");
  if (nseg) *nseg = b->nseg;
  if (n_cells) *n_cells = b->n_cells;
  if (nf) *nf = b->nf;
  SV_CATCH
}

// the X v block size (cells per block) the autotuner chose for this batch's shape
SV_API int sv_batch_tuning(const sv_batch* b, int64_t* cells_per_block) {
  SV_TRY
  SV_REQUIRE(b, "null handle");
  if (cells_per_block) *cells_per_block = b->xcells;
  SV_CATCH
}

// per-(sample, feature) statistics, sample-major (nseg x nf): mu = mean/std,
// mean, std
SV_API int sv_batch_stats(sv_context* ctx, const sv_batch* b, double* mu, double* mean, double* sd) {
  SV_TRY
  sv_ctx_check(ctx);
  SV_REQUIRE(b && b->ctx == ctx, "bad batch handle");
  size_t bytes = (size_t)b->nseg * b->nf * 8;
  if (mu) sv_d2h(ctx, mu, b->mu.get(), bytes);
  if (mean) sv_d2h(ctx, mean, b->mean.get(), bytes);
  if (sd) sv_d2h(ctx, sd, b->std_.get(), bytes);
  SV_CATCH
}

SV_API int sv_batch_free(sv_batch* b) {
  if (b) {
    sv_centered_free(b->base);
    delete b;
  }
  return SV_OK;
}

// W step of the batched Lanczos: for every active sample, y = X_s v_s - csub[s] z
// (double-float in and out, stacked)
void sv_batch_apply_N_df(sv_context* ctx, const sv_batch* b, const float* xh, const float* xl,
                         float* yh, float* yl, const double* csub, const float* zh, const float* zl,
                         const int* active) {
  const sv_centered* S = b->base;
  size_t smem = ((size_t)b->nf * 8 + 15) & ~(size_t)15;
#define LAUNCH_BCSR(VT, IT, COL)                                                                  \
  sv_launch(ctx, "spmv_csr_h", k_spmv_csr_df<VT, IT>, dim3(b->nxblk), dim3(256), smem,            \
            (const int64_t*)S->h_rowptr.get(), (const IT*)COL, (const VT*)S->h_val.get(),          \
            (const int64_t*)nullptr, b->nf, xh, xl, (const float*)b->inv_f.get(), (const float*)b->clip_f.get(), \
            (const float*)b->mu_h.get(), (const float*)b->mu_l.get(), yh, yl, csub, zh, zl,         \
            (const BlkRange*)b->xblk.get(), active)
  bool small = b->nf <= 65536;
  if (b->data->dtype == SV_F32) {
    if (small) LAUNCH_BCSR(float, uint16_t, S->h_col16.get());
    else LAUNCH_BCSR(float, int32_t, S->h_col32.get());
  } else {
    if (small) LAUNCH_BCSR(__nv_bfloat16, uint16_t, S->h_col16.get());
    else LAUNCH_BCSR(__nv_bfloat16, int32_t, S->h_col32.get());
  }
#undef LAUNCH_BCSR
}

// V step of the batched Lanczos: for every active sample, y_s = X_s^T u_s -
// csub[s] z_s (FP64, stacked by sample: index s * nf + f)
void sv_batch_apply_T(sv_context* ctx, const sv_batch* b, const double* u, double* y,
                      const double* csub, const double* z, const int* active) {
  sv_batch* bm = const_cast<sv_batch*>(b);
  sv_centered* S = b->base;
  sv_launch(ctx, "spmv_csc_uprep", k_bu_prep, dim3((unsigned)b->n_rb), dim3(256), 0, u,
            (const int64_t*)b->rb_row0.get(), S->u_f32.get(), bm->upart.get());
  int resident = ctx->num_sms * 3;
  int fg = (int)std::max<int64_t>(1, std::min<int64_t>(b->nf, (3 * resident + b->n_rb - 1) / b->n_rb));
  dim3 grid((unsigned)b->n_rb, (unsigned)fg);
  size_t smem = RB_ROWS * sizeof(float);
  if (b->data->dtype == SV_F32)
    sv_launch(ctx, "spmv_rb", k_spmv_rb<float>, grid, dim3(RB_THREADS), smem,
              (const int64_t*)b->rb_ptr.get(), (const unsigned long long*)b->rb_idx.get(), (const float*)b->rb_val.get(),
              b->nf, b->n_cells, (const float*)b->inv_f.get(), (const float*)b->clip_f.get(),
              (const float*)S->u_f32.get(), bm->rb_partial.get(), (const int64_t*)b->rb_row0.get(),
              (const int*)b->rb_seg.get(), active);
  else
    sv_launch(ctx, "spmv_rb", k_spmv_rb<__nv_bfloat16>, grid, dim3(RB_THREADS), smem,
              (const int64_t*)b->rb_ptr.get(), (const unsigned long long*)b->rb_idx.get(),
              (const __nv_bfloat16*)b->rb_val.get(), b->nf, b->n_cells, (const float*)b->inv_f.get(),
              (const float*)b->clip_f.get(), (const float*)S->u_f32.get(), bm->rb_partial.get(),
              (const int64_t*)b->rb_row0.get(), (const int*)b->rb_seg.get(), active);
  dim3 fgrid((unsigned)sv_grid_for(ctx, b->nf, 256, 1), (unsigned)b->nseg);
  sv_launch(ctx, "spmv_rb_finish", k_rb_finish_seg, fgrid, dim3(256), 0, (const float*)bm->rb_partial.get(),
            (const int64_t*)b->rb_first.get(), b->nf, (const double*)b->mu.get(),
            (const double*)bm->upart.get(), y, csub, z, active);
}

sv_counts* sv_counts_upload_positions(sv_context* ctx, int64_t n_rows, int64_t n_cols, int64_t nnz,
                                      const int64_t* colptr, const int64_t* rowval);

namespace {
template <typename T>
__global__ void k_gather_vals(const double* __restrict__ src, const int32_t* __restrict__ pos,
                              int64_t nnz, T* __restrict__ dst_csr, T* __restrict__ dst_csc) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nnz;
       e += (int64_t)gridDim.x * blockDim.x) {
    dst_csr[e] = (T)src[pos[e]];
    dst_csc[e] = (T)src[e];
  }
}
}  // namespace

SV_API int sv_centered_create(sv_context* ctx, int64_t n_rows, int64_t n_cols, int64_t nnz,
                              const int64_t* colptr, const int64_t* rowval, const double* nzval,
                              const double* mu, int dtype, sv_centered** out) {
  SV_TRY
  sv_ctx_check(ctx);
  SV_REQUIRE(out && colptr && mu && (nnz == 0 || (rowval && nzval)), "null argument");
  SV_REQUIRE(dtype == SV_F64 || dtype == SV_F32, "dtype must be F64 or F32");
  SV_REQUIRE(nnz < (1ll << 31), "nnz must fit Int32 positions");
  sv_counts* C = sv_counts_upload_positions(ctx, n_rows, n_cols, nnz, colptr, rowval);
  sv_data* D = nullptr;
  try {
    D = new sv_data();
    D->ctx = ctx;
    D->counts = C;
    D->dtype = dtype;
    size_t es = sv_elem_size(dtype);
    D->csc_val.alloc(std::max<int64_t>(1, nnz) * es);
    D->csr_val.alloc(std::max<int64_t>(1, nnz) * es);
    DevBuf<double> src(std::max<int64_t>(1, nnz));
    sv_h2d(ctx, src.get(), nzval, nnz * 8);
    if (dtype == SV_F64)
      sv_launch(ctx, "centered_gather", k_gather_vals<double>, dim3(sv_grid_for(ctx, nnz, 256, 8)),
                dim3(256), 0, (const double*)src.get(), (const int32_t*)C->csr_count.get(), nnz,
                (double*)D->csr_val.get(), (double*)D->csc_val.get());
    else
      sv_launch(ctx, "centered_gather", k_gather_vals<float>, dim3(sv_grid_for(ctx, nnz, 256, 8)),
                dim3(256), 0, (const double*)src.get(), (const int32_t*)C->csr_count.get(), nnz,
                (float*)D->csr_val.get(), (float*)D->csc_val.get());
    std::vector<int32_t> fg(n_cols);
    for (int64_t f = 0; f < n_cols; ++f) fg[f] = (int32_t)f;
    sv_centered* S = make_centered(ctx, D, fg, INFINITY, mu);
    S->own_counts = C;
    S->own_data = D;
    *out = S;
  } catch (...) {
    delete D;
    delete C;
    throw;
  }
  SV_CATCH
}

// Per-gene mean and standard deviation (n - 1) of the raw counts, implicit
// zeros included (mean_std on the count matrix, src/scaling.jl:18-44): device
// arrays of n_genes.
void sv_count_moments(sv_context* ctx, const sv_counts* C, double* mean, double* sd) {
  int64_t ng = C->n_genes;
  DevBuf<double> mu(ng), invd(ng), clipd(ng);
  DevBuf<float> invf(ng), clipf(ng);
  launch_moments<int32_t>(ctx, "gene_moments", (const int32_t*)C->csc_count.get(),
                          (const int64_t*)C->csc_colptr.get(), (const int64_t*)C->csc_colptr.get() + 1,
                          ng, C->n_cells, (double)INFINITY, mean, sd, mu.get(), invf.get(),
                          clipf.get(), invd.get(), clipd.get(), C->nnz);
}

SV_API int sv_gene_moments(sv_context* ctx, const sv_data* data, double* mean, double* var) {
  SV_TRY
  sv_ctx_check(ctx);
  SV_REQUIRE(data && data->ctx == ctx && (mean || var), "bad argument");
  const sv_counts* C = data->counts;
  SV_REQUIRE(C->n_cells >= 2, "need at least two cells for a variance");
  int64_t ng = C->n_genes;
  DevBuf<int64_t> fs(ng), fe(ng);
  DevBuf<double> m(ng), sd(ng), mu(ng), invd(ng), clipd(ng);
  DevBuf<float> invf(ng), clipf(ng);
  SV_CUDA(cudaMemcpyAsync(fs.get(), C->csc_colptr.get(), ng * 8, cudaMemcpyDeviceToDevice, ctx->stream));
  SV_CUDA(cudaMemcpyAsync(fe.get(), C->csc_colptr.get() + 1, ng * 8, cudaMemcpyDeviceToDevice,
                          ctx->stream));
#define LAUNCH_MOM(VT)                                                                           \
  launch_moments<VT>(ctx, "gene_moments", (const VT*)data->csc_val.get(), (const int64_t*)fs.get(), \
                     (const int64_t*)fe.get(), ng, C->n_cells, (double)INFINITY, m.get(), sd.get(), \
                     mu.get(), invf.get(), clipf.get(), invd.get(), clipd.get(), C->nnz)
  switch (data->dtype) {
    case SV_F64: LAUNCH_MOM(double); break;
    case SV_F32: LAUNCH_MOM(float); break;
    default: LAUNCH_MOM(__nv_bfloat16); break;
  }
#undef LAUNCH_MOM
  if (mean) sv_d2h(ctx, mean, m.get(), ng * 8);
  if (var) {
    std::vector<double> s(ng);
    sv_d2h(ctx, s.data(), sd.get(), ng * 8);
    for (int64_t g = 0; g < ng; ++g) var[g] = s[g] * s[g];
  }
  SV_CATCH
}

SV_API int sv_centered_info(const sv_centered* s, int64_t* n_cells, int64_t* nf, int64_t* nnz) {
  SV_TRY
  SV_REQUIRE(s, "null handle");
  if (n_cells) *n_cells = s->n_cells;
  if (nf) *nf = s->nf;
  if (nnz) *nnz = s->nnz_h;
  SV_CATCH
}

SV_API int sv_centered_stats(sv_context* ctx, const sv_centered* s, double* mu, double* mean,
                             double* sd) {
  SV_TRY
  sv_ctx_check(ctx);
  SV_REQUIRE(s && s->ctx == ctx, "bad handle");
  if (mu) sv_d2h(ctx, mu, s->mu.get(), s->nf * 8);
  if (mean) sv_d2h(ctx, mean, s->mean.get(), s->nf * 8);
  if (sd) sv_d2h(ctx, sd, s->std_.get(), s->nf * 8);
  SV_CATCH
}

SV_API int sv_centered_mul(sv_context* ctx, const sv_centered* s, char trans, int64_t ncols,
                           double alpha, const double* x, int64_t ldx, double beta, double* y,
                           int64_t ldy) {
  SV_TRY
  sv_ctx_check(ctx);
  SV_REQUIRE(s && s->ctx == ctx, "bad handle");
  SV_REQUIRE(trans == 'N' || trans == 'T', "trans must be 'N' or 'T'");
  SV_REQUIRE(ncols >= 0 && x && y, "bad arguments");
  int64_t nx = trans == 'N' ? s->nf : s->n_cells;
  int64_t ny = trans == 'N' ? s->n_cells : s->nf;
  SV_REQUIRE(ldx >= nx && ldy >= ny, "leading dimension too small");
  DevBuf<double> dx(nx), dy(ny);
  for (int64_t j = 0; j < ncols; ++j) {
    sv_h2d(ctx, dx.get(), x + j * ldx, nx * 8);
    if (beta != 0.0) sv_h2d(ctx, dy.get(), y + j * ldy, ny * 8);
    sv_centered_apply(ctx, s, trans, dx.get(), dy.get(), alpha, beta, nullptr, nullptr);
    sv_d2h(ctx, y + j * ldy, dy.get(), ny * 8);
  }
  SV_CATCH
}

SV_API int sv_centered_free(sv_centered* s) {
  if (s) {
    sv_data* d = s->own_data;
    sv_counts* c = s->own_counts;
    delete s;
    delete d;
    delete c;
  }
  return SV_OK;
}
