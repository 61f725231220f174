// Fuzzy-kNN graph construction on the device: the UMAP fuzzy simplicial set
// the crate consumes, built as its fixture generator builds it
// (tests/generate_fixtures.py:70-182 of the reference):
//   1. exact kNN, Euclidean, self excluded, ascending (ties by index);
//   2. smooth-kNN sigma / rho (umap-learn 0.5.11 smooth_knn_dist, as the
//      generator ran it: bisection for sum_{j>0} exp(-max(d - rho, 0) / sigma)
//      = log2(k) from sigma = 1, taking the midpoint against an infinite upper
//      bound, so a row whose root lies above 1 keeps sigma = +inf; floor
//      1e-3 x the row's (or all rows') mean distance);
//   3. membership strengths exp(-(d - rho) / sigma), 1 at or below rho;
//   4. the fuzzy union A + A^T - A∘A^T;
//   5. pruning below max / n_epochs (500 for n <= 10000, else 200).
// Distances in f64, reported as f32 like the generator's; sigma / rho f32
// with the bisection in f64; memberships f32.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>

#include "si_internal.h"

namespace si {
namespace {

constexpr int kKnnMax = 32;
constexpr int kKnnThreads = 128;
constexpr int kKnnQ = 128;      // queries per CTA
constexpr int kKnnC = 64;       // candidates per tile
constexpr int kKnnF = 16;       // features staged at a time
constexpr int kKnnBuf = 32;     // accepted candidates buffered per query: half a tile
constexpr int kSortWarp = 256;  // longest row sorted by one warp

int grid_items(const Exec& ex, int64_t items, int threads = 256) {
  const int64_t need = (items + threads - 1) / threads;
  return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(need, int64_t(ex.sms) * 16)));
}

// Stage 1, exact kNN.  A CTA takes 128 queries against one split of the
// candidates, 64 at a time: a thread forms the squared distances of 8 queries
// to 8 candidates in registers (16 shared-memory reads for 128 FP64
// operations a feature; every distance is the sum of (x_f - y_f)^2 in feature
// order by one chain of fma).  The registers leave eight warps an SM, so the FP64
// pipe, at 28 % at n = 4000 and 41 % at n = 20011, waits for fixed latencies, the
// panels' loads and the insertions.  Distances below the query's current k-th are
// buffered and inserted by the query's own thread; a few per query and tile after
// the first tiles.  Kept: the k smallest by
// (distance, index).  One query a thread, with both rows read again for every
// distance, took 55.3 ms at n = 20011, d = 50, k = 15; this takes 5.4 ms
// (FP64 alone: 2.2 ms).
struct KnnSmem {
  double q[kKnnF][kKnnQ + 2];
  double c[kKnnF][kKnnC + 2];
  double buf_s[kKnnQ][kKnnBuf];
  uint8_t buf_c[kKnnQ][kKnnBuf];
  double thr[kKnnQ];
  int cnt[kKnnQ];
  // then, dynamic: list_s [k][kKnnQ], list_i [k][kKnnQ]
};

__device__ __forceinline__ bool knn_before(double s, int32_t i, double t, int32_t j) {
  return s < t || (s == t && i < j);
}

__global__ void __launch_bounds__(kKnnThreads, 2) k_knn_exact(const double* __restrict__ x, int64_t n, int d, int k,
                                                              int tiles_per_split, double* __restrict__ ps,
                                                              int32_t* __restrict__ pi) {
  extern __shared__ __align__(16) unsigned char knn_raw[];
  KnnSmem& sm = *reinterpret_cast<KnnSmem*>(knn_raw);
  double* list_s = reinterpret_cast<double*>(knn_raw + sizeof(KnnSmem));
  int32_t* list_i = reinterpret_cast<int32_t*>(list_s + static_cast<size_t>(k) * kKnnQ);
  const int tid = threadIdx.x;
  const int tx = tid & 7, ty = tid >> 3;  // candidates 2 tx + 16 b + {0, 1}, queries 2 ty + 32 a + {0, 1}
  const int64_t q0 = static_cast<int64_t>(blockIdx.x) * kKnnQ;
  const int64_t t0 = static_cast<int64_t>(blockIdx.y) * tiles_per_split;
  const int64_t ntile = (n + kKnnC - 1) / kKnnC;
  const int64_t t1 = min(t0 + tiles_per_split, ntile);
  for (int t = 0; t < k; ++t) {
    list_s[t * kKnnQ + tid] = INFINITY;
    list_i[t * kKnnQ + tid] = -1;
  }
  sm.thr[tid] = INFINITY;
  sm.cnt[tid] = 0;
  for (int64_t tile = t0; tile < t1; ++tile) {
    const int64_t c0 = tile * kKnnC;
    double acc[8][8];
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
      for (int b = 0; b < 8; ++b) acc[a][b] = 0.0;
    for (int f0 = 0; f0 < d; f0 += kKnnF) {
      const int nf = min(kKnnF, d - f0);
      __syncthreads();
      const int f = tid & (kKnnF - 1);
      const bool fin = f < nf;
#pragma unroll 8
      for (int r = tid / kKnnF; r < kKnnQ; r += kKnnThreads / kKnnF)
        sm.q[f][r] = (fin && q0 + r < n) ? __ldg(x + (q0 + r) * d + f0 + f) : 0.0;
#pragma unroll 8
      for (int r = tid / kKnnF; r < kKnnC; r += kKnnThreads / kKnnF)
        sm.c[f][r] = (fin && c0 + r < n) ? __ldg(x + (c0 + r) * d + f0 + f) : 0.0;
      __syncthreads();
#pragma unroll 1
      for (int g = 0; g < nf; ++g) {
        double qv[8], cv[8];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const double2 t = *reinterpret_cast<const double2*>(&sm.q[g][2 * ty + 32 * a]);
          qv[2 * a] = t.x;
          qv[2 * a + 1] = t.y;
        }
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const double2 t = *reinterpret_cast<const double2*>(&sm.c[g][2 * tx + 16 * b]);
          cv[2 * b] = t.x;
          cv[2 * b + 1] = t.y;
        }
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
          for (int b = 0; b < 8; ++b) {
            const double df = qv[a] - cv[b];
            acc[a][b] = fma(df, df, acc[a][b]);
          }
      }
    }
    // candidates 32 h .. 32 h + 31 of the tile
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      __syncthreads();  // the insertions before this are done: thresholds are current
#pragma unroll
      for (int a = 0; a < 8; ++a) {
        const int q = 2 * ty + 32 * (a >> 1) + (a & 1);
        const double thr = sm.thr[q];
#pragma unroll
        for (int b = 4 * h; b < 4 * h + 4; ++b) {
          const int c = 2 * tx + 16 * (b >> 1) + (b & 1);
          if (acc[a][b] < thr && c0 + c < n && c0 + c != q0 + q) {
            const int p = atomicAdd(&sm.cnt[q], 1);
            sm.buf_s[q][p] = acc[a][b];
            sm.buf_c[q][p] = static_cast<uint8_t>(c);
          }
        }
      }
      __syncthreads();
      const int m = sm.cnt[tid];
      if (m > 0) {
        for (int e = 0; e < m; ++e) {
          const double s = sm.buf_s[tid][e];
          const int32_t i = static_cast<int32_t>(c0 + sm.buf_c[tid][e]);
          int p = k - 1;
          if (!knn_before(s, i, list_s[p * kKnnQ + tid], list_i[p * kKnnQ + tid]) && list_i[p * kKnnQ + tid] >= 0)
            continue;
          while (p > 0 && (list_i[(p - 1) * kKnnQ + tid] < 0 ||
                           knn_before(s, i, list_s[(p - 1) * kKnnQ + tid], list_i[(p - 1) * kKnnQ + tid]))) {
            list_s[p * kKnnQ + tid] = list_s[(p - 1) * kKnnQ + tid];
            list_i[p * kKnnQ + tid] = list_i[(p - 1) * kKnnQ + tid];
            --p;
          }
          list_s[p * kKnnQ + tid] = s;
          list_i[p * kKnnQ + tid] = i;
        }
        sm.thr[tid] = list_s[(k - 1) * kKnnQ + tid];
        sm.cnt[tid] = 0;
      }
    }
  }
  if (q0 + tid >= n) return;
  const int64_t o = (static_cast<int64_t>(blockIdx.y) * n + q0 + tid) * k;
  for (int t = 0; t < k; ++t) {
    ps[o + t] = list_s[t * kKnnQ + tid];
    pi[o + t] = list_i[t * kKnnQ + tid];
  }
}

// The splits' lists of a query into one; *zero_row is set when some row has
// only zero distances (its floor below needs the mean over all rows).
__global__ void k_knn_merge(const double* __restrict__ ps, const int32_t* __restrict__ pi, int64_t n, int k, int splits,
                            int32_t* __restrict__ idx, float* __restrict__ dist, int* __restrict__ zero_row) {
  const int64_t q = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (q >= n) return;
  double bd[kKnnMax];
  int32_t bi[kKnnMax];
#pragma unroll
  for (int t = 0; t < kKnnMax; ++t) {
    bd[t] = t < k ? ps[q * k + t] : INFINITY;
    bi[t] = t < k ? pi[q * k + t] : -1;
  }
  for (int sp = 1; sp < splits; ++sp) {
    const int64_t o = (static_cast<int64_t>(sp) * n + q) * k;
    for (int e = 0; e < k; ++e) {
      double cd = ps[o + e];
      int32_t ci = pi[o + e];
      if (ci < 0) break;
      // later splits hold larger indices: an equal distance goes after the kept ones
      bool in = false;
#pragma unroll
      for (int t = 0; t < kKnnMax; ++t) {
        if (t < k && (in || bi[t] < 0 || cd < bd[t])) {
          in = true;
          const double td = bd[t];
          const int32_t ti = bi[t];
          bd[t] = cd;
          bi[t] = ci;
          cd = td;
          ci = ti;
        }
      }
      if (!in) break;  // the split's list ascends
    }
  }
  bool zero = true;
#pragma unroll
  for (int t = 0; t < kKnnMax; ++t)
    if (t < k) {
      const float v = static_cast<float>(sqrt(bd[t]));
      idx[q * k + t] = bi[t];
      dist[q * k + t] = v;
      zero = zero && !(v > 0.0f);
    }
  if (zero) *zero_row = 1;
}

// mean of all distances (f64 sum in row order, one block); only rows without
// a positive distance read it
__global__ void k_dist_mean(const float* __restrict__ dist, int64_t total, const int* __restrict__ zero_row,
                            double* __restrict__ out) {
  __shared__ double red[256];
  if (*zero_row == 0) return;
  double s = 0.0;
  for (int64_t e = threadIdx.x; e < total; e += blockDim.x) s += static_cast<double>(dist[e]);
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = red[0] / static_cast<double>(total > 0 ? total : 1);
}

// Stage 2: L lanes a row (16, 32 when k > 16), a lane a distance: the
// exponentials of a bisection step, which are its cost, run side by side; the
// lanes then all add them in neighbour order, so the sum is the sequential one.
template <int L>
__global__ void k_smooth_knn(const float* __restrict__ dist, int64_t n, int k, const double* __restrict__ mean_all,
                             float* __restrict__ sigma, float* __restrict__ rho) {
  const double target = log2(static_cast<double>(k));
  const int lane = threadIdx.x & (L - 1);
  const unsigned mask = L == 32 ? 0xffffffffu : (0xffffu << (threadIdx.x & 16));
  const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x / L;
  for (int64_t i = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / L; i < n; i += step) {
    const float own = lane < k ? dist[i * k + lane] : 0.0f;
    float r = 0.0f;
    double rsum = 0.0;
    for (int j = 0; j < k; ++j) {
      const float v = __shfl_sync(mask, own, j, L);
      rsum += static_cast<double>(v);
      if (r == 0.0f && v > 0.0f) r = v;
    }
    const float dd = own - r;
    double lo = 0.0, hi = INFINITY, mid = 1.0;
    for (int it = 0; it < 64; ++it) {
      const double term = dd > 0.0f ? exp(-(static_cast<double>(dd) / mid)) : 1.0;
      double psum = 0.0;
      for (int j = 1; j < k; ++j) psum += __shfl_sync(mask, term, j, L);
      if (fabs(psum - target) < 1e-5) break;
      if (psum > target) {
        hi = mid;
        mid = (lo + hi) / 2.0;
      } else {
        lo = mid;
        mid = (lo + hi) / 2.0;  // an infinite upper bound keeps mid infinite (see above)
      }
    }
    if (lane == 0) {
      const double floor = 1e-3 * (r > 0.0f ? rsum / k : mean_all[0]);
      sigma[i] = static_cast<float>(mid < floor ? floor : mid);
      rho[i] = r;
    }
  }
}

// Stage 3: membership of neighbour t of row i (0 for the row itself)
__device__ __forceinline__ float membership_of(const int32_t* idx, const float* dist, const float* sigma,
                                               const float* rho, int k, int64_t i, int t) {
  const int32_t j = idx[i * k + t];
  if (j == i || j < 0) return 0.0f;
  const float diff = dist[i * k + t] - rho[i];
  const float sg = sigma[i];
  if (diff <= 0.0f || sg == 0.0f) return 1.0f;
  return expf(-(diff / sg));
}

// membership of the reverse edge j -> i (0 when i is not among j's neighbours)
__device__ __forceinline__ float reverse_membership(const int32_t* idx, const float* dist, const float* sigma,
                                                    const float* rho, int k, int64_t i, int64_t j) {
  for (int t = 0; t < k; ++t)
    if (idx[j * k + t] == i) return membership_of(idx, dist, sigma, rho, k, j, t);
  return 0.0f;
}

// Stage 4, counting: every directed edge i -> j with a > 0 gives (i, j); it
// also gives (j, i) when j -> i is absent (its union value is then a).  Each
// (row, column) pair of the union arises exactly once.
__global__ void k_union_count(const int32_t* __restrict__ idx, const float* __restrict__ dist,
                              const float* __restrict__ sigma, const float* __restrict__ rho, int64_t n, int k,
                              unsigned long long* __restrict__ counts) {
  const int64_t total = n * k;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < total; e += stride) {
    const int64_t i = e / k;
    const int t = static_cast<int>(e % k);
    const float a = membership_of(idx, dist, sigma, rho, k, i, t);
    if (a == 0.0f) continue;
    const int64_t j = idx[e];
    atomicAdd(counts + i, 1ull);
    if (reverse_membership(idx, dist, sigma, rho, k, i, j) == 0.0f) atomicAdd(counts + j, 1ull);
  }
}

// Stage 4, filling: union value (a + b) - a b in f32 as scipy forms it
__global__ void k_union_fill(const int32_t* __restrict__ idx, const float* __restrict__ dist,
                             const float* __restrict__ sigma, const float* __restrict__ rho, int64_t n, int k,
                             const uint64_t* __restrict__ ptr, unsigned long long* __restrict__ cursor,
                             uint32_t* __restrict__ cols, float* __restrict__ vals) {
  const int64_t total = n * k;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < total; e += stride) {
    const int64_t i = e / k;
    const int t = static_cast<int>(e % k);
    const float a = membership_of(idx, dist, sigma, rho, k, i, t);
    if (a == 0.0f) continue;
    const int64_t j = idx[e];
    const float b = reverse_membership(idx, dist, sigma, rho, k, i, j);
    const float u = (a + b) - a * b;
    const uint64_t p = ptr[i] + atomicAdd(cursor + i, 1ull);
    cols[p] = static_cast<uint32_t>(j);
    vals[p] = u;
    if (b == 0.0f) {
      const uint64_t q = ptr[j] + atomicAdd(cursor + j, 1ull);
      cols[q] = static_cast<uint32_t>(i);
      vals[q] = u;
    }
  }
}

// Each row's entries in column order (the fill order above is not fixed),
// into a second pair of arrays: an entry's place is the number of smaller
// columns of its row (columns are unique).  A warp a row up to kSortWarp
// entries, columns in shared memory; longer rows (hubs) go to a list that
// k_sort_long takes a CTA a row.  An insertion sort by one thread a row took
// 1.2 ms at n = 20011 for the hubs' sake.
__global__ void __launch_bounds__(256) k_sort_rows(int64_t n, const uint64_t* __restrict__ ptr,
                                                   const uint32_t* __restrict__ cols, const float* __restrict__ vals,
                                                   uint32_t* __restrict__ ocols, float* __restrict__ ovals,
                                                   uint32_t* __restrict__ long_rows, unsigned* __restrict__ n_long) {
  __shared__ uint32_t sc[8][kSortWarp];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t warps = static_cast<int64_t>(gridDim.x) * 8;
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * 8 + warp; r < n; r += warps) {
    const uint64_t s = ptr[r];
    const int64_t len = static_cast<int64_t>(ptr[r + 1] - s);
    if (len > kSortWarp) {
      if (lane == 0) long_rows[atomicAdd(n_long, 1u)] = static_cast<uint32_t>(r);
      continue;
    }
    __syncwarp();
    for (int e = lane; e < len; e += 32) sc[warp][e] = cols[s + e];
    __syncwarp();
    for (int e = lane; e < len; e += 32) {
      const uint32_t c = sc[warp][e];
      int rank = 0;
      for (int o = 0; o < len; ++o) rank += sc[warp][o] < c ? 1 : 0;
      ocols[s + rank] = c;
      ovals[s + rank] = vals[s + e];
    }
  }
}

__global__ void __launch_bounds__(256) k_sort_long(const uint32_t* __restrict__ long_rows,
                                                   const unsigned* __restrict__ n_long,
                                                   const uint64_t* __restrict__ ptr, const uint32_t* __restrict__ cols,
                                                   const float* __restrict__ vals, uint32_t* __restrict__ ocols,
                                                   float* __restrict__ ovals) {
  __shared__ uint32_t sc[2048];
  const unsigned m = *n_long;
  for (unsigned t = blockIdx.x; t < m; t += gridDim.x) {
    const int64_t r = long_rows[t];
    const uint64_t s = ptr[r];
    const int64_t len = static_cast<int64_t>(ptr[r + 1] - s);
    for (int64_t e0 = 0; e0 < len; e0 += 256) {  // all threads stay in step for the staged tiles
      const int64_t e = e0 + threadIdx.x;
      const uint32_t c = e < len ? cols[s + e] : 0u;
      int64_t rank = 0;
      for (int64_t o0 = 0; o0 < len; o0 += 2048) {
        const int on = static_cast<int>(min(static_cast<int64_t>(2048), len - o0));
        __syncthreads();
        for (int o = threadIdx.x; o < on; o += 256) sc[o] = cols[s + o0 + o];
        __syncthreads();
        int part = 0;
        for (int o = 0; o < on; ++o) part += sc[o] < c ? 1 : 0;
        rank += part;
      }
      if (e < len) {
        ocols[s + rank] = c;
        ovals[s + rank] = vals[s + e];
      }
    }
    __syncthreads();
  }
}

// max of non-negative values (zero on entry in out): their bit patterns order
// as integers
__global__ void k_max_f32(const float* __restrict__ v, int64_t count, float* __restrict__ out) {
  float m = 0.0f;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < count; e += stride)
    m = fmaxf(m, v[e]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0 && m > 0.0f) atomicMax(reinterpret_cast<int*>(out), __float_as_int(m));
}

// Stage 5a: entries kept per row, then the compacted CSR
__global__ void k_prune_count(int64_t n, const uint64_t* __restrict__ ptr, const float* __restrict__ vals,
                              const float* __restrict__ vmax, float n_epochs, unsigned long long* __restrict__ keep) {
  const float thr = vmax[0] / n_epochs;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r <= n; r += stride) {
    if (r == n) {
      keep[n] = 0;
      continue;
    }
    unsigned long long c = 0;
    for (uint64_t p = ptr[r]; p < ptr[r + 1]; ++p) c += (vals[p] < thr) ? 0 : 1;
    keep[r] = c;
  }
}

__global__ void k_prune_fill(int64_t n, const uint64_t* __restrict__ ptr, const uint32_t* __restrict__ cols,
                             const float* __restrict__ vals, const float* __restrict__ vmax, float n_epochs,
                             const uint64_t* __restrict__ optr, uint32_t* __restrict__ ocols,
                             float* __restrict__ ovals) {
  const float thr = vmax[0] / n_epochs;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < n; r += stride) {
    uint64_t o = optr[r];
    for (uint64_t p = ptr[r]; p < ptr[r + 1]; ++p) {
      if (vals[p] < thr) continue;
      ocols[o] = cols[p];
      ovals[o] = vals[p];
      ++o;
    }
  }
}

}  // namespace

void fuzzy_graph_dev(const Exec& ex, const double* x, int64_t n, int d, int k, int32_t* knn_idx, float* knn_dist,
                     float* sigma, float* rho, uint64_t* indptr, uint32_t* indices, float* data, uint64_t capacity,
                     uint64_t* nnz_out) {
  SI_REQUIRE(n >= 2 && d >= 1 && k >= 1 && k < n, SI_INVALID_ARGUMENT, "fuzzy graph: need n >= 2, d >= 1, 1 <= k < n");
  SI_REQUIRE(k <= kKnnMax, SI_INVALID_ARGUMENT, "fuzzy graph: k must be at most 32");
  SI_REQUIRE(d <= 256, SI_INVALID_ARGUMENT, "fuzzy graph: at most 256 features");
  SI_REQUIRE(n < (int64_t(1) << 31), SI_INVALID_ARGUMENT, "fuzzy graph: n must fit in int32");
  // 1. exact kNN: the splits that fill the last wave of 2 CTAs an SM best (a
  // split costs about four tiles more: its first tiles insert nearly everything)
  const int64_t ntile = (n + kKnnC - 1) / kKnnC, nq = (n + kKnnQ - 1) / kKnnQ;
  int64_t splits = 1, best = INT64_MAX;
  for (int64_t sp = 1; sp <= std::min<int64_t>({32, ntile, (int64_t(1) << 24) / std::max<int64_t>(n * k, 1) + 1}); ++sp) {
    const int64_t waves = (nq * sp + 2 * ex.sms - 1) / (2 * ex.sms);
    const int64_t cost = waves * ((ntile + sp - 1) / sp + 4);
    if (cost < best) {
      best = cost;
      splits = sp;
    }
  }
  const int per = static_cast<int>((ntile + splits - 1) / splits);
  splits = (ntile + per - 1) / per;
  const int smem = static_cast<int>(sizeof(KnnSmem)) + k * kKnnQ * 12;
  SI_CUDA(cudaFuncSetAttribute(k_knn_exact, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(sizeof(KnnSmem)) + kKnnMax * kKnnQ * 12));
  DevBuf<double> ps(static_cast<size_t>(splits) * n * k, ex.stream);
  DevBuf<int32_t> pi(static_cast<size_t>(splits) * n * k, ex.stream);
  DevBuf<int> flags(3, ex.stream);  // a row without a positive distance; long rows; the largest weight
  flags.zero();
  const dim3 grid(static_cast<unsigned>(nq), static_cast<unsigned>(splits));
  k_knn_exact<<<grid, kKnnThreads, smem, ex.stream>>>(x, n, d, k, per, ps.get(), pi.get());
  SI_LAUNCH_CHECK();
  k_knn_merge<<<static_cast<unsigned>((n + 127) / 128), 128, 0, ex.stream>>>(ps.get(), pi.get(), n, k,
                                                                             static_cast<int>(splits), knn_idx,
                                                                             knn_dist, flags.get());
  SI_LAUNCH_CHECK();
  // 2. smooth-kNN
  DevBuf<double> mean_all(1, ex.stream);
  k_dist_mean<<<1, 256, 0, ex.stream>>>(knn_dist, n * k, flags.get(), mean_all.get());
  SI_LAUNCH_CHECK();
  if (k <= 16)
    k_smooth_knn<16><<<grid_items(ex, n * 16), 256, 0, ex.stream>>>(knn_dist, n, k, mean_all.get(), sigma, rho);
  else
    k_smooth_knn<32><<<grid_items(ex, n * 32), 256, 0, ex.stream>>>(knn_dist, n, k, mean_all.get(), sigma, rho);
  SI_LAUNCH_CHECK();
  // 3 + 4. memberships and their fuzzy union as CSR
  DevBuf<unsigned long long> cnt(static_cast<size_t>(n + 1), ex.stream);
  cnt.zero();
  k_union_count<<<grid_items(ex, n * k), 256, 0, ex.stream>>>(knn_idx, knn_dist, sigma, rho, n, k, cnt.get());
  SI_LAUNCH_CHECK();
  DevBuf<uint64_t> uptr(static_cast<size_t>(n + 1), ex.stream);
  const uint64_t unnz = exclusive_scan_u64(ex, reinterpret_cast<const uint64_t*>(cnt.get()), uptr.get(), n);
  DevBuf<uint32_t> fcols(std::max<uint64_t>(unnz, 1), ex.stream), ucols(std::max<uint64_t>(unnz, 1), ex.stream);
  DevBuf<float> fvals(std::max<uint64_t>(unnz, 1), ex.stream), uvals(std::max<uint64_t>(unnz, 1), ex.stream);
  DevBuf<uint32_t> long_rows(static_cast<size_t>(n), ex.stream);
  cnt.zero();
  k_union_fill<<<grid_items(ex, n * k), 256, 0, ex.stream>>>(knn_idx, knn_dist, sigma, rho, n, k, uptr.get(),
                                                               cnt.get(), fcols.get(), fvals.get());
  SI_LAUNCH_CHECK();
  unsigned* n_long = reinterpret_cast<unsigned*>(flags.get() + 1);
  k_sort_rows<<<grid_items(ex, n * 32), 256, 0, ex.stream>>>(n, uptr.get(), fcols.get(), fvals.get(), ucols.get(),
                                                             uvals.get(), long_rows.get(), n_long);
  SI_LAUNCH_CHECK();
  k_sort_long<<<ex.sms, 256, 0, ex.stream>>>(long_rows.get(), n_long, uptr.get(), fcols.get(), fvals.get(),
                                             ucols.get(), uvals.get());
  SI_LAUNCH_CHECK();
  // 5a. pruning
  float* vmax = reinterpret_cast<float*>(flags.get() + 2);
  k_max_f32<<<grid_items(ex, static_cast<int64_t>(unnz)), 256, 0, ex.stream>>>(uvals.get(), static_cast<int64_t>(unnz),
                                                                               vmax);
  SI_LAUNCH_CHECK();
  const float n_epochs = n <= 10000 ? 500.0f : 200.0f;
  k_prune_count<<<grid_items(ex, n + 1), 256, 0, ex.stream>>>(n, uptr.get(), uvals.get(), vmax, n_epochs,
                                                              cnt.get());
  SI_LAUNCH_CHECK();
  const uint64_t pnnz = exclusive_scan_u64(ex, reinterpret_cast<const uint64_t*>(cnt.get()), indptr, n);
  SI_REQUIRE(pnnz <= capacity, SI_INVALID_ARGUMENT, "fuzzy graph: output capacity too small (need 2 n k entries)");
  k_prune_fill<<<grid_items(ex, n), 256, 0, ex.stream>>>(n, uptr.get(), ucols.get(), uvals.get(), vmax, n_epochs,
                                                        indptr, indices, data);
  SI_LAUNCH_CHECK();
  SI_CUDA(cudaStreamSynchronize(ex.stream));
  *nnz_out = pnnz;
}

}  // namespace si
