// Dense symmetric eigensolver on the device for the k smallest eigenpairs
// (dense_evd, src/solvers/dense.rs:9-46; Levels 0 and 5 of the chain).
//
//   1. densify the operator (lower triangle mirrored, like faer's Side::Lower);
//   2. Householder tridiagonalisation T = Q^T A Q (dsytd2-style): one launch
//      with the matrix spread over the shared memory of co-resident CTAs (a
//      cluster up to 512 rows, a cooperative launch up to 2048), and three
//      launches per column above that;
//   3. up to 2048 rows the k smallest pairs of T directly, a CTA each:
//      Sturm-count multisection and a twisted factorisation, then one CTA
//      orthonormalises and tests the vectors;
//   4. where that test fails (pairs that agree to rounding, a T that splits) and
//      above 2048 rows: T split where off-diagonals are negligible, for every
//      block the smallest eigenvalues by multisection (bisection when there are
//      many blocks) to LAPACK dstebz's default tolerance eps |T|, the k smallest
//      overall kept, and their vectors by inverse iteration restricted to the
//      block (LU with partial pivoting of T - lambda I), re-orthogonalised within
//      clusters of close eigenvalues (modified Gram-Schmidt), stopped as LAPACK's
//      dstein once the growth shows a rounding-level residual;
//   5. back-transformation v = Q y with the stored reflectors in compact-WY
//      blocks of eight: a CTA a vector up to 2048 rows, one CTA above while Y and
//      a block fit in shared memory, reflector by reflector beyond.
#include <cooperative_groups.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdlib>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "si_internal.h"

namespace si {
namespace {

constexpr int DT = 1024;
constexpr int TE_MS_ITEMS = 32;   // multisection when at most this many (block, index) items
constexpr int TE_MS_POINTS = 96;  // at most this many Sturm points per item and round

__global__ void k_densify(int64_t n, const uint64_t* __restrict__ indptr, const uint32_t* __restrict__ indices,
                          const double* __restrict__ vals, double diag, double* __restrict__ A) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n; i += stride) {
    for (uint64_t k = indptr[i]; k < indptr[i + 1]; ++k) A[i * n + indices[k]] += vals[k];
    A[i * n + i] += diag;
  }
}

// A[i][j] = A[j][i] for i < j (use the lower triangle).
__global__ void k_mirror_lower(int64_t n, double* A) {
  const int64_t total = n * n;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < total; t += stride) {
    const int64_t i = t / n, j = t % n;
    if (i < j) A[i * n + j] = A[j * n + i];
  }
}

__device__ double block_sum_all(double v, double* red) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  const int nw = blockDim.x >> 5;
  for (int i = 0; i < nw; ++i) t += red[i];
  __syncthreads();
  return t;
}

// ---- multi-launch tridiagonalisation: each Householder step three launches
// so the trailing-matrix passes use the whole GPU.
// Step j:  (1) one CTA forms the reflector of column j (d, e, tau; v in vbuf
// and in row j of A); (2) w = tau A v over the trailing rows, one warp per
// row, per-CTA partial dots w.v, the last CTA subtracts K v with
// K = tau (w.v) / 2 (deterministic order); (3) A -= v w^T + w v^T.
__global__ void __launch_bounds__(256) k_tri_house(double* A, int n, int j, double* d, double* e, double* tau,
                                                   double* vbuf) {
  __shared__ double red[32];
  __shared__ double s_tau, s_scal;
  const int tid = threadIdx.x;
  double part = 0.0;
  for (int i = j + 2 + tid; i < n; i += blockDim.x) {
    const double x = A[static_cast<int64_t>(i) * n + j];
    part += x * x;
  }
  const double sigma = block_sum_all(part, red);
  if (tid == 0) {
    const double alpha = A[static_cast<int64_t>(j + 1) * n + j];
    double t = 0.0, beta = alpha, scal = 0.0;
    if (sigma > 0.0) {
      const double nrm = sqrt(alpha * alpha + sigma);
      beta = alpha >= 0.0 ? -nrm : nrm;
      t = (beta - alpha) / beta;
      scal = 1.0 / (alpha - beta);
    }
    s_tau = t;
    s_scal = scal;
    e[j] = beta;
    tau[j] = t;
    d[j] = A[static_cast<int64_t>(j) * n + j];
  }
  __syncthreads();
  if (s_tau == 0.0) return;
  const double scal = s_scal;
  for (int i = j + 1 + tid; i < n; i += blockDim.x) {
    const double vi = (i == j + 1) ? 1.0 : A[static_cast<int64_t>(i) * n + j] * scal;
    vbuf[i] = vi;
    if (i >= j + 2) A[static_cast<int64_t>(j) * n + i] = vi;  // keep the reflector in row j
  }
}

__global__ void __launch_bounds__(256) k_tri_matvec(const double* __restrict__ A, int n, int j,
                                                    const double* __restrict__ tau, const double* __restrict__ vbuf,
                                                    double* __restrict__ wbuf, double* __restrict__ partial,
                                                    unsigned* __restrict__ counter) {
  __shared__ double red[8];
  __shared__ bool last;
  const double t = tau[j];
  if (t == 0.0) return;  // uniform for the grid
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = j + 1 + blockIdx.x * 8 + warp;
  double wv = 0.0;
  if (r < n) {
    double acc = 0.0;
    const double* row = A + static_cast<int64_t>(r) * n;
    for (int c = j + 1 + lane; c < n; c += 32) acc = fma(row[c], vbuf[c], acc);
    acc = warp_sum(acc);
    if (lane == 0) {
      wbuf[r] = t * acc;
      wv = t * acc * vbuf[r];
    }
  }
  if (lane == 0) red[warp] = wv;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < 8; ++w) s += red[w];
    partial[blockIdx.x] = s;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(counter, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  __shared__ double s_k;
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int b = 0; b < static_cast<int>(gridDim.x); ++b) s += __ldcg(&partial[b]);
    s_k = 0.5 * t * s;
    *counter = 0u;
  }
  __syncthreads();
  const double K = s_k;
  for (int i = j + 1 + threadIdx.x; i < n; i += blockDim.x) wbuf[i] = __ldcg(&wbuf[i]) - K * vbuf[i];
}

__global__ void __launch_bounds__(256) k_tri_update(double* __restrict__ A, int n, int j,
                                                    const double* __restrict__ tau, const double* __restrict__ vbuf,
                                                    const double* __restrict__ wbuf) {
  if (tau[j] == 0.0) return;
  for (int r = j + 1 + blockIdx.x; r < n; r += gridDim.x) {
    const double vr = vbuf[r], wr = wbuf[r];
    double* row = A + static_cast<int64_t>(r) * n;
    for (int c = j + 1 + threadIdx.x; c < n; c += blockDim.x) row[c] -= vr * wbuf[c] + wr * vbuf[c];
  }
}

__global__ void k_tri_last(const double* A, int n, double* d, double* e, double* tau) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  if (n >= 2) {
    d[n - 2] = A[static_cast<int64_t>(n - 2) * n + n - 2];
    e[n - 2] = A[static_cast<int64_t>(n - 1) * n + n - 2];
    tau[n - 2] = 0.0;
  }
  d[n - 1] = A[static_cast<int64_t>(n - 1) * n + n - 1];
}

// ---- single-launch tridiagonalisation (n <= kTriCoopMax) ----
// Householder steps with the matrix in the shared memory of G co-resident
// CTAs: row r lives in CTA r % G, slot r / G; a thread owns the columns
// c = tid + q * 256.  A step is one exchange between the CTAs:
//   pass    every CTA applies the previous step's A -= v w^T + w v^T to its
//           rows r > j and, in the same pass over shared memory, forms
//           p_r = (A v_j)_r; a_r = A(r, j + 1) is then up to step j - 1;
//   gather  every CTA publishes (p_r, a_r) of its rows and reads everybody's;
//   local   every CTA then knows p and column j + 1 and forms for itself
//           K = tau^2 (p.v) / 2, w = tau p - K v, the updated column
//           a - v w_{j+1} - w v_{j+1}, and from it the next reflector.
// The exchange is what bounds a step (the pass reads and writes at most
// 200 KB of shared memory a CTA, on average a third of that), and one is what
// it takes: publishing the reflector and w each with a grid-wide wait of its
// own measured 11 us a column at n = 1873, this 6.1 us; one CTA alone
// took 6.6 us a column at n = 150, a cluster here 2.1 us.
//   CLUSTER (n <= kTriClusterMax): up to 16 CTAs of one thread-block cluster;
//   a CTA stores its pairs into every peer's shared memory, the exchange is
//   one cluster barrier.  Small solves leave the other SMs to concurrent ones.
//   Otherwise (cooperative launch, up to one CTA an SM): pairs go through L2
//   as 16-byte words (value, step number), stored and loaded as single 128-bit
//   accesses, so that a word carries its own arrival flag and nothing has to be
//   ordered against it.  Words are double-buffered by step parity, and a word
//   is rewritten two steps later.  Its readers at step j are the CTAs with a row
//   > j.  Each of them has a row >= j + 1 and publishes it at step j + 1, after
//   its reads of step j; the gather of step j + 1 waits for the words of all rows
//   >= j + 1, so nobody is at step j + 2 before.  The word of row j + 1 itself
//   holds nothing then: it says that its owner is through step j, which no other
//   word may (a CTA whose last row is j + 1 has none below).  With it published
//   and the reflector stored, a CTA whose rows are all finished leaves.  Every
//   wait is bounded: a thread that waits longer than the limit sets the error
//   word, every CTA returns, and the host redoes the matrix with the
//   multi-launch steps.
constexpr int CT_THREADS = 256;
constexpr int CT_WARPS = CT_THREADS / 32;
constexpr int CT_CHUNK = 16;                                     // rows a pass accumulates at a time
constexpr int CT_RMAX = 32;                                      // rows per CTA
constexpr int CT_CMAX = 8;                                       // columns per thread
constexpr int64_t kTriCoopMax = int64_t(CT_THREADS) * CT_CMAX;   // 2048
constexpr int kTriClusterMax = 512;                              // 16 CTAs x 32 rows
constexpr uint64_t kCoopWaitNs = 2000000000ull;                  // 2 s per wait

struct CoopTri {
  double* A;  // n x n, symmetric on entry; reflector of step j goes to row j
  int n, G, R;
  double *d, *e, *tau;
  ulonglong2* words;  // [2][n][2]: (p_r, step), (a_r, step); zero on entry (cooperative launch)
  int* err;
  uint64_t wait_ns;   // limit of every wait
};

__device__ __forceinline__ uint64_t coop_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ ulonglong2 ld_word(const ulonglong2* p) {
  ulonglong2 v;
  asm volatile("{ .reg .b128 q; ld.relaxed.gpu.global.b128 q, [%2]; mov.b128 {%0, %1}, q; }"
               : "=l"(v.x), "=l"(v.y)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ void st_word(ulonglong2* p, double value, uint64_t step) {
  asm volatile("{ .reg .b128 q; mov.b128 q, {%1, %2}; st.relaxed.gpu.global.b128 [%0], q; }" ::"l"(p),
               "l"(__double_as_longlong(value)), "l"(step)
               : "memory");
}

// Sums of 16 values over the warp at once: every level halves the values a
// lane carries.  Lane l returns the sum of value l / 2.
__device__ __forceinline__ double warp_sum16(double (&a)[CT_CHUNK], int lane) {
#pragma unroll
  for (int h = CT_CHUNK / 2; h >= 1; h >>= 1) {
    const bool up = (lane & (2 * h)) != 0;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const double send = up ? a[i] : a[i + h];
      const double keep = up ? a[i + h] : a[i];
      a[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * h);
    }
  }
  return a[0] + __shfl_xor_sync(0xffffffffu, a[0], 1);
}

template <int CMAX, bool CLUSTER>
__global__ void __launch_bounds__(CT_THREADS, 1) k_tridiag_coop(CoopTri p) {
  // [R][n + 1] (cluster: [R + 1], a spare row), then (cluster) [2][n] pairs
  extern __shared__ __align__(16) double rows[];
  __shared__ double pr[CT_WARPS][CT_RMAX];        // row products, a partial per warp
  __shared__ double vr[CT_RMAX + CT_CHUNK], wr[CT_RMAX + CT_CHUNK];
  __shared__ __align__(16) double red_s[CT_WARPS], red_d[CT_WARPS];
  __shared__ double s_alpha, s_p1;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = p.n, G = p.G, R = p.R, b = blockIdx.x;
  const int ns = n + 1;
  double2* pairs = reinterpret_cast<double2*>(rows + ((static_cast<size_t>(R + 1) * ns + 1) & ~size_t(1)));
  for (int l = 0; l < (CLUSTER ? R + 1 : R); ++l) {
    const int r = l * G + b;
    const bool held = l < R && r < n;
    for (int c = tid; c <= n; c += CT_THREADS)
      rows[l * ns + c] = held && c < n ? p.A[static_cast<int64_t>(r) * n + c] : 0.0;
  }
  // x: column j from the diagonal down; v, w of the previous step; v of this one
  double x[CMAX], vp[CMAX], wp[CMAX], vc[CMAX];
#pragma unroll
  for (int q = 0; q < CMAX; ++q) {
    const int c = tid + q * CT_THREADS;
    x[q] = c < n ? p.A[c] : 0.0;
    vp[q] = 0.0;
    wp[q] = 0.0;
  }
  int slot[CMAX];  // where this CTA keeps row c, -1: it does not
  int col[CMAX];
#pragma unroll
  for (int q = 0; q < CMAX; ++q) {
    const int c = tid + q * CT_THREADS;
    col[q] = min(c, n);
    slot[q] = c < n && c % G == b ? c / G : -1;
  }
  if (tid < CT_RMAX + CT_CHUNK) {
    vr[tid] = 0.0;
    wr[tid] = 0.0;
  }
  if constexpr (CLUSTER) cooperative_groups::this_cluster().sync();  // peers' shared memory is live
  for (int j = 0; j + 2 < n; ++j) {
    const bool owner = j % G == b;
    // reflector of column j, in every CTA
    double sq = 0.0;
#pragma unroll
    for (int q = 0; q < CMAX; ++q) {
      const int c = tid + q * CT_THREADS;
      if (c > j + 1 && c < n) sq = fma(x[q], x[q], sq);
      if (c == j + 1) s_alpha = x[q];
      if (c == j && owner) p.d[j] = x[q];
    }
    sq = warp_sum(sq);
    if (lane == 0) red_s[warp] = sq;
    __syncthreads();
    double sigma = 0.0;
#pragma unroll
    for (int w = 0; w < CT_WARPS; w += 2) {
      const double2 t = *reinterpret_cast<const double2*>(red_s + w);
      sigma += t.x + t.y;
    }
    // H = I - tau v v^T, v = S (alpha - beta, x_{j+2}, ..) unnormalised: its
    // division is not needed before w.  S, a power of two from the exponents of
    // alpha and sigma (beta's square root is not waited for), puts the column's
    // norm into [1, 3) and v's first element into [1, 5), so that tau^2 is in
    // range whatever the column's size (a sigma below the normal numbers leaves
    // them above 2^-26).
    const double alpha = s_alpha;
    const int ea = (__double2hiint(alpha) >> 20 & 0x7ff) - 1023;
    const int eg = ((__double2hiint(sigma) >> 20 & 0x7ff) - 1023) >> 1;
    const double S = __hiloint2double((1023 - min(max(ea, eg), 1022)) << 20, 0);
    double beta = alpha, v1 = 0.0, tau_inv = 0.0;
    if (sigma > 0.0) {
      const double nrm = sqrt(fma(alpha, alpha, sigma));
      beta = alpha >= 0.0 ? -nrm : nrm;
      v1 = (alpha - beta) * S;
      tau_inv = -(beta * S) * v1;
    }
#pragma unroll
    for (int q = 0; q < CMAX; ++q) {
      const int c = tid + q * CT_THREADS;
      vc[q] = c == j + 1 ? v1 : (c > j + 1 ? x[q] * S : 0.0);  // x is zero past the end
    }
    // pass: slots below l0 hold finished rows (r <= j)
    const int l0 = j >= b ? (j - b) / G + 1 : 0;
    const int live = (n - b + G - 1) / G;  // slots that hold a row
    bool on[CMAX], any = false;
#pragma unroll
    for (int q = 0; q < CMAX; ++q) {
      const int c = warp * 32 + q * CT_THREADS;  // the group's first column
      on[q] = c + 31 > j && c < n;
      any = any || on[q];
    }
    if (!any && lane < CT_RMAX) pr[warp][lane] = 0.0;
    for (int lb = any ? l0 : live; lb < live; lb += CT_CHUNK) {
      double acc[CT_CHUNK];
      // Finished columns need no guard (v and w are zero there); a warp skips
      // a column group that is finished as a whole, and columns past the end
      // go to a pad column.  GR rows are loaded together: the stores of one
      // row could alias the loads of the next as far as the compiler knows;
      // with two columns a thread, rows past the end go to a spare row.
      constexpr int GR = CMAX == 2 ? 4 : 1;
#pragma unroll
      for (int g = 0; g < CT_CHUNK; g += GR) {
#pragma unroll
        for (int i = 0; i < GR; ++i) acc[g + i] = 0.0;
        if (lb + g >= live) continue;
        double a[GR][CMAX];
        double* row[GR];
#pragma unroll
        for (int i = 0; i < GR; ++i) {
          row[i] = rows + min(lb + g + i, GR > 1 ? live : R - 1) * ns;
#pragma unroll
          for (int q = 0; q < CMAX; ++q) a[i][q] = on[q] ? row[i][col[q]] : 0.0;
        }
#pragma unroll
        for (int i = 0; i < GR; ++i) {
          const double nv = -vr[lb + g + i], nw = -wr[lb + g + i];
#pragma unroll
          for (int q = 0; q < CMAX; ++q) {
            a[i][q] = fma(nv, wp[q], fma(nw, vp[q], a[i][q]));
            acc[g + i] = fma(a[i][q], vc[q], acc[g + i]);
          }
        }
#pragma unroll
        for (int i = 0; i < GR; ++i)
#pragma unroll
          for (int q = 0; q < CMAX; ++q)
            if (on[q]) row[i][col[q]] = a[i][q];
      }
      const double sum = warp_sum16(acc, lane);
      if ((lane & 1) == 0 && lb + (lane >> 1) < live) pr[warp][lb + (lane >> 1)] = sum;
    }
    __syncthreads();
    // publish own rows
    const uint64_t step = static_cast<uint64_t>(j) + 1;
    const int nl = live - l0;
    if constexpr (CLUSTER) {
      // a thread a (row, peer) pair
      for (int t = tid; t < CT_RMAX * G; t += CT_THREADS) {
        const int peer = t / CT_RMAX, l = l0 + (t & (CT_RMAX - 1));
        if (l >= live) continue;
        double sum = 0.0;
#pragma unroll
        for (int w = 0; w < CT_WARPS; ++w) sum += pr[w][l];
        *cooperative_groups::this_cluster().map_shared_rank(pairs + (j & 1) * n + l * G + b, peer) =
            make_double2(sum, rows[l * ns + j + 1]);
      }
    } else if (tid < nl + (owner ? 1 : 0)) {
      const bool done = tid == nl;  // row j, in slot l0 - 1
      const int l = done ? l0 - 1 : l0 + tid;
      double sum = 0.0;
#pragma unroll
      for (int w = 0; w < CT_WARPS; ++w) sum += pr[w][l];
      ulonglong2* out = p.words + (static_cast<size_t>(j & 1) * n + l * G + b) * 2;
      st_word(out, done ? 0.0 : sum, step);
      st_word(out + 1, done ? 0.0 : rows[l * ns + j + 1], step);
    }
    const double tau = tau_inv != 0.0 ? 1.0 / tau_inv : 0.0;
    // Row j of A takes the reflector, normalised to a first element of one as
    // the back-transformation reads it, while the other CTAs' words are on
    // their way (row 0, which every CTA read at the start, after they came).
    auto keep_reflector = [&] {
      if (!owner) return;
      const double inv = v1 != 0.0 ? 1.0 / v1 : 0.0;
#pragma unroll
      for (int q = 0; q < CMAX; ++q) {
        const int c = tid + q * CT_THREADS;
        if (c > j + 1 && c < n) p.A[static_cast<int64_t>(j) * n + c] = vc[q] * inv;
      }
      if (tid == 0) {
        p.e[j] = beta;
        p.tau[j] = tau * v1 * v1;
      }
    };
    if (j > 0) keep_reflector();
    if (!CLUSTER && nl == 0) return;  // j > 0 here: every CTA starts with three rows or more
    // gather
    double pc[CMAX], ac[CMAX];
    int fail = 0;
    if constexpr (CLUSTER) {
      cooperative_groups::this_cluster().sync();
#pragma unroll
      for (int q = 0; q < CMAX; ++q) {
        const int c = tid + q * CT_THREADS;
        const double2 t = (c > j && c < n) ? pairs[(j & 1) * n + c] : make_double2(0.0, 0.0);
        pc[q] = t.x;
        ac[q] = t.y;
      }
    } else {
      const ulonglong2* in = p.words + static_cast<size_t>(j & 1) * n * 2;
      unsigned missing = 0;
#pragma unroll
      for (int q = 0; q < CMAX; ++q) {
        const int c = tid + q * CT_THREADS;
        pc[q] = 0.0;
        ac[q] = 0.0;
        if (c >= j && c < n) missing |= 1u << q;
      }
      uint64_t t0 = 0;
      unsigned fails = 0;
      while (missing != 0) {
        ulonglong2 wa[CMAX], wb[CMAX];
#pragma unroll
        for (int q = 0; q < CMAX; ++q) {
          if (missing >> q & 1u) {
            const ulonglong2* at = in + static_cast<size_t>(tid + q * CT_THREADS) * 2;
            wa[q] = ld_word(at);
            wb[q] = ld_word(at + 1);
          }
        }
#pragma unroll
        for (int q = 0; q < CMAX; ++q) {
          if ((missing >> q & 1u) && wa[q].y == step && wb[q].y == step) {
            pc[q] = __longlong_as_double(static_cast<long long>(wa[q].x));
            ac[q] = __longlong_as_double(static_cast<long long>(wb[q].x));
            missing &= ~(1u << q);
          }
        }
        // the clock and the error word cost as much as a poll: every 64 rounds
        if (missing != 0 && ((++fails & 63u) == 0 || p.wait_ns == 0)) {
          const uint64_t now = coop_ns();
          if (t0 == 0) t0 = now;
          if (now - t0 >= p.wait_ns || *reinterpret_cast<volatile int*>(p.err) != 0) {
            if (now - t0 >= p.wait_ns) atomicExch(p.err, 1);
            fail = 1;
            break;
          }
        }
      }
    }
    if (j == 0) keep_reflector();
    // w and column j + 1
    double dot = 0.0;
#pragma unroll
    for (int q = 0; q < CMAX; ++q) {
      dot = fma(pc[q], vc[q], dot);
      if (tid + q * CT_THREADS == j + 1) s_p1 = pc[q];
    }
    dot = warp_sum(dot);
    if (lane == 0) red_d[warp] = dot;
    if constexpr (CLUSTER) {
      __syncthreads();
    } else {
      if (__syncthreads_or(fail)) return;
    }
    double pv = 0.0;
#pragma unroll
    for (int w = 0; w < CT_WARPS; w += 2) {
      const double2 t = *reinterpret_cast<const double2*>(red_d + w);
      pv += t.x + t.y;
    }
    const double K = 0.5 * tau * tau * pv;
    const double w1 = fma(tau, s_p1, -K * v1);  // w_{j+1}
#pragma unroll
    for (int q = 0; q < CMAX; ++q) {
      vp[q] = tau != 0.0 ? vc[q] : 0.0;
      wp[q] = tau != 0.0 ? fma(tau, pc[q], -K * vc[q]) : 0.0;
      x[q] = tau != 0.0 ? ac[q] - fma(vp[q], w1, wp[q] * v1) : ac[q];
      if (slot[q] >= l0) {
        vr[slot[q]] = vp[q];
        wr[slot[q]] = wp[q];
      }
    }
  }
  // x: column n - 2; the last diagonal entry still lacks the last update
#pragma unroll
  for (int q = 0; q < CMAX; ++q) {
    const int c = tid + q * CT_THREADS;
    if (n >= 2 && (n - 2) % G == b) {
      if (c == n - 2) {
        p.d[c] = x[q];
        p.tau[c] = 0.0;
      }
      if (c == n - 1) p.e[n - 2] = x[q];
    }
    if ((n - 1) % G == b && c == n - 1) p.d[c] = fma(-2.0 * vp[q], wp[q], rows[(c / G) * ns + c]);
  }
  if constexpr (CLUSTER) cooperative_groups::this_cluster().sync();  // no peer stores into a CTA that has left
}

// ---- the k smallest eigenpairs of T directly (n <= kTriDirectMax) ----
// One CTA an eigenpair: multisection of eigenvalue blockIdx.x (kTdThreads
// points a round, so eight rounds to eps |T|), then its vector from the
// twisted factorisation of T - theta (Parlett and Dhillon, "Fernando's
// solution to Wilkinson's problem", LAA 267, 1997): pivots from both ends as
// ratios of successive leading / trailing minors, the twist where their sum is
// smallest, running products away from it.  No division is on a chain: a step
// of a count is one dependent multiply-add; four warps keep the shared-memory
// reads of T (16 bytes a step, the same for every lane) below that chain.
// k_tri_polish then orthonormalises the k vectors and tests them; where two
// wanted eigenvalues agree to rounding (a matrix that splits, multiplicities)
// the test fails and k_tri_eig, whose inverse iteration handles those, runs
// instead.  Measured at n = 1873, k = 4: 0.51 ms against 4.6 ms for
// k_tri_eig alone.
constexpr int kTdThreads = 128;
constexpr int64_t kTriDirectMax = 2048;
constexpr int kTdPad = 4;

// Rescale a pair of successive minors towards one (exact; ratios and signs stay).
__device__ __forceinline__ void td_rescale(double& p0, double& p1) {
  const double m = fmax(fabs(p0), fabs(p1));
  if (m < 0x1p-300 || m > 0x1p300) {
    const double f = m < 1.0 ? 0x1p300 : 0x1p-300;
    p0 *= f;
    p1 *= f;
  }
}

// eigenvalues of T below x: sign changes of the leading minors of T - x;
// de[i] = (d_i, e_{i-1}^2) scaled to a norm in [1/2, 1), padded with (2, 0)
__device__ __forceinline__ int td_count(const double2* de, int n, double x) {
  double p0 = 0.0, p1 = 1.0;
  unsigned signs = 0;
  int cnt = 0;
  for (int i = 0; i < n; i += 4) {
    double2 t[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) t[u] = de[i + u];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const double p2 = fma(t[u].x - x, p1, -t[u].y * p0);
      signs = __funnelshift_l(static_cast<unsigned>(__double2hiint(p2)), signs, 1);
      p0 = p1;
      p1 = p2;
    }
    cnt += __popc((signs ^ (signs >> 1)) & 15u);
    td_rescale(p0, p1);
  }
  return cnt;
}

__global__ void __launch_bounds__(kTdThreads) k_tri_direct(const double* __restrict__ d, const double* __restrict__ e,
                                                           int n, double* __restrict__ theta, double* __restrict__ Y,
                                                           int ld) {
  extern __shared__ __align__(16) double td_sm[];
  double2* de = reinterpret_cast<double2*>(td_sm);      // [n + 4]
  double2* fw = de + n + kTdPad;                        // [n] (minor before i, minor at i) from the top
  double2* bw = fw + n;                                 // [n] the same from the bottom
  __shared__ double red[kTdThreads / 32];
  __shared__ int redk[kTdThreads / 32];
  __shared__ int s_cnt[kTdThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int want = blockIdx.x;
  // power-of-two scale to a Gershgorin bound in [1/2, 1)
  double b = 0.0;
  for (int i = tid; i < n; i += kTdThreads)
    b = fmax(b, fabs(d[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < n ? fabs(e[i]) : 0.0));
  b = warp_max(b);
  if (lane == 0) red[warp] = b;
  __syncthreads();
  b = fmax(fmax(red[0], red[1]), fmax(red[2], red[3]));
  const int be = (__double2hiint(b) >> 20) & 0x7ff;
  const int ex = be > 32 && be < 2014 ? be - 1022 : 0;
  const double sc = __hiloint2double((1023 - ex) << 20, 0);
  for (int i = tid; i < n + kTdPad; i += kTdThreads) {
    const double es = (i > 0 && i < n) ? e[i - 1] * sc : 0.0;
    de[i] = i < n ? make_double2(d[i] * sc, es * es) : make_double2(2.0, 0.0);
  }
  __syncthreads();
  double lo = -1.0, hi = 1.0;
  for (int round = 0; round < 12 && hi - lo > 0.5 * DBL_EPSILON; ++round) {
    const double h = (hi - lo) * (1.0 / (kTdThreads + 1));
    const bool above = td_count(de, n, fma(h, tid + 1.0, lo)) > want;
    // first point with more than `want` eigenvalues below it
    const unsigned m = __ballot_sync(0xffffffffu, above);
    if (lane == 0) s_cnt[warp] = m ? warp * 32 + __ffs(m) - 1 : kTdThreads;
    __syncthreads();
    const int l = min(min(s_cnt[0], s_cnt[1]), min(s_cnt[2], s_cnt[3]));
    const double nlo = l > 0 ? fma(h, static_cast<double>(l), lo) : lo;
    if (l < kTdThreads) hi = fma(h, l + 1.0, lo);
    lo = nlo;
    __syncthreads();
  }
  const double t = 0.5 * (lo + hi);
  const double tiny = 0.0625 * DBL_EPSILON * DBL_EPSILON;
  // minors from both ends, warps 0 and 1
  if (lane == 0 && warp < 2) {
    double2* out = warp == 0 ? fw : bw;
    double p0 = 0.0, p1 = 1.0;
    for (int c0 = 0; c0 < n; c0 += 4) {
      double dd[4], ee[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int c = min(c0 + u, n - 1);
        dd[u] = de[warp == 0 ? c : n - 1 - c].x - t;
        ee[u] = warp == 0 ? de[c].y : (c > 0 ? de[n - c].y : 0.0);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const double p2 = fma(dd[u], p1, -ee[u] * p0);
        if (c0 + u < n) out[warp == 0 ? c0 + u : n - 1 - c0 - u] = make_double2(p1, p2);
        p0 = p1;
        p1 = p2;
      }
      td_rescale(p0, p1);
    }
  }
  __syncthreads();
  double gmin = DBL_MAX;
  int kmin = 0;
  for (int i = tid; i < n; i += kTdThreads) {
    const double2 f = fw[i], g = bw[i];
    double df = f.y / f.x, dg = g.y / g.x;
    if (!(fabs(df) >= tiny)) df = tiny;
    if (!(fabs(dg) >= tiny)) dg = tiny;
    const double gam = fabs(df + dg - (de[i].x - t));
    if (gam < gmin) {
      gmin = gam;
      kmin = i;
    }
    // z_i = fw.x z_{i+1} above the twist, bw.x z_{i-1} below it
    const double ei = i + 1 < n ? e[i] * sc : 0.0, em = i > 0 ? e[i - 1] * sc : 0.0;
    fw[i].x = -ei / df;
    bw[i].x = -em / dg;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double g = __shfl_xor_sync(0xffffffffu, gmin, o);
    const int k = __shfl_xor_sync(0xffffffffu, kmin, o);
    if (g < gmin || (g == gmin && k < kmin)) {
      gmin = g;
      kmin = k;
    }
  }
  if (lane == 0) {
    red[warp] = gmin;
    redk[warp] = kmin;
  }
  __syncthreads();
  gmin = red[0];
  kmin = redk[0];
  for (int w = 1; w < kTdThreads / 32; ++w)
    if (red[w] < gmin || (red[w] == gmin && redk[w] < kmin)) {
      gmin = red[w];
      kmin = redk[w];
    }
  // running products into fw.y
  if (lane == 0 && warp < 2) {
    double z = 1.0;
    if (warp == 0) {
      fw[kmin].y = 1.0;
#pragma unroll 8
      for (int i = kmin - 1; i >= 0; --i) {
        z *= fw[i].x;
        fw[i].y = z;
      }
    } else {
#pragma unroll 8
      for (int i = kmin + 1; i < n; ++i) {
        z *= bw[i].x;
        fw[i].y = z;
      }
    }
  }
  __syncthreads();
  double n2 = 0.0;
  for (int i = tid; i < n; i += kTdThreads) n2 = fma(fw[i].y, fw[i].y, n2);
  n2 = warp_sum(n2);
  if (lane == 0) red[warp] = n2;
  __syncthreads();
  const double inv = 1.0 / sqrt(((red[0] + red[1]) + red[2]) + red[3]);
  for (int i = tid; i < n; i += kTdThreads) Y[static_cast<int64_t>(i) * ld + want] = fw[i].y * inv;
  if (tid == 0) theta[want] = t * __hiloint2double((1023 + ex) << 20, 0);
}

// Y <- Y (3/2 I - G/2), G = Y^T Y, until G is the identity to rounding
// (quadratic; the vectors of pairs a gap g apart start eps / g from
// orthogonal, and the rotation that mends it moves T's projection by eps), and
// the residual test, at what inverse iteration ends with (graph Laplacians and
// random matrices of 10 to 2048 rows: at most 3 eps |T|).  ok[0] = 1 when the pairs stand, 0 when k_tri_eig has to
// find them.  One CTA.
constexpr int kTpThreads = 512;
__global__ void __launch_bounds__(kTpThreads) k_tri_polish(const double* __restrict__ d, const double* __restrict__ e,
                                                           int n, int k, const double* __restrict__ theta,
                                                           double* __restrict__ Y, int ld, int* __restrict__ ok) {
  __shared__ double G[MAXM * MAXM], red[kTpThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NW = kTpThreads / 32;
  double b = 0.0;
  for (int i = tid; i < n; i += kTpThreads)
    b = fmax(b, fabs(d[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < n ? fabs(e[i]) : 0.0));
  b = warp_max(b);
  if (lane == 0) red[warp] = b;
  __syncthreads();
  double tnorm = 0.0;
  for (int w = 0; w < NW; ++w) tnorm = fmax(tnorm, red[w]);
  bool fine = false;
  for (int it = 0; it < 4 && !fine; ++it) {
    for (int t = warp; t < k * k; t += NW) {
      const int i = t / k, j = t % k;
      if (j < i) continue;
      double g = 0.0;
      for (int r = lane; r < n; r += 32)
        g = fma(Y[static_cast<int64_t>(r) * ld + i], Y[static_cast<int64_t>(r) * ld + j], g);
      g = warp_sum(g);
      if (lane == 0) {
        G[i * k + j] = g;
        G[j * k + i] = g;
      }
    }
    __syncthreads();
    int bad = 0, big = 0;
    for (int t = tid; t < k * k; t += kTpThreads) {
      const double off = fabs(t / k == t % k ? G[t] - 1.0 : G[t]);
      if (!(off <= 16.0 * DBL_EPSILON)) bad = 1;
      if (!(off <= 0.05)) big = 1;
    }
    if (__syncthreads_or(big)) break;
    fine = !__syncthreads_or(bad);
    if (fine) break;
    for (int r = tid; r < n; r += kTpThreads) {
      double y[MAXM];
#pragma unroll
      for (int j = 0; j < MAXM; ++j) y[j] = j < k ? Y[static_cast<int64_t>(r) * ld + j] : 0.0;
      for (int i = 0; i < k; ++i) {
        double v = 0.0;
#pragma unroll
        for (int j = 0; j < MAXM; ++j)
          if (j < k) v = fma(-0.5 * y[j], G[j * k + i] - (i == j ? 3.0 : 0.0), v);
        Y[static_cast<int64_t>(r) * ld + i] = v;
      }
    }
    __syncthreads();
  }
  int off = fine ? 0 : 1;
  for (int r = tid; r < n && fine; r += kTpThreads) {
    for (int q = 0; q < k; ++q) {
      double v = (d[r] - theta[q]) * Y[static_cast<int64_t>(r) * ld + q];
      if (r > 0) v = fma(e[r - 1], Y[static_cast<int64_t>(r - 1) * ld + q], v);
      if (r + 1 < n) v = fma(e[r], Y[static_cast<int64_t>(r + 1) * ld + q], v);
      if (!(fabs(v) <= 16.0 * DBL_EPSILON * tnorm)) off = 1;
    }
  }
  off = __syncthreads_or(off);
  if (tid == 0) ok[0] = off ? 0 : 1;
  if (!off) return;
  for (int t = tid; t < n * k; t += kTpThreads) Y[static_cast<int64_t>(t / k) * ld + t % k] = 0.0;  // as k_tri_eig expects
}

// number of eigenvalues of T[l..r] smaller than x (Sturm sequence; e2 holds
// the squared off-diagonals)
__device__ int sturm_count(const double* d, const double* e2, int l, int r, double x, double pivmin) {
  int cnt = 0;
  double q = d[l] - x;
  if (fabs(q) < pivmin) q = -pivmin;
  if (q < 0.0) ++cnt;
  for (int i = l + 1; i <= r; ++i) {
    q = d[i] - x - e2[i - 1] / q;
    if (fabs(q) < pivmin) q = -pivmin;
    if (q < 0.0) ++cnt;
  }
  return cnt;
}

struct TriWork {
  int* bstart;      // [n + 1]
  double* es;       // [n] split off-diagonals
  double* e2;       // [n] their squares
  double* cand;     // [n * k]
  int* cand_blk;    // [n * k]
  double* lu;       // [5 * n]
  int* piv;         // [n]
  double* xv;       // [n]
  int* sel_blk;     // [k]
  double* sel_val;  // [k]
};

__global__ void __launch_bounds__(DT) k_tri_eig(const double* __restrict__ d, const double* __restrict__ e, int n,
                                                int k, TriWork w, double* evals_out, double* Y, int ld,
                                                int use_smem, const int* __restrict__ skip) {
  if (skip != nullptr && *skip != 0) return;  // the direct route's pairs stand
  __shared__ int s_nb;
  __shared__ double s_tnorm;
  __shared__ double s_red[32];
  extern __shared__ double te_sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // diagonal, split off-diagonals and their squares: in shared memory behind
  // the inverse-iteration arrays when it fits
  const double* dd = d;
  double* es = w.es;
  double* e2 = w.e2;
  if (use_smem) {
    double* dsm = te_sm + 6 * n;
    for (int i = tid; i < n; i += blockDim.x) dsm[i] = d[i];
    dd = dsm;
    es = te_sm + 7 * n;
    e2 = te_sm + 8 * n;
  }
  // |T| (row sums) and the splits where an off-diagonal is negligible
  double part = 0.0;
  for (int i = tid; i < n; i += blockDim.x) {
    part = fmax(part, fabs(d[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < n ? fabs(e[i]) : 0.0));
    if (i + 1 < n) {
      const double off = fabs(e[i]);
      const bool split = off <= DBL_EPSILON * (fabs(d[i]) + fabs(d[i + 1])) || off <= 1e-300;
      es[i] = split ? 0.0 : e[i];
      e2[i] = split ? 0.0 : e[i] * e[i];
    }
  }
  part = warp_max(part);
  if (lane == 0) s_red[warp] = part;
  __syncthreads();
  // block starts in order (one warp: ballot and prefix count per 32 entries)
  if (warp == 0) {
    double tn = 0.0;
    for (int i = lane; i < static_cast<int>(blockDim.x >> 5); i += 32) tn = fmax(tn, s_red[i]);
    tn = warp_max(tn);
    int cnt = 0;
    for (int base = 0; base + 1 < n; base += 32) {
      const int i = base + lane;
      const bool f = i + 1 < n && es[i] == 0.0;
      const unsigned bal = __ballot_sync(0xffffffffu, f);
      if (f) w.bstart[1 + cnt + __popc(bal & ((1u << lane) - 1u))] = i + 1;
      cnt += __popc(bal);
    }
    if (lane == 0) {
      w.bstart[0] = 0;
      w.bstart[cnt + 1] = n;
      s_nb = cnt + 1;
      s_tnorm = tn;
    }
  }
  __syncthreads();
  const int nb = s_nb;
  const double tnorm = s_tnorm;
  const double pivmin = fmax(DBL_MIN, tnorm * tnorm * DBL_MIN);
  // absolute tolerance of the eigenvalue intervals: eps |T| (the default of
  // LAPACK's dstebz); relative eps for eigenvalues away from zero
  const double atol = DBL_EPSILON * tnorm + pivmin;
  const int nitems = nb * k;
  // Gershgorin interval of item q's block; false if the block has no t-th eigenvalue
  auto item_interval = [&](int q, double& lo, double& hi) {
    const int b = q / k, t = q % k;
    const int l = w.bstart[b], r = w.bstart[b + 1] - 1;
    w.cand_blk[q] = b;
    if (t > r - l) {
      w.cand[q] = DBL_MAX;
      return false;
    }
    lo = DBL_MAX;
    hi = -DBL_MAX;
    for (int i = l; i <= r; ++i) {
      const double rad = (i > l ? fabs(es[i - 1]) : 0.0) + (i < r ? fabs(es[i]) : 0.0);
      lo = fmin(lo, dd[i] - rad);
      hi = fmax(hi, dd[i] + rad);
    }
    lo -= 2.0 * DBL_EPSILON * tnorm + pivmin;
    hi += 2.0 * DBL_EPSILON * tnorm + pivmin;
    return true;
  };
  auto converged = [&](double lo, double hi) {
    const double mid = 0.5 * (lo + hi);
    return hi - lo <= 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)) + atol || mid == lo || mid == hi;
  };
  if (nitems <= TE_MS_ITEMS) {
    // multisection: the P threads of an item count eigenvalues below P interior
    // points of its interval per round, and the interval shrinks to the gap
    // between the two points around the wanted index (a factor P + 1 a round)
    __shared__ double s_lo[TE_MS_ITEMS], s_hi[TE_MS_ITEMS];
    __shared__ int s_live[TE_MS_ITEMS];
    __shared__ int s_cnt[DT];
    // points per item: each Sturm count is a chain of n FP64 divisions, so past
    // ~96 points per item the SM's FP64 pipe, not the chain, sets the round time
    const int P = min(static_cast<int>(blockDim.x) / nitems, TE_MS_POINTS);
    if (tid < nitems) {
      double lo = 0.0, hi = 0.0;
      const bool ok = item_interval(tid, lo, hi);
      s_lo[tid] = lo;
      s_hi[tid] = hi;
      s_live[tid] = ok && !converged(lo, hi);
      if (ok && !s_live[tid]) w.cand[tid] = 0.5 * (lo + hi);
    }
    __syncthreads();
    const int item = tid / P, pi = tid % P;
    auto point = [&](double lo, double hi, int p) { return lo + (hi - lo) * (static_cast<double>(p + 1) / (P + 1)); };
    for (int round = 0; round < 200; ++round) {
      if (item < nitems && s_live[item]) {
        const int b = item / k;
        s_cnt[tid] = sturm_count(dd, e2, w.bstart[b], w.bstart[b + 1] - 1, point(s_lo[item], s_hi[item], pi), pivmin);
      }
      __syncthreads();
      int more = 0;
      if (tid < nitems && s_live[tid]) {
        const int t = tid % k;
        const double lo = s_lo[tid], hi = s_hi[tid];
        int p = 0;
        while (p < P && s_cnt[tid * P + p] <= t) ++p;
        // count(point p - 1) <= t < count(point p)
        const double nlo = p == 0 ? lo : point(lo, hi, p - 1);
        const double nhi = p == P ? hi : point(lo, hi, p);
        s_lo[tid] = nlo;
        s_hi[tid] = nhi;
        if (converged(nlo, nhi) || (nlo == lo && nhi == hi)) {
          s_live[tid] = 0;
          w.cand[tid] = 0.5 * (nlo + nhi);
        } else {
          more = 1;
        }
      }
      if (!__syncthreads_or(more)) break;
    }
    if (tid < nitems && s_live[tid]) w.cand[tid] = 0.5 * (s_lo[tid] + s_hi[tid]);
  } else {
    // one thread per item, bisection
    for (int q = tid; q < nitems; q += blockDim.x) {
      double lo = 0.0, hi = 0.0;
      if (!item_interval(q, lo, hi)) continue;
      const int b = q / k, t = q % k;
      const int l = w.bstart[b], r = w.bstart[b + 1] - 1;
      for (int it = 0; it < 200 && !converged(lo, hi); ++it) {
        const double mid = 0.5 * (lo + hi);
        if (sturm_count(dd, e2, l, r, mid, pivmin) > t) hi = mid; else lo = mid;
      }
      w.cand[q] = 0.5 * (lo + hi);
    }
  }
  __syncthreads();
  // k smallest candidates (stable)
  __shared__ int s_nsel;
  if (tid == 0) {
    int nsel = 0;
    for (int s = 0; s < k; ++s) {
      int best = -1;
      for (int q = 0; q < nb * k; ++q) {
        if (w.cand[q] == DBL_MAX) continue;
        bool taken = false;
        for (int u = 0; u < nsel; ++u)
          if (w.sel_blk[u] == q) taken = true;
        if (taken) continue;
        if (best < 0 || w.cand[q] < w.cand[best]) best = q;
      }
      if (best < 0) break;
      w.sel_blk[nsel++] = best;
    }
    for (int s = 0; s < nsel; ++s) {
      const int q = w.sel_blk[s];
      evals_out[s] = w.cand[q];
      w.sel_val[s] = w.cand[q];
    }
    s_nsel = nsel;
  }
  __syncthreads();
  const int nsel = s_nsel;
  // Eigenvectors by inverse iteration.  The LU factorisation and the two
  // triangular sweeps are sequential (thread 0, working arrays in shared
  // memory when they fit, reciprocals of the pivots formed in parallel);
  // re-orthogonalisation and normalisation use the whole CTA.  Iteration stops
  // after the second solve once the growth ||y|| shows a residual at rounding
  // level (as LAPACK's dstein), at the latest after the fourth.
  double* D = use_smem ? te_sm : w.lu;
  double* DL = D + n;
  double* DU = D + 2 * n;
  double* DU2 = D + 3 * n;
  double* RD = D + 4 * n;  // 1 / D
  double* x = use_smem ? te_sm + 5 * n : w.xv;
  int* piv = use_smem ? reinterpret_cast<int*>(te_sm + 9 * n) : w.piv;
  double* red = s_red;
  const double tiny = DBL_EPSILON * fmax(tnorm, DBL_MIN);
  for (int s = 0; s < nsel; ++s) {
    const int q = w.sel_blk[s];
    const int b = w.cand_blk[q];
    const int l = w.bstart[b], r = w.bstart[b + 1] - 1, sz = r - l + 1;
    const double lam = w.cand[q];
    double bpart = 0.0;
    for (int i = l + tid; i <= r; i += blockDim.x)
      bpart = fmax(bpart, fabs(dd[i]) + (i > l ? fabs(es[i - 1]) : 0.0) + (i < r ? fabs(es[i]) : 0.0));
    bpart = warp_max(bpart);
    if ((tid & 31) == 0) red[tid >> 5] = bpart;
    __syncthreads();
    double bnorm = 0.0;
    for (int i = 0; i < static_cast<int>(blockDim.x >> 5); ++i) bnorm = fmax(bnorm, red[i]);
    // T_b - lam I, and the start vector
    for (int i = tid; i < sz; i += blockDim.x) {
      D[i] = dd[l + i] - lam;
      DU[i] = (i + 1 < sz) ? es[l + i] : 0.0;
      DL[i] = DU[i];
      DU2[i] = 0.0;
      double z0, z1;
      philox_normal2(0x0de75eedull + s, 7, static_cast<uint64_t>(i), z0, z1);
      x[i] = z0;
    }
    __syncthreads();
    // LU with partial pivoting
    if (tid == 0) {
      for (int i = 0; i + 1 < sz; ++i) {
        if (fabs(D[i]) >= fabs(DL[i])) {
          if (D[i] == 0.0) D[i] = tiny;
          const double f = DL[i] / D[i];
          DL[i] = f;
          D[i + 1] -= f * DU[i];
          piv[i] = 0;
        } else {
          const double f = D[i] / DL[i];
          D[i] = DL[i];
          DL[i] = f;
          const double tmp = DU[i];
          DU[i] = D[i + 1];
          D[i + 1] = tmp - f * D[i + 1];
          if (i + 2 < sz) {
            DU2[i] = DU[i + 1];
            DU[i + 1] = -f * DU[i + 1];
          }
          piv[i] = 1;
        }
      }
    }
    __syncthreads();
    for (int i = tid; i < sz; i += blockDim.x) {
      if (fabs(D[i]) < tiny) D[i] = D[i] < 0.0 ? -tiny : tiny;
      RD[i] = 1.0 / D[i];
    }
    __syncthreads();
    const double grow_ok = 1.0 / (static_cast<double>(sz) * DBL_EPSILON * fmax(bnorm, DBL_MIN));
    for (int it = 0; it < 4; ++it) {
      // solve (T - lam I) y = x in place
      if (tid == 0) {
        for (int i = 0; i + 1 < sz; ++i) {
          if (piv[i] == 0) {
            x[i + 1] -= DL[i] * x[i];
          } else {
            const double tmp = x[i];
            x[i] = x[i + 1];
            x[i + 1] = tmp - DL[i] * x[i];
          }
        }
        x[sz - 1] *= RD[sz - 1];
        if (sz >= 2) x[sz - 2] = (x[sz - 2] - DU[sz - 2] * x[sz - 1]) * RD[sz - 2];
        for (int i = sz - 3; i >= 0; --i) x[i] = (x[i] - DU[i] * x[i + 1] - DU2[i] * x[i + 2]) * RD[i];
      }
      __syncthreads();
      // re-orthogonalise against earlier vectors of the same block in the cluster
      for (int u = 0; u < s; ++u) {
        const int qu = w.sel_blk[u];
        if (w.cand_blk[qu] != b) continue;
        if (fabs(w.sel_val[u] - lam) > 1e-3 * bnorm) continue;
        double part = 0.0;
        for (int i = tid; i < sz; i += blockDim.x) part += Y[static_cast<int64_t>(l + i) * ld + u] * x[i];
        const double dot = block_sum_all(part, red);
        for (int i = tid; i < sz; i += blockDim.x) x[i] -= dot * Y[static_cast<int64_t>(l + i) * ld + u];
        __syncthreads();
      }
      double part = 0.0;
      for (int i = tid; i < sz; i += blockDim.x) part += x[i] * x[i];
      double nrm = sqrt(block_sum_all(part, red));
      const bool degenerate = !(nrm > 0.0);
      const double inv = degenerate ? 1.0 : 1.0 / nrm;
      for (int i = tid; i < sz; i += blockDim.x) x[i] = degenerate ? ((i == s % sz) ? 1.0 : 0.0) : x[i] * inv;
      __syncthreads();
      if (it >= 1 && nrm >= grow_ok) break;  // uniform: nrm is the same in every thread
    }
    for (int i = tid; i < sz; i += blockDim.x) Y[static_cast<int64_t>(l + i) * ld + s] = x[i];
    __syncthreads();
  }
}

// Y <- Q Y with Q = H_0 H_1 ... H_{n-3}; reflector j: u = (1, A[j][j+2..n)) on rows j+1..n-1.
__global__ void __launch_bounds__(DT) k_backtransform(const double* __restrict__ A, const double* __restrict__ tau,
                                                      int n, double* Y, int ld, int k) {
  __shared__ double dots[MAXM];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  for (int j = n - 3; j >= 0; --j) {
    const double t = tau[j];
    if (t == 0.0) continue;
    for (int v = warp; v < k; v += nwarps) {
      double acc = 0.0;
      for (int r = j + 1 + lane; r < n; r += 32) {
        const double u = (r == j + 1) ? 1.0 : A[static_cast<int64_t>(j) * n + r];
        acc = fma(u, Y[static_cast<int64_t>(r) * ld + v], acc);
      }
      acc = warp_sum(acc);
      if (lane == 0) dots[v] = t * acc;
    }
    __syncthreads();
    const int len = n - j - 1;
    for (int idx = tid; idx < len * k; idx += blockDim.x) {
      const int r = j + 1 + idx / k, v = idx % k;
      const double u = (r == j + 1) ? 1.0 : A[static_cast<int64_t>(j) * n + r];
      Y[static_cast<int64_t>(r) * ld + v] -= dots[v] * u;
    }
    __syncthreads();
  }
}

// The same product, blocked: reflectors are applied eight at a time from the
// last block down, each block as one compact-WY product (the forward,
// column-wise form of LAPACK's dlarft):
//   H_j0 H_j0+1 ... H_j0+7 = I - V T V^T,   T upper triangular,
//   T[i][i] = tau_i,  T[0:i, i] = -tau_i T[0:i, 0:i] (V^T V)[0:i, i],
// so a block costs one pass of dot products (V^T V and V^T Y, one warp per
// product, lanes over rows), a small triangular product and one pass
// Y -= V (T V^T Y).  Y (n x k) and the block's reflectors stay in shared
// memory; a reflector with tau = 0 gets a zero row and column of T.
constexpr int BW_NB = 8;
constexpr int BW_THREADS = 512;

__global__ void __launch_bounds__(BW_THREADS) k_backtransform_wy(const double* __restrict__ A,
                                                                 const double* __restrict__ tau, int n,
                                                                 double* __restrict__ Y, int ld, int k) {
  extern __shared__ double bw_sm[];
  double* ys = bw_sm;          // [n][k]
  double* U = bw_sm + n * k;   // [BW_NB][n]
  __shared__ double G[BW_NB][BW_NB], T[BW_NB][BW_NB], Wt[BW_NB][MAXM], Wp[BW_NB][MAXM], st[BW_NB];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NW = BW_THREADS / 32;
  for (int idx = tid; idx < n * k; idx += BW_THREADS) ys[idx] = Y[static_cast<int64_t>(idx / k) * ld + idx % k];
  const int nref = n - 2;  // reflectors 0 .. n - 3
  for (int bi = (nref + BW_NB - 1) / BW_NB - 1; bi >= 0; --bi) {
    const int j0 = bi * BW_NB, nb = min(BW_NB, nref - j0);
    const int r0 = j0 + 1, len = n - r0;  // rows where the block's reflectors can be nonzero
    for (int idx = tid; idx < nb * len; idx += BW_THREADS) {
      const int i = idx / len, r = r0 + idx % len;
      const int j = j0 + i;
      U[i * n + r] = r == j + 1 ? 1.0 : (r > j + 1 ? A[static_cast<int64_t>(j) * n + r] : 0.0);
    }
    if (tid < nb) st[tid] = tau[j0 + tid];
    __syncthreads();
    const int ng = nb * (nb + 1) / 2, nd = ng + nb * k;
    for (int dd = warp; dd < nd; dd += NW) {
      double acc = 0.0;
      int a = 0, b = 0, v = 0;
      if (dd < ng) {
        int e = dd;
        while (e >= nb - a) {
          e -= nb - a;
          ++a;
        }
        b = a + e;
        for (int r = r0 + lane; r < n; r += 32) acc = fma(U[a * n + r], U[b * n + r], acc);
      } else {
        a = (dd - ng) / k;
        v = (dd - ng) % k;
        for (int r = r0 + lane; r < n; r += 32) acc = fma(U[a * n + r], ys[r * k + v], acc);
      }
      acc = warp_sum(acc);
      if (lane == 0) {
        if (dd < ng) G[a][b] = acc;
        else Wt[a][v] = acc;
      }
    }
    __syncthreads();
    if (tid == 0) {
      for (int i = 0; i < nb; ++i) {
        T[i][i] = st[i];
        for (int p = 0; p < i; ++p) {
          double sum = 0.0;
          for (int q = p; q < i; ++q) sum = fma(T[p][q], G[q][i], sum);
          T[p][i] = -st[i] * sum;
        }
      }
      for (int a = 0; a < nb; ++a)
        for (int v = 0; v < k; ++v) {
          double sum = 0.0;
          for (int b = a; b < nb; ++b) sum = fma(T[a][b], Wt[b][v], sum);
          Wp[a][v] = sum;
        }
    }
    __syncthreads();
    for (int idx = tid; idx < len * k; idx += BW_THREADS) {
      const int r = r0 + idx / k, v = idx % k;
      double sum = 0.0;
      for (int a = 0; a < nb; ++a) sum = fma(U[a * n + r], Wp[a][v], sum);
      ys[r * k + v] -= sum;
    }
    __syncthreads();
  }
  for (int idx = tid; idx < n * k; idx += BW_THREADS) Y[static_cast<int64_t>(idx / k) * ld + idx % k] = ys[idx];
}

// The same blocks of eight for n <= kBcMax, one CTA a vector, two launches:
// k_wy_factors forms every block's T at once (a warp a block pair of rows),
// k_backtransform_cols walks the blocks with y and the block in registers (a
// thread owns rows tid + q * 512) and the next block's rows already in flight,
// so the reflectors are read once a vector and a block costs two barriers.
// Forming T on the way, by one thread, took most of k_backtransform_wy's 26 us
// a block at n = 1873; this takes 2.2 us.
constexpr int BC_THREADS = 512;
constexpr int BC_RPT = 4;
constexpr int kBcMax = BC_THREADS * BC_RPT;

__global__ void __launch_bounds__(256) k_wy_factors(const double* __restrict__ A, const double* __restrict__ tau,
                                                    int n, double* __restrict__ Tout) {
  __shared__ double G[BW_NB][BW_NB], T[BW_NB][BW_NB];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nref = n - 2, j0 = blockIdx.x * BW_NB, nb = min(BW_NB, nref - j0);
  // row `warp` of the strict upper triangle of U U^T
  if (warp < nb) {
    double acc[BW_NB];
#pragma unroll
    for (int i = 0; i < BW_NB; ++i) acc[i] = 0.0;
    for (int r = j0 + 1 + lane; r < n; r += 32) {
      const int ja = j0 + warp;
      const double ua = r == ja + 1 ? 1.0 : (r > ja + 1 ? A[static_cast<int64_t>(ja) * n + r] : 0.0);
#pragma unroll
      for (int i = 1; i < BW_NB; ++i) {
        const int ji = j0 + i;
        if (i > warp && i < nb && r > ji)
          acc[i] = fma(ua, r == ji + 1 ? 1.0 : A[static_cast<int64_t>(ji) * n + r], acc[i]);
      }
    }
#pragma unroll
    for (int i = 1; i < BW_NB; ++i) {
      const double g = warp_sum(acc[i]);
      if (lane == 0) G[warp][i] = g;
    }
  }
  for (int t = threadIdx.x; t < BW_NB * BW_NB; t += 256) T[t / BW_NB][t % BW_NB] = 0.0;
  __syncthreads();
  if (warp == 0) {
    for (int i = 0; i < nb; ++i) {
      const double ti = tau[j0 + i];
      if (lane < i) {
        double sum = 0.0;
        for (int q = lane; q < i; ++q) sum = fma(T[lane][q], G[q][i], sum);
        T[lane][i] = -ti * sum;
      } else if (lane == i) {
        T[i][i] = ti;
      }
      __syncwarp();
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < BW_NB * BW_NB; t += 256)
    Tout[static_cast<int64_t>(blockIdx.x) * BW_NB * BW_NB + t] = T[t / BW_NB][t % BW_NB];
}

__global__ void __launch_bounds__(BC_THREADS) k_backtransform_cols(const double* __restrict__ A,
                                                                   const double* __restrict__ Tf, int n,
                                                                   double* __restrict__ Y, int ld) {
  constexpr int NW = BC_THREADS / 32;
  __shared__ double part[2][NW][BW_NB];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nref = n - 2, nblk = (nref + BW_NB - 1) / BW_NB;
  double y[BC_RPT], u[BW_NB][BC_RPT];
#pragma unroll
  for (int q = 0; q < BC_RPT; ++q) {
    const int r = tid + q * BC_THREADS;
    y[q] = r < n ? Y[static_cast<int64_t>(r) * ld + blockIdx.x] : 0.0;
  }
  auto load = [&](int bi) {
#pragma unroll
    for (int i = 0; i < BW_NB; ++i) {
      const int j = bi * BW_NB + i;
#pragma unroll
      for (int q = 0; q < BC_RPT; ++q) {
        const int r = tid + q * BC_THREADS;
        u[i][q] = (j < nref && r > j + 1 && r < n) ? __ldg(A + static_cast<int64_t>(j) * n + r) : 0.0;
      }
    }
  };
  load(nblk - 1);
  for (int bi = nblk - 1; bi >= 0; --bi) {
    const int j0 = bi * BW_NB;
    // lane i + 8 g: entries 2 g, 2 g + 1 of row i of T
    const int ti = lane & 7, tg = lane >> 3;
    const double t0 = __ldg(Tf + static_cast<int64_t>(bi) * 64 + ti * 8 + 2 * tg);
    const double t1 = __ldg(Tf + static_cast<int64_t>(bi) * 64 + ti * 8 + 2 * tg + 1);
    double a[BW_NB];
#pragma unroll
    for (int i = 0; i < BW_NB; ++i) {
      a[i] = 0.0;
#pragma unroll
      for (int q = 0; q < BC_RPT; ++q) {
        const int r = tid + q * BC_THREADS;
        if (r == j0 + i + 1 && j0 + i < nref) u[i][q] = 1.0;
        a[i] = fma(u[i][q], y[q], a[i]);
      }
    }
    // eight sums over the warp, halving what a lane carries: lane l ends with value l / 4
#pragma unroll
    for (int h = BW_NB / 2; h >= 1; h >>= 1) {
      const bool up = (lane & (4 * h)) != 0;
#pragma unroll
      for (int i = 0; i < h; ++i) {
        const double send = up ? a[i] : a[i + h];
        const double keep = up ? a[i + h] : a[i];
        a[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * h);
      }
    }
    double v = a[0];
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    double(*pt)[BW_NB] = part[bi & 1];
    if ((lane & 3) == 0) pt[warp][lane >> 2] = v;
    __syncthreads();
    // every warp: w_i = sum over warps (lane i + 8 g adds warps g, g + 4, ..), c = T w
    double w = 0.0;
#pragma unroll
    for (int g = 0; g < NW / 4; ++g) w += pt[tg + 4 * g][ti];
    w += __shfl_xor_sync(0xffffffffu, w, 8);
    w += __shfl_xor_sync(0xffffffffu, w, 16);
    const double wa = __shfl_sync(0xffffffffu, w, 2 * tg), wb = __shfl_sync(0xffffffffu, w, 2 * tg + 1);
    double c = fma(t0, wa, t1 * wb);
    c += __shfl_xor_sync(0xffffffffu, c, 8);
    c += __shfl_xor_sync(0xffffffffu, c, 16);
#pragma unroll
    for (int i = 0; i < BW_NB; ++i) {
      const double ci = __shfl_sync(0xffffffffu, c, i);
#pragma unroll
      for (int q = 0; q < BC_RPT; ++q) y[q] = fma(-ci, u[i][q], y[q]);
    }
    if (bi > 0) load(bi - 1);
  }
#pragma unroll
  for (int q = 0; q < BC_RPT; ++q) {
    const int r = tid + q * BC_THREADS;
    if (r < n) Y[static_cast<int64_t>(r) * ld + blockIdx.x] = y[q];
  }
}

}  // namespace

namespace {

void densify(const Exec& ex, const OpDev& op, double* A) {
  const int64_t n = op.n;
  SI_CUDA(cudaMemsetAsync(A, 0, sizeof(double) * n * n, ex.stream));
  const int grid = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, int64_t(ex.sms) * 8)));
  k_densify<<<grid, 256, 0, ex.stream>>>(n, op.indptr, op.indices, op.v64, op.diag, A);
  SI_LAUNCH_CHECK();
  k_mirror_lower<<<static_cast<int>(std::min<int64_t>((n * n + 255) / 256, int64_t(ex.sms) * 16)), 256, 0,
                   ex.stream>>>(n, A);
  SI_LAUNCH_CHECK();
}

// The multi-launch steps (three launches per column).
void tridiag_steps(const Exec& ex, double* A, int n, double* d, double* e, double* tau) {
  DevBuf<double> vbuf(n, ex.stream), wbuf(n, ex.stream), partial((n + 7) / 8, ex.stream);
  DevBuf<unsigned> counter(1, ex.stream);
  counter.zero();
  for (int j = 0; j + 2 < n; ++j) {
    const int len = n - j - 1;
    k_tri_house<<<1, 256, 0, ex.stream>>>(A, n, j, d, e, tau, vbuf.get());
    SI_LAUNCH_CHECK();
    k_tri_matvec<<<(len + 7) / 8, 256, 0, ex.stream>>>(A, n, j, tau, vbuf.get(), wbuf.get(), partial.get(),
                                                       counter.get());
    SI_LAUNCH_CHECK();
    k_tri_update<<<std::min(len, ex.sms * 8), 256, 0, ex.stream>>>(A, n, j, tau, vbuf.get(), wbuf.get());
    SI_LAUNCH_CHECK();
  }
  k_tri_last<<<1, 32, 0, ex.stream>>>(A, n, d, e, tau);
  SI_LAUNCH_CHECK();
}

// Dynamic shared memory a kernel of this file may use on a device (the
// opt-in limit less its static shared memory), with the attribute raised to
// it on first use.
template <class F>
int smem_limit(int device, F* kernel) {
  static std::mutex mu;
  static std::vector<std::pair<std::pair<int, const void*>, int>> known;
  SI_REQUIRE(device >= 0 && device < 128, SI_INVALID_ARGUMENT, "dense_evd: device ordinal");
  const void* key = reinterpret_cast<const void*>(kernel);
  std::lock_guard<std::mutex> lk(mu);
  for (const auto& kv : known)
    if (kv.first.first == device && kv.first.second == key) return kv.second;
  int smem = 0;
  SI_CUDA(cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
  cudaFuncAttributes fa{};
  SI_CUDA(cudaFuncGetAttributes(&fa, kernel));
  const int dyn = smem - static_cast<int>(fa.sharedSizeBytes);
  SI_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn));
  known.push_back({{device, key}, dyn});
  return dyn;
}

// Limit of every wait of the single-launch tridiagonalisation: 2 s, or less
// through SPECTRAL_INIT_COOP_WAIT_NS (a test seam: a limit of 0 makes the
// first wait that is not already satisfied give up, which exercises the
// recovery path -- every CTA leaves at its next wait and the multi-launch
// steps redo the matrix).
uint64_t coop_wait_limit_ns() {
  const char* v = std::getenv("SPECTRAL_INIT_COOP_WAIT_NS");
  if (v == nullptr) return kCoopWaitNs;
  char* end = nullptr;
  const unsigned long long x = std::strtoull(v, &end, 10);
  return (end != v) ? static_cast<uint64_t>(std::min<unsigned long long>(x, kCoopWaitNs)) : kCoopWaitNs;
}

// SPECTRAL_INIT_TRIDIAG=steps selects the multi-launch steps for every n
// (read on every call, so one process can exercise both paths).
bool coop_disabled() {
  const char* v = std::getenv("SPECTRAL_INIT_TRIDIAG");
  return v != nullptr && std::string(v) == "steps";
}

// Launch the single-launch tridiagonalisation if the matrix fits in the shared
// memory of co-resident CTAs; false (nothing launched) otherwise.
//   n <= 512: one cluster, as few CTAs as hold 16 rows each (one chunk of the
//   pass), 16 at most;
//   above: a cooperative launch, about 96 KB of rows per CTA (fewer CTAs leave
//   SMs to concurrent solves; the largest matrices use every SM).
bool tridiag_cluster(const Exec& ex, const CoopTri& base) {
  CoopTri p = base;
  const int n = p.n;
  p.G = 1;
  while (p.G < 16 && p.G * CT_CHUNK < n) p.G *= 2;
  p.R = ceil_div(n, p.G);
  const size_t smem =
      sizeof(double) * ((static_cast<size_t>(p.R + 1) * (n + 1) + 1) & ~size_t(1)) + sizeof(double2) * 2 * n;
  auto* kernel = k_tridiag_coop<2, true>;
  if (p.R > CT_RMAX || smem > static_cast<size_t>(smem_limit(ex.device, kernel))) return false;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(p.G);
  cfg.blockDim = dim3(CT_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ex.stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = p.G;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (p.G > 8) SI_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  int clusters = 0;
  SI_CUDA(cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg));
  if (clusters < 1) return false;
  SI_CUDA(cudaLaunchKernelEx(&cfg, kernel, p));
  SI_LAUNCH_CHECK();
  return true;
}

bool tridiag_single(const Exec& ex, double* A, int n, double* d, double* e, double* tau,
                    DevBuf<unsigned char>& work, const int** err) {
  *err = nullptr;
  if (n > kTriCoopMax || coop_disabled()) return false;
  CoopTri p{};
  p.A = A;
  p.n = n;
  p.d = d;
  p.e = e;
  p.tau = tau;
  p.wait_ns = coop_wait_limit_ns();
  if (n <= kTriClusterMax && tridiag_cluster(ex, p)) return true;
  int coop = 0;
  SI_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ex.device));
  if (!coop) return false;
  const double bytes = 8.0 * n * n;
  int G = static_cast<int>(std::ceil(bytes / (96.0 * 1024.0)));
  G = std::max(G, ceil_div(n, CT_CHUNK));
  G = std::min({G, n, ex.sms});
  const int R = ceil_div(n, G);
  G = ceil_div(n, R);
  const size_t smem = sizeof(double) * static_cast<size_t>(R) * (n + 1);
  auto* kernel = n <= 4 * CT_THREADS ? k_tridiag_coop<4, false> : k_tridiag_coop<CT_CMAX, false>;
  if (R > CT_RMAX || smem > static_cast<size_t>(smem_limit(ex.device, kernel))) return false;
  int occ = 0;
  SI_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, CT_THREADS, smem));
  if (G > occ * ex.sms) return false;
  const size_t words = sizeof(ulonglong2) * 4 * static_cast<size_t>(n);
  work.alloc(words + 128, ex.stream);  // the error word on a line of its own
  work.zero();
  p.G = G;
  p.R = R;
  p.words = reinterpret_cast<ulonglong2*>(work.get());
  p.err = reinterpret_cast<int*>(work.get() + words);
  *err = p.err;
  void* args[] = {&p};
  SI_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kernel), dim3(G), dim3(CT_THREADS), args, smem,
                                      ex.stream));
  SI_LAUNCH_CHECK();
  return true;
}

}  // namespace

void dense_evd_dev(const Exec& ex, const OpDev& op, int k, double* evals_host, double* evecs, int ld) {
  const int64_t n = op.n;
  SI_REQUIRE(n >= 1 && k >= 1 && k <= n && k <= MAXM, SI_INVALID_ARGUMENT, "dense_evd: bad sizes");
  SI_REQUIRE(op.v64 != nullptr || op.nnz == 0, SI_INVALID_ARGUMENT, "dense_evd: f64 values required");
  DevBuf<double> A(static_cast<size_t>(n) * n, ex.stream), d(n, ex.stream), e(n, ex.stream), tau(n, ex.stream),
      ev(MAXM, ex.stream);
  DevBuf<int> bstart(n + 1, ex.stream), cand_blk(static_cast<size_t>(n) * k, ex.stream), piv(n, ex.stream),
      sel_blk(MAXM + 1, ex.stream);  // the last word: whether the direct route's pairs stand
  DevBuf<double> es(n, ex.stream), e2(n, ex.stream), cand(static_cast<size_t>(n) * k, ex.stream),
      lu(5 * n, ex.stream), xv(n, ex.stream), sel_val(MAXM, ex.stream);
  TriWork w{bstart.get(), es.get(), e2.get(), cand.get(), cand_blk.get(), lu.get(), piv.get(), xv.get(), sel_blk.get(),
            sel_val.get()};
  const int ni = static_cast<int>(n);
  auto finish = [&] {
    SI_CUDA(cudaMemsetAsync(evecs, 0, sizeof(double) * n * ld, ex.stream));
    const size_t te_smem = (sizeof(double) * 9 + sizeof(int)) * static_cast<size_t>(n);
    const bool te_in_smem = te_smem <= static_cast<size_t>(smem_limit(ex.device, k_tri_eig));
    const int* skip = nullptr;
    if (n >= 2 && n <= kTriDirectMax) {
      const size_t td_smem = sizeof(double2) * (3 * static_cast<size_t>(n) + kTdPad);
      smem_limit(ex.device, k_tri_direct);
      k_tri_direct<<<k, kTdThreads, td_smem, ex.stream>>>(d.get(), e.get(), ni, ev.get(), evecs, ld);
      SI_LAUNCH_CHECK();
      k_tri_polish<<<1, kTpThreads, 0, ex.stream>>>(d.get(), e.get(), ni, k, ev.get(), evecs, ld, sel_blk.get() + MAXM);
      SI_LAUNCH_CHECK();
      skip = sel_blk.get() + MAXM;
    }
    k_tri_eig<<<1, DT, te_in_smem ? te_smem : 0, ex.stream>>>(d.get(), e.get(), ni, k, w, ev.get(), evecs, ld,
                                                              te_in_smem ? 1 : 0, skip);
    SI_LAUNCH_CHECK();
    const size_t wy_smem = sizeof(double) * static_cast<size_t>(n) * (k + BW_NB);
    if (n >= 3 && n <= kBcMax) {
      const int nblk = ceil_div(n - 2, BW_NB);
      DevBuf<double> tf(static_cast<size_t>(nblk) * BW_NB * BW_NB, ex.stream);
      k_wy_factors<<<nblk, 256, 0, ex.stream>>>(A.get(), tau.get(), ni, tf.get());
      SI_LAUNCH_CHECK();
      k_backtransform_cols<<<k, BC_THREADS, 0, ex.stream>>>(A.get(), tf.get(), ni, evecs, ld);
    } else if (n >= 3 && wy_smem <= static_cast<size_t>(smem_limit(ex.device, k_backtransform_wy))) {
      k_backtransform_wy<<<1, BW_THREADS, wy_smem, ex.stream>>>(A.get(), tau.get(), ni, evecs, ld, k);
    } else {
      k_backtransform<<<1, DT, 0, ex.stream>>>(A.get(), tau.get(), ni, evecs, ld, k);
    }
    SI_LAUNCH_CHECK();
    SI_CUDA(cudaMemcpyAsync(evals_host, ev.get(), sizeof(double) * k, cudaMemcpyDeviceToHost, ex.stream));
  };
  densify(ex, op, A.get());
  DevBuf<unsigned char> work;
  const int* err_dev = nullptr;
  if (tridiag_single(ex, A.get(), ni, d.get(), e.get(), tau.get(), work, &err_dev)) {
    finish();
    int err = 0;
    if (err_dev != nullptr)
      SI_CUDA(cudaMemcpyAsync(&err, err_dev, sizeof(int), cudaMemcpyDeviceToHost, ex.stream));
    SI_CUDA(cudaStreamSynchronize(ex.stream));
    if (err == 0) return;
    // a wait of the cooperative launch ran out: redo with the multi-launch steps
    densify(ex, op, A.get());
  }
  tridiag_steps(ex, A.get(), ni, d.get(), e.get(), tau.get());
  finish();
  SI_CUDA(cudaStreamSynchronize(ex.stream));
}

}  // namespace si
