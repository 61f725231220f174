// Small dense linear algebra in one CTA (matrices in shared memory and
// registers): Cholesky, a direct eigensolver of the wanted pairs, a parallel
// cyclic Jacobi eigensolver for what that refuses, and on top of them the
// per-iteration "small step" of block LOBPCG.
//
// LOBPCG small step (restatement of one iteration of the linfa-linalg 0.2
// LOBPCG loop that src/solvers/lobpcg.rs:327-358 calls; algorithm of Knyazev,
// SIAM J. Sci. Comput. 23(2), 2001):
//   1. residual norms of the current block from diag(R^T R) of the Gram,
//      best-iterate tracking (smallest sum of wanted residual norms), soft
//      locking (a wanted column stays locked once its norm <= tol), and the
//      convergence / iteration-cap decision;
//   2. Rayleigh-Ritz on span{X, R_active, P_active} as the generalised
//      problem (S^T A S) y = theta (S^T S) y, made well-scaled by the diagonal
//      of S^T S and reduced with a Cholesky factor; when the factor fails
//      with P present the step is retried on span{X, R_active} (the same
//      fallback as the reference iteration);
//   3. the coefficients Cx, Cr, Cp of the new X and P for the block update.
// The Gram matrices come from the fused device pass over the blocks, so the
// residuals never need an explicit orthogonalisation pass.
#include <cfloat>
#include <cstddef>
#include <cstdlib>
#include <string>

#include "si_internal.h"

namespace si {
namespace {

constexpr int ST = 128;       // threads of the small-step CTA (blocks of up to 8 columns)
constexpr int ST_WIDE = 512;  // threads of the small-step CTA for wider blocks

struct SmallSmem {
  double* A;
  double* B;
  double* V;
  double* Z;
  double* T;  // second buffer of A for the double-buffered Jacobi
  int ld;
  double* W;  // scratch of cta_tri_select (kTriWork doubles; parallel form only)
};

// Sweep stopping test of the Jacobi eigensolvers: the off-diagonal Frobenius
// mass against (4 s eps)^2 times the diagonal mass.  Rounding keeps a
// rotated s x s matrix's off-diagonal part at about eps * ||A|| per entry, so
// a test at eps^2 alone is rarely met and runs sweeps to the cap; at this
// level the eigenvalues are exact to rounding and the eigenvectors to
// s eps ||A|| / gap.
__device__ __forceinline__ double jacobi_stop2(int s) {
  const double t = 4.0 * static_cast<double>(s) * DBL_EPSILON;
  return t * t;
}

__device__ void cta_identity(double* V, int s, int ld) {
  for (int i = threadIdx.x; i < s * s; i += blockDim.x) V[(i / s) * ld + i % s] = (i / s == i % s) ? 1.0 : 0.0;
}

// In-place lower Cholesky; returns false if a pivot is <= tol.
__device__ bool cta_cholesky(double* B, int s, int ld, double tol, int* sflag) {
  for (int j = 0; j < s; ++j) {
    if (threadIdx.x == 0) {
      const double d = B[j * ld + j];
      if (!(d > tol)) {
        *sflag = 1;
      } else {
        B[j * ld + j] = sqrt(d);
        *sflag = 0;
      }
    }
    __syncthreads();
    if (*sflag) return false;
    const double piv = B[j * ld + j];
    for (int i = j + 1 + threadIdx.x; i < s; i += blockDim.x) B[i * ld + j] /= piv;
    __syncthreads();
    const int w = s - j - 1;
    for (int t = threadIdx.x; t < w * w; t += blockDim.x) {
      const int i = j + 1 + t / w, k = j + 1 + t % w;
      if (k <= i) B[i * ld + k] -= B[i * ld + j] * B[k * ld + j];
    }
    __syncthreads();
  }
  return true;
}

// M <- L^-1 M   (M: s x ncol), one thread per column.
__device__ void cta_trsm_left_lower(const double* L, double* M, int s, int ncol, int ld) {
  for (int c = threadIdx.x; c < ncol; c += blockDim.x) {
    for (int i = 0; i < s; ++i) {
      double v = M[i * ld + c];
      for (int k = 0; k < i; ++k) v -= L[i * ld + k] * M[k * ld + c];
      M[i * ld + c] = v / L[i * ld + i];
    }
  }
  __syncthreads();
}

// M <- M L^-T   (M: nrow x s), one thread per row.
__device__ void cta_trsm_right_lowerT(const double* L, double* M, int s, int nrow, int ld) {
  for (int r = threadIdx.x; r < nrow; r += blockDim.x) {
    for (int j = 0; j < s; ++j) {
      double v = M[r * ld + j];
      for (int k = 0; k < j; ++k) v -= M[r * ld + k] * L[j * ld + k];
      M[r * ld + j] = v / L[j * ld + j];
    }
  }
  __syncthreads();
}

// M <- L^-T M   (M: s x ncol), one thread per column (back substitution).
__device__ void cta_trsm_left_lowerT(const double* L, double* M, int s, int ncol, int ld) {
  for (int c = threadIdx.x; c < ncol; c += blockDim.x) {
    for (int i = s - 1; i >= 0; --i) {
      double v = M[i * ld + c];
      for (int k = i + 1; k < s; ++k) v -= L[k * ld + i] * M[k * ld + c];
      M[i * ld + c] = v / L[i * ld + i];
    }
  }
  __syncthreads();
}

__device__ double cta_sum(double v, double* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) red[w] = v;
  __syncthreads();
  double t = 0.0;
  for (int i = 0; i < static_cast<int>(blockDim.x >> 5); ++i) t += red[i];
  __syncthreads();
  return t;
}

// Scales a finite A by a power of two (exact) to a largest entry in [1, 2): the
// Jacobi iteration below forms its angles in single precision and sums squares.
// Returns the factor that takes eigenvalues back, zero where A is not finite.  A
// function of its own: part of the iteration, it cost the direct route's callers
// 2.4 us a step of 48 columns.
__device__ __noinline__ double cta_unit_scale(double* A, int s, int ld, double* red) {
  double big = 0.0;
  int bad = 0;
  for (int t = threadIdx.x; t < s * s; t += blockDim.x) {
    const double a = fabs(A[(t / s) * ld + t % s]);
    big = fmax(big, a);
    if (!(a <= DBL_MAX)) bad = 1;
  }
  big = warp_max(big);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = big;
  if (__syncthreads_or(bad)) return 0.0;
  for (int i = 0; i < static_cast<int>(blockDim.x >> 5); ++i) big = fmax(big, red[i]);
  const int ex = min(max(__double2hiint(big) >> 20, 1), 2045);  // exponent field
  const double sc = __hiloint2double((2046 - ex) << 20, 0);
  for (int t = threadIdx.x; t < s * s; t += blockDim.x) A[(t / s) * ld + t % s] *= sc;
  __syncthreads();
  return __hiloint2double(ex << 20, 0);
}

// Parallel cyclic Jacobi with one update phase per round: the round's
// disjoint rotations J are applied as A' = J^T A J and V' = V J in a single
// pass into second buffers (every element of A' depends on a 2 x 2 block of
// A), so a round is two barriers.  The rotation angle is taken in single
// precision,
//   t = h sgn(d) / (|d| + sqrt(d^2 + h^2)),  d = a_qq - a_pp, h = 2 a_pq,
//   c = 1/sqrt(1 + t^2), s = t c     (the smaller root of t^2 + 2 (d/h) t - 1),
// and (c, s) are then normalised in double precision by two Newton steps
// (c, s) *= 1.5 - (c^2 + s^2)/2, so every rotation is orthogonal to rounding:
// A and V stay exactly similar / orthogonal, and an angle off by ~1e-7 only
// leaves ~1e-7 of a_pq for the next sweep (quadratic convergence down to that
// level, then a factor ~1e-7 per sweep).  No f64 square root or division on
// the round's critical path.  On return A (diagonal) and V hold the result.
// Wants finite entries of order one (cta_unit_scale).
__device__ void cta_jacobi_db(double* A, double* V, double* A2, double* V2, int s, int ld, double* red) {
  __shared__ double al[3 * MAXM + 2], be[3 * MAXM + 2];
  __shared__ int pq[3 * MAXM + 2];
  constexpr int kItems = 9;  // per-thread update items resolved once when 2 s^2 <= 9 * threads
  const int s2 = s + (s & 1);
  const int np = s2 / 2;
  const int nitems = 2 * s * s;
  const bool pre = nitems <= kItems * static_cast<int>(blockDim.x);
  int it_i[kItems], it_j[kItems];
#pragma unroll
  for (int q = 0; q < kItems; ++q) {
    const int t = threadIdx.x + q * blockDim.x;
    const int u = t < s * s ? t : t - s * s;
    it_i[q] = u / s;
    it_j[q] = u - (u / s) * s;
  }
  double* cur = A;
  double* nxt = A2;
  double* vc = V;
  double* vn = V2;
  auto update_item = [&](int t, int i, int j) {
    if (t < s * s) {
      const int qi = pq[i], qj = pq[j];
      nxt[i * ld + j] = al[i] * (al[j] * cur[i * ld + j] + be[j] * cur[i * ld + qj]) +
                        be[i] * (al[j] * cur[qi * ld + j] + be[j] * cur[qi * ld + qj]);
    } else {
      vn[i * ld + j] = al[j] * vc[i * ld + j] + be[j] * vc[i * ld + pq[j]];
    }
  };
  for (int sweep = 0; sweep < 40; ++sweep) {
    double off = 0.0, dia = 0.0;
    for (int t = threadIdx.x; t < s * s; t += blockDim.x) {
      const int i = t / s, j = t - (t / s) * s;
      const double a = cur[i * ld + j];
      if (i == j) dia += a * a; else off += a * a;
    }
    off = cta_sum(off, red);
    dia = cta_sum(dia, red);
    if (!(off > jacobi_stop2(s) * dia)) break;
    for (int r = 0; r < s2 - 1; ++r) {
      for (int p = threadIdx.x; p < np; p += blockDim.x) {
        int a, b;
        if (p == 0) {
          a = r;
          b = s2 - 1;
        } else {
          a = (r + p) % (s2 - 1);
          b = (r - p + s2 - 1) % (s2 - 1);
        }
        if (a > b) {
          const int t = a;
          a = b;
          b = t;
        }
        double c = 1.0, sn = 0.0;
        if (b < s) {
          const double apq = cur[a * ld + b];
          const double app = cur[a * ld + a], aqq = cur[b * ld + b];
          const double tiny = DBL_EPSILON * 1e-3;
          if (fabs(apq) > 1e-300 && apq * apq > tiny * tiny * fabs(app * aqq)) {
            const float d = static_cast<float>(aqq - app), h = static_cast<float>(2.0 * apq);
            const float tf = (d >= 0.0f ? h : -h) / (fabsf(d) + sqrtf(fmaf(d, d, h * h)));
            const float cf = rsqrtf(fmaf(tf, tf, 1.0f));
            c = static_cast<double>(cf);
            sn = static_cast<double>(tf) * static_cast<double>(cf);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const double f = fma(-0.5, fma(c, c, sn * sn), 1.5);
              c *= f;
              sn *= f;
            }
          }
        }
        // new row/column a = c a - s b ; new b = s a + c b
        al[a] = c;
        be[a] = -sn;
        pq[a] = (b < s) ? b : a;
        if (b < s) {
          al[b] = c;
          be[b] = sn;
          pq[b] = a;
        }
      }
      __syncthreads();
      if (pre) {
#pragma unroll
        for (int q = 0; q < kItems; ++q) {
          const int t = threadIdx.x + q * blockDim.x;
          if (t < nitems) update_item(t, it_i[q], it_j[q]);
        }
      } else {
        for (int t = threadIdx.x; t < nitems; t += blockDim.x) {
          const int u = t < s * s ? t : t - s * s;
          update_item(t, u / s, u - (u / s) * s);
        }
      }
      __syncthreads();
      double* tmp = cur;
      cur = nxt;
      nxt = tmp;
      tmp = vc;
      vc = vn;
      vn = tmp;
    }
  }
  if (cur != A) {
    for (int t = threadIdx.x; t < s * s; t += blockDim.x) {
      const int i = t / s, j = t - (t / s) * s;
      A[i * ld + j] = cur[i * ld + j];
      V[i * ld + j] = vc[i * ld + j];
    }
  }
  __syncthreads();
}

// Parallel cyclic Jacobi (round-robin pairing): A <- diag, V <- eigenvectors
// (columns).  A is symmetric s x s; V must hold the identity on entry.
__device__ void cta_jacobi(double* A, double* V, int s, int ld, double* red, double* rc, double* rs, int* ra,
                           int* rb) {
  const int s2 = s + (s & 1);
  const int np = s2 / 2;
  // this thread's (pair, index) items of a round, resolved once per call
  constexpr int MAXIT = 12;
  int itp[MAXIT], itk[MAXIT];
  int nit = 0;
  for (int t = threadIdx.x; t < np * s && nit < MAXIT; t += blockDim.x) {
    itp[nit] = t / s;
    itk[nit] = t % s;
    ++nit;
  }
  const bool fast = np * s <= MAXIT * static_cast<int>(blockDim.x);
  for (int sweep = 0; sweep < 40 && fast; ++sweep) {
    double off = 0.0, dia = 0.0;
    for (int t = threadIdx.x; t < s * s; t += blockDim.x) {
      const int i = t / s, j = t % s;
      const double a = A[i * ld + j];
      if (i == j) dia += a * a; else off += a * a;
    }
    off = cta_sum(off, red);
    dia = cta_sum(dia, red);
    if (!(off > jacobi_stop2(s) * dia)) return;
    for (int r = 0; r < s2 - 1; ++r) {
      for (int p = threadIdx.x; p < np; p += blockDim.x) {
        int a, b;
        if (p == 0) {
          a = r;
          b = s2 - 1;
        } else {
          a = (r + p) % (s2 - 1);
          b = (r - p + s2 - 1) % (s2 - 1);
        }
        if (a > b) {
          const int t = a;
          a = b;
          b = t;
        }
        double c = 1.0, sn = 0.0;
        if (b < s) {
          const double apq = A[a * ld + b];
          const double app = A[a * ld + a], aqq = A[b * ld + b];
          if (fabs(apq) > 1e-300 && fabs(apq) > DBL_EPSILON * 1e-3 * sqrt(fabs(app * aqq))) {
            const double theta = (aqq - app) / (2.0 * apq);
            const double t = (theta >= 0.0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
            c = 1.0 / sqrt(t * t + 1.0);
            sn = t * c;
          }
        }
        rc[p] = c;
        rs[p] = sn;
        ra[p] = a;
        rb[p] = (b < s && sn != 0.0) ? b : -1;
      }
      __syncthreads();
      for (int q = 0; q < nit; ++q) {  // rows a, b
        const int p = itp[q], k = itk[q];
        const int a = ra[p], b = rb[p];
        if (b < 0) continue;
        const double x = A[a * ld + k], y = A[b * ld + k];
        A[a * ld + k] = rc[p] * x - rs[p] * y;
        A[b * ld + k] = rs[p] * x + rc[p] * y;
      }
      __syncthreads();
      for (int q = 0; q < nit; ++q) {  // columns a, b (the annihilated pair set to exact zero)
        const int p = itp[q], k = itk[q];
        const int a = ra[p], b = rb[p];
        if (b < 0) continue;
        const double x = A[k * ld + a], y = A[k * ld + b];
        A[k * ld + a] = (k == b) ? 0.0 : rc[p] * x - rs[p] * y;
        A[k * ld + b] = (k == a) ? 0.0 : rs[p] * x + rc[p] * y;
        const double vx = V[k * ld + a], vy = V[k * ld + b];
        V[k * ld + a] = rc[p] * vx - rs[p] * vy;
        V[k * ld + b] = rs[p] * vx + rc[p] * vy;
      }
      __syncthreads();
    }
  }
  if (fast) return;
  // wide problems (more items than the per-thread table holds): plain loops
  for (int sweep = 0; sweep < 40; ++sweep) {
    double off = 0.0, dia = 0.0;
    for (int t = threadIdx.x; t < s * s; t += blockDim.x) {
      const int i = t / s, j = t % s;
      const double a = A[i * ld + j];
      if (i == j) dia += a * a; else off += a * a;
    }
    off = cta_sum(off, red);
    dia = cta_sum(dia, red);
    if (!(off > jacobi_stop2(s) * dia)) break;
    for (int r = 0; r < s2 - 1; ++r) {
      for (int p = threadIdx.x; p < np; p += blockDim.x) {
        int a, b;
        if (p == 0) {
          a = r;
          b = s2 - 1;
        } else {
          a = (r + p) % (s2 - 1);
          b = (r - p + s2 - 1) % (s2 - 1);
        }
        if (a > b) {
          const int t = a;
          a = b;
          b = t;
        }
        double c = 1.0, sn = 0.0;
        if (b < s) {
          const double apq = A[a * ld + b];
          const double app = A[a * ld + a], aqq = A[b * ld + b];
          if (fabs(apq) > 1e-300 && fabs(apq) > DBL_EPSILON * 1e-3 * sqrt(fabs(app * aqq))) {
            const double theta = (aqq - app) / (2.0 * apq);
            const double t = (theta >= 0.0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
            c = 1.0 / sqrt(t * t + 1.0);
            sn = t * c;
          }
        }
        rc[p] = c;
        rs[p] = sn;
        ra[p] = a;
        rb[p] = b < s ? b : -1;
      }
      __syncthreads();
      for (int t = threadIdx.x; t < np * s; t += blockDim.x) {
        const int p = t / s, k = t % s;
        const int a = ra[p], b = rb[p];
        if (b < 0 || rs[p] == 0.0) continue;
        const double x = A[a * ld + k], y = A[b * ld + k];
        A[a * ld + k] = rc[p] * x - rs[p] * y;
        A[b * ld + k] = rs[p] * x + rc[p] * y;
      }
      __syncthreads();
      for (int t = threadIdx.x; t < np * s; t += blockDim.x) {
        const int p = t / s, k = t % s;
        const int a = ra[p], b = rb[p];
        if (b < 0 || rs[p] == 0.0) continue;
        const double x = A[k * ld + a], y = A[k * ld + b];
        A[k * ld + a] = rc[p] * x - rs[p] * y;
        A[k * ld + b] = rs[p] * x + rc[p] * y;
        const double vx = V[k * ld + a], vy = V[k * ld + b];
        V[k * ld + a] = rc[p] * vx - rs[p] * vy;
        V[k * ld + b] = rs[p] * vx + rc[p] * vy;
      }
      __syncthreads();
      // the rotation annihilates a_pq: store the exact zero (the two-phase
      // update leaves O(eps) rounding there, which would never drop below the
      // skip threshold and would keep every sweep rotating)
      for (int p = threadIdx.x; p < np; p += blockDim.x) {
        if (rb[p] >= 0 && rs[p] != 0.0) {
          A[ra[p] * ld + rb[p]] = 0.0;
          A[rb[p] * ld + ra[p]] = 0.0;
        }
      }
      __syncthreads();
    }
  }
}

// order[0..s) = indices of diag(A) ascending (stable); thread 0 only.
__device__ void sort_eigs(const double* A, int s, int ld, int* order) {
  for (int i = 0; i < s; ++i) order[i] = i;
  for (int i = 1; i < s; ++i) {
    const int v = order[i];
    const double key = A[v * ld + v];
    int j = i - 1;
    while (j >= 0 && A[order[j] * ld + order[j]] > key) {
      order[j + 1] = order[j];
      --j;
    }
    order[j + 1] = v;
  }
}

// Generalised Rayleigh-Ritz on the Gram sub-matrices selected by idx[0..s):
// (D GA D) y = theta (D GB D) y.  On success Z[0..s) x [0..nsel) holds
// D L^-T V_sel and theta_out the selected Ritz values.
__device__ bool cta_rr_general(const double* gb, const double* ga, int P, const int* idx, int s, int nsel,
                               int largest, double chol_tol, SmallSmem sm, double* dsc, double* theta_out,
                               double* red, double* rc, double* rs, int* ra, int* rb, int* order, int* sflag) {
  const int ld = sm.ld;
  for (int t = threadIdx.x; t < s * s; t += blockDim.x) {
    const int i = t / s, j = t % s;
    sm.B[i * ld + j] = gb[idx[i] * P + idx[j]];
    sm.A[i * ld + j] = ga[idx[i] * P + idx[j]];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int bad = 0;
    for (int i = 0; i < s; ++i) {
      const double d = sm.B[i * ld + i];
      if (!(d > 0.0) || !isfinite(d)) bad = 1;
      dsc[i] = (d > 0.0) ? 1.0 / sqrt(d) : 0.0;
    }
    *sflag = bad;
  }
  __syncthreads();
  if (*sflag) return false;
  for (int t = threadIdx.x; t < s * s; t += blockDim.x) {
    const int i = t / s, j = t % s;
    const double f = dsc[i] * dsc[j];
    sm.B[i * ld + j] *= f;
    sm.A[i * ld + j] *= f;
  }
  __syncthreads();
  if (!cta_cholesky(sm.B, s, ld, chol_tol, sflag)) return false;
  // A <- L^-1 A L^-T
  cta_trsm_left_lower(sm.B, sm.A, s, s, ld);
  cta_trsm_right_lowerT(sm.B, sm.A, s, s, ld);
  // symmetrise
  for (int t = threadIdx.x; t < s * s; t += blockDim.x) {
    const int i = t / s, j = t % s;
    if (i < j) {
      const double v = 0.5 * (sm.A[i * ld + j] + sm.A[j * ld + i]);
      sm.A[i * ld + j] = v;
      sm.A[j * ld + i] = v;
    }
  }
  __syncthreads();
  cta_identity(sm.V, s, ld);
  __syncthreads();
  const double unscale = cta_unit_scale(sm.A, s, ld, red);
  if (unscale == 0.0) return false;
  if (s <= 3 * MAXM) cta_jacobi_db(sm.A, sm.V, sm.T, sm.Z, s, ld, red);
  else cta_jacobi(sm.A, sm.V, s, ld, red, rc, rs, ra, rb);
  if (threadIdx.x == 0) {
    sort_eigs(sm.A, s, ld, order);
    if (largest) {
      for (int i = 0; i < s / 2; ++i) {
        const int t = order[i];
        order[i] = order[s - 1 - i];
        order[s - 1 - i] = t;
      }
    }
    for (int q = 0; q < nsel; ++q) theta_out[q] = sm.A[order[q] * ld + order[q]] * unscale;
  }
  __syncthreads();
  // Z = V[:, order[0..nsel)]
  for (int t = threadIdx.x; t < s * nsel; t += blockDim.x) {
    const int i = t / nsel, q = t % nsel;
    sm.Z[i * ld + q] = sm.V[i * ld + order[q]];
  }
  __syncthreads();
  cta_trsm_left_lowerT(sm.B, sm.Z, s, nsel, ld);
  for (int t = threadIdx.x; t < s * nsel; t += blockDim.x) {
    const int i = t / nsel, q = t % nsel;
    sm.Z[i * ld + q] *= dsc[i];
  }
  __syncthreads();
  return true;
}

// ---------------------------------------------------------------------------
// The same generalised Rayleigh-Ritz for s <= 16 in one warp, in registers:
// lane j < 16 holds column j of B (then L) and of A (then C = L^-1 A L^-T),
// lane 16 + j holds column j of the eigenvector matrix V.  Every step is
// lane-local arithmetic and warp shuffles; no CTA barrier is involved.
//   * Cholesky, right-looking: at step k lane k forms column k of L, which is
//     broadcast by shuffles, and every lane j > k updates its own column;
//   * C = L^-1 (L^-1 A)^T (A symmetric), each lane solving for its column
//     with L read from shared memory, the transpose through shared memory,
//     then symmetrised;
//   * cyclic Jacobi with the round-robin pairing of 16 columns (15 rounds of
//     8 disjoint rotations per sweep; the round and pair indices are
//     compile-time constants, so every register index is static): a lane
//     exchanges its column with its partner lane for the column rotation and
//     applies the row rotations of all 8 pairs locally.  Rotation angles as in
//     cta_jacobi_db (f32 angle, two f64 Newton normalisation steps: every
//     rotation exactly orthogonal, a_pq left at ~1e-7 of itself for the next
//     sweep, never forced to zero), the same sweep stopping test;
//   * Z = D L^-T V_sel by back substitution, one lane per selected column.
// Padded columns (j >= s) carry B = I, A = 0 and are never selected.
constexpr int WRR = 16;

__device__ __forceinline__ double sel16(const double (&a)[WRR], int i) {
  double v = a[0];
#pragma unroll
  for (int t = 1; t < WRR; ++t)
    if (t == i) v = a[t];
  return v;
}

// One Jacobi sweep over 16 columns as 15 rounds of one fixed shape: the pairs
// are always the positions (2p, 2p + 1), and after every round the content
// moves to new positions by the fixed permutation sigma of the circle method
// (the player at position p goes to sigma[p]), so that every pair of columns
// meets once per sweep and after 15 rounds every column is back where it
// started.  With fixed pair positions every register index is a compile-time
// constant while the round loop stays a runtime loop (one copy of the code).
//   lane k < 16: column of C at position k (rows indexed by position);
//   lane 16 + k: column of V at position k (rows in the original basis).
// Moving to the next round permutes C's rows (a compile-time renaming of the
// registers, C lanes only) and the columns of C and V (one shuffle per row).
__device__ __constant__ int kJacSigmaInv[16] = {2, 1, 4, 0, 6, 3, 8, 5, 10, 7, 12, 9, 14, 11, 15, 13};

__device__ __forceinline__ void warp_jacobi_sweep(double (&col)[WRR], int k, bool isv, int src_lane) {
  const unsigned full = 0xffffffffu;
#pragma unroll 1
  for (int round = 0; round < WRR - 1; ++round) {
    // rotation of the pair (k & ~1, k | 1), formed by its even C lane
    const double dkk = sel16(col, k);
    const double dqq = __shfl_xor_sync(full, dkk, 1);
    const double akq = sel16(col, k ^ 1);
    double c = 1.0, sn = 0.0;
    if (!isv && (k & 1) == 0) {
      const double app = dkk, aqq = dqq, apq = akq;
      const double tiny = DBL_EPSILON * 1e-3;
      if (fabs(apq) > 1e-300 && apq * apq > tiny * tiny * fabs(app * aqq)) {
        const float d = static_cast<float>(aqq - app), h = static_cast<float>(2.0 * apq);
        const float tf = (d >= 0.0f ? h : -h) / (fabsf(d) + sqrtf(fmaf(d, d, h * h)));
        const float cf = rsqrtf(fmaf(tf, tf, 1.0f));
        c = static_cast<double>(cf);
        sn = static_cast<double>(tf) * static_cast<double>(cf);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const double f = fma(-0.5, fma(c, c, sn * sn), 1.5);
          c *= f;
          sn *= f;
        }
      }
    }
    // column rotation: new even = c even - s odd ; new odd = s even + c odd
    const double cp = __shfl_sync(full, c, k & ~1);
    const double sp = __shfl_sync(full, sn, k & ~1);
    const bool even = (k & 1) == 0;
#pragma unroll
    for (int i = 0; i < WRR; ++i) {
      const double o = __shfl_xor_sync(full, col[i], 1);
      col[i] = even ? fma(cp, col[i], -sp * o) : fma(sp, o, cp * col[i]);
    }
    // row rotations of the 8 pairs (C lanes)
#pragma unroll
    for (int p = 0; p < WRR / 2; ++p) {
      const double cc = __shfl_sync(full, c, 2 * p);
      const double ss = __shfl_sync(full, sn, 2 * p);
      if (!isv) {
        const double x = col[2 * p], y = col[2 * p + 1];
        col[2 * p] = fma(cc, x, -ss * y);
        col[2 * p + 1] = fma(ss, x, cc * y);
      }
    }
    // next round's positions: rows of C renamed (row q takes row kJacSigmaInv[q]),
    // columns of C and V moved
    double t[WRR];
    t[0] = isv ? col[0] : col[2];
    t[1] = isv ? col[1] : col[1];
    t[2] = isv ? col[2] : col[4];
    t[3] = isv ? col[3] : col[0];
    t[4] = isv ? col[4] : col[6];
    t[5] = isv ? col[5] : col[3];
    t[6] = isv ? col[6] : col[8];
    t[7] = isv ? col[7] : col[5];
    t[8] = isv ? col[8] : col[10];
    t[9] = isv ? col[9] : col[7];
    t[10] = isv ? col[10] : col[12];
    t[11] = isv ? col[11] : col[9];
    t[12] = isv ? col[12] : col[14];
    t[13] = isv ? col[13] : col[11];
    t[14] = isv ? col[14] : col[15];
    t[15] = isv ? col[15] : col[13];
#pragma unroll
    for (int i = 0; i < WRR; ++i) col[i] = __shfl_sync(full, t[i], src_lane);
  }
}

// sh: 2 * 16 * 16 doubles of shared memory; Z (ldz) and theta_out in shared memory.
__device__ bool warp_rr_general(const double* gb, const double* ga, int P, const int* idx, int s, int nsel,
                                int largest, double chol_tol, double* Z, int ldz, double* sh, double* theta_out) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int j = lane & (WRR - 1);
  const bool isv = lane >= WRR;
  const bool live = j < s;
  // D scaling from diag(B)
  double dj = 0.0;
  int bad = 0;
  if (!isv && live) {
    const double d = gb[idx[j] * P + idx[j]];
    bad = (!(d > 0.0) || !isfinite(d)) ? 1 : 0;
    dj = d > 0.0 ? 1.0 / sqrt(d) : 0.0;
  }
  if (__any_sync(full, bad)) return false;
  double colB[WRR], col[WRR];
#pragma unroll
  for (int i = 0; i < WRR; ++i) {
    const double di = __shfl_sync(full, dj, i);
    if (!isv && live && i < s) {
      const double f = di * dj;
      colB[i] = gb[idx[i] * P + idx[j]] * f;
      col[i] = ga[idx[i] * P + idx[j]] * f;
    } else {
      colB[i] = (!isv && i == j) ? 1.0 : 0.0;
      col[i] = 0.0;
    }
  }
  // Cholesky B = L L^T (lanes 0..15; the V lanes follow the shuffles)
  int fail = 0;
#pragma unroll
  for (int k = 0; k < WRR; ++k) {
    const double pk = __shfl_sync(full, colB[k], k);
    if (k < s && !(pk > chol_tol)) fail = 1;
    const double piv = sqrt(fmax(pk, 1e-300));
    const double inv = 1.0 / piv;
    if (j == k && !isv) {
      colB[k] = piv;
#pragma unroll
      for (int i = k + 1; i < WRR; ++i) colB[i] *= inv;
    }
    double lk[WRR];
#pragma unroll
    for (int i = k + 1; i < WRR; ++i) lk[i] = __shfl_sync(full, colB[i], k);
    double ljk = 0.0;
#pragma unroll
    for (int i = k + 1; i < WRR; ++i)
      if (i == j) ljk = lk[i];
    if (!isv && j > k) {
#pragma unroll
      for (int i = k + 1; i < WRR; ++i) colB[i] = fma(-lk[i], ljk, colB[i]);
    }
  }
  if (fail) return false;
  double* Ls = sh;              // L, row-major 16 x 16 (lower part)
  double* Ts = sh + WRR * WRR;  // transpose staging
  if (!isv) {
#pragma unroll
    for (int i = 0; i < WRR; ++i) Ls[i * WRR + j] = (i >= j) ? colB[i] : 0.0;
  }
  __syncwarp();
  // Y = L^-1 A (column j), then C = L^-1 Y^T
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {
    if (!isv) {
      double y[WRR];
#pragma unroll
      for (int i = 0; i < WRR; ++i) {
        double v = col[i];
#pragma unroll
        for (int k = 0; k < i; ++k) v = fma(-Ls[i * WRR + k], y[k], v);
        y[i] = v / Ls[i * WRR + i];
      }
#pragma unroll
      for (int i = 0; i < WRR; ++i) Ts[i * WRR + j] = y[i];
    }
    __syncwarp();
    if (!isv) {
#pragma unroll
      for (int i = 0; i < WRR; ++i) col[i] = Ts[j * WRR + i];  // column j of Y^T = row j of Y
    }
    __syncwarp();
  }
  // symmetrise C (col holds row j of C)
  if (!isv) {
#pragma unroll
    for (int i = 0; i < WRR; ++i) Ts[i * WRR + j] = col[i];
  }
  __syncwarp();
  if (!isv) {
#pragma unroll
    for (int i = 0; i < WRR; ++i) col[i] = 0.5 * (col[i] + Ts[j * WRR + i]);
  } else {
#pragma unroll
    for (int i = 0; i < WRR; ++i) col[i] = (i == j) ? 1.0 : 0.0;  // V = I
  }
  __syncwarp();
  // a power of two to entries of order one, as in cta_jacobi_db
  double big = 0.0;
  bad = 0;
#pragma unroll
  for (int i = 0; i < WRR; ++i) {
    big = isv ? big : fmax(big, fabs(col[i]));
    if (!(fabs(col[i]) <= DBL_MAX)) bad = 1;
  }
  if (__any_sync(full, bad)) return false;
  big = warp_max(big);
  const int ex = min(max(__double2hiint(big) >> 20, 1), 2045);
  const double sc = __hiloint2double((2046 - ex) << 20, 0);
#pragma unroll
  for (int i = 0; i < WRR; ++i)
    if (!isv) col[i] *= sc;
  const int src_lane = (isv ? WRR : 0) + kJacSigmaInv[j];
  for (int sweep = 0; sweep < 40; ++sweep) {
    double off = 0.0, dia = 0.0;
    if (!isv) {
#pragma unroll
      for (int i = 0; i < WRR; ++i) {
        const double v = col[i] * col[i];
        if (i == j) dia += v; else off += v;
      }
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      off += __shfl_xor_sync(full, off, o);
      dia += __shfl_xor_sync(full, dia, o);
    }
    if (!(off > jacobi_stop2(s) * dia)) break;
    warp_jacobi_sweep(col, j, isv, src_lane);
  }
  // eigenvalues (the diagonal) ranked among the live columns
  const double lam = isv ? 0.0 : sel16(col, j) * __hiloint2double(ex << 20, 0);
  int rank = 0;
#pragma unroll
  for (int i = 0; i < WRR; ++i) {
    const double li = __shfl_sync(full, lam, i);
    if (i < s && live && !isv) {
      const bool before = largest ? (li > lam || (li == lam && i < j)) : (li < lam || (li == lam && i < j));
      if (before) ++rank;
    }
  }
  int* ord = reinterpret_cast<int*>(Ts);
  if (!isv && live && rank < nsel) {
    ord[rank] = j;
    theta_out[rank] = lam;
  }
  __syncwarp();
  // Z[:, q] = D L^-T V[:, ord[q]]: lane q < nsel takes column ord[q] from the V lanes
  const int src = WRR + ((lane < nsel) ? ord[lane] : 0);
  double v[WRR], dall[WRR];
#pragma unroll
  for (int i = 0; i < WRR; ++i) {
    v[i] = __shfl_sync(full, col[i], src);
    dall[i] = __shfl_sync(full, dj, i);
  }
  if (lane < nsel) {
    double z[WRR];
#pragma unroll
    for (int i = WRR - 1; i >= 0; --i) {
      double t = v[i];
#pragma unroll
      for (int k = i + 1; k < WRR; ++k) t = fma(-Ls[k * WRR + i], z[k], t);
      z[i] = t / Ls[i * WRR + i];
    }
#pragma unroll
    for (int i = 0; i < WRR; ++i)
      if (i < s) Z[i * ldz + lane] = z[i] * dall[i];
  }
  __syncwarp();
  return true;
}

// ---------------------------------------------------------------------------
// The nsel smallest (largest) eigenpairs of a symmetric s x s matrix, s <= 48,
// by the direct route: Householder tridiagonalisation, multisection of the
// wanted eigenvalues (one warp each), eigenvectors from twisted
// factorisations of T - theta (Parlett and Dhillon, "Fernando's solution to
// Wilkinson's problem", LAA 267, 1997), a symmetric (Newton-Schulz)
// orthonormalisation and the back-transformation.  The Rayleigh-Ritz step
// wants at most a third of the pairs, and a cyclic Jacobi pays about four
// sweeps of s - 1 two-barrier rounds for all of them: the chain here is s - 2
// reflectors, 11 counts and one factorisation long.  Measured (whole small
// step, B200): 12 x 12 49 -> 22 us; 16-wide blocks (up to
// 48 x 48) 493 -> 78 us on average over a solve.
//
// The result is backward stable (a computed vector is off by eps / gap along
// a neighbour, which moves the projected matrix by eps) unless two wanted
// eigenvalues agree to about 1e-14 of the norm; then the vectors come out
// nearly parallel, the orthonormality or the residual test fails and false is
// returned: the caller falls back to the Jacobi iteration.
//   A (ld): destroyed (rows keep the reflectors); V (ld): s x nsel vectors;
//   work: kTriWork doubles, 16-byte aligned; theta: nsel values, ascending (descending for
//   `largest`).
constexpr int kTriMax = 3 * MAXM;
constexpr int kTriWarps = 16;  // warps that take an eigenpair each
constexpr int kTriWork = kTriWarps * 4 * kTriMax;  // doubles of scratch

// Householder tridiagonalisation, the matrix in registers throughout.
// H_j = I - tau v v^T with v = (alpha - beta, x_{j+2}, ...) unnormalised: its
// division, tau = 1 / (beta (beta - alpha)), overlaps the product A v.  Row j
// of A receives v, d / e / tau the tridiagonal and the factors.
struct Reflector {
  double beta, v1, tau_inv;  // v1: v's first element; tau_inv = 0: H = I
};
__device__ __forceinline__ Reflector make_reflector(double alpha, double sigma) {
  Reflector r{alpha, 0.0, 0.0};
  if (sigma > 0x1p-930) {  // below, tau_inv would underflow: entries of 1e-140 are zeros here
    const double nrm = sqrt(fma(alpha, alpha, sigma));
    r.beta = alpha >= 0.0 ? -nrm : nrm;
    r.v1 = alpha - r.beta;
    r.tau_inv = -r.beta * r.v1;
  }
  return r;
}

// Up to N <= 32 columns in one warp: lane l holds column l, a[k] = A(j + k, l)
// with the rows moved up by one register per column, so that every index is
// static while the column loop stays a loop.  A column costs two round trips
// through shared memory (row j, then p = A v, each read by every lane, which
// then forms the sums, v and w itself) and no shuffle: 0.55 k cycles at 12 x
// 12 against 1.7 k with the matrix in shared memory and shuffle reductions.
template <int N>
__device__ void warp_householder(double* A, int s, int ld, double* d, double* e, double* tau, double* xs, double* ps) {
  const int l = threadIdx.x & 31;
  double a[N];
#pragma unroll
  for (int k = 0; k < N; ++k) a[k] = (k < s && l < s) ? A[k * ld + l] : 0.0;
  __syncwarp();
#pragma unroll 1
  for (int j = 0; j + 2 < s; ++j) {
    const int at = l >= j ? l - j : l - j + N;  // slot 0: the diagonal, 1: alpha, 2 ..: below; zero past the end
    if (l < N) xs[at] = l >= j ? a[0] : 0.0;
    __syncwarp();
    double v[N];
#pragma unroll
    for (int k = 0; k < N; k += 2) {
      const double2 t = *reinterpret_cast<const double2*>(xs + k);
      v[k] = t.x;
      v[k + 1] = t.y;
    }
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int k = 2; k < N; k += 2) {
      s0 = fma(v[k], v[k], s0);
      s1 = fma(v[k + 1], v[k + 1], s1);
    }
    const Reflector r = make_reflector(v[1], s0 + s1);
    const double diag = v[0];
    const bool on = r.tau_inv != 0.0;
    const double own = l == j + 1 ? r.v1 : (l > j ? a[0] : 0.0);
    const double tj = on ? 1.0 / r.tau_inv : 0.0;
    v[1] = r.v1;
    s0 = 0.0;
    s1 = 0.0;
#pragma unroll
    for (int k = 1; k + 1 < N; k += 2) {
      s0 = fma(a[k], v[k], s0);
      s1 = fma(a[k + 1], v[k + 1], s1);
    }
    s0 = fma(a[N - 1], v[N - 1], s0);
    const double p = l > j ? s0 + s1 : 0.0;
    if (l < N) ps[at] = p;
    __syncwarp();
    double w[N];
#pragma unroll
    for (int k = 0; k < N; k += 2) {
      const double2 t = *reinterpret_cast<const double2*>(ps + k);
      w[k] = t.x;
      w[k + 1] = t.y;
    }
    s0 = 0.0;
    s1 = 0.0;
#pragma unroll
    for (int k = 1; k + 1 < N; k += 2) {
      s0 = fma(w[k], v[k], s0);
      s1 = fma(w[k + 1], v[k + 1], s1);
    }
    s0 = fma(w[N - 1], v[N - 1], s0);
    // A - v w^T - w v^T with w = tau p - h v, in p: A - v (w - h v)^T - p (tau v)^T
    const double h = 0.5 * tj * tj * (s0 + s1);
    const double c1 = fma(tj, p, -2.0 * h * own), c2 = tj * own;
#pragma unroll
    for (int k = 1; k < N; ++k) a[k - 1] = fma(-v[k], c1, fma(-w[k], c2, a[k]));
    a[N - 1] = 0.0;
    if (l > j && l < s) A[j * ld + l] = on ? own : 0.0;
    if (l == 0) {
      d[j] = diag;
      e[j] = r.beta;
      tau[j] = tj;
    }
    __syncwarp();
  }
  // the last two rows: a[0], a[1] of lanes s - 2, s - 1
  if (l == s - 2) d[s - 2] = a[0];
  if (l == s - 1) {
    e[s - 2] = a[0];
    d[s - 1] = a[1];
  }
}

// Sum over the warp of four values at once: every level halves the values a
// lane carries, 6 shuffles (of doubles) for all four instead of 20.  On return
// lane l holds the sum of value ((l >> 4) & 1) * 2 + ((l >> 3) & 1).
__device__ __forceinline__ double warp_sum4(double v0, double v1, double v2, double v3, int lane) {
  const bool h = lane & 16;
  double k0 = (h ? v2 : v0) + __shfl_xor_sync(0xffffffffu, h ? v0 : v2, 16);
  const double k1 = (h ? v3 : v1) + __shfl_xor_sync(0xffffffffu, h ? v1 : v3, 16);
  const bool g = lane & 8;
  k0 = (g ? k1 : k0) + __shfl_xor_sync(0xffffffffu, g ? k0 : k1, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) k0 += __shfl_xor_sync(0xffffffffu, k0, o);
  return k0;
}

// Up to 48 columns over 16 warps: warp w holds rows w, w + 16, w + 32, lane l
// columns l and l + 32.  The warp that owns the next row forms its reflector
// and publishes it; p = A v is a row sum, v^T p a sum of one partial per warp:
// two barriers a column and few shuffles, which bound this kernel (one a cycle
// for the SM: every warp summing for itself cost 2.1 k cycles a column).
__device__ void cta_householder48(double* A, int s, int ld, double* d, double* e, double* tau, double* xs, double* ps) {
  constexpr int NW = ST_WIDE / 32;
  static_assert(3 * NW == kTriMax, "three rows a warp");
  __shared__ __align__(16) double part[NW];
  __shared__ Reflector refl;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int l1 = lane + 32;
  double a0[3], a1[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int r = warp + q * NW;
    a0[q] = (r < s && lane < s) ? A[r * ld + lane] : 0.0;
    a1[q] = (r < s && l1 < s) ? A[r * ld + l1] : 0.0;
  }
  // row r (x0, x1 on its lanes), its reflector and its diagonal entry
  auto publish = [&](int r, double x0, double x1) {
    double sq = lane > r + 1 ? x0 * x0 : 0.0;
    if (l1 > r + 1) sq = fma(x1, x1, sq);
    const double sigma = warp_sum(sq);
    const double alpha = __shfl_sync(0xffffffffu, r + 1 < 32 ? x0 : x1, (r + 1) & 31);
    const double diag = __shfl_sync(0xffffffffu, r < 32 ? x0 : x1, r & 31);
    const Reflector f = make_reflector(alpha, sigma);
    const bool on = f.tau_inv != 0.0;
    x0 = lane == r + 1 ? f.v1 : (on && lane > r ? x0 : 0.0);
    x1 = l1 == r + 1 ? f.v1 : (on && l1 > r ? x1 : 0.0);
    xs[lane] = x0;
    if (l1 < kTriMax) xs[l1] = x1;
    if (lane > r && lane < s) A[r * ld + lane] = x0;
    if (l1 > r && l1 < s) A[r * ld + l1] = x1;
    if (lane == 0) {
      refl = f;
      d[r] = diag;
      e[r] = f.beta;
    }
  };
  if (warp == 0) publish(0, a0[0], a1[0]);
  __syncthreads();
#pragma unroll 1
  for (int j = 0; j + 2 < s; ++j) {
    const double x0 = xs[lane], x1 = l1 < kTriMax ? xs[l1] : 0.0;
    const double ti = refl.tau_inv;
    const double tj = ti != 0.0 ? 1.0 / ti : 0.0;
    double vr[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) vr[q] = xs[warp + q * NW];
    const double sum = warp_sum4(fma(a0[0], x0, a1[0] * x1), fma(a0[1], x0, a1[1] * x1), fma(a0[2], x0, a1[2] * x1),
                                 0.0, lane);
    double p[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) p[q] = __shfl_sync(0xffffffffu, sum, q * 8);
    if (lane == 0) {
#pragma unroll
      for (int q = 0; q < 3; ++q) ps[warp + q * NW] = p[q];
      part[warp] = fma(p[0], vr[0], fma(p[1], vr[1], p[2] * vr[2]));  // v is zero at rows <= j
    }
    __syncthreads();
    const double q0 = ps[lane], q1 = l1 < kTriMax ? ps[l1] : 0.0;
    double h0 = 0.0, h1 = 0.0;
#pragma unroll
    for (int w = 0; w < NW; w += 2) {
      const double2 t = *reinterpret_cast<const double2*>(part + w);
      h0 += t.x;
      h1 += t.y;
    }
    const double h = 0.5 * tj * tj * (h0 + h1);  // w = tau p - h v
    // rows and columns <= j keep whatever they hold: nothing reads them again
    const double w0 = fma(tj, q0, -h * x0), w1 = fma(tj, q1, -h * x1);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const double wr = fma(tj, p[q], -h * vr[q]);
      a0[q] -= fma(vr[q], w0, wr * x0);
      a1[q] -= fma(vr[q], w1, wr * x1);
    }
    if (threadIdx.x == 0) tau[j] = tj;
    if (j + 3 < s) {
#pragma unroll
      for (int q = 0; q < 3; ++q)
        if (warp + q * NW == j + 1) publish(j + 1, a0[q], a1[q]);
      __syncthreads();
    }
  }
  // the last two rows from their owners
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int r = warp + q * NW;
    if (r == s - 2 || r == s - 1) {
      if (lane == (r & 31)) d[r] = r < 32 ? a0[q] : a1[q];
      if (r == s - 2 && lane == ((s - 1) & 31)) e[r] = s - 1 < 32 ? a0[q] : a1[q];
    }
  }
}

// Eigenvalues of T below x: sign changes of the leading minors of T - x
// (d, e2 scaled to a norm of about one; two minors a step are rescaled
// together before they could underflow).  de[i] = (d_i, e_{i-1}^2), padded
// with (2, 0), a positive pivot, to a multiple of four: four steps' loads are
// in flight before their chain of products.
__device__ __forceinline__ int tri_count_below(const double2* de, int s, double x) {
  double p0 = 0.0, p1 = 1.0;
  unsigned signs = 0;  // one bit a step, the previous step's sign in the bit above
  int cnt = 0;
  for (int i = 0; i < s; i += 4) {
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
    if (fabs(p0) < 0x1p-300 && fabs(p1) < 0x1p-300) {
      p0 *= 0x1p300;
      p1 *= 0x1p300;
    }
  }
  return cnt;
}

__device__ bool cta_tri_select(double* A, int s, int ld, int nsel, int largest, double* theta, double* V,
                               double* work) {
  __shared__ double d[kTriMax], e[kTriMax], tau[kTriMax];
  __shared__ __align__(16) double vs[kTriMax], ws[kTriMax];
  __shared__ __align__(16) double2 de[kTriMax];
  __shared__ double th[MAXM], G[MAXM * MAXM], sscale;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int nw = static_cast<int>(blockDim.x >> 5);
  const int nt = static_cast<int>(blockDim.x);
  if (nt == ST_WIDE) cta_householder48(A, s, ld, d, e, tau, vs, ws);
  else if (warp == 0 && s <= 16) warp_householder<16>(A, s, ld, d, e, tau, vs, ws);
  else if (warp == 0) warp_householder<24>(A, s, ld, d, e, tau, vs, ws);
  __syncthreads();
  // scale by a power of two (exact) to a Gershgorin bound in [1/2, 1)
  if (warp == 0) {
    double b = 0.0;
    for (int i = lane; i < s; i += 32)
      b = fmax(b, fabs(d[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < s ? fabs(e[i]) : 0.0));
    b = warp_max(b);
    // Bounds of 2^+-240 and beyond are left to the caller's Jacobi iteration: a
    // column of norm 2^256 would take tau^2 out of range, and what the reflectors
    // dropped (norms below 2^-465) is no longer nothing beside a bound of 2^-400.
    // A column whose tau^2 overflows (a norm below 2^-256 beside a bound in
    // range) leaves T without finite entries, which the tests below refuse.
    const int be = (__double2hiint(b) >> 20) & 0x7ff;
    const bool fit = be > 1023 - 240 && be < 1023 + 240;
    const int ex = fit ? be - 1022 : 0;
    const double sc = __hiloint2double((1023 - ex) << 20, 0);
    __syncwarp();
    for (int i = lane; i < ((s + 3) & ~3); i += 32) {
      const double es = (i > 0 && i < s) ? e[i - 1] * sc : 0.0;
      de[i] = i < s ? make_double2(d[i] * sc, es * es) : make_double2(2.0, 0.0);
    }
    __syncwarp();
    for (int i = lane; i < s; i += 32) {
      d[i] *= sc;
      if (i + 1 < s) e[i] *= sc;
    }
    if (lane == 0) sscale = fit ? __hiloint2double((1023 + ex) << 20, 0) : 0.0;
  }
  __syncthreads();
  // ---- eigenvalues and vectors, one warp each ----
  double2* Lp = reinterpret_cast<double2*>(work) + warp * 2 * kTriMax;  // per warp: two rows
  for (int q = warp; q < nsel; q += nw) {
    const int want = largest ? s - 1 - q : q;
    double lo = -1.0, hi = 1.0;  // the scaled spectrum lies inside
    for (int round = 0; round < 13 && hi - lo > 0.5 * DBL_EPSILON; ++round) {
      const double x = fma(hi - lo, (lane + 1) * (1.0 / 33.0), lo);
      const unsigned m = __ballot_sync(0xffffffffu, tri_count_below(de, s, x) > want);
      const int l = m ? __ffs(m) - 1 : 32;
      const double xl = __shfl_sync(0xffffffffu, x, l & 31), xp = __shfl_sync(0xffffffffu, x, (l + 31) & 31);
      if (l < 32) hi = xl;
      if (l > 0) lo = xp;
    }
    const double t = 0.5 * (lo + hi);
    // twisted factorisation: the pivots from the top (lane 0) and from the
    // bottom (lane 1) as ratios of successive minors, whose recurrences need
    // no division; out[i] = (minor before i, minor at i) in one scale
    const double tiny = 0.0625 * DBL_EPSILON * DBL_EPSILON;
    __syncwarp();
    if (lane < 2) {
      double2* out = Lp + lane * kTriMax;
      double p0 = 0.0, p1 = 1.0;
      for (int c0 = 0; c0 < s; c0 += 4) {
        double dd[4], ee[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int c = min(c0 + u, s - 1);
          dd[u] = de[lane == 0 ? c : s - 1 - c].x - t;
          ee[u] = lane == 0 ? de[c].y : (c > 0 ? de[s - c].y : 0.0);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const double p2 = fma(dd[u], p1, -ee[u] * p0);
          if (c0 + u < s) out[lane == 0 ? c0 + u : s - 1 - c0 - u] = make_double2(p1, p2);
          p0 = p1;
          p1 = p2;
        }
        if (fabs(p0) < 0x1p-300 && fabs(p1) < 0x1p-300) {
          p0 *= 0x1p300;
          p1 *= 0x1p300;
        }
      }
    }
    __syncwarp();
    double gmin = DBL_MAX;
    int kmin = 0;
    double lo_r[2], up_r[2];  // z_i = lo z_{i+1} above the twist, z_i = up z_{i-1} below
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int i = lane + 32 * c;
      lo_r[c] = 0.0;
      up_r[c] = 0.0;
      if (i < s) {
        const double2 f = Lp[i], g = Lp[kTriMax + i];
        double df = f.y / f.x, dg = g.y / g.x;
        if (!(fabs(df) >= tiny)) df = tiny;
        if (!(fabs(dg) >= tiny)) dg = tiny;
        const double gam = fabs(df + dg - (de[i].x - t));
        if (gam < gmin) {
          gmin = gam;
          kmin = i;
        }
        if (i + 1 < s) lo_r[c] = -e[i] / df;
        if (i > 0) up_r[c] = -e[i - 1] / dg;
      }
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
    // z = 1 at the twist, a running product away from it on either side (the
    // factors on the other side are one)
    double zl[2], zu[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      zl[c] = lane + 32 * c < kmin ? lo_r[c] : 1.0;
      zu[c] = lane + 32 * c > kmin && lane + 32 * c < s ? up_r[c] : 1.0;
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (c == 1 && s <= 32) break;
        const double dn = __shfl_down_sync(0xffffffffu, zl[c], o), up = __shfl_up_sync(0xffffffffu, zu[c], o);
        if (lane + o < 32) zl[c] *= dn;
        if (lane >= o) zu[c] *= up;
      }
    }
    if (s > 32) {
      zl[0] *= __shfl_sync(0xffffffffu, zl[1], 0);
      zu[1] *= __shfl_sync(0xffffffffu, zu[0], 31);
    }
    double n2 = 0.0;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      zl[c] *= zu[c];
      if (lane + 32 * c < s) n2 = fma(zl[c], zl[c], n2);
    }
    n2 = 1.0 / sqrt(warp_sum(n2));
#pragma unroll
    for (int c = 0; c < 2; ++c)
      if (lane + 32 * c < s) V[(lane + 32 * c) * ld + q] = zl[c] * n2;
    if (lane == 0) th[q] = t;
  }
  __syncthreads();
  // ---- orthonormalise: V <- V (3/2 I - G/2), quadratic in |G - I| ----
  bool fine = false;
  for (int it = 0; it < 4 && !fine; ++it) {
    int bad = 0, big = 0;
    for (int t = threadIdx.x; t < nsel * nsel; t += nt) {
      const int i = t / nsel, j = t - (t / nsel) * nsel;
      double g = 0.0;
      for (int k = 0; k < s; ++k) g = fma(V[k * ld + i], V[k * ld + j], g);
      G[t] = g;
      const double off = fabs(i == j ? g - 1.0 : g);
      if (!(off <= 8.0 * DBL_EPSILON)) bad = 1;
      if (!(off <= 0.05)) big = 1;
    }
    if (__syncthreads_or(big)) return false;
    fine = !__syncthreads_or(bad);
    if (fine) break;
    double nv[2];  // s nsel <= 2 x the CTA's threads (s = 3 nsel: 12 x 4, 24 x 8 on 128; 48 x 16 on 512)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int t = threadIdx.x + c * nt;
      nv[c] = 0.0;
      if (t < s * nsel) {
        const int k = t / nsel, i = t - (t / nsel) * nsel;
        double v = 1.5 * V[k * ld + i];
        for (int j = 0; j < nsel; ++j) v = fma(-0.5 * V[k * ld + j], G[j * nsel + i], v);
        nv[c] = v;
      }
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int t = threadIdx.x + c * nt;
      if (t < s * nsel) V[(t / nsel) * ld + t - (t / nsel) * nsel] = nv[c];
    }
    __syncthreads();
  }
  // ---- residual test in the tridiagonal basis, at what Jacobi ends with (750
  // steps of solves at 1e-10, widths 4 to 48: at most 0.7 eps) ----
  int off = fine && sscale != 0.0 ? 0 : 1;
  for (int t = threadIdx.x; t < s * nsel; t += nt) {
    const int i = t / nsel, q = t - (t / nsel) * nsel;
    double r = (d[i] - th[q]) * V[i * ld + q];
    if (i > 0) r = fma(e[i - 1], V[(i - 1) * ld + q], r);
    if (i + 1 < s) r = fma(e[i], V[(i + 1) * ld + q], r);
    if (!(fabs(r) <= 8.0 * DBL_EPSILON)) off = 1;
  }
  if (__syncthreads_or(off)) return false;
  // ---- back-transformation: eight lanes a vector, element i on lane i % 8 ----
  for (int q0 = warp * 4; q0 < nsel; q0 += nw * 4) {
    const int g = lane & 7, q = q0 + (lane >> 3);
    const bool mine = q < nsel;
    double z[kTriMax / 8];
#pragma unroll
    for (int c = 0; c < kTriMax / 8; ++c) z[c] = (mine && g + 8 * c < s) ? V[(g + 8 * c) * ld + q] : 0.0;
#pragma unroll 1
    for (int j = s - 3; j >= 0; --j) {
      double v[kTriMax / 8], t0 = 0.0, t1 = 0.0;
#pragma unroll
      for (int c = 0; c < kTriMax / 8; ++c) {
        const int i = g + 8 * c;
        v[c] = (i > j && i < s) ? A[j * ld + i] : 0.0;
        if (c & 1) t1 = fma(v[c], z[c], t1);
        else t0 = fma(v[c], z[c], t0);
      }
      t0 += t1;
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) t0 += __shfl_xor_sync(0xffffffffu, t0, o);
      t0 *= tau[j];
#pragma unroll
      for (int c = 0; c < kTriMax / 8; ++c) z[c] = fma(-t0, v[c], z[c]);
    }
#pragma unroll
    for (int c = 0; c < kTriMax / 8; ++c)
      if (mine && g + 8 * c < s) V[(g + 8 * c) * ld + q] = z[c];
    if (mine && g == 0) theta[q] = th[q] * sscale;
  }
  __syncthreads();
  return true;
}

// In-place elimination of [B | I] (B symmetric positive definite, ld) to
// M = L^-1, B = L L^T: rows in registers (warp w holds rows w + q NW, lane l
// columns l and, WIDE, l + 32; column c <= j of row i already holds L^-1 at
// pivot j, the rest the trailing matrix), the pivot row published in shared
// memory, one barrier a pivot.  False when a pivot is <= tol.
template <int NW, int RW, bool WIDE>
__device__ bool cta_inverse_cholesky(double* B, int s, int ld, double tol, double (*rowbuf)[kTriMax]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int l1 = lane + 32;
  double a0[RW], a1[RW];
#pragma unroll
  for (int q = 0; q < RW; ++q) {
    const int r = warp + q * NW;
    a0[q] = (r < s && lane < s) ? B[r * ld + lane] : 0.0;
    a1[q] = (WIDE && r < s && l1 < s) ? B[r * ld + l1] : 0.0;
  }
  if (warp == 0) {
    rowbuf[0][lane] = a0[0];
    if (WIDE && l1 < kTriMax) rowbuf[0][l1] = a1[0];
  }
  __syncthreads();
#pragma unroll 1
  for (int j = 0; j < s; ++j) {
    const double* row = rowbuf[j & 1];
    const double piv = row[j];
    if (!(piv > tol)) return false;  // the same value in every thread
    const double inv = 1.0 / piv;
    const double r0 = row[lane], r1 = WIDE && l1 < kTriMax ? row[l1] : 0.0;
#pragma unroll
    for (int q = 0; q < RW; ++q) {
      const int i = warp + q * NW;
      const double f = __shfl_sync(0xffffffffu, !WIDE || j < 32 ? a0[q] : a1[q], j & 31) * inv;
      if (i > j) {
        a0[q] = lane == j ? -f : fma(-f, r0, a0[q]);
        if (WIDE) a1[q] = l1 == j ? -f : fma(-f, r1, a1[q]);
        if (i == j + 1) {
          double* nr = rowbuf[(j + 1) & 1];
          nr[lane] = a0[q];
          if (WIDE && l1 < kTriMax) nr[l1] = a1[q];
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < RW; ++q) {
    const int i = warp + q * NW;
    const double piv = __shfl_sync(0xffffffffu, !WIDE || i < 32 ? a0[q] : a1[q], i & 31);
    if (i >= s) break;
    const double f = 1.0 / sqrt(piv);
    if (lane < s) B[i * ld + lane] = lane < i ? a0[q] * f : (lane == i ? f : 0.0);
    if (WIDE && l1 < s) B[i * ld + l1] = l1 < i ? a1[q] * f : (l1 == i ? f : 0.0);
  }
  return true;
}

// The nsel smallest (largest) eigenpairs of sm.A by the Jacobi iteration over all:
// theta_out the values, order their columns of sm.V.  False where A is not finite.
// Not inlined: it is the rare branch of a kernel that spills.
__device__ __noinline__ bool cta_jacobi_pairs(SmallSmem sm, int s, int nsel, int largest, double* theta_out, double* red,
                                              int* order) {
  const int ld = sm.ld, nt = blockDim.x;
  cta_identity(sm.V, s, ld);
  for (int t = threadIdx.x; t < s * s; t += nt) {  // C to exact symmetry
    const int i = t / s, j = t - (t / s) * s;
    if (j > i) sm.T[i * ld + j] = 0.5 * (sm.A[i * ld + j] + sm.A[j * ld + i]);
  }
  __syncthreads();
  for (int t = threadIdx.x; t < s * s; t += nt) {
    const int i = t / s, j = t - (t / s) * s;
    if (j > i) {
      sm.A[i * ld + j] = sm.T[i * ld + j];
      sm.A[j * ld + i] = sm.T[i * ld + j];
    }
  }
  __syncthreads();
  const double unscale = cta_unit_scale(sm.A, s, ld, red);
  if (unscale == 0.0) return false;  // no order: the ranks below would not cover it
  cta_jacobi_db(sm.A, sm.V, sm.T, sm.Z, s, ld, red);
  // ---- selection by ranks (ascending, or descending for `largest`; ties by index) ----
  for (int i = threadIdx.x; i < s; i += nt) {
    const double di = sm.A[i * ld + i];
    int rank = 0;
    for (int j = 0; j < s; ++j) {
      const double dj = sm.A[j * ld + j];
      // ascending and stable; for `largest` the reverse of that order
      const bool before = largest ? (dj > di || (dj == di && j > i)) : (dj < di || (dj == di && j < i));
      rank += before ? 1 : 0;
    }
    order[rank] = i;
  }
  __syncthreads();
  for (int q = threadIdx.x; q < nsel; q += nt) theta_out[q] = sm.A[order[q] * ld + order[q]] * unscale;
  __syncthreads();
  return true;
}

// The generalised Rayleigh-Ritz of cta_rr_general with its serial sections
// made parallel (rows over warps, columns over lanes: no index division): the
// D-scale factors one per thread; the elimination of [B | I] in place, one
// barrier a pivot, which leaves the unit lower L^-1 below the diagonal and the
// pivots on it, so that M = L^-1 needs no pass of its own; C = M A M^T and the
// Ritz vectors D M^T V_sel as parallel products; the wanted pairs of C by
// cta_tri_select.  Same results as cta_rr_general up to rounding.
__device__ bool cta_rr_general_par(const double* gb, const double* ga, int P, const int* idx, int s, int nsel,
                                   int largest, double chol_tol, SmallSmem sm, double* dsc, double* theta_out,
                                   double* red, int* order, int* sflag) {
  __shared__ double rowbuf[2][kTriMax];
  const int ld = sm.ld;
  const int nt = blockDim.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = nt >> 5;
  int bad = 0;
  for (int i = threadIdx.x; i < s; i += nt) {
    const double d = gb[idx[i] * (P + 1)];
    const bool ok = d > 0.0 && isfinite(d);
    if (!ok) bad = 1;
    dsc[i] = ok ? 1.0 / sqrt(d) : 0.0;
  }
  if (__syncthreads_or(bad)) return false;
  for (int i = warp; i < s; i += nw) {
    const double di = dsc[i];
    for (int j = lane; j < s; j += 32) {
      const int src = idx[i] * P + idx[j];
      const double f = di * dsc[j];
      sm.B[i * ld + j] = gb[src] * f;
      sm.A[i * ld + j] = ga[src] * f;
    }
  }
  __syncthreads();
  // ---- M = L^-1 in place of B ----
  const bool spd = nt == ST_WIDE ? cta_inverse_cholesky<ST_WIDE / 32, 3, true>(sm.B, s, ld, chol_tol, rowbuf)
                   : s <= 12     ? cta_inverse_cholesky<ST / 32, 3, false>(sm.B, s, ld, chol_tol, rowbuf)
                                 : cta_inverse_cholesky<ST / 32, 8, false>(sm.B, s, ld, chol_tol, rowbuf);
  if (!spd) return false;
  __syncthreads();
  // ---- C = M A M^T: Y = M A, kept transposed in Z with row r rotated by r
  // (both the transposed store and the row reads are free of bank conflicts),
  // then C = M Y^T, to A and to T (the copy that the direct route destroys) ----
  for (int i0 = warp; i0 < s; i0 += 3 * nw) {
    const int i1 = min(i0 + nw, s - 1), i2 = min(i0 + 2 * nw, s - 1);
    const double *m0 = sm.B + i0 * ld, *m1 = sm.B + i1 * ld, *m2 = sm.B + i2 * ld;
    double v0[2] = {0.0, 0.0}, v1[2] = {0.0, 0.0}, v2[2] = {0.0, 0.0};
    const int c0 = min(lane, s - 1), c1 = min(lane + 32, s - 1);
#pragma unroll 2
    for (int k = 0; k <= i2; ++k) {
      const double b0 = m0[k], b1 = m1[k], b2 = m2[k];
      const double a = sm.A[k * ld + c0];
      v0[0] = fma(b0, a, v0[0]);
      v1[0] = fma(b1, a, v1[0]);
      v2[0] = fma(b2, a, v2[0]);
      if (s > 32) {
        const double h = sm.A[k * ld + c1];
        v0[1] = fma(b0, h, v0[1]);
        v1[1] = fma(b1, h, v1[1]);
        v2[1] = fma(b2, h, v2[1]);
      }
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int c = lane + 32 * t;
      if (c >= s) break;
      double* z = sm.Z + c * ld;
      z[i0 + c < s ? i0 + c : i0 + c - s] = v0[t];
      if (i0 + nw < s) z[i1 + c < s ? i1 + c : i1 + c - s] = v1[t];
      if (i0 + 2 * nw < s) z[i2 + c < s ? i2 + c : i2 + c - s] = v2[t];
    }
  }
  __syncthreads();
  for (int i0 = warp; i0 < s; i0 += 3 * nw) {
    const int i1 = min(i0 + nw, s - 1), i2 = min(i0 + 2 * nw, s - 1);
    const double *m0 = sm.B + i0 * ld, *m1 = sm.B + i1 * ld, *m2 = sm.B + i2 * ld;
    double v0[2] = {0.0, 0.0}, v1[2] = {0.0, 0.0}, v2[2] = {0.0, 0.0};
    const int c0 = min(lane, s - 1), c1 = min(lane + 32, s - 1);
#pragma unroll 2
    for (int k = 0; k <= i2; ++k) {
      const double b0 = m0[k], b1 = m1[k], b2 = m2[k];
      const double y = sm.Z[k * ld + (c0 + k < s ? c0 + k : c0 + k - s)];
      v0[0] = fma(b0, y, v0[0]);
      v1[0] = fma(b1, y, v1[0]);
      v2[0] = fma(b2, y, v2[0]);
      if (s > 32) {
        const double h = sm.Z[k * ld + (c1 + k < s ? c1 + k : c1 + k - s)];
        v0[1] = fma(b0, h, v0[1]);
        v1[1] = fma(b1, h, v1[1]);
        v2[1] = fma(b2, h, v2[1]);
      }
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int c = lane + 32 * t;
      if (c >= s) break;
      sm.A[i0 * ld + c] = v0[t];
      sm.T[i0 * ld + c] = v0[t];
      if (i0 + nw < s) {
        sm.A[i1 * ld + c] = v1[t];
        sm.T[i1 * ld + c] = v1[t];
      }
      if (i0 + 2 * nw < s) {
        sm.A[i2 * ld + c] = v2[t];
        sm.T[i2 * ld + c] = v2[t];
      }
    }
  }
  __syncthreads();
  // the wanted pairs directly (T: a copy of C to destroy, Z: scratch); Jacobi
  // on C where that route does not apply or its tests fail (pairs that agree
  // to rounding)
  bool direct = false;
  if (s >= 3 && s <= (nt == ST_WIDE ? kTriMax : 24) && s * nsel <= 2 * nt) {
    direct = cta_tri_select(sm.T, s, ld, nsel, largest, theta_out, sm.V, sm.W);
  }
  if (direct) {
    for (int q = threadIdx.x; q < nsel; q += nt) order[q] = q;
    __syncthreads();
  } else {
    if (!cta_jacobi_pairs(sm, s, nsel, largest, theta_out, red, order)) return false;
  }
  // ---- Z = D M^T V_sel ----
  for (int t = threadIdx.x; t < s * nsel; t += nt) {
    const int i = t / nsel, q = t - (t / nsel) * nsel;
    const int c = order[q];
    double v = 0.0;
#pragma unroll 4
    for (int k = i; k < s; ++k) v = fma(sm.B[k * ld + i], sm.V[k * ld + c], v);
    sm.Z[i * ld + q] = v * dsc[i];
  }
  __syncthreads();
  return true;
}

// Rayleigh-Ritz of the small step: the shared-memory CTA routines (PAR: the
// parallel form, the default for the CTA kernels; on a single-warp CTA their
// barriers are warp-cheap), or, with REG, the register-resident warp version
// (SPECTRAL_INIT_SMALL_STEP=reg).
template <int NT, bool REG, bool PAR>
__device__ bool rr_general(const double* gb, const double* ga, int P, const int* idx, int s, int nsel, int largest,
                           double chol_tol, SmallSmem sm, double* dsc, double* theta_out, double* red, double* rc,
                           double* rs, int* ra, int* rb, int* order, int* sflag) {
  if constexpr (NT == 32 && REG) {
    if (s <= WRR)
      return warp_rr_general(gb, ga, P, idx, s, nsel, largest, chol_tol, sm.Z, sm.ld, sm.T, theta_out);
  }
  if constexpr (PAR) {
    if (s <= (NT == ST_WIDE ? 3 * MAXM : 32))
      return cta_rr_general_par(gb, ga, P, idx, s, nsel, largest, chol_tol, sm, dsc, theta_out, red, order, sflag);
  }
  return cta_rr_general(gb, ga, P, idx, s, nsel, largest, chol_tol, sm, dsc, theta_out, red, rc, rs, ra, rb, order,
                        sflag);
}

// `ctrl` points to the CTA's shared-memory copy of the control block's header;
// the coefficients, which the step only writes, go to `gctrl` in global memory.
template <int NT, bool REG, bool PAR>
__device__ void small_step_body(LobpcgCtrl* ctrl, LobpcgCtrl* gctrl, const double* gram, int ns, int mode,
                                double* smem) {
  __shared__ double red[ST_WIDE / 32];
  __shared__ double rc[SMAX / 2 + 1], rs[SMAX / 2 + 1], dsc[3 * MAXM], theta[MAXM], rn[MAXM];
  __shared__ int ra[SMAX / 2 + 1], rb[SMAX / 2 + 1], order[3 * MAXM], idx[3 * MAXM], inv[3 * MAXM];
  __shared__ int sflag, sdone, s_na, s_withp;
  const int LDS = 3 * MAXM;
  SmallSmem sm{smem, smem + LDS * LDS, smem + 2 * LDS * LDS, smem + 3 * LDS * LDS, smem + 4 * LDS * LDS, LDS,
               smem + 5 * LDS * LDS};
  const int m = ctrl->m;
  const int P = ns * m;
  const double* gb = gram;
  const double* ga = gram + P * P;
  if (mode == SM_ITER) {
    if constexpr (PAR) {
      // both Gram matrices to shared memory in one go, in flight with the
      // residual norms below (V and T are free until the eigensolve)
      for (int t = threadIdx.x; t < P * P; t += blockDim.x) {
        sm.V[t] = gb[t];
        sm.T[t] = ga[t];
      }
    }
    for (int c = threadIdx.x; c < m; c += blockDim.x) {
      const double g = gb[(m + c) * P + (m + c)];
      rn[c] = sqrt(g > 0.0 ? g : 0.0);
    }
  }
  if (threadIdx.x == 0) {
    sdone = ctrl->done;
    // iterations queued after convergence: the final best copy already happened
    if (sdone && mode == SM_ITER) ctrl->copy_best = 0;
  }
  __syncthreads();
  if (sdone) return;

  if (mode == SM_INIT) {
    for (int i = threadIdx.x; i < m; i += blockDim.x) idx[i] = i;
    __syncthreads();
    const bool ok = rr_general<NT, REG, PAR>(gb, ga, P, idx, m, m, ctrl->largest, ctrl->chol_tol, sm, dsc, theta, red, rc,
                                   rs, ra, rb, order, &sflag);
    if (threadIdx.x == 0) {
      ctrl->iter = 0;
      ctrl->copy_best = 0;
      ctrl->has_p = 0;
      ctrl->p_valid = 0;
      ctrl->best_sum = DBL_MAX;
      ctrl->best_iter = -1;
      ctrl->n_active = m;
      for (int c = 0; c < MAXM; ++c) ctrl->active[c] = c < m ? 1 : 0;
      if (!ok) {
        ctrl->done = 1;
        ctrl->status = ST_BREAKDOWN;
      } else {
        for (int q = 0; q < m; ++q) ctrl->lam[q] = theta[q];
      }
    }
    __syncthreads();
    if (ok) {
      for (int t = threadIdx.x; t < MAXM * MAXM; t += blockDim.x) {
        const int i = t / MAXM, q = t % MAXM;
        gctrl->Cx[t] = (i < m && q < m) ? sm.Z[i * LDS + q] : 0.0;
        gctrl->Cr[t] = 0.0;
        gctrl->Cp[t] = 0.0;
      }
    }
    return;
  }

  if (mode == SM_RR_PLAIN) {
    for (int t = threadIdx.x; t < m * m; t += blockDim.x) sm.A[(t / m) * LDS + t % m] = ga[t];
    __syncthreads();
    cta_identity(sm.V, m, LDS);
    __syncthreads();
    const double unscale = cta_unit_scale(sm.A, m, LDS, red);
    if (unscale != 0.0) cta_jacobi_db(sm.A, sm.V, sm.T, sm.Z, m, LDS, red);
    if (threadIdx.x == 0) {
      sort_eigs(sm.A, m, LDS, order);
      for (int q = 0; q < m; ++q) ctrl->lam[q] = sm.A[order[q] * LDS + order[q]] * (unscale != 0.0 ? unscale : 1.0);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < MAXM * MAXM; t += blockDim.x) {
      const int i = t / MAXM, q = t % MAXM;
      gctrl->Cx[t] = (i < m && q < m) ? sm.V[i * LDS + order[q]] : 0.0;
    }
    return;
  }

  if (mode == SM_CHOLQR) {
    for (int t = threadIdx.x; t < m * m; t += blockDim.x) sm.B[(t / m) * LDS + t % m] = gb[t];
    __syncthreads();
    const bool ok = cta_cholesky(sm.B, m, LDS, 0.0, &sflag);
    if (ok) {
      cta_identity(sm.Z, m, LDS);
      __syncthreads();
      cta_trsm_left_lowerT(sm.B, sm.Z, m, m, LDS);
    }
    for (int t = threadIdx.x; t < MAXM * MAXM; t += blockDim.x) {
      const int i = t / MAXM, q = t % MAXM;
      gctrl->Cx[t] = (ok && i < m && q < m) ? sm.Z[i * LDS + q] : 0.0;
    }
    if (threadIdx.x == 0) ctrl->status = ok ? ST_CONVERGED : ST_BREAKDOWN;
    return;
  }

  // ---- SM_ITER --------------------------------------------------------------
  if (threadIdx.x < 32) {  // warp 0, lane c = column c
    const int k = ctrl->k_wanted;
    const int c = threadIdx.x;
    const bool mine = c < m;
    double sum = 0.0;
    for (int j = 0; j < k; ++j) sum += rn[j];
    const bool copy = ctrl->best_sum > sum;
    const bool capped = ctrl->iter >= ctrl->maxiter;
    const int act = mine && (c >= k || (ctrl->active[c] && rn[c] > ctrl->tol)) ? 1 : 0;
    const unsigned am = __ballot_sync(0xffffffffu, act);
    const unsigned wanted = k < 32 ? (1u << k) - 1u : 0xffffffffu;
    const bool conv = (am & wanted) == 0u;
    if (mine) {
      ctrl->rnorm[c] = rn[c];
      ctrl->active[c] = act;
      if (copy) {
        ctrl->best_lam[c] = ctrl->lam[c];
        ctrl->best_rnorm[c] = rn[c];
      }
      idx[c] = c;
      if (act) {
        const int at = m + __popc(am & ((1u << c) - 1u));
        idx[at] = m + c;                  // R, then P, of the active columns
        idx[at + __popc(am)] = 2 * m + c;
      }
    }
    __syncwarp();
    if (c == 0) {
      if (copy) {
        ctrl->best_sum = sum;
        ctrl->best_iter = ctrl->iter;
      }
      ctrl->copy_best = copy ? 1 : 0;
      if (conv) ctrl->status = ST_CONVERGED;
      else if (capped) ctrl->status = ST_MAXITER;
      const int done = conv || capped ? 1 : 0;
      ctrl->done = done;
      sdone = done;
      if (!done) ctrl->iter += 1;
      s_na = __popc(am);
      s_withp = ctrl->p_valid;
    }
  }
  __syncthreads();
  if (sdone) return;
  const int na = s_na;
  bool ok = false;
  int withp = s_withp;
  if (withp) {
    ok = rr_general<NT, REG, PAR>(PAR ? sm.V : gb, PAR ? sm.T : ga, P, idx, m + 2 * na, m, ctrl->largest,
                                  ctrl->chol_tol, sm, dsc, theta, red, rc, rs, ra, rb, order, &sflag);
    if (!ok) withp = 0;
  }
  if (!ok) {
    ok = rr_general<NT, REG, PAR>(gb, ga, P, idx, m + na, m, ctrl->largest, ctrl->chol_tol, sm, dsc, theta, red, rc, rs, ra,
                        rb, order, &sflag);
  }
  if (!ok) {
    if (threadIdx.x == 0) {
      ctrl->done = 1;
      ctrl->status = ST_BREAKDOWN;
    }
    return;
  }
  // the coefficients of X, R, P from the rows of Z (zero for what the step left
  // out; the entries outside m x m were zeroed by the initial step)
  const int rows = m + na * (withp ? 2 : 1);
  for (int t = threadIdx.x; t < 3 * MAXM; t += blockDim.x) inv[t] = -1;
  __syncthreads();
  for (int t = threadIdx.x; t < rows; t += blockDim.x) inv[idx[t]] = t;
  __syncthreads();
  for (int t = threadIdx.x; t < 3 * m * MAXM; t += blockDim.x) {
    const int c = t / MAXM, q = t % MAXM;
    const int blk = c < m ? 0 : (c < 2 * m ? 1 : 2);
    const int row = inv[c];
    double* dst = blk == 0 ? gctrl->Cx : (blk == 1 ? gctrl->Cr : gctrl->Cp);
    if (q < m) dst[(c - blk * m) * MAXM + q] = row >= 0 ? sm.Z[row * LDS + q] : 0.0;
  }
  if (threadIdx.x == 0) {
    for (int q = 0; q < m; ++q) ctrl->lam[q] = theta[q];
    ctrl->has_p = withp;
    ctrl->p_valid = 1;
  }
}

// The control block's header is staged in shared memory for the whole step
// (the step is a long chain of small dependent updates) and written back at
// the end.
template <int NT, bool REG = false, bool PAR = false>
__global__ void __launch_bounds__(NT, 1) k_small_step(LobpcgCtrl* ctrl, const double* gram, int ns,
                                                   int mode) {
  extern __shared__ double smem[];
  __shared__ LobpcgCtrl sctrl;
  constexpr int W = offsetof(LobpcgCtrl, Cx) / sizeof(double);
  static_assert(offsetof(LobpcgCtrl, Cx) % sizeof(double) == 0, "the header must be a whole number of words");
  double* dst = reinterpret_cast<double*>(&sctrl);
  const double* src = reinterpret_cast<const double*>(ctrl);
  // complete since the previous step (the kernels between have waited for it)
  for (int i = threadIdx.x; i < W; i += blockDim.x) dst[i] = __ldcg(src + i);
  kernel_begin();
  __syncthreads();
  small_step_body<NT, REG, PAR>(&sctrl, ctrl, gram, ns, mode, smem);
  __syncthreads();
  double* back = reinterpret_cast<double*>(ctrl);
  for (int i = threadIdx.x; i < W; i += blockDim.x) back[i] = dst[i];
}

__global__ void __launch_bounds__(ST) k_small_dense(const double* __restrict__ a, int s, int mode, double* evals,
                                                    double* evecs) {
  extern __shared__ double smem[];
  __shared__ double red[ST / 32];
  __shared__ double rc[SMAX / 2 + 1], rs[SMAX / 2 + 1];
  __shared__ int ra[SMAX / 2 + 1], rb[SMAX / 2 + 1], order[SMAX];
  __shared__ int sflag;
  const int ld = SMAX;
  double* A = smem;
  double* V = smem + SMAX * SMAX;
  for (int t = threadIdx.x; t < s * s; t += blockDim.x) A[(t / s) * ld + t % s] = a[t];
  __syncthreads();
  if (mode == SM_RR_PLAIN) {
    cta_identity(V, s, ld);
    __syncthreads();
    cta_jacobi(A, V, s, ld, red, rc, rs, ra, rb);
    if (threadIdx.x == 0) {
      sort_eigs(A, s, ld, order);
      for (int q = 0; q < s; ++q) evals[q] = A[order[q] * ld + order[q]];
    }
    __syncthreads();
    for (int t = threadIdx.x; t < s * s; t += blockDim.x) {
      const int i = t / s, q = t % s;
      evecs[t] = V[i * ld + order[q]];
    }
  } else {
    const bool ok = cta_cholesky(A, s, ld, 0.0, &sflag);
    if (ok) {
      cta_identity(V, s, ld);
      __syncthreads();
      cta_trsm_left_lowerT(A, V, s, s, ld);
      for (int t = threadIdx.x; t < s * s; t += blockDim.x) evecs[t] = V[(t / s) * ld + t % s];
    }
    if (threadIdx.x == 0) evals[0] = ok ? 1.0 : 0.0;
  }
}

}  // namespace

// SPECTRAL_INIT_SMALL_STEP, read on every launch so that one process can compare
// them: serial (the CTA with one-thread-per-column triangular solves and the
// Jacobi iteration over all pairs), warp (one warp running the shared-memory
// routines, up to 16 columns), reg (one warp, register-resident Rayleigh-Ritz, up
// to 16 columns); anything else, or unset: the CTA with the direct pairs, 22 us a
// step at 12 x 12 where the others take 49 and more.
int small_step_variant() {
  const char* e = std::getenv("SPECTRAL_INIT_SMALL_STEP");
  if (e == nullptr) return 1;
  const std::string v(e);
  return v == "warp" ? 0 : (v == "reg" ? 2 : (v == "serial" ? 3 : 1));
}

void small_step_dev(const Exec& ex, LobpcgCtrl* ctrl, const double* gram, int ns, int mode, int m) {
  const int LDS = 3 * MAXM;
  const size_t smem = sizeof(double) * (5 * LDS * LDS + kTriWork);
  static std::atomic<bool> attr_set[128];
  if (ex.device >= 0 && ex.device < 128 && !attr_set[ex.device]) {
    SI_CUDA(cudaFuncSetAttribute(k_small_step<ST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem)));
    SI_CUDA(cudaFuncSetAttribute(k_small_step<ST_WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem)));
    SI_CUDA(cudaFuncSetAttribute(k_small_step<ST, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem)));
    SI_CUDA(cudaFuncSetAttribute(k_small_step<ST_WIDE, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem)));
    SI_CUDA(cudaFuncSetAttribute(k_small_step<32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem)));
    SI_CUDA(cudaFuncSetAttribute(k_small_step<32, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem)));
    attr_set[ex.device] = true;
  }
  // the Rayleigh-Ritz problem has up to ns * m rows; above 24 the CTA gets 512
  // threads (the one-warp variants take up to 16)
  const int variant = small_step_variant();
  const bool par = variant != 3;
  auto launch = [&](auto kernel, int threads) {
    launch_after(ex.stream, kernel, 1, threads, smem, ctrl, gram, ns, mode);
  };
  if (ns * m > 24) {
    if (par) launch(k_small_step<ST_WIDE, false, true>, ST_WIDE);
    else launch(k_small_step<ST_WIDE>, ST_WIDE);
  } else if (ns * m > WRR || variant == 1 || variant == 3) {
    if (par) launch(k_small_step<ST, false, true>, ST);
    else launch(k_small_step<ST>, ST);
  } else if (variant == 2) {
    launch(k_small_step<32, true>, 32);
  } else {
    launch(k_small_step<32>, 32);
  }
  SI_LAUNCH_CHECK();
}

void small_dense_dev(const Exec& ex, const double* a, int s, int mode, double* evals, double* evecs) {
  SI_REQUIRE(s >= 1 && s <= SMAX, SI_INVALID_ARGUMENT, "small_dense: size out of range");
  const size_t smem = sizeof(double) * 2 * SMAX * SMAX;
  static std::atomic<bool> attr_set[128];
  if (ex.device >= 0 && ex.device < 128 && !attr_set[ex.device]) {
    SI_CUDA(cudaFuncSetAttribute(k_small_dense, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    attr_set[ex.device] = true;
  }
  k_small_dense<<<1, ST, smem, ex.stream>>>(a, s, mode, evals, evecs);
  SI_LAUNCH_CHECK();
}

}  // namespace si
