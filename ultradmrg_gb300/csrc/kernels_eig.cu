// Batched symmetric eigen-solver of the truncated SVD (Gram matrices of the
// bond sectors and the Rayleigh-Ritz matrices of the randomized SVD).
//
// FP64 throughput per SM is low on this GPU, so the solver does as little
// FP64 work as the problem allows:
//   1. Householder reduction to tridiagonal form (n^3 FMAs; the rows stay in
//      the shared memory of one CTA, or of several co-resident ones; the
//      reflectors stay in the matrix's upper triangle);
//   2. every eigenvalue by Sturm-sequence bisection (O(n) per step and
//      eigenvalue, all eigenvalues of all matrices in parallel);
//   3. only the eigenvectors the caller needs, by inverse iteration on the
//      tridiagonal matrix (one thread per cluster of close eigenvalues;
//      modified Gram-Schmidt inside a cluster);
//   4. orthonormalisation by Newton-Schulz steps (grouped GEMMs, host side);
//   5. back-transformation by the Householder reflectors (one CTA per matrix).
// These are the textbook methods (Golub & Van Loan ch. 8; Wilkinson's
// inverse iteration; Givens' Sturm sequence), written
// for this batch layout.
#include <algorithm>
#include <cmath>

#include "svd.hpp"
#include "vecops.hpp"

namespace udmrg {

namespace {

constexpr int kTriThreads = 256;

// x 2^k by the exponent field (zero where it would leave the normal range)
__device__ __forceinline__ double exp_shift(double x, int k) {
  const int hi = __double2hiint(x), ex = ((hi >> 20) & 0x7FF) + k;
  return ex > 0 ? __hiloint2double(hi + (k << 20), __double2loint(x)) : 0.0;
}

// Number of eigenvalues of the tridiagonal (diagonal d, squared off-diagonal
// e2) below x: sign changes of the leading principal minors p_k(x) = (d_k - x)
// p_{k-1} - e2_{k-1} p_{k-2} (Givens' Sturm sequence), rescaled by their
// exponents every four steps.  Three FP64 instructions per entry instead of
// the fourteen of the quotient form's division, and a chain of one FMA; signs
// and scaling run on the integer pipes (64 sectors of a D = 2000 bond: 4.6 ->
// 1.4 ms).  A zero minor counts as a sign change and goes on as -1e-30 of its
// predecessor.  Up to 32 rows the quotients q_k = d_k - x - e2_{k-1} / q_{k-1}
// themselves (Barth, Martin and Wilkinson).  The product form is the faster one
// there too (64 matrices of 32 rows, values and vectors: 1.48 against 1.66 ms; of
// 8 rows: 0.43 against 0.47), but with the ordered reduction the quotients give a
// few-state sector's eigenvalues bit for bit, and a noised sweep adapts its noise
// by the sign of an energy difference that can be rounding alone.
constexpr int kSturmQuotient = 32;
__device__ __forceinline__ int sturm_count(const double *d, const double *e2, int n, double x) {
  if (n <= kSturmQuotient) {
    const double pivmin = 1e-290;
    int c = 0;
    double q = 0.0;
    for (int k = 0; k < n; ++k) {
      q = k == 0 ? d[0] - x : d[k] - x - e2[k - 1] / q;
      if (fabs(q) < pivmin) q = -pivmin;
      c += q < 0.0;
    }
    return c;
  }
  double p0 = 1.0, p1 = d[0] - x;
  int cnt = 0, neg = 0;
  auto sign = [&]() {  // counts the change from p0 to p1
    const int hi = __double2hiint(p1);
    if (((hi << 1) | __double2loint(p1)) == 0) {
      p1 = p0 * -1e-30;
      neg ^= 1;
      ++cnt;
    } else {
      const int s = (int)((unsigned)hi >> 31);
      cnt += s ^ neg;
      neg = s;
    }
  };
  sign();
  for (int k0 = 1; k0 < n; k0 += 4) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int k = k0 + q;
      if (k < n) {
        const double p2 = fma(d[k] - x, p1, -(e2[k - 1] * p0));
        p0 = p1;
        p1 = p2;
        sign();
      }
    }
    const int m = max(__double2hiint(p0) & 0x7FFFFFFF, __double2hiint(p1) & 0x7FFFFFFF) >> 20;
    p0 = exp_shift(p0, 1023 - m);
    p1 = exp_shift(p1, 1023 - m);
  }
  return cnt;
}

// Eigenvalues by multisection; lam[lam_off + i] (descending) = scale * value.
// A warp handles kBisectEigs eigenvalues of one job, kBisectLanes lanes each:
// per step the lanes of an eigenvalue take Sturm counts at the kBisectLanes
// interior points that cut its interval into kBisectLanes + 1 equal parts,
// and the part holding the eigenvalue is kept (a Sturm count is a
// serial chain, so points side by side shorten the chain of steps; eight lanes
// per eigenvalue fill the chip's FP64 pipes with one warp each at 2,000
// eigenvalues).
// Block b handles eigenvalues i0 .. i0 + kBisectEigs - 1 (ascending index) of
// job chunk[b].x, i0 = chunk[b].y.
// With the threshold grid of the leading-eigenvalue path (top, cnt; see
// grid_count_kernel) each eigenvalue starts from its grid cell, a factor 1.34
// wide, instead of the Gershgorin interval: up to ~40% fewer steps for the
// small eigenvalues of a Gram matrix.
constexpr int kBisectLanes = 8;
constexpr int kBisectEigs = 32 / kBisectLanes;
constexpr int kGrid = 256;             // grid points
constexpr double kGridDecades = 32.0;  // the grid spans top .. top * 1e-32
__device__ __forceinline__ double grid_point(double top, int k) {
  return top * exp10(-(double)k * kGridDecades / (kGrid - 1));
}
__global__ void __launch_bounds__(32)
    bisect_kernel(const EigJob *__restrict__ jobs, const int2 *__restrict__ chunk,
                  const double *__restrict__ d_all, const double *__restrict__ e_all,
                  const double *__restrict__ scale_all, double *__restrict__ lam_all,
                  const double *__restrict__ grid_top, const int *__restrict__ grid_cnt) {
  extern __shared__ double sm[];
  const int jb = chunk[blockIdx.x].x, i0 = chunk[blockIdx.x].y;
  const EigJob job = jobs[jb];
  const int n = job.n;
  if (n == 0) return;
  const int lane = threadIdx.x, grp = lane / kBisectLanes, k = lane % kBisectLanes;
  double *d = sm, *e = sm + n;  // e: first the off-diagonal, then its squares
  for (int i = lane; i < n; i += 32) {
    d[i] = d_all[job.lam_off + i];
    e[i] = i + 1 < n ? e_all[job.lam_off + i] : 0.0;
  }
  __syncwarp();
  // Gershgorin interval (warp reduction)
  double glo = 1e308, ghi = -1e308;
  for (int i = lane; i < n; i += 32) {
    const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < n ? fabs(e[i]) : 0.0);
    glo = fmin(glo, d[i] - r);
    ghi = fmax(ghi, d[i] + r);
  }
  for (int o = 16; o > 0; o >>= 1) {
    glo = fmin(glo, __shfl_xor_sync(0xffffffffu, glo, o));
    ghi = fmax(ghi, __shfl_xor_sync(0xffffffffu, ghi, o));
  }
  __syncwarp();
  for (int i = lane; i < n; i += 32) e[i] *= e[i];
  __syncwarp();
  const double pad = 2.2e-16 * fmax(fabs(glo), fabs(ghi)) * n + 1e-300;
  const double lo0 = glo - pad, hi0 = ghi + pad;
  const double scale = scale_all[jb];
  // absolute accuracy far below the eps * |T| the reduction itself achieves
  const double atol = 1e-18 * fmax(fabs(lo0), fabs(hi0));
  const int i = i0 + grp;  // i-th smallest
  double lo = lo0, hi = hi0;
  bool done = i >= n;
  if (grid_cnt && !done && scale > 0.0 && grid_top[0] > 0.0) {
    // cnt[k] = eigenvalues not below x_k (decreasing x_k); the first k with
    // cnt[k] >= n - i bounds eigenvalue i from below by x_k, and x_{k-1}
    // from above (the counts come from the same Sturm sequence)
    const int *cnt = grid_cnt + (int64_t)jb * (kGrid + 1);
    int k = 0;
    while (k < kGrid && cnt[k] < n - i) ++k;
    if (k < kGrid) lo = fmax(lo, grid_point(grid_top[0], k) / scale);
    if (k > 0) hi = fmin(hi, grid_point(grid_top[0], k - 1) / scale);
    if (!(lo < hi)) {  // inconsistent rounding at a cell edge: the full interval
      lo = lo0;
      hi = hi0;
    }
  }
  for (int it = 0; it < 64; ++it) {
    if (!done && hi - lo <= 4.4e-16 * fmax(fabs(lo), fabs(hi)) + atol) done = true;
    if (__all_sync(0xffffffffu, done)) break;
    const double w = (hi - lo) / (kBisectLanes + 1);
    const double x = lo + w * (k + 1);
    const bool above = !done && x > lo && x < hi && sturm_count(d, e, n, x) > i;
    const unsigned m = (__ballot_sync(0xffffffffu, above) >> (grp * kBisectLanes)) &
                       ((1u << kBisectLanes) - 1);
    if (!done) {
      // first point with more than i eigenvalues below it bounds eigenvalue i
      const int f = m ? __ffs(m) - 1 : kBisectLanes;
      const double nlo = f == 0 ? lo : lo + w * f, nhi = f == kBisectLanes ? hi : lo + w * (f + 1);
      if (nlo <= lo && nhi >= hi) {
        done = true;  // no representable point inside the interval
      } else {
        lo = nlo;
        hi = nhi;
      }
    }
  }
  if (i < n && k == 0) lam_all[job.lam_off + (n - 1 - i)] = scale * 0.5 * (lo + hi);
}

// ---- leading eigenvalues only (positive semi-definite jobs) ----
//
// A truncated SVD keeps at most Dmax states of all bond sectors together, and
// the weight of the discarded ones follows from each Gram matrix's trace, so
// only the leading eigenvalues of every sector need bisection.  A common
// threshold is read off Sturm counts at a logarithmic grid of points below
// the largest Gershgorin bound of all jobs.
// top[0] = max over jobs of scale * (Gershgorin upper bound of its tridiagonal)
__global__ void grid_top_kernel(const EigJob *__restrict__ jobs, int nj,
                                const double *__restrict__ d_all, const double *__restrict__ e_all,
                                const double *__restrict__ scale_all, double *__restrict__ top) {
  __shared__ double red[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  double m = 0.0;
  for (int q = warp; q < nj; q += nwarp) {
    const EigJob job = jobs[q];
    const int n = job.n;
    const double *d = d_all + job.lam_off, *e = e_all + job.lam_off;
    double h = 0.0;
    for (int i = lane; i < n; i += 32)
      h = fmax(h, d[i] + (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < n ? fabs(e[i]) : 0.0));
    for (int o = 16; o > 0; o >>= 1) h = fmax(h, __shfl_down_sync(0xffffffffu, h, o));
    if (lane == 0) m = fmax(m, scale_all[q] * h);
  }
  if (lane == 0) red[warp] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < nwarp; ++w) t = fmax(t, red[w]);
    top[0] = t;
  }
}

// cnt[q * (kGrid + 1) + k] = number of eigenvalues of job q not below
// x_k = top * 10^(-k * kGridDecades / (kGrid - 1)) for k < kGrid, and n for
// k = kGrid; tr[q] = scale * sum of the diagonal (the trace).  One block per
// job, one grid point per thread.
__global__ void grid_count_kernel(const EigJob *__restrict__ jobs,
                                  const double *__restrict__ d_all,
                                  const double *__restrict__ e_all,
                                  const double *__restrict__ scale_all,
                                  const double *__restrict__ top, int *__restrict__ cnt,
                                  double *__restrict__ tr) {
  extern __shared__ double sm[];
  __shared__ double pm;
  const int q = blockIdx.x;
  const EigJob job = jobs[q];
  const int n = job.n;
  double *d = sm, *e = sm + n;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    d[i] = d_all[job.lam_off + i];
    const double x = i + 1 < n ? e_all[job.lam_off + i] : 0.0;
    e[i] = x * x;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    double t = 0.0;
    for (int i = threadIdx.x; i < n; i += 32) t += d[i];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (threadIdx.x == 0) pm = t;
  }
  __syncthreads();
  const double sc = scale_all[q];
  if (threadIdx.x == 0) tr[q] = sc * pm;
  for (int k = threadIdx.x; k <= kGrid; k += blockDim.x) {
    int c;
    if (k == kGrid || n == 0) {
      c = n;
    } else if (sc <= 0.0 || top[0] <= 0.0) {
      c = 0;  // a zero matrix: no eigenvalue reaches x_k > 0
    } else {
      c = n - sturm_count(d, e, n, grid_point(top[0], k) / sc);
    }
    cnt[(int64_t)q * (kGrid + 1) + k] = c;
  }
}

__device__ __forceinline__ double start_entry(uint64_t seed, int i) {
  uint64_t z = seed + 0x9E3779B97F4A7C15ull * (uint64_t)(i + 1);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return (double)(z >> 11) * (2.0 / 9007199254740992.0) - 1.0;
}

// Inverse iteration: one thread per cluster of eigenvalues (descending
// positions first .. first+count-1 of job `job`), each eigenvector found with
// an LU factorisation (partial pivoting) of T - lambda I and three solves,
// orthogonalised against the cluster's earlier vectors (modified
// Gram-Schmidt).  Vector of position p goes to column p of Z (row-major
// n x ld at z_off).  Work arrays are interleaved by thread (coalesced).
//
// Bound: a serial chain of about 40 FP64 instructions per row, 64 clocks each
// (a few hundred warps cannot fill the chip).  The factors of eight rows are
// loaded together, ahead of the recurrences that use them, so the chain does
// not wait for L2; two divisions per row (a multiplier from the pivot's reciprocal
// would be rounded twice); the norm is summed from the first row on, its factor
// applied by the next pass.
constexpr int kInvB = 8;
__global__ void __launch_bounds__(32)
    invit_kernel(const EigCluster *__restrict__ cl, int ncl, const EigJob *__restrict__ jobs,
                 const double *__restrict__ d_all, const double *__restrict__ e_all,
                 const double *__restrict__ scale_all, const double *__restrict__ lam_all,
                 double *__restrict__ Z, double *__restrict__ work, int nmax) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ncl) return;
  const EigCluster c = cl[t];
  const EigJob job = jobs[c.job];
  const int n = job.n;
  const double *d = d_all + job.lam_off, *e = e_all + job.lam_off;
  const int64_t T = ncl, A = (int64_t)nmax * T;
  // l: multipliers (an interchange in the lowest bit of pv), u0: reciprocal
  // diagonal of U, u1, u2: its superdiagonals, y: the vector
  double *l = work + t, *u0 = l + A, *u1 = u0 + A, *u2 = u1 + A, *y = u2 + A, *pv = y + A;
  double tnorm = 0.0;
  for (int i = 0; i < n; ++i)
    tnorm = fmax(tnorm, fabs(d[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0) +
                            (i + 1 < n ? fabs(e[i]) : 0.0));
  const double tiny = 2.2e-16 * (tnorm > 0.0 ? tnorm : 1.0);  // zero matrix: any basis
  const double inv_scale = scale_all[c.job] > 0.0 ? 1.0 / scale_all[c.job] : 0.0;
  double *zc = Z + c.z_off;
  for (int k = 0; k < c.count; ++k) {
    const int p = c.first + k;
    const double lam = lam_all[job.lam_off + p] * inv_scale;
    if (n == 1) {
      zc[p] = 1.0;
      continue;
    }
    // LU of T - lam I with row interchanges: row i of U holds u0 (the
    // reciprocal of the diagonal, kept away from zero), u1, u2 (the two
    // superdiagonals); l the multipliers; pv the interchanges
    auto rinv = [&](double v) {
      return 1.0 / (fabs(v) > tiny ? v : (v < 0 ? -tiny : tiny));
    };
    double a = d[0] - lam, b = e[0];
    double sub = e[0], dn = d[1], sup = n > 2 ? e[1] : 0.0;
    for (int i = 0; i + 1 < n; ++i) {
      const double s0 = sub, dl = dn - lam, s1 = sup;
      if (i + 2 < n) {  // the next row's entries
        sub = s1;
        dn = d[i + 2];
        sup = i + 3 < n ? e[i + 2] : 0.0;
      }
      const bool keep = fabs(a) >= fabs(s0);
      const double r = rinv(keep ? a : s0);
      const double f = (keep ? s0 : a) / (keep ? (a != 0.0 ? a : tiny) : s0);
      const int64_t at = i * T;
      u0[at] = r;
      u1[at] = keep ? b : dl;
      u2[at] = keep ? 0.0 : s1;
      l[at] = f;
      pv[at] = keep ? 0.0 : 1.0;
      a = keep ? fma(-f, b, dl) : fma(-f, dl, b);
      b = keep ? s1 : -f * s1;
    }
    u0[(n - 1) * T] = rinv(a);
    const uint64_t seed = c.seed + 7919ull * (uint64_t)p;
    double fac = 1.0;  // factor of the stored y still to be applied
    for (int it = 0; it < 3; ++it) {
      // forward: apply the interchanges and multipliers
      double cur = it == 0 ? start_entry(seed, 0) : y[0] * fac;
      for (int i0 = 0; i0 + 1 < n; i0 += kInvB) {
        double lv[kInvB], pq[kInvB], yv[kInvB];
#pragma unroll
        for (int q = 0; q < kInvB; ++q) {
          const int i = i0 + q;
          if (i + 1 < n) {
            lv[q] = l[i * T];
            pq[q] = pv[i * T];
            yv[q] = it == 0 ? start_entry(seed, i + 1) : y[(i + 1) * T];
          }
        }
#pragma unroll
        for (int q = 0; q < kInvB; ++q) {
          const int i = i0 + q;
          if (i + 1 < n) {
            const double nx = it == 0 ? yv[q] : yv[q] * fac;
            const bool sw = __double2hiint(pq[q]) != 0;
            const double top = sw ? nx : cur, bot = sw ? cur : nx;
            y[i * T] = top;
            cur = fma(-lv[q], top, bot);
          }
        }
      }
      // back substitution with U
      double y1 = cur * u0[(n - 1) * T], y2 = 0.0;
      y[(n - 1) * T] = y1;
      for (int i0 = n - 2; i0 >= 0; i0 -= kInvB) {
        double av[kInvB], bv[kInvB], cv[kInvB], yv[kInvB];
#pragma unroll
        for (int q = 0; q < kInvB; ++q) {
          const int i = i0 - q;
          if (i >= 0) {
            av[q] = u0[i * T];
            bv[q] = u1[i * T];
            cv[q] = u2[i * T];
            yv[q] = y[i * T];
          }
        }
#pragma unroll
        for (int q = 0; q < kInvB; ++q) {
          const int i = i0 - q;
          if (i >= 0) {
            const double s = fma(-cv[q], y2, fma(-bv[q], y1, yv[q])) * av[q];
            y[i * T] = s;
            y2 = y1;
            y1 = s;
          }
        }
      }
      // orthogonalise against the cluster's earlier vectors
      for (int q = c.first; q < p; ++q) {
        double s = 0.0;
        for (int i = 0; i < n; ++i) s += zc[(int64_t)i * c.ld + q] * y[i * T];
        for (int i = 0; i < n; ++i) y[i * T] -= s * zc[(int64_t)i * c.ld + q];
      }
      double nrm = 0.0;
#pragma unroll 8
      for (int i = 0; i < n; ++i) nrm = fma(y[i * T], y[i * T], nrm);
      nrm = sqrt(nrm);
      fac = nrm > 0.0 ? 1.0 / nrm : 0.0;
    }
#pragma unroll 8
    for (int i = 0; i < n; ++i) zc[(int64_t)i * c.ld + p] = y[i * T] * fac;
  }
}

// Back transformation: Z (row-major n x k, leading dimension ld, at z_off)
// <- Q Z with Q = H_0 H_1 ... H_{n-3}, H_j = I - tau_j v_j v_j^T acting on
// rows j+1 ...  Block b transforms columns c0 .. c0 + cw - 1 of job
// bt[b].job (columns are independent).
struct BackChunk {
  int64_t z_off, ld;
  int32_t job, c0, cw, pad;
};


__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cmulc(double2 a, double2 b) {  // conj(a) * b
  return make_double2(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) {
  return make_double2(a.x + b.x, a.y + b.y);
}

// ---- Householder tridiagonalisation of one large matrix by several CTAs ----
//
// A matrix too large for one SM's shared memory is reduced by P co-resident
// CTAs (a cooperative launch): CTA p owns the rows i with i % P == p and keeps
// them in its shared memory (in the global matrix where they do not fit).
// Step j uses the reflector v_j of row j and w_j = t_j A v_j - K v_j; one fused
// pass over each CTA's own rows applies the rank-2 update of step j and forms
// the matrix-vector product of step j + 1, and the owner of the next pivot row
// publishes it.  Per step the CTAs meet once, at a counter barrier; then every
// CTA reads w_j's entries, the partial sums and the pivot row together, applies
// step j's update to that row (the same arithmetic in every CTA) and forms the
// next reflector.  The barrier gives up after kTriTimeoutNs and sets status 3.
// Partial sums are added in CTA order, so the result does not depend on timing.
//
// A matrix of at most tri_one() rows is one CTA's, and ordered: every sum and
// every entry's update has the order of a row per warp (32 interleaved chains and
// their tree), whatever the lanes that compute it, and nothing fused across the
// two terms of an update.  A Gram matrix's small sectors hold kept vectors whose
// eigenvalue is near the rounding of the largest (a 9 x 9 one with s_7 / s_1 =
// 5e-6: 4e-6 of the vector), so a state's small parts follow this kernel's last
// bit.  Costs four FP64 instructions per entry and step instead of three.
//
// Bound: 3 m^2 FP64 FMAs per step at two per clock and SM (n^3 in all, shared
// out over the CTAs), plus about 5.5 us per step of barrier, L2 and scalar
// latency.  A warp's FP64 instruction holds its quarter's pipe for
// 64 clocks, so a warp takes four rows at a time with eight lanes each (their
// sums reduced by three additions) and nothing scalar is computed by more than
// one warp.
struct TriPart {
  int32_t job, p, P, slot;
  int64_t wb_off;  // 4 n scalars: w entries and pivot rows (double-buffered by step parity)
  int64_t part_off;  // slice sums in the w buffer (-1: in shared memory)
  int32_t resident, ordered;  // the own rows are kept in shared memory; one CTA, fixed order
};
struct TriSlot {  // one per matrix, zeroed before the launch
  unsigned int arrive;
  int pad[3];
};
constexpr int kTriMaxParts = 64;
constexpr unsigned long long kTriTimeoutNs = 2000000000ull;

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ double cj(double a) { return a; }
__device__ __forceinline__ double2 cj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double smul(double a, double b) { return a * b; }
__device__ __forceinline__ double2 smul(double2 a, double2 b) { return cmul(a, b); }
__device__ __forceinline__ double sadd(double a, double b) { return a + b; }
__device__ __forceinline__ double2 sadd(double2 a, double2 b) { return cadd(a, b); }
__device__ __forceinline__ double ssub(double a, double b) { return a - b; }
__device__ __forceinline__ double2 ssub(double2 a, double2 b) {
  return make_double2(a.x - b.x, a.y - b.y);
}
// s + a x and s - a x.  Complex data form the product first: two fused steps
// would round at s's size twice (measured: a third more error in a ladder SVD).
__device__ __forceinline__ double smadd(double s, double a, double x) { return fma(a, x, s); }
__device__ __forceinline__ double2 smadd(double2 s, double2 a, double2 x) {
  return cadd(s, cmul(a, x));
}
__device__ __forceinline__ double smsub(double s, double a, double x) { return fma(-a, x, s); }
__device__ __forceinline__ double2 smsub(double2 s, double2 a, double2 x) {
  const double2 p = cmul(a, x);
  return make_double2(s.x - p.x, s.y - p.y);
}
// a - v w - u x, the rank-2 update of one entry.  Complex data form the products'
// sum first: four fused subtractions would round at a's size four times
// (measured: twice the error of a ladder SVD's state).
__device__ __forceinline__ double rank2(double a, double v, double w, double u, double x) {
  return fma(-u, x, fma(-v, w, a));
}
__device__ __forceinline__ double2 rank2(double2 a, double2 v, double2 w, double2 u, double2 x) {
  const double2 p = cadd(cmul(v, w), cmul(u, x));
  return make_double2(a.x - p.x, a.y - p.y);
}
// The same in the fixed order: a - (v w + u x), real data with the first product
// fused into the second's rounding, complex data (a - v w) - u x.
__device__ __forceinline__ double rank2_ordered(double a, double v, double w, double u, double x) {
  return __dsub_rn(a, fma(v, w, __dmul_rn(u, x)));
}
__device__ __forceinline__ double2 rank2_ordered(double2 a, double2 v, double2 w, double2 u,
                                                 double2 x) {
  const double2 p = cmul(v, w), q = cmul(u, x);
  return make_double2(a.x - p.x - q.x, a.y - p.y - q.y);
}
__device__ __forceinline__ double sinv(double a) { return 1.0 / a; }
__device__ __forceinline__ double2 sinv(double2 a) {
  const double dd = a.x * a.x + a.y * a.y;
  return make_double2(a.x / dd, -a.y / dd);
}
__device__ __forceinline__ double sre(double a) { return a; }
__device__ __forceinline__ double sre(double2 a) { return a.x; }
__device__ __forceinline__ double sim(double) { return 0.0; }
__device__ __forceinline__ double sim(double2 a) { return a.y; }
__device__ __forceinline__ double sabs2(double a) { return a * a; }
__device__ __forceinline__ double sabs2(double2 a) { return a.x * a.x + a.y * a.y; }
__device__ __forceinline__ double samax(double a) { return fabs(a); }
__device__ __forceinline__ double samax(double2 a) { return fmax(fabs(a.x), fabs(a.y)); }
__device__ __forceinline__ bool sfinite(double a) { return isfinite(a); }
__device__ __forceinline__ bool sfinite(double2 a) { return isfinite(a.x) && isfinite(a.y); }
template <typename T> __device__ __forceinline__ T smake(double re, double im);
template <> __device__ __forceinline__ double smake<double>(double re, double) { return re; }
template <> __device__ __forceinline__ double2 smake<double2>(double re, double im) {
  return make_double2(re, im);
}
__device__ __forceinline__ double sscale(double s, double a) { return s * a; }
__device__ __forceinline__ double2 sscale(double s, double2 a) {
  return make_double2(s * a.x, s * a.y);
}
__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double2 warp_sum(double2 v) {
  return make_double2(warp_sum(v.x), warp_sum(v.y));
}

// Sum over each group of eight lanes.
__device__ __forceinline__ double oct_sum(double v) {
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  return v + __shfl_xor_sync(0xffffffffu, v, 1);
}
__device__ __forceinline__ double2 oct_sum(double2 v) {
  return make_double2(oct_sum(v.x), oct_sum(v.y));
}

// All CTAs of the matrix arrive; false (status 3) if the others do not
// arrive within the time limit.  The release of one thread covers the block's
// writes (ordered before it by the block barrier), the acquire the reads after.
__device__ bool tri_barrier(TriSlot *sl, int P, unsigned target, int *status) {
  __shared__ int ok;
  __syncthreads();
  if (P == 1) return true;
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&sl->arrive) : "memory");
    int good = 1;
    unsigned long long t0 = 0;
    for (unsigned spin = 0;; ++spin) {
      unsigned got;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(got) : "l"(&sl->arrive) : "memory");
      if (got >= target) break;
      if ((spin & 63) == 63) {
        const unsigned long long t = global_ns();
        if (t0 == 0) t0 = t;
        if (t - t0 > kTriTimeoutNs) {
          good = 0;
          atomicExch(status, 3);
          break;
        }
      }
    }
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

// Leading dimension of resident rows: four rows by eight lanes of a warp fall
// into different shared-memory banks where it is 8 modulo 16 doubles.
template <typename T>
__host__ __device__ constexpr int tri_ld(int n) {
  return sizeof(T) == 8 ? (n + 7) / 16 * 16 + 8 : (n | 1);
}
// Largest matrix of the ordered one-CTA reduction (square and two rows within
// 200 KB; the resident rows then fit an SM).
template <typename T>
__host__ __device__ constexpr int tri_one() {
  return sizeof(T) == 8 ? 159 : 112;
}
// Slice sums of the row pass: one per own row of the full rounds, at most eight
// for each of the 4 x 7 rows left over.
__host__ __device__ constexpr int tri_parts(int n, int P) { return 224 + (n + P - 1) / P + 4; }

template <typename T>
__global__ void __launch_bounds__(kTriThreads)
    tridiag_mc_kernel(const EigJob *__restrict__ jobs, const TriPart *__restrict__ parts,
                      T *__restrict__ G_all, double *__restrict__ d_all,
                      double *__restrict__ e_all, T *__restrict__ tau_all,
                      double *__restrict__ scale_all, TriSlot *__restrict__ slots,
                      T *__restrict__ wbuf_all, T *__restrict__ red_all,
                      int *__restrict__ status) {
  extern __shared__ __align__(16) unsigned char tri_sm[];
  __shared__ double red[33];
  __shared__ T sh_k, sh_t, sh_sc;
  __shared__ T wpart[kTriThreads / 32];
  const TriPart pt = parts[blockIdx.x];
  const EigJob job = jobs[pt.job];
  const int n = job.n, p = pt.p, P = pt.P;
  TriSlot *sl = slots + pt.slot;
  T *A = G_all + job.g_off;
  T *wb = wbuf_all + pt.wb_off;      // w entries, two buffers by step parity
  T *pb = wb + 2 * (int64_t)n;       // published pivot rows, likewise
  T *rd = red_all + (int64_t)pt.slot * 2 * kTriMaxParts;
  double *d = d_all + job.lam_off, *e = e_all + job.lam_off;
  T *tau = tau_all + job.lam_off;
  T *vA = (T *)tri_sm, *vB = vA + n, *wA = vB + n, *rb = wA + n;  // rb: the next pivot row
  T *part = pt.part_off < 0 ? rb + n : wbuf_all + pt.part_off;
  const int kown = p < n ? (n - p + P - 1) / P : 0;  // own rows p, p + P, ...
  T *rows = pt.resident ? rb + n + tri_parts(n, P) : A + (int64_t)p * n;
  const int64_t rld = pt.resident ? tri_ld<T>(n) : (int64_t)P * n;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const int nwarp = nt >> 5;
  const bool ordered = pt.ordered != 0;
  // the thread's first vector entry: the ordered sums start at entry 2
  const int r0 = ordered ? (tid + 2) & (kTriThreads - 1) : tid;
  unsigned nbar = 0;

  // 1. max-abs and finiteness of the upper triangle of the own rows; partials
  //    in the w buffer
  double mx = 0.0;
  int nf = 0;
  for (int k = warp; k < kown; k += nwarp) {
    const int i = p + k * P;
    for (int c = i + lane; c < n; c += 32) {
      const T g = A[(int64_t)i * n + c];
      nf |= !sfinite(g);
      mx = fmax(mx, samax(g));
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, o));
    nf |= __shfl_down_sync(0xffffffffu, nf, o);
  }
  __syncthreads();
  if (lane == 0) red[warp] = nf ? -1.0 : mx;
  __syncthreads();
  double *pw = (double *)wb;  // 2 P doubles (P <= n / 4)
  if (tid == 0) {
    double m = 0.0;
    int bad = 0;
    for (int i = 0; i < nwarp; ++i) {
      bad |= red[i] < 0.0;
      m = fmax(m, red[i]);
    }
    pw[p] = m;
    pw[P + p] = bad;
  }
  if (!tri_barrier(sl, P, ++nbar * P, status)) return;
  if (warp == 0) {
    double m = 0.0;
    int bad = 0;
    for (int q = lane; q < P; q += 32) {
      m = fmax(m, __ldcg(&pw[q]));
      bad |= __ldcg(&pw[P + q]) != 0.0;
    }
    for (int o = 16; o > 0; o >>= 1) {
      m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
      bad |= __shfl_down_sync(0xffffffffu, bad, o);
    }
    if (lane == 0) red[32] = bad ? -1.0 : m;
  }
  __syncthreads();
  const double scale = red[32];
  if (scale < 0.0) {  // every CTA sees the same flag and leaves
    if (tid == 0 && p == 0) atomicExch(status, 2);
    return;
  }
  if (tid == 0 && p == 0) scale_all[pt.job] = scale;
  const double inv = scale > 0.0 ? 1.0 / scale : 0.0;
  // 2. own rows scaled, their lower parts the conjugate of the upper triangle
  //    (exactly Hermitian).  In the global matrix the lower parts come first:
  //    nobody reads them, and the upper ones are overwritten after a barrier.
  for (int k = warp; k < kown; k += nwarp) {
    const int i = p + k * P;
    T *ar = rows + k * rld;
    for (int c = lane; c < i; c += 32) ar[c] = sscale(inv, cj(__ldcg(&A[(int64_t)c * n + i])));
  }
  if (!pt.resident && !tri_barrier(sl, P, ++nbar * P, status)) return;
  for (int k = warp; k < kown; k += nwarp) {
    const int i = p + k * P;
    T *ar = rows + k * rld;
    for (int c = i + lane; c < n; c += 32) {
      const T g = sscale(inv, A[(int64_t)i * n + c]);
      ar[c] = c == i ? smake<T>(sre(g), 0.0) : g;
    }
  }
  if (n == 1) {
    if (tid == 0) {
      d[0] = sre(rows[0]);
      e[0] = 0.0;
      tau[0] = smake<T>(0.0, 0.0);
    }
    return;
  }
  if (p == 0) {  // row 0 for the first reflector
    __syncthreads();
    for (int c = tid; c < n; c += nt) pb[n + c] = rows[c];
  }
  // (also: the reflectors overwrite rows of A once every CTA has read them)
  if (!tri_barrier(sl, P, ++nbar * P, status)) return;

  // Reflector of step j from the pivot row in rb (rb[c - j] = A[j][c]; its
  // entries rb[2 ..] already squared into x2): v (v_0 = 1) into v[0 .. m), tau
  // into sh_t.
  auto reflector = [&](int j, double x2, T *v) {
    for (int o = 16; o > 0; o >>= 1) x2 += __shfl_down_sync(0xffffffffu, x2, o);
    if (lane == 0) red[warp] = x2;
    __syncthreads();
    const int m = n - j - 1;
    if (warp == 0) {
      double s;
      if (ordered) {
        s = red[0];
        for (int q = 1; q < (tri_one<T>() + 31) / 32; ++q) s += red[q];
      } else {
        s = lane < nwarp ? red[lane] : 0.0;
        for (int o = kTriThreads / 64; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      }
      const T alpha = cj(rb[1]);
      const bool refl = s > 0.0 || sim(alpha) != 0.0;
      double beta = sre(alpha);
      T t = smake<T>(0.0, 0.0), sc = smake<T>(0.0, 0.0);
      if (refl) {
        beta = -copysign(sqrt(sabs2(alpha) + s), sre(alpha));
        t = smake<T>((beta - sre(alpha)) / beta, -sim(alpha) / beta);
        sc = sinv(smake<T>(sre(alpha) - beta, sim(alpha)));
      }
      if (lane == 0) {
        sh_t = t;
        sh_sc = sc;
        if (p == 0) {
          d[j] = sre(rb[0]);
          e[j] = beta;
          tau[j] = t;
        }
      }
    }
    __syncthreads();
    const T sc = sh_sc;  // zero without a reflection
    for (int r = tid; r < m; r += nt)
      v[r] = r == 0 ? smake<T>(1.0, 0.0) : smul(cj(rb[1 + r]), sc);
    __syncthreads();
  };

  // Own rows i >= lo: optional rank-2 update with (vA, wA) of step j = lo - 2,
  // then w[i - lo] = t * (row i, columns lo ..) . vn into wout, and the CTA's
  // partial sum of conj(w_i) vn_i into rout; row lo goes to prow.  A warp takes
  // four rows at a time, eight lanes each (three additions reduce the four
  // sums); the groups left over after full rounds of all warps are cut into Q
  // interleaved column slices, so that every warp gets the same number of items.
  auto rows_pass = [&](int lo, bool upd, const T *vn, T t, T *wout, T *rout, T *prow) {
    constexpr int W = kTriThreads / 32;
    const int k0 = lo <= p ? 0 : (lo - p + P - 1) / P;
    const int cnt = kown - k0, g4 = (cnt + 3) >> 2;
    const int gfull = ordered ? g4 : g4 / W * W, rem = g4 - gfull;
    int lq = 0;  // log2 Q: the smallest with rem Q a multiple of the warps
    while (((rem << lq) & (W - 1)) != 0) ++lq;
    const int Q = 1 << lq, len = n - lo;
    const T *va = vA + 1, *wa = wA + 1;  // va[c] belongs to column lo + c
    for (int it = warp; it < gfull + (rem << lq); it += W) {
      const bool whole = it < gfull;
      const int g = whole ? it : gfull + ((it - gfull) >> lq);
      const int q = whole ? 0 : (it - gfull) & (Q - 1), step = whole ? 8 : 8 << lq;
      const int k = k0 + 4 * g + (lane >> 3), i = p + k * P;
      const bool ok = k < kown, first = i == lo;
      T s = smake<T>(0.0, 0.0);
      T *ar = rows + (ok ? k : k0) * rld + lo;
      const T vi = ok && upd ? va[i - lo] : s, wi = ok && upd ? wa[i - lo] : s;
      if (ordered) {  // chains over columns 32 apart, four per lane, then their tree
        T sq[4] = {s, s, s, s};
        for (int c0 = lane & 7; c0 < len; c0 += 32) {
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const int c = c0 + 8 * b;
            if (c >= len) break;
            T a = ar[c];
            if (upd) {
              a = rank2_ordered(a, vi, cj(wa[c]), wi, cj(va[c]));
              if (ok) ar[c] = a;
            }
            if (first) prow[c] = a;
            sq[b] = smadd(sq[b], a, vn[c]);
          }
        }
        s = sadd(sadd(sq[0], sq[2]), sadd(sq[1], sq[3]));
      } else if (upd) {
#pragma unroll 4
        for (int c = q * 8 + (lane & 7); c < len; c += step) {
          const T a = rank2(ar[c], vi, cj(wa[c]), wi, cj(va[c]));
          if (ok) ar[c] = a;
          if (first) prow[c] = a;
          s = smadd(s, a, vn[c]);
        }
      } else {
#pragma unroll 4
        for (int c = q * 8 + (lane & 7); c < len; c += step) {
          const T a = ar[c];
          if (first) prow[c] = a;
          s = smadd(s, a, vn[c]);
        }
      }
      s = oct_sum(s);
      if ((lane & 7) == 0) {
        const int r = k - k0;  // rows of sliced groups hold Q sums each
        part[whole ? r : 4 * gfull + (r - 4 * gfull) * Q + q] = s;
      }
    }
    __syncthreads();
    T acc = smake<T>(0.0, 0.0);
    for (int k = tid; k < cnt; k += nt) {
      const bool whole = k < 4 * gfull;
      const T *pk = part + (whole ? k : 4 * gfull + (k - 4 * gfull) * Q);
      T s = pk[0];
      if (!whole && Q == 8)
        s = sadd(sadd(sadd(s, pk[1]), sadd(pk[2], pk[3])),
                 sadd(sadd(pk[4], pk[5]), sadd(pk[6], pk[7])));
      else if (!whole && Q == 4)
        s = sadd(sadd(s, pk[1]), sadd(pk[2], pk[3]));
      else if (!whole && Q == 2)
        s = sadd(s, pk[1]);
      const int r = p + (k0 + k) * P - lo;
      const T w = smul(t, s);
      wout[r] = w;
      acc = sadd(acc, smul(cj(w), vn[r]));
    }
    if (cnt <= 32) {
      if (warp == 0) {
        acc = warp_sum(acc);
        if (lane == 0) rout[p] = acc;
      }
    } else {
      acc = warp_sum(acc);
      if (lane == 0) wpart[warp] = acc;
      __syncthreads();
      if (tid == 0) {
        T s = wpart[0];
        for (int q = 1; q < nwarp; ++q) s = sadd(s, wpart[q]);
        rout[p] = s;
      }
    }
  };

  // step 0: reflector and products of the own rows
  {
    double x2 = 0.0;
    for (int c = r0; c < n; c += nt) {
      rb[c] = __ldcg(&pb[n + c]);
      if (c >= 2) x2 += sabs2(rb[c]);
    }
    reflector(0, x2, vA);
  }
  T t = sh_t;
  rows_pass(1, false, vA, t, wb, rd, pb);
  for (int j = 0; j + 1 < n; ++j) {
    const int m = n - j - 1, par = j & 1;
    if (!tri_barrier(sl, P, ++nbar * P, status)) return;
    // w's entries, the pivot row and the partial sums, one L2 round trip
    const T *wj = wb + par * n, *pj = pb + par * n;
    constexpr int kPer = 4;  // entries per thread held in registers (n <= 1024)
    T we[kPer], pe[kPer];
    const T w0raw = __ldcg(&wj[0]);
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      const int r = r0 + q * nt;
      if (r < m) {
        we[q] = __ldcg(&wj[r]);
        pe[q] = __ldcg(&pj[r]);
      }
    }
    if (warp == 0) {  // the P partials: lane q holds q and q + 32, tree sum in lane order
      T s = smake<T>(0.0, 0.0);
      if (lane < P) s = __ldcg(&rd[par * kTriMaxParts + lane]);
      if (lane + 32 < P) s = sadd(s, __ldcg(&rd[par * kTriMaxParts + lane + 32]));
      s = warp_sum(s);
      if (lane == 0) sh_k = smul(sscale(-0.5, t), s);  // K = -t (w^H v) / 2
    }
    if (j % P == p)  // reflector storage
      for (int c = j + 2 + tid; c < n; c += nt) A[(int64_t)j * n + c] = vA[c - j - 1];
    __syncthreads();
    const T K = sh_k;
    const T w0 = sadd(w0raw, K);  // v_0 = 1
    // w = w + K v; row j + 1 (updated through step j - 1 by its owner) with
    // step j's update
    double x2 = 0.0;
    auto entry = [&](int r, T wr, T ar) {
      const T v = vA[r];
      const T w = smadd(wr, K, v);
      wA[r] = w;
      const T one = smake<T>(1.0, 0.0);
      const T a = ordered ? rank2_ordered(ar, one, cj(w), w0, cj(v))
                          : rank2(ar, one, cj(w), w0, cj(v));
      rb[r] = a;
      if (r >= 2) x2 += sabs2(a);
    };
#pragma unroll
    for (int q = 0; q < kPer; ++q)
      if (r0 + q * nt < m) entry(r0 + q * nt, we[q], pe[q]);
    for (int r = r0 + kPer * nt; r < m; r += nt) entry(r, __ldcg(&wj[r]), __ldcg(&pj[r]));
    if (j + 2 == n) {  // the trailing block is the last diagonal entry
      if (p == 0 && r0 == 0) {  // the thread that wrote it
        d[n - 1] = sre(rb[0]);
        e[n - 1] = 0.0;
        tau[n - 1] = smake<T>(0.0, 0.0);
      }
      break;
    }
    reflector(j + 1, x2, vB);
    const T tn = sh_t;
    rows_pass(j + 2, true, vB, tn, wb + (par ^ 1) * n, rd + (par ^ 1) * kTriMaxParts,
              pb + (par ^ 1) * n);
    T *x = vA;
    vA = vB;
    vB = x;
    t = tn;
  }
}

// One warp per chunk of C columns (two real, one complex), held in shared memory
// for all reflectors; lanes walk the rows.  One pass applies reflector j and
// forms the products with reflector j - 1, whose vector was copied to shared
// memory meanwhile (cp.async), so neither L2 nor a block barrier is waited for.
// FP64 bound: a warp's FP64 instruction holds its quarter's pipe for 64 clocks,
// four per row of C columns and nine additions per reflector.  A column's
// product is summed over rows 32 apart in two chains, over the lanes by fours
// and then over these: small sectors' vectors keep this order.
template <typename T>
struct BackShape;
template <>
struct BackShape<double> {
  static constexpr int kCols = 2;
};
template <>
struct BackShape<double2> {
  static constexpr int kCols = 1;
};
// sum of x over the warp in lanes 0 .. 15, of y in lanes 16 .. 31 (the parts of a
// complex column)
__device__ __forceinline__ double pair_sum(double x, double y) {
  const bool up = threadIdx.x & 16;
  double v = (up ? y : x) + __shfl_xor_sync(0xffffffffu, up ? x : y, 16);
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Two real columns: sums over four lanes (x in the even ones, y in the odd ones),
// then over the eight quads in order.
__device__ __forceinline__ void back_weights(const double (&s)[2], double t, double (&w)[2]) {
  const bool odd = threadIdx.x & 1;
  double v = (odd ? s[1] : s[0]) + __shfl_xor_sync(0xffffffffu, odd ? s[0] : s[1], 1);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  double sum = __shfl_sync(0xffffffffu, v, odd);
#pragma unroll
  for (int q = 1; q < 8; ++q) sum += __shfl_sync(0xffffffffu, v, 4 * q + odd);
  sum *= t;
  w[0] = __shfl_sync(0xffffffffu, sum, 0);
  w[1] = __shfl_sync(0xffffffffu, sum, 1);
}
__device__ __forceinline__ void back_weights(const double2 (&s)[1], double2 t, double2 (&w)[1]) {
  const double v = pair_sum(s[0].x, s[0].y);
  w[0] = cmul(t, make_double2(__shfl_sync(0xffffffffu, v, 0), __shfl_sync(0xffffffffu, v, 16)));
}

template <typename T>
__global__ void __launch_bounds__(32)
    backtransform_kernel(const EigJob *__restrict__ jobs, const BackChunk *__restrict__ bt,
                         const T *__restrict__ G_all, const T *__restrict__ tau_all,
                         T *__restrict__ Z) {
  constexpr int C = BackShape<T>::kCols;
  extern __shared__ __align__(16) unsigned char back_sm[];
  const BackChunk ch = bt[blockIdx.x];
  const EigJob job = jobs[ch.job];
  const int n = job.n, lane = threadIdx.x;
  if (n < 2 || ch.cw == 0) return;
  // C columns of n, then the reflectors of two consecutive steps (entry r of
  // row j's vector at index j + 1 + r)
  T *zs = (T *)back_sm, *vb = zs + C * n;
  T *z = Z + ch.z_off + ch.c0;
  const T *A = G_all + job.g_off;
  const T *tau = tau_all + job.lam_off;
  auto fetch = [&](int j) {  // the vector of step j
    T *dst = vb + (j & 1) * n;
    const T *src = A + (int64_t)j * n;
    if (lane == 0) dst[j + 1] = smake<T>(1.0, 0.0);
    for (int c = j + 2 + lane; c < n; c += 32)
      asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(
                       (uint32_t)__cvta_generic_to_shared(dst + c)),
                   "l"(src + c), "n"(sizeof(T))
                   : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int r = lane; r < n; r += 32)
#pragma unroll
    for (int c = 0; c < C; ++c)
      zs[c * n + r] = c < ch.cw ? z[(int64_t)r * ch.ld + c] : smake<T>(0.0, 0.0);
  fetch(n - 2);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncwarp();
  // products with the first reflector: rows n - 1 only
  T s[C];
#pragma unroll
  for (int c = 0; c < C; ++c)
    s[c] = lane == 0 ? smul(cj(vb[((n - 2) & 1) * n + n - 1]), zs[c * n + n - 1])
                     : smake<T>(0.0, 0.0);
  T t = tau[n - 2];
  for (int j = n - 2; j >= 0; --j) {
    const T *v = vb + (j & 1) * n, *vn = vb + ((j + 1) & 1) * n;  // vn: step j - 1
    if (j > 0) fetch(j - 1);
    const T tn = j > 0 ? tau[j - 1] : t;
    T w[C];
    back_weights(s, t, w);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    T s2[C][2];  // rows from j on, 32 apart, in two chains
#pragma unroll
    for (int c = 0; c < C; ++c) s2[c][0] = s2[c][1] = smake<T>(0.0, 0.0);
#pragma unroll 2
    for (int r0 = j + lane; r0 < n; r0 += 64) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = r0 + 32 * h;
        if (r >= n) break;
        // row j takes part in the products only
        const T x = r > j ? v[r] : smake<T>(0.0, 0.0);
        const T y = j > 0 ? cj(vn[r]) : smake<T>(0.0, 0.0);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const T a = smsub(zs[c * n + r], x, w[c]);
          zs[c * n + r] = a;
          s2[c][h] = smadd(s2[c][h], y, a);
        }
      }
    }
    __syncwarp();
#pragma unroll
    for (int c = 0; c < C; ++c) s[c] = sadd(s2[c][0], s2[c][1]);
    t = tn;
  }
  for (int r = lane; r < n; r += 32)
#pragma unroll
    for (int c = 0; c < C; ++c)
      if (c < ch.cw) z[(int64_t)r * ch.ld + c] = zs[c * n + r];
}

}  // namespace

bool eig_ordered(int64_t n, bool cplx) {
  return n <= (cplx ? tri_one<double2>() : tri_one<double>());
}

// Shared memory a CTA of the reduction may use, and the matrices that leave
// room for a second CTA on the SM.
constexpr size_t kTriSmemBytes = 226 * 1024;
constexpr size_t kTriSmallBytes = 110 * 1024;
// Time model of the reduction: 5.5 us per step, and n^3 FMAs (four per complex
// one) at 3e9 per second and CTA (80% of its FP64 pipe).
constexpr double kTriStep = 5.5e-6, kTriRate = 3e9;

template <typename T>
static size_t tri_smem(int n, int P) {  // with the own rows resident
  return (4 * (size_t)n + tri_parts(n, P) + (size_t)((n + P - 1) / P) * tri_ld<T>(n)) * sizeof(T);
}

// Householder reduction of every job.  Matrices of which two fit one SM's
// shared memory run on one CTA each, on the side stream; the larger ones run in
// one cooperative launch (more if they do not fit), the SMs shared out so that
// all are expected to end together (ordered ones: one CTA).
template <typename T>
static void tridiag_all(Ctx &ctx, DeviceScratch &scratch, const std::vector<EigJob> &jobs,
                        const SymEigWork &wk, double *G, int *dstat) {
  std::vector<int> big, small;
  for (int q = 0; q < (int)jobs.size(); ++q) {
    if (jobs[q].n == 0) continue;
    (tri_smem<T>(jobs[q].n, 1) <= kTriSmallBytes ? small : big).push_back(q);
  }
  auto larger = [&](int x, int y) { return jobs[x].n > jobs[y].n; };
  std::stable_sort(big.begin(), big.end(), larger);
  std::stable_sort(small.begin(), small.end(), larger);
  const void *kern = (const void *)tridiag_mc_kernel<T>;
  size_t max_smem = kTriSmemBytes;
  if (!big.empty()) max_smem = std::max(max_smem, 4 * (size_t)jobs[big[0]].n * sizeof(T));
  UDMRG_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)max_smem));
  const int reserve = std::min((int)(small.size() + 1) / 2, ctx.num_sms / 6);
  const int budget = ctx.num_sms - (big.empty() ? 0 : reserve);
  // the parts of every launch, their slots and buffers in one upload
  std::vector<TriPart> parts;
  struct Launch {
    size_t part0, nparts, smem;
    bool coop;
  };
  std::vector<Launch> launches;
  int64_t wb_tot = 0;
  int slot = 0;
  // returns the shared memory of the job's CTAs
  auto add = [&](int q, int P) {
    const int n = jobs[q].n;
    const bool resident = tri_smem<T>(n, P) <= kTriSmemBytes;
    const int64_t np = tri_parts(n, P), wb = wb_tot;
    wb_tot += 4 * (int64_t)n;
    size_t bytes = tri_smem<T>(n, P);
    if (!resident) bytes = (4 * (size_t)n + np) * sizeof(T);
    const bool gpart = bytes > kTriSmemBytes;
    if (gpart) bytes = 4 * (size_t)n * sizeof(T);
    for (int p = 0; p < P; ++p) {
      parts.push_back(TriPart{q, p, P, slot, wb, gpart ? wb_tot : -1, resident ? 1 : 0,
                              n <= tri_one<T>() ? 1 : 0});
      if (gpart) wb_tot += np;
    }
    ++slot;
    return bytes;
  };
  const double rate = kTriRate / (sizeof(T) / sizeof(double) == 2 ? 4.0 : 1.0);
  for (size_t at = 0; at < big.size();) {
    // as many matrices as fit with the fewest CTAs that keep their rows resident
    std::vector<int> pmin, cap;
    size_t end = at;
    int sum = 0;
    for (; end < big.size(); ++end) {
      const int n = jobs[big[end]].n;
      const int c = n <= tri_one<T>() ? 1 : std::min({kTriMaxParts, n / 8, budget});
      int P = 1;
      while (P < c && tri_smem<T>(n, P) > kTriSmemBytes) ++P;
      if (end > at && sum + P > budget) break;
      sum += P;
      pmin.push_back(P);
      cap.push_back(c);
    }
    auto share = [&](double t, size_t i) {
      const double n = jobs[big[at + i]].n, left = t - n * kTriStep;
      const double P = left > 0 ? std::ceil(n * n * n / rate / left) : 1e9;
      return (int)std::min<double>(cap[i], std::max<double>(pmin[i], P));
    };
    double lo = 0.0, hi = 10.0;  // seconds
    for (int it = 0; it < 60; ++it) {
      const double t = 0.5 * (lo + hi);
      int s = 0;
      for (size_t i = 0; i < pmin.size(); ++i) s += share(t, i);
      (s <= budget ? hi : lo) = t;
    }
    Launch L{parts.size(), 0, 0, true};
    for (size_t i = 0; i < pmin.size(); ++i) {
      L.smem = std::max(L.smem, add(big[at + i], share(hi, i)));
    }
    L.nparts = parts.size() - L.part0;
    launches.push_back(L);
    at = end;
  }
  if (!small.empty()) {
    Launch L{parts.size(), small.size(), 0, false};
    for (int q : small) L.smem = std::max(L.smem, add(q, 1));
    launches.push_back(L);
  }
  if (parts.empty()) return;
  TriPart *dparts = scratch.get<TriPart>(parts.size());
  TriSlot *dslots = scratch.get<TriSlot>(slot);
  T *dwb = scratch.get<T>(wb_tot);
  T *dred = scratch.get<T>((int64_t)slot * 2 * kTriMaxParts);
  ctx.upload(dparts, parts.data(), parts.size() * sizeof(TriPart));
  UDMRG_CHECK_CUDA(cudaMemsetAsync(dslots, 0, slot * sizeof(TriSlot), ctx.stream));
  // the side stream starts after the uploads and the Gram products, and the
  // main stream goes on after it
  struct Events {
    cudaEvent_t a = nullptr, b = nullptr;
    ~Events() {
      if (a) cudaEventDestroy(a);
      if (b) cudaEventDestroy(b);
    }
  } ev;
  const bool side = launches.size() > 1 && !launches.back().coop;
  if (side) {
    UDMRG_CHECK_CUDA(cudaEventCreateWithFlags(&ev.a, cudaEventDisableTiming));
    UDMRG_CHECK_CUDA(cudaEventCreateWithFlags(&ev.b, cudaEventDisableTiming));
    UDMRG_CHECK_CUDA(cudaEventRecord(ev.a, ctx.stream));
  }
  const EigJob *djobs = wk.jobs;
  T *g = (T *)G, *tau = (T *)wk.tau;
  double *d = wk.d, *e = wk.e, *sc = wk.scale;
  auto launch = [&](const Launch &L, cudaStream_t st) {
    const TriPart *dp = dparts + L.part0;
    void *args[] = {&djobs, &dp, &g, &d, &e, &tau, &sc, &dslots, &dwb, &dred, &dstat};
    if (L.coop)
      UDMRG_CHECK_CUDA(cudaLaunchCooperativeKernel(kern, dim3((unsigned)L.nparts),
                                                   dim3(kTriThreads), args, L.smem, st));
    else
      UDMRG_CHECK_CUDA(
          cudaLaunchKernel(kern, dim3((unsigned)L.nparts), dim3(kTriThreads), args, L.smem, st));
    ctx.launches++;
  };
  launch(launches[0], ctx.stream);
  if (side) {
    UDMRG_CHECK_CUDA(cudaStreamWaitEvent(ctx.side, ev.a, 0));
    launch(launches.back(), ctx.side);
    UDMRG_CHECK_CUDA(cudaEventRecord(ev.b, ctx.side));
  }
  for (size_t i = 1; i + (side ? 1 : 0) < launches.size(); ++i) launch(launches[i], ctx.stream);
  if (side) UDMRG_CHECK_CUDA(cudaStreamWaitEvent(ctx.stream, ev.b, 0));
}

int sym_eig_values(Ctx &ctx, DeviceScratch &scratch, std::vector<EigJob> &jobs, double *G,
                   double *lam, SymEigWork &wk, bool cplx, int64_t need, int64_t floor,
                   const std::vector<int64_t> *rank_cap) {
  const int nj = (int)jobs.size();
  if (nj == 0) return 0;
  int64_t ltot = 0;
  int nmax = 0;
  for (auto &j : jobs) {
    ltot = std::max<int64_t>(ltot, j.lam_off + j.n);
    nmax = std::max(nmax, j.n);
  }
  UDMRG_REQUIRE(nmax <= 4096, "eigensolver: matrix larger than 4096 is not supported");
  wk.d = scratch.get<double>(std::max<int64_t>(ltot, 1));
  wk.e = scratch.get<double>(std::max<int64_t>(ltot, 1));
  wk.tau = scratch.get<double>((cplx ? 2 : 1) * std::max<int64_t>(ltot, 1));
  wk.scale = scratch.get<double>(nj);
  wk.cplx = cplx;
  wk.jobs = scratch.get<EigJob>(nj);
  int *dstat = scratch.get<int>(1);
  UDMRG_CHECK_CUDA(cudaMemsetAsync(dstat, 0, sizeof(int), ctx.stream));
  ctx.upload(wk.jobs, jobs.data(), nj * sizeof(EigJob));
  if (cplx)
    tridiag_all<double2>(ctx, scratch, jobs, wk, G, dstat);
  else
    tridiag_all<double>(ctx, scratch, jobs, wk, G, dstat);
  const size_t bsmem = 2 * (size_t)nmax * sizeof(double);
  if (bsmem > 48 * 1024) {
    UDMRG_CHECK_CUDA(cudaFuncSetAttribute(bisect_kernel,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bsmem));
    UDMRG_CHECK_CUDA(cudaFuncSetAttribute(grid_count_kernel,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bsmem));
  }
  // how many leading eigenvalues of each job to compute
  wk.computed.assign(nj, 0);
  wk.trace.clear();
  int64_t ntot = 0;
  for (int q = 0; q < nj; ++q) {
    wk.computed[q] = jobs[q].n;
    ntot += jobs[q].n;
  }
  double *dtop = nullptr;
  int *dcnt = nullptr;
  if (need > 0 && need < ntot) {
    dtop = scratch.get<double>(1);
    double *dtr = scratch.get<double>(nj);
    dcnt = scratch.get<int>((size_t)nj * (kGrid + 1));
    grid_top_kernel<<<1, 1024, 0, ctx.stream>>>(wk.jobs, nj, wk.d, wk.e, wk.scale, dtop);
    grid_count_kernel<<<nj, kGrid, bsmem, ctx.stream>>>(wk.jobs, wk.d, wk.e, wk.scale, dtop, dcnt,
                                                        dtr);
    UDMRG_CHECK_CUDA(cudaGetLastError());
    ctx.launches += 2;
    std::vector<int> cnt((size_t)nj * (kGrid + 1));
    wk.trace.assign(nj, 0.0);
    UDMRG_CHECK_CUDA(cudaMemcpyAsync(cnt.data(), dcnt, cnt.size() * sizeof(int),
                                     cudaMemcpyDeviceToHost, ctx.stream));
    UDMRG_CHECK_CUDA(cudaMemcpyAsync(wk.trace.data(), dtr, nj * sizeof(double),
                                     cudaMemcpyDeviceToHost, ctx.stream));
    ctx.sync();
    // the first grid point with `need` eigenvalues above it, then one point
    // lower (a factor 1.34: near-ties and rounding at the threshold)
    int ks = -1;
    for (int k = 0; k <= kGrid; ++k) {
      int64_t t = 0;
      for (int q = 0; q < nj; ++q) {
        const int64_t c = cnt[(size_t)q * (kGrid + 1) + k];
        t += rank_cap ? std::min<int64_t>(c, (*rank_cap)[q]) : c;
      }
      if (t >= need) {
        ks = k;
        break;
      }
    }
    // fewer than `need` usable eigenvalues above the lowest grid point (a
    // rank-deficient set, and a Dmin asking for its null states too): every
    // eigenvalue
    if (ks >= 0) {
      ks = std::min(ks + 1, kGrid);
      for (int q = 0; q < nj; ++q) {
        const int64_t n = jobs[q].n;
        const int64_t c =
            std::max<int64_t>(cnt[(size_t)q * (kGrid + 1) + ks], std::min(n, floor));
        wk.computed[q] = std::min(c, n);
      }
    }
  }
  std::vector<int2> chunks;
  for (int q = 0; q < nj; ++q)
    for (int i0 = jobs[q].n - (int)wk.computed[q]; i0 < jobs[q].n; i0 += kBisectEigs)
      chunks.push_back(make_int2(q, i0));
  int2 *dch = scratch.get<int2>(chunks.size());
  ctx.upload(dch, chunks.data(), chunks.size() * sizeof(int2));
  if (!chunks.empty())
    bisect_kernel<<<(int)chunks.size(), 32, bsmem, ctx.stream>>>(
        wk.jobs, dch, wk.d, wk.e, wk.scale, lam, dtop, dcnt);
  UDMRG_CHECK_CUDA(cudaGetLastError());
  ctx.launches += 2;
  int hstat = 0;
  UDMRG_CHECK_CUDA(cudaMemcpyAsync(&hstat, dstat, sizeof(int), cudaMemcpyDeviceToHost, ctx.stream));
  ctx.sync();
  return hstat;
}

void sym_eig_vectors(Ctx &ctx, DeviceScratch &scratch, const std::vector<EigJob> &jobs,
                     const double *G, const double *lam, const std::vector<double> &hlam,
                     const std::vector<int64_t> &k, const std::vector<int64_t> &z_off_out,
                     const std::vector<int64_t> &z_ld_out, double *Zout, const SymEigWork &wk,
                     uint64_t seed) {
  const int nj = (int)jobs.size();
  // the eigenvectors of the (real) tridiagonal matrix: in place for real
  // matrices, in a packed real buffer for complex ones
  double *Z = Zout;
  std::vector<int64_t> z_off = z_off_out, z_ld = z_ld_out;
  int64_t zr_tot = 0;
  if (wk.cplx) {
    for (int q = 0; q < nj; ++q) {
      z_off[q] = zr_tot;
      z_ld[q] = std::max<int64_t>(k[q], 1);
      zr_tot += (int64_t)jobs[q].n * k[q];
    }
    Z = scratch.get<double>(std::max<int64_t>(zr_tot, 1));
  }
  // clusters: descending neighbours closer than 1e-9 of the matrix's largest |eigenvalue|
  std::vector<EigCluster> cl;
  int nmax = 0;
  for (int q = 0; q < nj; ++q) {
    const int n = jobs[q].n;
    nmax = std::max(nmax, n);
    if (k[q] == 0) continue;
    const double *h = hlam.data() + jobs[q].lam_off;
    const int64_t nc = q < (int)wk.computed.size() ? wk.computed[q] : n;  // computed values
    const double big = std::max(std::fabs(h[0]), std::fabs(h[std::max<int64_t>(nc, 1) - 1]));
    const double tol = 1e-9 * big;
    int first = 0;
    for (int p = 1; p <= k[q]; ++p) {
      if (p == k[q] || h[p - 1] - h[p] > tol) {
        cl.push_back(EigCluster{z_off[q], z_ld[q], seed + 1000003ull * (uint64_t)q, q, first,
                                p - first, 0});
        first = p;
      }
    }
  }
  if (!cl.empty()) {
    const int ncl = (int)cl.size();
    EigCluster *dcl = scratch.get<EigCluster>(ncl);
    double *work = scratch.get<double>(6 * (int64_t)nmax * ncl);
    ctx.upload(dcl, cl.data(), ncl * sizeof(EigCluster));
    invit_kernel<<<(ncl + 31) / 32, 32, 0, ctx.stream>>>(dcl, ncl, wk.jobs, wk.d, wk.e, wk.scale,
                                                        lam, Z, work, nmax);
    UDMRG_CHECK_CUDA(cudaGetLastError());
    ctx.launches++;
  }
  // Newton-Schulz: Z <- 1.5 Z - 0.5 Z (Z^T Z), twice (grouped GEMMs)
  {
    int64_t stot = 0, ztot = 0;
    std::vector<int64_t> soff(nj), zc_off(nj);
    for (int q = 0; q < nj; ++q) {
      soff[q] = stot;
      stot += k[q] * k[q];
      zc_off[q] = ztot;
      ztot += (int64_t)jobs[q].n * k[q];
    }
    if (stot > 0) {
      DeviceScratch ns(ctx);
      double *S = ns.get<double>(stot), *Zc = ns.get<double>(ztot);
      GemmPlan gs, gz;
      gs.ctx = gz.ctx = &ctx;
      for (int q = 0; q < nj; ++q) {
        if (k[q] == 0) continue;
        const int64_t n = jobs[q].n, kk = k[q];
        // S = Z^T Z (k x k): A = Z^T (ms 1, ks ld), B = Z (ks ld, ns 1)
        gemm_add_simple(gs, soff[q], kk, kk, n, z_off[q], 1, z_ld[q], z_off[q], z_ld[q], 1, false);
        // Zc = Z S (n x k, packed)
        gemm_add_simple(gz, zc_off[q], n, kk, kk, z_off[q], z_ld[q], 1, soff[q], kk, 1, false);
      }
      gemm_finalize(gs);
      gemm_finalize(gz);
      std::vector<Copy2D> upd;  // Z = 1.5 Z - 0.5 Zc
      for (int q = 0; q < nj; ++q)
        if (k[q] > 0)
          upd.push_back(
              Copy2D{zc_off[q], z_off[q], jobs[q].n, (int32_t)k[q], k[q], 1, z_ld[q], 1});
      for (int it = 0; it < 2; ++it) {
        (ctx.svd_dw ? run_gemm_dw : run_gemm)(ctx, gs, kF64, Z, Z, S, 1.0, 0.0);
        (ctx.svd_dw ? run_gemm_dw : run_gemm)(ctx, gz, kF64, Z, S, Zc, 1.0, 0.0);
        run_axpby2d(ctx, upd, Zc, Z, 1.5, -0.5);
      }
    }
  }
  if (wk.cplx && zr_tot > 0) {  // real eigenvectors of T -> complex, into the caller's layout
    double *Zc = scratch.get<double>(2 * zr_tot);
    real_to_complex(ctx, Z, Zc, zr_tot);
    std::vector<Copy2D> ops;
    for (int q = 0; q < nj; ++q)
      if (k[q] > 0)
        ops.push_back(Copy2D{z_off[q], z_off_out[q], jobs[q].n, (int32_t)k[q], k[q], 1,
                             z_ld_out[q], 1});
    run_copy2d(ctx, ops, Zc, Zout, true);
  }
  // back-transformation by the reflectors, the largest matrices first
  {
    const int width = wk.cplx ? BackShape<double2>::kCols : BackShape<double>::kCols;
    std::vector<int> order(nj);
    for (int q = 0; q < nj; ++q) order[q] = q;
    std::stable_sort(order.begin(), order.end(),
                     [&](int x, int y) { return jobs[x].n > jobs[y].n; });
    std::vector<BackChunk> bt;
    for (int q : order)
      for (int64_t c0 = 0; c0 < k[q]; c0 += width)
        bt.push_back(BackChunk{z_off_out[q], z_ld_out[q], q, (int32_t)c0,
                               (int32_t)std::min<int64_t>(width, k[q] - c0), 0});
    if (!bt.empty()) {
      BackChunk *dbt = scratch.get<BackChunk>(bt.size());
      ctx.upload(dbt, bt.data(), bt.size() * sizeof(BackChunk));
      const size_t smem = wk.cplx
                              ? (size_t)nmax * (BackShape<double2>::kCols + 2) * sizeof(double2)
                              : (size_t)nmax * (BackShape<double>::kCols + 2) * sizeof(double);
      UDMRG_REQUIRE(smem <= 227 * 1024, "back transformation: matrix too large");
      const void *kern = wk.cplx ? (const void *)backtransform_kernel<double2>
                                 : (const void *)backtransform_kernel<double>;
      if (smem > 48 * 1024)
        UDMRG_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)smem));
      if (wk.cplx)
        backtransform_kernel<double2><<<(int)bt.size(), 32, smem, ctx.stream>>>(
            wk.jobs, dbt, (const double2 *)G, (const double2 *)wk.tau, (double2 *)Zout);
      else
        backtransform_kernel<double><<<(int)bt.size(), 32, smem, ctx.stream>>>(wk.jobs, dbt, G,
                                                                              wk.tau, Zout);
      UDMRG_CHECK_CUDA(cudaGetLastError());
      ctx.launches++;
    }
  }
}

}  // namespace udmrg
