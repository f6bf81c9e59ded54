// vca_tri.cuh -- lowest eigenpair of a Lanczos tridiagonal, one warp.
//
// T_k has diagonal A[0..k-1] and off-diagonal Bt[1..k-1] (Bt[j] = beta_{j+1}
// couples rows j-1 and j); the Lanczos residual estimate is |beta_{k+1}
// s_{k-1}|.  GB300's FP64 pipe takes ~64 cycles per warp instruction, so a
// serial FP64 recurrence over k rows costs k * 64 cycles per operation in it
// and the test is split by what it has to decide:
//  * tri_estimate (FP32): the lowest eigenvalue by warp multisection on the
//    leading minors of T - x (all positive below it; two FMAs a row), a peak
//    row r of its eigenvector (a small |gamma_r|, see below), and the tail
//    component from the backward pivots, whose ratios keep their relative
//    accuracy however small the component is.  A run whose estimate is 64
//    times the tolerance or more goes on without FP64 work; that is nearly
//    every test.
//  * tri_newton (FP64): Newton's method on gamma_r(x) = (a_r - x) -
//    b_r^2 / f_{r-1}(x) - b_{r+1}^2 / d_{r+1}(x), f the forward and d the
//    backward pivots of T - x.  While all of them are positive (x below the
//    spectra of the rows above and below r) gamma_r is decreasing and concave,
//    so the iterates fall monotonically onto the lowest eigenvalue; its slope,
//    minus the squared norm of the vector with s_r = 1, comes with the same
//    pass, and so do the ratios |s_j / s_{j-1}| down to the tail.  One lane
//    runs each direction.
//  * tri_bisect (FP64): Sturm multisection, where a pivot is not positive (a
//    lowest level that is nearly repeated) or the estimate is not finite.
//  * tri_invit (FP64): the eigenvector, where a caller reads it, by inverse
//    iteration (Wilkinson, The Algebraic Eigenvalue Problem, ch. 5).
// One test of a 100-row problem took 0.80 ms by bisection and inverse iteration
// with the LU formed at each of its steps, at every test; the estimate takes
// about 20 us.
// All 32 lanes call.  s needs 5*k doubles (eigenvector + LU work).  k <= 512.
#pragma once

#include <cuda_runtime.h>

namespace vca {

#define TRI_MAX 512

__device__ __forceinline__ int sturm_count_tri(const double* a, const double* b1, int k, double x) {
  int cnt = 0;
  double q = a[0] - x;
  if (q < 0) cnt++;
  for (int j = 1; j < k; j++) {
    if (q == 0.0) q = 1e-300;
    q = a[j] - x - b1[j] * b1[j] / q;
    if (q < 0) cnt++;
  }
  return cnt;
}

// the lowest eigenvalue to adjacent doubles; the value is returned to every lane
static __device__ double tri_bisect(const double* A, const double* Bt, int k) {
  const int lane = threadIdx.x & 31;
  double lo = A[0], hi = A[0];
  for (int j = 0; j < k; j++) {  // Gershgorin bounds (every lane, same values)
    double r = (j > 0 ? fabs(Bt[j]) : 0.0) + (j < k - 1 ? fabs(Bt[j + 1]) : 0.0);
    lo = fmin(lo, A[j] - r);
    hi = fmax(hi, A[j] + r);
  }
  for (int round = 0; round < 100; round++) {
    const double x = lo + (hi - lo) * (double)(lane + 1) / 33.0;
    const int c = (x > lo && x < hi) ? sturm_count_tri(A, Bt, k, x) : (x >= hi ? 1 : 0);
    const unsigned ball = __ballot_sync(0xffffffffu, c >= 1);
    const int f = ball ? (__ffs(ball) - 1) : 32;  // first point above the lowest eigenvalue
    double nlo = (f == 0) ? lo : lo + (hi - lo) * (double)f / 33.0;
    double nhi = (f == 32) ? hi : lo + (hi - lo) * (double)(f + 1) / 33.0;
    if (nlo < lo) nlo = lo;
    if (nhi > hi) nhi = hi;
    const bool stop = (nhi - nlo <= 2.220446049250313e-16 * fmax(fabs(nlo), fabs(nhi))) || !(nlo < nhi) ||
                      (nlo == lo && nhi == hi);
    lo = nlo;
    hi = nhi;
    if (stop) break;
  }
  if (lane == 0)
    for (int it = 0; it < 200; it++) {
      const double mid = 0.5 * (lo + hi);
      if (mid <= lo || mid >= hi) break;
      if (sturm_count_tri(A, Bt, k, mid) >= 1) hi = mid; else lo = mid;
    }
  return __shfl_sync(0xffffffffu, 0.5 * (lo + hi), 0);
}

// Eigenvector s[0..k-1] of the eigenvalue th: one partially pivoted LU of
// T - th, three steps of inverse iteration from all ones, the serial
// recurrences on lane 0, reciprocals and norms on all lanes.  (A single solve
// with the twisted pivots would be off by eps / gap where T holds a second,
// not yet converged copy of the lowest level; repeated steps are not.)
static __device__ void tri_invit(const double* A, const double* Bt, int k, double th, double* s) {
  const int lane = threadIdx.x & 31;
  double* y = s;
  double *dl = s + k, *dd = s + 2 * k, *du = s + 3 * k, *du2 = s + 4 * k;
  for (int j = lane; j < k; j += 32) {
    y[j] = 1.0;
    dd[j] = A[j] - th;
    if (j < k - 1) { dl[j] = Bt[j + 1]; du[j] = Bt[j + 1]; du2[j] = 0.0; }
  }
  __syncwarp();
  unsigned long long piv[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (lane == 0) {
    for (int j = 0; j < k - 1; j++) {
      if (fabs(dd[j]) >= fabs(dl[j])) {
        if (dd[j] == 0.0) dd[j] = 1e-300;
        const double f = dl[j] / dd[j];
        dl[j] = f;
        dd[j + 1] -= f * du[j];
      } else {
        const double f = dd[j] / dl[j];
        dd[j] = dl[j];
        dl[j] = f;
        const double t = du[j];
        du[j] = dd[j + 1];
        dd[j + 1] = t - f * dd[j + 1];
        if (j < k - 2) { du2[j] = du[j + 1]; du[j + 1] = -f * du[j + 1]; }
        piv[j >> 6] |= 1ull << (j & 63);
      }
    }
    if (dd[k - 1] == 0.0) dd[k - 1] = 1e-300;
  }
  __syncwarp();
  for (int j = lane; j < k; j += 32) dd[j] = 1.0 / dd[j];
  __syncwarp();
  for (int it = 0; it < 3; it++) {
    if (lane == 0) {
      for (int j = 0; j < k - 1; j++) {
        if (!((piv[j >> 6] >> (j & 63)) & 1ull)) y[j + 1] -= dl[j] * y[j];
        else { const double t = y[j]; y[j] = y[j + 1]; y[j + 1] = t - dl[j] * y[j]; }
      }
      y[k - 1] *= dd[k - 1];
      if (k > 1) y[k - 2] = (y[k - 2] - du[k - 2] * y[k - 1]) * dd[k - 2];
      for (int j = k - 3; j >= 0; j--) y[j] = (y[j] - du[j] * y[j + 1] - du2[j] * y[j + 2]) * dd[j];
    }
    __syncwarp();
    double nr = 0.0;
    for (int j = lane; j < k; j += 32) nr = fma(y[j], y[j], nr);
    for (int off = 16; off > 0; off >>= 1) nr += __shfl_xor_sync(0xffffffffu, nr, off);
    const double inv = 1.0 / sqrt(nr);
    for (int j = lane; j < k; j += 32) y[j] *= inv;
    __syncwarp();
  }
  const double sg = y[0] < 0 ? -1.0 : 1.0;
  __syncwarp();
  for (int j = lane; j < k; j += 32) y[j] *= sg;
  __syncwarp();
}

// FP32 estimate of the residual |btail s_{k-1}| of the lowest pair and of the
// eigenvalue itself; false where the pivots do not allow one.  w: 2*TRI_MAX
// float2 of the warp's own (diagonal, squared off-diagonal; forward pivots).
__device__ __forceinline__ bool tri_estimate(const double* A, const double* Bt, int k, double btail, float2* w,
                                             float& theta, int& peak, float& resid) {
  float2* fm = w + TRI_MAX;
  const int lane = threadIdx.x & 31;
  const unsigned all = 0xffffffffu;
  // rows scaled by a power of two to magnitudes of order 1
  double big = 0.0;
  for (int j = lane; j < k; j += 32) big = fmax(big, fabs(A[j]) + (j ? fabs(Bt[j]) : 0.0));
  for (int off = 16; off > 0; off >>= 1) big = fmax(big, __shfl_xor_sync(all, big, off));
  if (!(big > 1e-30 && big < 1e30)) return false;
  int e;
  frexp(big, &e);
  const double down = ldexp(1.0, -e);
  float lo = 3.0e38f, hi = 3.0e38f;
  for (int j = lane; j < k; j += 32) {
    const float a = (float)(A[j] * down), b = j ? (float)(Bt[j] * down) : 0.f;
    const float bn = j < k - 1 ? (float)(Bt[j + 1] * down) : 0.f;
    w[j] = make_float2(a, b * b);
    lo = fminf(lo, a - fabsf(b) - fabsf(bn));
    hi = fminf(hi, a);  // the lowest eigenvalue is at most any diagonal entry
  }
  for (int off = 16; off > 0; off >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(all, lo, off));
    hi = fminf(hi, __shfl_xor_sync(all, hi, off));
  }
  __syncwarp();
  const float pad = 1e-6f * fmaxf(fabsf(lo), fabsf(hi)) + 1e-30f;
  lo -= pad;
  hi += pad;
  for (int round = 0; round < 8 && hi - lo > 4e-7f * fmaxf(fabsf(lo), fabsf(hi)); round++) {
    const float x = lo + (hi - lo) * ((float)(lane + 1) * (1.f / 33.f));
    float pp = 1.f, p = w[0].x - x, low = p;
#pragma unroll 4
    for (int j = 1; j < k; j++) {
      const float2 ab = w[j];
      const float pn = fmaf(ab.x - x, p, -ab.y * pp);
      pp = p;
      p = pn;
      low = fminf(low, p);
      if ((j & 3) == 0) {  // keep the minors near 1: scale by a power of two
        const int ex = (__float_as_int(fmaxf(fabsf(p), fabsf(pp))) >> 23) & 255;
        const float sc = __int_as_float((254 - min(253, max(1, ex))) << 23);
        p *= sc;
        pp *= sc;
      }
    }
    const unsigned above = __ballot_sync(all, !(low > 0.f));  // points not below the lowest eigenvalue
    const int f = above ? __ffs(above) - 1 : 32;
    const float nlo = f == 0 ? lo : lo + (hi - lo) * ((float)f * (1.f / 33.f));
    const float nhi = f == 32 ? hi : lo + (hi - lo) * ((float)(f + 1) * (1.f / 33.f));
    if (!(nhi < hi || nlo > lo)) break;
    lo = nlo;
    hi = nhi;
  }
  const float th = 0.5f * (lo + hi);
  // forward pivots f_j and m_j = 1 + sum_{i<j} (s_i / s_j)^2 (every lane, same values)
  float f = w[0].x - th, m = 1.f;
  for (int j = 0; j < k; j++) {
    if (lane == 0) fm[j] = make_float2(f, m);
    if (j + 1 < k) {
      const float gi = __fdividef(1.f, f), t = w[j + 1].y * gi;
      m = fmaf(t * gi, m, 1.f);
      f = (w[j + 1].x - th) - t;
    }
  }
  __syncwarp();
  // backward pivots; the twist row is the one of smallest |gamma|, and among
  // rows that FP32 cannot tell from null the one of the smallest tail: where T
  // holds a second copy of the level, FP64 decides on the converged one
  float d = w[k - 1].x - th, lg = 0.f, n = 1.f, best = 3.0e38f, lgr = 0.f, nr = 0.f;
  float low = 3.0e38f, lowr = 0.f;  // smallest backward pivot so far; below the twist row
  peak = 0;
  for (int j = k - 1; j >= 0; j--) {
    const float2 x = fm[j];
    const float gam = fabsf(x.x + d - (w[j].x - th)), nj = n + x.y - 1.f, tail = lg - __log2f(nj);
    const bool null = gam < 1e-5f;  // s_j is a sizeable part of a null vector in FP32
    if (null ? !(best == 0.f && tail >= lgr - __log2f(nr)) : gam < best) {
      best = null ? 0.f : gam;
      peak = j;
      lgr = lg;
      nr = nj;
      lowr = low;
    }
    if (j) {
      low = fminf(low, d);
      const float gi = __fdividef(1.f, d), t = w[j].y * gi, r2 = t * gi;
      n = fmaf(r2, n, 1.f);
      lg += __log2f(r2);
      d = (w[j - 1].x - th) - t;
    }
  }
  float up = 3.0e38f;  // smallest forward pivot above the twist row
  for (int j = lane; j < peak; j += 32) up = fminf(up, fm[j].x);
  for (int off = 16; off > 0; off >>= 1) up = fminf(up, __shfl_xor_sync(all, up, off));
  resid = fabsf((float)btail) * exp2f(0.5f * (lgr - __log2f(nr)));
  theta = ldexpf(th, e);
  return fminf(up, lowr) > 0.f && lgr == lgr && nr < 3e38f && resid == resid;
}

// reciprocal of a positive normal double in FP32 range: the FP32 estimate and
// one cubic Newton step (relative error 2^-66 before rounding)
__device__ __forceinline__ double tri_recip(double d) {
  const double g = (double)__frcp_rn((float)d);
  const double e = fma(-d, g, 1.0);
  return fma(g, fma(e, e, e), g);
}

// theta and the residual; lane 0 runs the backward pivots, lane 1 the forward
// ones, the outcome is returned to every lane.  s: k doubles of scratch.
static __device__ bool tri_newton(const double* A, const double* Bt, int k, double btail, float start, int r,
                                  double* theta_out, double* s, double* resid) {
  const int lane = threadIdx.x & 31;
  const unsigned all = 0xffffffffu;
  const bool fwd = lane == 1;
  const int cnt = lane == 0 ? k - 1 - r : fwd ? r : 0;  // rows on this side of r
  const int dir = fwd ? 1 : -1, j0 = fwd ? 0 : k - 1;
  double th = (double)start, n = 1.0;
  bool last = false;
  for (int it = 0; it < 12; it++) {
    double d = cnt ? A[j0] - th : 1.0, t = 0.0;
    bool pos = true;
    n = 1.0;
    for (int i = 0; i < cnt; i++) {
      const int j = j0 + dir * i;
      const double b = fwd ? Bt[j + 1] : Bt[j], a = A[j + dir];
      if (!(d > 1e-30 && d < 1e30)) { pos = false; break; }
      const double q = b * tri_recip(d);  // |s_j / s_{j+dir}|
      t = b * q;
      if (!fwd) s[j] = q;
      n = fma(q * q, n, 1.0);
      d = (a - th) - t;
    }
    const bool ok = __all_sync(all, pos && n < 1e200);
    if (!ok) return false;
    const double tb = __shfl_sync(all, t, 0), tf = __shfl_sync(all, t, 1);
    const double nb = __shfl_sync(all, n, 0), nf = __shfl_sync(all, n, 1);
    n = nb + (nf - 1.0);
    const double step = ((A[r] - th) - tb - tf) / n;  // gamma / |gamma'|
    th += step;
    if (last) break;
    if (it == 11) return false;
    // quadratic from here: this step's square is below rounding
    last = fabs(step) <= 1e-9 * fmax(1.0, fabs(th));
  }
  double y = 1.0 / sqrt(n);  // |s_r|, then |s_{k-1}|
  if (lane == 0) {
    for (int j = r + 1; j < k; j++) y *= s[j];
    theta_out[0] = th;
    resid[0] = fabs(btail * y);
  }
  return true;
}

// The convergence test of a Lanczos run of k steps: false = not converged at
// tol and must_finish not set (theta and resid hold FP32 estimates, resid
// above tol), true = theta and resid (want_vec: and s) written in FP64.
static __device__ bool warp_tri_lowest(const double* A, const double* Bt, int k, double btail, double tol,
                                       bool must_finish, bool want_vec, float2* w, double* theta_out, double* s,
                                       double* resid) {
  const int lane = threadIdx.x & 31;
  if (k == 1) {
    if (lane == 0) { theta_out[0] = A[0]; s[0] = 1.0; resid[0] = fabs(btail); }
    __syncwarp();
    return true;
  }
  float th, rs;
  int peak;
  const bool est = tri_estimate(A, Bt, k, btail, w, th, peak, rs);
  if (est && !must_finish && rs > 64.f * (float)tol * fmaxf(1.f, fabsf(th))) {
    if (lane == 0) { theta_out[0] = th; resid[0] = rs; }
    __syncwarp();
    return false;
  }
  const bool fast = est && tri_newton(A, Bt, k, btail, th, peak, theta_out, s, resid);
  if (!fast) {
    const double t = tri_bisect(A, Bt, k);
    if (lane == 0) theta_out[0] = t;
  }
  __syncwarp();
  if (!fast || (want_vec && (must_finish || resid[0] <= tol * fmax(1.0, fabs(theta_out[0]))))) {
    tri_invit(A, Bt, k, theta_out[0], s);
    if (lane == 0) resid[0] = fabs(btail * s[k - 1]);
    __syncwarp();
  }
  return true;
}

}  // namespace vca
