// Device Rys roots and weights.
//
// For order n and parameter x the n roots t_r^2 (ascending) and weights w_r of
//     int_0^1 exp(-x t^2) P(t^2) dt = sum_r w_r P(t_r^2)
// are the quantities libcint's CINTrys_roots computes (rys_roots.c:57; it returns
// u = t^2/(1-t^2)).  Here they come from a piecewise polynomial table (unit-width intervals
// in x, degree CINTX_RYS_DEG in d = x - i - 1/2, generated in 50-digit arithmetic by
// gen_rys_table.py) for x < xmax[n], and from the exact large-x limit
// t_r^2 = h_r^2 / x, w_r = W_r / sqrt(x) (positive Gauss-Hermite nodes of order 2n) beyond.
#pragma once
#include "common.h"

// Device layout (rys_table_image): per order n, interval i, function f the DEG+1 monomial coefficients
// are contiguous (16-byte aligned), so one function costs (DEG+1)/2 vector loads.  Interval xmax[n] holds
// the constants h_r^2 and W_r of the large-x form as polynomials of degree 0.
constexpr int RYS_NC = CINTX_RYS_DEG + 1;  // coefficients per function (even)

// Doubles per interval of an order-n coefficient block staged in shared memory: the 2n*RYS_NC
// coefficients plus 2 of padding, so that the interval stride is an odd number of 16-byte units
// (12n + 1) and the 16-byte loads of lanes reading different intervals spread over the banks
// (unpadded, stride 12n units: lanes 2 intervals apart, n odd, or any two lanes, n even, collide).
__host__ __device__ constexpr int rys_stage_stride(int n) { return 2 * n * RYS_NC + 2; }
// Intervals of an order-n block, the large-x constants included.
__host__ __device__ constexpr int rys_intervals(int n) { return cintx_rys_xmax(n) + 1; }

// Interval of y = x - 1/2 and the distance d from its centre, by rounding y to an integer with the
// largest-integer addition (two double-precision additions in place of the conversions to an integer and
// back, which run at a quarter of their rate).
__device__ __forceinline__ int rys_interval(double y, double& d) {
  constexpr double kInt = 6755399441055744.0;  // 1.5 * 2^52: adding it leaves the integer in the low word
  const double t = y + kInt;
  d = y - (t - kInt);
  return __double2loint(t);
}

// Where a primitive quartet's roots come from, without a branch.  With s = a_ij + a_kl,
// n = a_ij a_kl |P-Q|^2 and x = n / s, the recurrences want t_r^2 / s and w_r / sqrt(s):
//   table:   poly(x) / s           and poly(x) / sqrt(s),
//   large x: (h_r^2 s / n) / s = h_r^2 / n  and  W_r / sqrt(n),
// i.e. both are table values (the large-x form's are the constants of interval xmax) times r^2 and r with
// r = 1/sqrt(s) or 1/sqrt(n): one reciprocal square root either way, and lanes of a warp on the two sides
// of the table's end do not part.  The large-x form starts 2^-20 before xmax, so that the rounding of x
// cannot lead past the last interval.
struct RysPoint {
  double r, r2;  // 1/sqrt(s) or 1/sqrt(n), and its square
  double d;      // argument of the interval's polynomials
  int i;         // interval
};
__device__ __forceinline__ RysPoint rys_point(double n, double s, int xmax) {
  RysPoint p;
  const bool big = !(n < ((double)xmax - 0x1p-20) * s);  // also routes NaN away from the table index
  p.r = rsqrt(big ? n : s);
  p.r2 = p.r * p.r;
  p.i = rys_interval(fma(n, p.r2, -0.5), p.d);
  if (big) {
    p.i = xmax;
    p.d = 0.0;
  }
  return p;
}

template <class LD>
__device__ __forceinline__ double rys_horner(const double* __restrict__ c, double d, LD ld) {
  const double2* c2 = reinterpret_cast<const double2*>(c);
  const double2 hi = ld(c2 + RYS_NC / 2 - 1);
  double acc = fma(hi.y, d, hi.x);
#pragma unroll
  for (int k = RYS_NC / 2 - 2; k >= 0; --k) {
    const double2 v = ld(c2 + k);
    acc = fma(acc, d, v.y);
    acc = fma(acc, d, v.x);
  }
  return acc;
}
__device__ __forceinline__ double rys_horner(const double* __restrict__ c, double d) {
  return rys_horner(c, d, [](const double2* q) { return __ldg(q); });
}

// Function f of order n at x: f < n -> t^2 of root f, else weight of root f - n.
__device__ __forceinline__ double rys_fn(const RysTable& c_rys, int n, int f, double x) {
  const int xmax = c_rys.xmax[n];
  if (!(x < (double)xmax)) {  // also routes NaN away from the table index
    const double* a = c_rys.asym[n];
    return f < n ? __ldg(a + f) / x : __ldg(a + f) * rsqrt(x);
  }
  double d;
  const int i = rys_interval(x - 0.5, d);
  return rys_horner(c_rys.poly[n] + ((size_t)i * 2 * n + f) * RYS_NC, d);
}

// Function f of order N at a primitive quartet's point: the table value to be scaled by p.r2 (roots) or
// p.r (weights).
template <int N>
__device__ __forceinline__ double rys_fn_at(const RysTable& c_rys, int f, const RysPoint& p) {
  return rys_horner(c_rys.poly[N] + (p.i * (2 * N) + f) * RYS_NC, p.d);
}

// All functions [F0, 2N) of order N at a point (one thread), from the global table; F0 = N gives the
// weights only.
template <int N, int F0 = 0>
__device__ __forceinline__ void rys_all_at(const RysTable& c_rys, const RysPoint& p, double* t2, double* w) {
  const double* c = c_rys.poly[N] + p.i * (2 * N * RYS_NC);
#pragma unroll
  for (int f = F0; f < 2 * N; ++f) {
    const double v = rys_horner(c + f * RYS_NC, p.d);
    if (f < N) t2[f] = v;
    else w[f - N] = v;
  }
}

// As rys_all_at, with the order-N coefficient block (rys_intervals(N) intervals, rys_stage_stride(N)
// doubles apart) staged in shared memory at `tab`.
template <int N, int F0 = 0>
__device__ __forceinline__ void rys_all_staged(const double* tab, const RysPoint& p, double* t2, double* w) {
  const double* c = tab + p.i * rys_stage_stride(N);
  auto horner = [&](int f) { return rys_horner(c + f * RYS_NC, p.d, [](const double2* q) { return *q; }); };
  // one root (its t^2 and weight polynomials) in flight at a time: the compiler barrier keeps
  // the other roots' coefficient loads from being hoisted into registers ahead of use
#pragma unroll
  for (int r = 0; r < N; ++r) {
    if (F0 <= r) t2[r] = horner(r);
    w[r] = horner(N + r);
    if (r + 1 < N) asm volatile("" ::: "memory");
  }
}

// As rys_fn_at, with the coefficient block staged in shared memory at `tab`.
template <int N>
__device__ __forceinline__ double rys_fn_staged(const double* tab, int f, const RysPoint& p) {
  return rys_horner(tab + p.i * rys_stage_stride(N) + f * RYS_NC, p.d, [](const double2* q) { return *q; });
}
