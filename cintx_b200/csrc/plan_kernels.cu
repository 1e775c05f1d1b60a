// Device-side quartet generation for screened plans.
//
// A tile (A, B) of a screened plan pairs every shell pair p of pair type A (sorted by
// decreasing Schwarz factor) with a run of the pairs of type B.  Quartets are numbered row-major;
// prefix[r] is the first quartet index of row r.  Out offsets are consecutive blocks.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "chain.cuh"
#include "common.h"

namespace cintx {
int device_sm_count();
}

// Multi-range generation: one launch fills records [rbegin, rend) of a chunk: of the whole chunk when
// it is run as one, of a single class segment when that is run alone.  ranges[] are the tile ranges that
// hold them, ordered by rec_off (a range's first record); record r belongs to the last range whose
// rec_off <= r.
//
// A warp writes `run` consecutive records (kGenRun, fewer where that would leave the chip idle), 32 at a
// time.  Its lanes search the range and the row of the warp's first record together (the same addresses for
// all lanes); a record a few places on is then usually in the same row, and where it is not, every row between
// holds at least one record, so its row lies within that many rows of the first one's and a short search ends
// there.  (One full search of both lists per record was bound by the latency of its dependent loads.)
// Records of a 40-atom s/p/d sweep: 362 us in a launch per class with one search per record, 80 us so; of 12
// atoms 157 and 11 us.
constexpr int kGenRun = 256;

__global__ void gen_range_quartets(const GenRange* __restrict__ ranges, int nranges, long long rbegin,
                                   long long rend, QuartetRec* __restrict__ recs, int run) {
  // last index in [lo, hi] whose value is <= x (the first one's is)
  auto last_le = [](const long long* v, int lo, int hi, long long x) {
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (v[mid] <= x) lo = mid;
      else hi = mid - 1;
    }
    return lo;
  };
  const int lane = threadIdx.x & 31;
  const long long warp = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long r0 = rbegin + warp * run; r0 < rend; r0 += nwarps * run) {
    int lo = 0, hi = nranges - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (ranges[mid].rec_off <= r0) lo = mid;
      else hi = mid - 1;
    }
    GenRange g = ranges[lo];
    long long next_off = lo + 1 < nranges ? ranges[lo + 1].rec_off : rend;  // first record past the range
    long long t_row = g.t0 + (r0 - g.rec_off);  // a quartet of the range and its row
    int row = last_le(g.prefix, 0, g.nrows - 1, t_row);
    long long row_start = g.prefix[row], row_end = g.prefix[row + 1];
    const long long rlast = r0 + run < rend ? r0 + run : rend;
    for (long long r = r0 + lane; r < rlast; r += 32) {
      if (r >= next_off) {  // into a later range: search its row afresh
        do {
          ++lo;
          next_off = lo + 1 < nranges ? ranges[lo + 1].rec_off : rend;
        } while (r >= next_off);
        g = ranges[lo];
        t_row = g.t0;
        row = last_le(g.prefix, 0, g.nrows - 1, t_row);
        row_start = g.prefix[row];
        row_end = g.prefix[row + 1];
      }
      const long long t = g.t0 + (r - g.rec_off);
      if (t >= row_end) {
        const long long far = row + (t - t_row);
        row = last_le(g.prefix, row + 1, far < g.nrows - 1 ? (int)far : g.nrows - 1, t);
        row_start = g.prefix[row];
        row_end = g.prefix[row + 1];
        t_row = t;
      }
      QuartetRec q;
      const int rw = g.rows[row], col = g.cols[(g.colstart ? g.colstart[row] : 0) + (t - row_start)];
      q.pij = g.swap ? col : rw;
      q.pkl = g.swap ? rw : col;
      q.out = g.out_off + (r - g.rec_off) * g.nout;
      recs[r] = q;
    }
  }
}

// x = a_ij a_kl / (a_ij + a_kl) |P - Q|^2 of every primitive quartet (b over the (kl) pair's
// primitives, a over the (ij) pair's, the ERI kernels' loop order) of nrec records, written at
// xout[pbase[r] + b * npij + a].  The kernels' own table roots are evaluated at an x that differs from
// this one by rounding (rys_point).
__global__ void prim_x_kernel(const QuartetRec* __restrict__ recs, long long nrec, const ShellPair* __restrict__ pairs,
                              const PrimPair* __restrict__ prims, const long long* __restrict__ pbase,
                              double* __restrict__ xout) {
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < nrec;
       r += (long long)gridDim.x * blockDim.x) {
    const QuartetRec rec = recs[r];
    const ShellPair pij = pairs[rec.pij], pkl = pairs[rec.pkl];
    for (int b = 0; b < pkl.nprim; ++b) {
      const PrimPair pk = prims[pkl.prim_off + b];
      for (int a = 0; a < pij.nprim; ++a) {
        const PrimPair pi = prims[pij.prim_off + a];
        const double aijkl = pi.aij + pk.aij;
        const double rs = rsqrt(aijkl);
        const double pqx = pi.px - pk.px, pqy = pi.py - pk.py, pqz = pi.pz - pk.pz;
        xout[pbase[r] + (long long)b * pij.nprim + a] =
            pi.aij * pk.aij * (rs * rs) * (pqx * pqx + pqy * pqy + pqz * pqz);
      }
    }
  }
}

// q[r] = sqrt(max |out[recs[r].out .. + len[r])|): one warp per record.
__global__ void block_absmax_sqrt_kernel(const QuartetRec* __restrict__ recs, long long nrec,
                                         const double* __restrict__ out, const long long* __restrict__ len,
                                         double* __restrict__ q) {
  const int lane = threadIdx.x & 31;
  for (long long r = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; r < nrec;
       r += ((long long)gridDim.x * blockDim.x) >> 5) {
    const double* o = out + recs[r].out;
    double m = 0.0;
    for (long long e = lane; e < len[r]; e += 32) m = fmax(m, fabs(o[e]));
    for (int s = 16; s > 0; s >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, s));
    if (lane == 0) q[r] = sqrt(m);
  }
}

// Division of a small non-negative number by a block extent: e / d for e < 2^16, d <= 15 (the error of
// the reciprocal, e (m d - 2^32) / 2^32 < e / 2^28, stays under 1 / d).
struct SmallDiv {
  unsigned d, m;  // m = ceil(2^32 / d), 0 for d == 1
};
static SmallDiv small_divisor(int d) {
  return SmallDiv{(unsigned)d, d == 1 ? 0u : (unsigned)(((1ull << 32) + d - 1) / d)};
}
__device__ __forceinline__ unsigned small_div(unsigned e, const SmallDiv& v) { return v.m ? __umulhi(e, v.m) : e; }

// The AO table of a plan's pairs: first functions of the pair's two shells (block axes 0 and 1), the
// second one's sign bit set where both are one shell (those blocks hold every element twice).
__device__ __forceinline__ int pair_ao(const int2& p) { return p.y & 0x7fffffff; }
__device__ __forceinline__ double pair_weight(const int2& p) { return p.y < 0 ? 0.5 : 1.0; }

// Coulomb/exchange contraction of one chunk of a unique-quartet sweep (a >= b, c >= d, ab >= cd):
// one warp per quartet block v[i + ni*(j + nj*(k + nk*l))] (shells a, b, c, d), with the 8-fold
// permutational symmetry of real integrals and a symmetric density D (row-major nao x nao):
//   A[i,j] += 2 s sum_kl v D[k,l],  A[k,l] += 2 s sum_ij v D[i,j]          (J = A + A^T)
//   B[i,k] += s sum_jl v D[j,l],  B[j,k] += s sum_il v D[i,l],
//   B[i,l] += s sum_jk v D[j,k],  B[j,l] += s sum_ik v D[i,k]               (K = B + B^T)
// with s = 1/2 for each of a == b, c == d, (ab) == (cd) (those blocks hold every element twice).
// Each (row, column) pair of a block reduces its sum first and adds it with one atomic.
__global__ void jk_contract_kernel(const QuartetRec* __restrict__ recs, long long nrec, const int2* __restrict__ pao,
                                   const double* __restrict__ out, const double* __restrict__ dm, int nao,
                                   double* __restrict__ A, double* __restrict__ B, int ni, int nj, int nk, int nl,
                                   int chain, int nblocks) {
  if (chain_begin(chain, nblocks)) return;
  const int lane = threadIdx.x & 31;
  for (long long r = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; r < nrec;
       r += ((long long)nblocks * blockDim.x) >> 5) {
    const QuartetRec rec = recs[r];
    const int2 ab = pao[rec.pij], cd = pao[rec.pkl];
    const int i0 = ab.x, j0 = pair_ao(ab), k0 = cd.x, l0 = pair_ao(cd);
    const double s = pair_weight(ab) * pair_weight(cd) * (rec.pij == rec.pkl ? 0.5 : 1.0);
    const double* v = out + rec.out;
    const int sj = ni, sk = ni * nj, sl = ni * nj * nk;
    if (A) {
      for (int e = lane; e < ni * nj; e += 32) {
        const int i = e % ni, j = e / ni;
        double t = 0.0;
        for (int l = 0; l < nl; ++l)
          for (int k = 0; k < nk; ++k) t += v[i + j * sj + k * sk + l * sl] * dm[(size_t)(k0 + k) * nao + l0 + l];
        atomicAdd(A + (size_t)(i0 + i) * nao + j0 + j, 2.0 * s * t);
      }
      for (int e = lane; e < nk * nl; e += 32) {
        const int k = e % nk, l = e / nk;
        double t = 0.0;
        for (int j = 0; j < nj; ++j)
          for (int i = 0; i < ni; ++i) t += v[i + j * sj + k * sk + l * sl] * dm[(size_t)(i0 + i) * nao + j0 + j];
        atomicAdd(A + (size_t)(k0 + k) * nao + l0 + l, 2.0 * s * t);
      }
    }
    if (B) {
      for (int e = lane; e < ni * nk; e += 32) {  // B[i,k] += s sum_jl v D[j,l]
        const int i = e % ni, k = e / ni;
        double t = 0.0;
        for (int l = 0; l < nl; ++l)
          for (int j = 0; j < nj; ++j) t += v[i + j * sj + k * sk + l * sl] * dm[(size_t)(j0 + j) * nao + l0 + l];
        atomicAdd(B + (size_t)(i0 + i) * nao + k0 + k, s * t);
      }
      for (int e = lane; e < nj * nk; e += 32) {  // B[j,k] += s sum_il v D[i,l]
        const int j = e % nj, k = e / nj;
        double t = 0.0;
        for (int l = 0; l < nl; ++l)
          for (int i = 0; i < ni; ++i) t += v[i + j * sj + k * sk + l * sl] * dm[(size_t)(i0 + i) * nao + l0 + l];
        atomicAdd(B + (size_t)(j0 + j) * nao + k0 + k, s * t);
      }
      for (int e = lane; e < ni * nl; e += 32) {  // B[i,l] += s sum_jk v D[j,k]
        const int i = e % ni, l = e / ni;
        double t = 0.0;
        for (int k = 0; k < nk; ++k)
          for (int j = 0; j < nj; ++j) t += v[i + j * sj + k * sk + l * sl] * dm[(size_t)(j0 + j) * nao + k0 + k];
        atomicAdd(B + (size_t)(i0 + i) * nao + l0 + l, s * t);
      }
      for (int e = lane; e < nj * nl; e += 32) {  // B[j,l] += s sum_ik v D[i,k]
        const int j = e % nj, l = e / nj;
        double t = 0.0;
        for (int k = 0; k < nk; ++k)
          for (int i = 0; i < ni; ++i) t += v[i + j * sj + k * sk + l * sl] * dm[(size_t)(i0 + i) * nao + k0 + k];
        atomicAdd(B + (size_t)(j0 + j) * nao + l0 + l, s * t);
      }
    }
  }
}

// Scatters a class segment (blocks ni x nj x nk x nl) of a unique-quartet sweep into an AO tensor, G lanes
// (the power of two from the block size up, at most a warp) per quartet block:
//   mode 1 (PySCF ao2mo's "s1"): eri[((p*nao + q)*nao + r)*nao + s] at the eight index orders the quartet
//          stands for;
//   mode 4 ("s4"): the pair-pair matrix eri[pq*npair + rs] and its transposed slot, pq = p*(p+1)/2 + q
//          over p >= q;
//   mode 8 ("s8"): eri[pq*(pq+1)/2 + rs], pq >= rs.
// Slots reached twice receive equal elements.  Bound: the scattered writes.  Each index order is written
// with the axis that is contiguous in it fastest over the lanes, so that a shell's 3 to 7 functions share
// memory sectors (one pass over the block per pair of orders; the block is read again from L1).  Clearing
// and scatter, beside the sweep itself: s8 of 24 atoms (2.0 GB) 863 -> 632 us, s4 of 18 (1.1 GB) 580 -> 496,
// s1 of 14 (1.9 GB, 254 of it the clearing) 980 -> 947.
template <int MODE>
__global__ void scatter_ao_kernel(const QuartetRec* __restrict__ recs, long long nrec, const int2* __restrict__ pao,
                                  const double* __restrict__ out, double* __restrict__ eri, long long nao,
                                  SmallDiv ni, SmallDiv nj, SmallDiv nk, SmallDiv nl, int G, int chain, int nblocks) {
  if (chain_begin(chain, nblocks)) return;
  const int g = threadIdx.x & (G - 1);
  const long long npair = nao * (nao + 1) / 2, n2 = nao * nao;
  const unsigned n = ni.d * nj.d * nk.d * nl.d;
  const unsigned sj = ni.d, sk = ni.d * nj.d, sl = ni.d * nj.d * nk.d;
  const long long ngroups = (long long)nblocks * blockDim.x / G;
  for (long long r = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / G; r < nrec; r += ngroups) {
    const QuartetRec rec = recs[r];
    const int2 ab = pao[rec.pij], cd = pao[rec.pkl];
    const long long i0 = ab.x, j0 = pair_ao(ab), k0 = cd.x, l0 = pair_ao(cd);
    const double* v = out + rec.out;
    if constexpr (MODE == 1) {
      for (unsigned e = g; e < n; e += G) {  // l fastest, then k, j, i
        const unsigned a = small_div(e, nl), b = small_div(a, nk), c = small_div(b, nj);
        const unsigned l = e - a * nl.d, k = a - b * nk.d, j = b - c * nj.d, i = c;
        const double x = v[i + j * sj + k * sk + l * sl];
        const long long uw = (k0 + k) * nao + l0 + l;
        eri[((i0 + i) * nao + j0 + j) * n2 + uw] = x;
        eri[((j0 + j) * nao + i0 + i) * n2 + uw] = x;
      }
      for (unsigned e = g; e < n; e += G) {  // k fastest, then l, j, i
        const unsigned a = small_div(e, nk), b = small_div(a, nl), c = small_div(b, nj);
        const unsigned k = e - a * nk.d, l = a - b * nl.d, j = b - c * nj.d, i = c;
        const double x = v[i + j * sj + k * sk + l * sl];
        const long long wu = (l0 + l) * nao + k0 + k;
        eri[((i0 + i) * nao + j0 + j) * n2 + wu] = x;
        eri[((j0 + j) * nao + i0 + i) * n2 + wu] = x;
      }
      for (unsigned e = g; e < n; e += G) {  // j fastest, then i, l, k
        const unsigned a = small_div(e, nj), b = small_div(a, ni), c = small_div(b, nl);
        const unsigned j = e - a * nj.d, i = a - b * ni.d, l = b - c * nl.d, k = c;
        const double x = v[i + j * sj + k * sk + l * sl];
        const long long pq = (i0 + i) * nao + j0 + j;
        eri[((k0 + k) * nao + l0 + l) * n2 + pq] = x;
        eri[((l0 + l) * nao + k0 + k) * n2 + pq] = x;
      }
      for (unsigned e = g; e < n; e += G) {  // i fastest, then j, l, k
        const unsigned a = small_div(e, ni), b = small_div(a, nj), c = small_div(b, nl);
        const unsigned i = e - a * ni.d, j = a - b * nj.d, l = b - c * nl.d, k = c;
        const double x = v[i + j * sj + k * sk + l * sl];
        const long long qp = (j0 + j) * nao + i0 + i;
        eri[((k0 + k) * nao + l0 + l) * n2 + qp] = x;
        eri[((l0 + l) * nao + k0 + k) * n2 + qp] = x;
      }
    } else {
      // an AO pair's packed index runs along its smaller function: fastest the smaller shell of each side
      // (a block of a diagonal pair, which reaches slots twice, in its own order in both: the last one stays)
      const bool twice = ab.y < 0 || cd.y < 0 || rec.pij == rec.pkl;
      const bool klow = twice || k0 < l0, ilow = twice || i0 < j0;
      const SmallDiv f1 = klow ? nk : nl, f2 = klow ? nl : nk, f3 = ilow ? ni : nj, f4 = ilow ? nj : ni;
      for (int pass = 0; pass < (MODE == 4 ? 2 : 1); ++pass) {
        // pass 0: the (kl) side fastest; pass 1 (s4's transposed slot): the (ij) side
        const bool ij_fast = pass || twice;
        const SmallDiv d1 = ij_fast ? f3 : f1, d2 = ij_fast ? f4 : f2, d3 = ij_fast ? f1 : f3;
        for (unsigned e = g; e < n; e += G) {
          const unsigned a = small_div(e, d1), b = small_div(a, d2), c = small_div(b, d3);
          const unsigned x1 = e - a * d1.d, x2 = a - b * d2.d, x3 = b - c * d3.d, x4 = c;
          const unsigned lo_kl = ij_fast ? x3 : x1, hi_kl = ij_fast ? x4 : x2;
          const unsigned lo_ij = ij_fast ? x1 : x3, hi_ij = ij_fast ? x2 : x4;
          const unsigned k = klow ? lo_kl : hi_kl, l = klow ? hi_kl : lo_kl;
          const unsigned i = ilow ? lo_ij : hi_ij, j = ilow ? hi_ij : lo_ij;
          const double x = v[i + j * sj + k * sk + l * sl];
          const long long p = i0 + i, q = j0 + j, u = k0 + k, w = l0 + l;
          const long long pq = p >= q ? p * (p + 1) / 2 + q : q * (q + 1) / 2 + p;
          const long long uw = u >= w ? u * (u + 1) / 2 + w : w * (w + 1) / 2 + u;
          if (MODE == 8) eri[pq >= uw ? pq * (pq + 1) / 2 + uw : uw * (uw + 1) / 2 + pq] = x;
          else if (pass == 0) eri[pq * npair + uw] = x;
          else eri[uw * npair + pq] = x;
        }
      }
    }
  }
}

// The same contraction with compile-time ket extents, each block element read once.  A group of G lanes
// (the power of two from nij = ni*nj up, at most a warp) takes one quartet: lane <-> (i,j) (several of
// them in turn where nij > 32), and walks the block's (k,l) elements, consecutive lanes reading
// consecutive doubles.  Per element x it adds x D[k,l] to its A[i,j] sum, x D[j,l] and x D[i,l] to two
// sums per k, x D[j,k] and x D[i,k] to two sums per l (all in registers), and the group reduces x D[i,j]
// over its lanes into A[k,l] (halving_sum: about NK shuffles per l).  The per-(i,j) sums then meet in
// shared memory, where they are reduced over j (i) before one atomic per element of B[i,kl] (B[j,kl]).
// Consecutive quartets of a tile row share their (ij) pair, so a group takes runs of `run` records (up to
// kJkRun, fewer where the records would not give every resident warp work) and adds A[i,j] once per run
// and pair.
//
// Bound: instructions and the gathers of the density; the atomics, about (nk + nl)(ni + nj) + nk nl per
// quartet, are not (leaving them all out: 2%).  J+K of 120 s/p/d/f atoms (5.7e9 integrals): 139 ms of
// contraction with six passes over each block, 68 ms so, 48 with jk_contract_thread_kernel and the rest.
constexpr int kJkRun = 16;
constexpr int kJkWarps = 4;

// doubles of shared memory per group: D[k,l], A[k,l], A[i,j] and the per-(i,j) sums
__host__ __device__ constexpr int jk_group_doubles(int nij, int nk, int nl) {
  return 2 * nk * nl + nij + nij * 2 * (nk + nl);
}

// Sums p[0..N) over the group of G lanes starting at a multiple of G: where G >= 2, each step sends one
// half of the values still held to the lane a power of two away and keeps the other half.  On return p[0]
// is the group's sum of value `*which`; lanes with equal `*which` hold the same sum.
template <int N>
__device__ __forceinline__ void halving_sum(double (&p)[N], int G, unsigned mask, int lane, int* which) {
  static_assert((N & (N - 1)) == 0, "padded to a power of two");
  int w = 0, o = G >> 1;
  if constexpr (N > 1) {
    double h[N / 2];
    if (o > 0) {
      const bool up = lane & o;
#pragma unroll
      for (int n = 0; n < N / 2; ++n) {
        const double keep = up ? p[n + N / 2] : p[n], send = up ? p[n] : p[n + N / 2];
        h[n] = keep + __shfl_xor_sync(mask, send, o);
      }
      w = up ? N / 2 : 0;
      int sub = 0;
      halving_sum<N / 2>(h, o, mask, lane, &sub);
      p[0] = h[0];
      *which = w + sub;
      return;
    }
    *which = 0;  // one lane left with several values: the caller reads p[0..N)
  } else {
    for (; o > 0; o >>= 1) p[0] += __shfl_xor_sync(mask, p[0], o);
    *which = 0;
  }
}

template <int NK, int NL>
__global__ void __launch_bounds__(32 * kJkWarps)
    jk_contract_group_kernel(const QuartetRec* __restrict__ recs, long long nrec, const int2* __restrict__ pao,
                             const double* __restrict__ out,
                             const double* __restrict__ dm, int nao, double* __restrict__ A, double* __restrict__ B,
                             SmallDiv di_, SmallDiv dj_, int G, int run, int chain, int nblocks) {
  if (chain_begin(chain, nblocks)) return;
  constexpr int NP = NK <= 1 ? 1 : NK <= 2 ? 2 : NK <= 4 ? 4 : NK <= 8 ? 8 : 16;
  constexpr int NKL = NK + NL;
  extern __shared__ double sm[];
  const int ni = (int)di_.d, nj = (int)dj_.d, nij = ni * nj;
  const int lane = threadIdx.x & 31, g = lane & (G - 1);
  const unsigned mask = G == 32 ? 0xffffffffu : (((1u << G) - 1u) << (lane & ~(G - 1)));
  double* s_dkl = sm + (size_t)(threadIdx.x / G) * jk_group_doubles(nij, NK, NL);
  double* s_akl = s_dkl + NK * NL;
  double* s_aij = s_akl + NK * NL;
  double* s_t = s_aij + nij;  // [2 * NKL][nij]: sums over l with D[j,l], over k with D[j,k]; with D[i,l], D[i,k]
  const long long gid = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / G;
  const long long ngroups = (long long)nblocks * blockDim.x / G;
  for (long long base = gid * run; base < nrec; base += ngroups * run) {
    const long long rend = base + run < nrec ? base + run : nrec;
    int cur = -1;  // the (ij) pair whose A[i,j] sums s_aij holds
    int i0 = 0, j0 = 0;
    double sij = 0;
    QuartetRec next = recs[base];
    int2 next_cd = pao[next.pkl];
    for (long long r = base; r < rend; ++r) {
      const QuartetRec rec = next;
      const int2 cd = next_cd;
      if (r + 1 < rend) {  // on its way while this quartet is contracted
        next = recs[r + 1];
        next_cd = pao[next.pkl];
      }
      const int k0 = cd.x, l0 = pair_ao(cd);
      if (rec.pij != cur) {
        if (cur >= 0 && A)
          for (int e = g; e < nij; e += G) {
            const int j = (int)small_div(e, di_);
            atomicAdd(A + (size_t)(i0 + e - j * ni) * nao + j0 + j, s_aij[e]);
          }
        const int2 ab = pao[rec.pij];
        i0 = ab.x;
        j0 = pair_ao(ab);
        sij = pair_weight(ab);
        cur = rec.pij;
        for (int e = g; e < nij; e += G) s_aij[e] = 0.0;
      }
      const double s = sij * pair_weight(cd) * (rec.pij == rec.pkl ? 0.5 : 1.0);
      for (int e = g; e < NK * NL; e += G) {
        s_dkl[e] = dm[(size_t)(k0 + e % NK) * nao + l0 + e / NK];
        s_akl[e] = 0.0;
      }
      __syncwarp(mask);
      for (int ij0 = 0; ij0 < nij; ij0 += G) {
        const int ij = ij0 + g;
        const bool on = ij < nij;
        const int j = on ? (int)small_div(ij, di_) : 0, i = on ? ij - j * ni : 0;
        const double* v = out + rec.out + (on ? ij : 0);
        const double* di = dm + (size_t)(i0 + i) * nao;
        const double* dj = dm + (size_t)(j0 + j) * nao;
        const double dij = on ? di[j0 + j] : 0.0;  // not 0 times an infinity in a lane without an element
        double djk[NK], dik[NK], t[NK], u[NK];
#pragma unroll
        for (int k = 0; k < NK; ++k) {
          djk[k] = dj[k0 + k];
          dik[k] = di[k0 + k];
          t[k] = u[k] = 0.0;
        }
        double aij = 0.0;
#pragma unroll
        for (int l = 0; l < NL; ++l) {
          const double djl = dj[l0 + l], dil = di[l0 + l];
          double sl = 0.0, wl = 0.0, p[NP];
#pragma unroll
          for (int k = 0; k < NK; ++k) {
            const double x = on ? v[(size_t)nij * (k + NK * l)] : 0.0;
            aij = fma(x, s_dkl[k + NK * l], aij);
            t[k] = fma(x, djl, t[k]);
            u[k] = fma(x, dil, u[k]);
            sl = fma(x, djk[k], sl);
            wl = fma(x, dik[k], wl);
            p[k] = x * dij;
          }
#pragma unroll
          for (int k = NK; k < NP; ++k) p[k] = 0.0;
          if (on) {
            s_t[(NK + l) * nij + ij] = sl;
            s_t[(NKL + NK + l) * nij + ij] = wl;
          }
          if (G >= NP) {  // one value per lane is left; the first lane of each value adds it up
            int w;
            halving_sum<NP>(p, G, mask, g, &w);
            if (w < NK && (g & (G / NP - 1)) == 0) s_akl[w + NK * l] += p[0];
          } else {
#pragma unroll
            for (int k = 0; k < NK; ++k) {
              for (int o = G >> 1; o > 0; o >>= 1) p[k] += __shfl_xor_sync(mask, p[k], o);
              if (g == 0) s_akl[k + NK * l] += p[k];
            }
          }
        }
        if (on) {
          s_aij[ij] = fma(2.0 * s, aij, s_aij[ij]);
#pragma unroll
          for (int k = 0; k < NK; ++k) {
            s_t[k * nij + ij] = t[k];
            s_t[(NKL + k) * nij + ij] = u[k];
          }
        }
      }
      __syncwarp(mask);
      if (A)
        for (int e = g; e < NK * NL; e += G)
          atomicAdd(A + (size_t)(k0 + e % NK) * nao + l0 + e / NK, 2.0 * s * s_akl[e]);
      if (B) {
        for (int e = g; e < ni * NKL; e += G) {  // B[i, k or l]: sums over j
          const int c = (int)small_div(e, di_), i = e - c * ni;
          const double* x = s_t + c * nij + i;
          double sum = 0.0;
          for (int j = 0; j < nj; ++j) sum += x[ni * j];
          atomicAdd(B + (size_t)(i0 + i) * nao + (c < NK ? k0 + c : l0 + c - NK), s * sum);
        }
        for (int e = g; e < nj * NKL; e += G) {  // B[j, k or l]: sums over i
          const int c = (int)small_div(e, dj_), j = e - c * nj;
          const double* x = s_t + (NKL + c) * nij + ni * j;
          double sum = 0.0;
          for (int i = 0; i < ni; ++i) sum += x[i];
          atomicAdd(B + (size_t)(j0 + j) * nao + (c < NK ? k0 + c : l0 + c - NK), s * sum);
        }
      }
      __syncwarp(mask);
    }
    if (cur >= 0 && A)
      for (int e = g; e < nij; e += G) {
        const int j = (int)small_div(e, di_);
        atomicAdd(A + (size_t)(i0 + e - j * ni) * nao + j0 + j, s_aij[e]);
      }
    __syncwarp(mask);
  }
}

// The same contraction for small kets (nk <= 3, nl = 1): one thread per quartet, consecutive lanes the
// consecutive quartets of a tile row.  A group of lanes per quartet (jk_contract_group_kernel) spends
// most of its instructions on handing three elements per lane around; here a thread walks its own block,
// j after j with the i axis unrolled, and keeps every exchange sum of the i axis in registers (nothing
// is shared), while D[i,j] is the same for the whole warp and A[i,j] is reduced over the warp (halving_sum)
// before one atomic per row and (i,j).  A warp whose lanes meet more than one (ij) pair (the end of a row)
// adds A[i,j] lane by lane.  J+K of 120 s/p/d/f atoms: 229.8 -> 217.0 ms.
template <int NI, int NK>
__global__ void __launch_bounds__(128)
    jk_contract_thread_kernel(const QuartetRec* __restrict__ recs, long long nrec, const int2* __restrict__ pao,
                              const double* __restrict__ out, const double* __restrict__ dm, int nao,
                              double* __restrict__ A, double* __restrict__ B, int nj, int chain, int nblocks) {
  if (chain_begin(chain, nblocks)) return;
  constexpr int NP = NI <= 1 ? 1 : NI <= 4 ? 4 : NI <= 8 ? 8 : 16;
  const int lane = threadIdx.x & 31;
  const long long stride = (long long)nblocks * blockDim.x;
  // whole warps run (lanes past the end repeat the last record with weight 0 and store nothing)
  for (long long r0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) - lane; r0 < nrec; r0 += stride) {
    const bool on = r0 + lane < nrec;
    const QuartetRec rec = recs[on ? r0 + lane : nrec - 1];
    const int2 ab = pao[rec.pij], cd = pao[rec.pkl];
    const int i0 = ab.x, j0 = pair_ao(ab), k0 = cd.x, l0 = pair_ao(cd);
    const double s = on ? pair_weight(ab) * pair_weight(cd) * (rec.pij == rec.pkl ? 0.5 : 1.0) : 0.0;
    const bool one_row = __all_sync(0xffffffffu, rec.pij == __shfl_sync(0xffffffffu, rec.pij, 0));
    const double* v = out + rec.out;
    double dkl[NK], akl[NK], dil[NI], dik[NI][NK], sil[NI], tik[NI][NK];
#pragma unroll
    for (int k = 0; k < NK; ++k) {
      dkl[k] = 2.0 * s * dm[(size_t)(k0 + k) * nao + l0];
      akl[k] = 0.0;
    }
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const double* di = dm + (size_t)(i0 + i) * nao;
      dil[i] = di[l0];
      sil[i] = 0.0;
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        dik[i][k] = di[k0 + k];
        tik[i][k] = 0.0;
      }
    }
    for (int j = 0; j < nj; ++j) {
      const double* dj = dm + (size_t)(j0 + j) * nao;
      const double djl = dj[l0];
      double djk[NK], ujk[NK], wjl = 0.0, p[NP];
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        djk[k] = dj[k0 + k];
        ujk[k] = 0.0;
      }
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const double dij = dm[(size_t)(i0 + i) * nao + j0 + j];
        double aij = 0.0;
#pragma unroll
        for (int k = 0; k < NK; ++k) {
          const double x = v[i + NI * (j + nj * k)];
          aij = fma(x, dkl[k], aij);
          akl[k] = fma(x, dij, akl[k]);
          tik[i][k] = fma(x, djl, tik[i][k]);
          ujk[k] = fma(x, dil[i], ujk[k]);
          sil[i] = fma(x, djk[k], sil[i]);
          wjl = fma(x, dik[i][k], wjl);
        }
        p[i] = on ? aij : 0.0;  // weight 0 times an infinite density is not 0
      }
      if (A) {
        if (one_row) {
#pragma unroll
          for (int i = NI; i < NP; ++i) p[i] = 0.0;
          int w;
          halving_sum<NP>(p, 32, 0xffffffffu, lane, &w);
          if (w < NI && (lane & (32 / NP - 1)) == 0) atomicAdd(A + (size_t)(i0 + w) * nao + j0 + j, p[0]);
        } else if (on) {
#pragma unroll
          for (int i = 0; i < NI; ++i) atomicAdd(A + (size_t)(i0 + i) * nao + j0 + j, p[i]);
        }
      }
      if (B && on) {
        double* bj = B + (size_t)(j0 + j) * nao;
#pragma unroll
        for (int k = 0; k < NK; ++k) atomicAdd(bj + k0 + k, s * ujk[k]);
        atomicAdd(bj + l0, s * wjl);
      }
    }
    if (!on) continue;
    if (A) {
#pragma unroll
      for (int k = 0; k < NK; ++k) atomicAdd(A + (size_t)(k0 + k) * nao + l0, 2.0 * s * akl[k]);
    }
    if (B) {
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        double* bi = B + (size_t)(i0 + i) * nao;
#pragma unroll
        for (int k = 0; k < NK; ++k) atomicAdd(bi + k0 + k, s * tik[i][k]);
        atomicAdd(bi + l0, s * sil[i]);
      }
    }
  }
}

// M[p,q] = X[p,q] + X[q,p] (n x n), for J = A + A^T and K = B + B^T.
__global__ void symmetrize_kernel(const double* __restrict__ X, double* __restrict__ M, int n) {
  const long long total = (long long)n * n;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int p = (int)(e / n), q = (int)(e % n);
    M[e] = X[e] + X[(size_t)q * n + p];
  }
}

namespace cintx {
cudaError_t launch_prim_x(const QuartetRec* recs, long long nrec, const ShellPair* pairs, const PrimPair* prims,
                          const long long* pbase, double* xout, cudaStream_t stream) {
  if (nrec <= 0) return cudaSuccess;
  long long blocks = (nrec + 127) / 128;
  if (blocks > 65535) blocks = 65535;
  prim_x_kernel<<<(unsigned)blocks, 128, 0, stream>>>(recs, nrec, pairs, prims, pbase, xout);
  return cudaGetLastError();
}

cudaError_t launch_block_absmax_sqrt(const QuartetRec* recs, long long nrec, const double* out, const long long* len,
                                     double* q, cudaStream_t stream) {
  if (nrec <= 0) return cudaSuccess;
  long long blocks = (nrec * 32 + 255) / 256;
  if (blocks > 65535) blocks = 65535;
  block_absmax_sqrt_kernel<<<(unsigned)blocks, 256, 0, stream>>>(recs, nrec, out, len, q);
  return cudaGetLastError();
}

// Most dynamic shared memory of a jk_contract_group_kernel block (of the 227 KB a block may have).
constexpr size_t kJkSmem = 200 * 1024;

static int jk_group_lanes(int nij) {
  int G = 1;
  while (G < 32 && G < nij) G *= 2;
  return G;
}
static size_t jk_group_smem(int nij, int nk, int nl) {
  return sizeof(double) * (size_t)jk_group_doubles(nij, nk, nl) * (32 * kJkWarps / jk_group_lanes(nij));
}

template <int NK, int NL>
static cudaError_t launch_jk_group(const QuartetRec* recs, long long nrec, const int2* pao, const double* out,
                                   const double* dm, int nao, double* A, double* B,
                                   cudaStream_t stream, int ni, int nj, int chain) {
  const int G = jk_group_lanes(ni * nj);
  const size_t smem = jk_group_smem(ni * nj, NK, NL);
  auto kern = jk_contract_group_kernel<NK, NL>;
  // The limit is a property of the kernel that all host threads share, and one instance serves bras of
  // several sizes: it is set to what the largest may take, never to this launch's own size.
  static std::atomic<int> attr_done[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !attr_done[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kJkSmem);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) attr_done[dev] = 1;
  }
  const long long resident = (long long)device_sm_count() * 16 * (32 / G);  // groups, 16 warps per SM
  const int run = (int)std::max(1LL, std::min<long long>(kJkRun, nrec / (2 * resident)));
  const long long per_block = 32LL * kJkWarps / G * run;
  long long blocks = (nrec + per_block - 1) / per_block;
  if (blocks > (long long)device_sm_count() * 64) blocks = (long long)device_sm_count() * 64;
  return chain_launch(kern, (unsigned)blocks, 32 * kJkWarps, smem, stream, chain, recs, nrec, pao, out, dm, nao, A, B,
                      small_divisor(ni), small_divisor(nj), G, run);
}

template <int NI, int NK>
static cudaError_t launch_jk_thread(const QuartetRec* recs, long long nrec, const int2* pao, const double* out,
                                    const double* dm, int nao, double* A, double* B, cudaStream_t stream, int nj,
                                    int chain) {
  const long long blocks = std::min((nrec + 127) / 128, (long long)device_sm_count() * 64);
  return chain_launch(jk_contract_thread_kernel<NI, NK>, (unsigned)blocks, 128, 0, stream, chain, recs, nrec, pao, out,
                      dm, nao, A, B, nj);
}

// One class segment, blocks ni x nj x nk x nl.  Small kets (nl = 1, nk <= 3) take a thread per quartet
// where its sums, 2 ni (nk + 1) doubles, fit the registers (ni <= 9 for nk = 1, 7 for nk = 3).  Other ket
// extents up to 10 have a kernel for groups of lanes (sph 1..9, cart 1..10); cartesian g kets (15
// functions: the sums of one lane no longer fit registers) keep the general kernel.
cudaError_t launch_jk_contract(const QuartetRec* recs, long long nrec, const int2* pao, const double* out,
                               const double* dm, int nao, double* A, double* B, cudaStream_t stream,
                               int ni, int nj, int nk, int nl, int chain) {
  if (nrec <= 0) return cudaSuccess;
#define CINTX_JK_THREAD(I, K) \
  if (ni == I && nk == K && nl == 1)  \
    return launch_jk_thread<I, K>(recs, nrec, pao, out, dm, nao, A, B, stream, nj, chain);
  CINTX_JK_THREAD(1, 1) CINTX_JK_THREAD(3, 1) CINTX_JK_THREAD(5, 1) CINTX_JK_THREAD(6, 1) CINTX_JK_THREAD(7, 1)
  CINTX_JK_THREAD(9, 1) CINTX_JK_THREAD(3, 3) CINTX_JK_THREAD(5, 3) CINTX_JK_THREAD(6, 3) CINTX_JK_THREAD(7, 3)
#undef CINTX_JK_THREAD
#define CINTX_JK(K, L) \
  if (nk == K && nl == L) return launch_jk_group<K, L>(recs, nrec, pao, out, dm, nao, A, B, stream, ni, nj, chain);
  if (jk_group_smem(ni * nj, nk, nl) <= kJkSmem) {
    CINTX_JK(1, 1) CINTX_JK(3, 1) CINTX_JK(3, 3)  // (1, 1): cartesian f and g first shells, (3, 1): spherical g too
    CINTX_JK(5, 1) CINTX_JK(5, 3) CINTX_JK(5, 5)
    CINTX_JK(6, 1) CINTX_JK(6, 3) CINTX_JK(6, 6)
    CINTX_JK(7, 1) CINTX_JK(7, 3) CINTX_JK(7, 5) CINTX_JK(7, 7)
    CINTX_JK(9, 1) CINTX_JK(9, 3) CINTX_JK(9, 5) CINTX_JK(9, 7) CINTX_JK(9, 9)
    CINTX_JK(10, 1) CINTX_JK(10, 3) CINTX_JK(10, 6) CINTX_JK(10, 10)
  }
#undef CINTX_JK
  long long blocks = (nrec * 32 + 255) / 256;
  if (blocks > (long long)device_sm_count() * 64) blocks = (long long)device_sm_count() * 64;
  return chain_launch(jk_contract_kernel, (unsigned)blocks, 256, 0, stream, chain, recs, nrec, pao, out, dm, nao, A, B,
                      ni, nj, nk, nl);
}

cudaError_t launch_scatter_ao(const QuartetRec* recs, long long nrec, const int2* pao, const double* out,
                              double* eri, int mode, long long nao, int ni, int nj, int nk, int nl,
                              cudaStream_t stream, int chain) {
  if (nrec <= 0) return cudaSuccess;
  int G = 1;
  while (G < 32 && G < ni * nj * nk * nl) G *= 2;
  long long blocks = (nrec * G + 255) / 256;
  if (blocks > (long long)device_sm_count() * 64) blocks = (long long)device_sm_count() * 64;
  auto kern = mode == 1 ? scatter_ao_kernel<1> : (mode == 4 ? scatter_ao_kernel<4> : scatter_ao_kernel<8>);
  return chain_launch(kern, (unsigned)blocks, 256, 0, stream, chain, recs, nrec, pao, out, eri, nao, small_divisor(ni),
                      small_divisor(nj), small_divisor(nk), small_divisor(nl), G);
}

cudaError_t launch_symmetrize(const double* X, double* M, int n, cudaStream_t stream) {
  const long long total = (long long)n * n;
  long long blocks = (total + 255) / 256;
  if (blocks > (long long)device_sm_count() * 32) blocks = (long long)device_sm_count() * 32;
  if (total > 0) symmetrize_kernel<<<(unsigned)blocks, 256, 0, stream>>>(X, M, n);
  return cudaGetLastError();
}

cudaError_t launch_gen_ranges(const GenRange* ranges, int nranges, long long rbegin, long long rend, QuartetRec* recs,
                              cudaStream_t stream) {
  const long long nrec = rend - rbegin;
  if (nrec <= 0) return cudaSuccess;
  const int run = 32 * (int)std::max(1LL, std::min<long long>(kGenRun / 32, nrec / (device_sm_count() * 64LL * 32)));
  long long blocks = (nrec + 8 * run - 1) / (8 * run);  // 8 warps per block
  if (blocks > 65535) blocks = 65535;
  gen_range_quartets<<<(unsigned)blocks, 256, 0, stream>>>(ranges, nranges, rbegin, rend, recs, run);
  return cudaGetLastError();
}
}  // namespace cintx
