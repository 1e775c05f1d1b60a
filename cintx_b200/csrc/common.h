// Shared host/device data layout of the B200 two-electron integral engine.
//
// The basis lives in HBM as structure-of-arrays records built once per CINTOpt
// (int2e_optimizer).  Everything the kernels need per primitive pair is precomputed into a
// 64-byte PrimPair record so the inner primitive loop reads one cache line per pair.
#pragma once
#include <stdint.h>

#define CINTX_LMAX 4          // highest angular momentum with compiled kernels (g)
#define CINTX_NRMAX 9         // highest Rys order: (4+4+4+4)/2 + 1
#define CINTX_RYS_DEG 11      // polynomial degree per unit-width x interval

// Table intervals per order (x < xmax uses the table; the file header must match).
__host__ __device__ constexpr int cintx_rys_xmax(int n) {
  return n == 1 ? 40 : n == 2 ? 52 : n == 3 ? 60 : n == 4 ? 64 : n == 5 ? 72 : n == 6 ? 76 : n == 7 ? 84
       : n == 8 ? 92 : 100;
}

// One primitive pair (a, b) of an oriented shell pair (i, j), after exponent screening.
// kab folds exp(-a_i a_j/a_ij |A-B|^2), both contraction coefficients (single contraction), 1 / a_ij
// and the pair's share of libcint's common factor sqrt(2 pi^2.5) * fac_sp(li) * fac_sp(lj), so that a
// primitive quartet's prefactor is kab_ij kab_kl / sqrt(a_ij + a_kl).
// When q is set, a shell pair's primitive pairs are sorted by decreasing q, so a primitive
// quartet loop can stop at the first pair whose bound q_ab * q_cd falls below its threshold.
struct __align__(64) PrimPair {
  double aij;         // a_i + a_j
  double px, py, pz;  // product centre P = (a_i A + a_j B) / a_ij
  double kab;         // prefactor described above
  double cce;         // libcint screening exponent of this pair (CINTset_pairdata)
  double half_inv;    // 0.5 / a_ij
  double q;           // primitive Schwarz factor |c_i c_j| sqrt(max|(ab|ab)|) (0: not computed)
};

// An oriented shell pair (i, j).  Its primitive pairs are prims[prim_off, prim_off+nprim).
struct __align__(16) ShellPair {
  double ax, ay, az;     // centre of shell i
  double abx, aby, abz;  // A - B
  int prim_off;
  int nprim;
  int ish, jsh;          // shell ids
};

// One shell quartet of a launch: pairs (ij) and (kl), the start of its output block (doubles) in the low
// 56 bits of `out`, and in the high 8 which of the launch's stride sets its block is laid out with (0 in
// every list but explicit ones, whose tuples may name the shells of a class in any order).
struct __align__(16) QuartetRec {
  int pij;
  int pkl;
  long long out;
};
__host__ __device__ inline long long rec_offset(const QuartetRec& r) { return r.out & ((1LL << 56) - 1); }
__host__ __device__ inline int rec_strides(const QuartetRec& r) { return (int)((unsigned long long)r.out >> 56); }

// A contiguous run [t0, t1) of one screened tile's row-major quartet numbering, generating
// records rec_off.. of its chunk, whose blocks start at out_off (doubles).
struct __align__(16) GenRange {
  const int* rows;
  const int* cols;
  const long long* prefix;
  int nrows;
  int swap;  // nonzero: the column pair is the kernel's first pair (pij)
  long long t0, t1;
  long long rec_off;
  long long out_off;
  long long nout;
  const int* colstart;  // per row: first column of the range's tile (nullptr: 0)
};

// Output placement of one launch group: the element (a, b, c, d) of the canonical block
// (a over shell i components fastest) goes to out + rec.out + a*s0 + b*s1 + c*s2 + d*s3.
struct OutStrides {
  long long s0, s1, s2, s3;
};

// The layouts of one launch's blocks, by rec_strides.
struct StrideSet {
  OutStrides s[8];
};
inline StrideSet one_stride(const OutStrides& st) {
  StrideSet r{};
  r.s[0] = st;
  return r;
}

// The eight index orders a tuple list can name a class's shells in: bit 0, the kernel's first pair is
// requested (second shell, first shell); bit 1, its second pair; bit 2, the kernel's second pair is
// requested first.  `extent` are the functions (contractions included) along the kernel's axes; the
// requested axes are laid out first fastest.
inline int order_code(const int (&src)[4]) {
  return (src[0] & 1) | ((src[2] & 1) << 1) | (src[0] >= 2 ? 4 : 0);
}
inline StrideSet order_strides(const long long (&extent)[4]) {
  StrideSet r{};
  for (int code = 0; code < 8; ++code) {
    long long st[4], n = 1;
    for (int x = 0; x < 4; ++x) {  // requested axis x: kernel pair and shell of it
      const int pair = (x >> 1) ^ (code >> 2), second = (x & 1) ^ ((code >> pair) & 1);
      st[2 * pair + second] = n;
      n *= extent[2 * pair + second];
    }
    r.s[code] = OutStrides{st[0], st[1], st[2], st[3]};
  }
  return r;
}

// Device Rys table (see gen_rys_table.py for the layout).
struct RysTable {
  const double* poly[CINTX_NRMAX + 1];  // [n] -> [xmax + 1][2n][DEG+1] (rys_roots.cuh)
  const double* asym[CINTX_NRMAX + 1];  // [n] -> h_r^2 (n), W_r (n)
  int xmax[CINTX_NRMAX + 1];
};

// libcint status semantics and cintx C-ABI status codes (cintx-capi errors.rs:9-21)
enum CintxStatus {
  CINTX_SUCCESS = 0,
  CINTX_INVALID_INPUT = 1,
  CINTX_UNSUPPORTED_API = 2,
  CINTX_UNSUPPORTED_REPRESENTATION = 3,
  CINTX_BUFFER_TOO_SMALL = 4,
  CINTX_MEMORY_LIMIT_EXCEEDED = 5,
  CINTX_ALLOCATION_FAILED = 6,
  CINTX_EXECUTION_FAILED = 7,
  CINTX_NULL_POINTER = 8,
  CINTX_PANIC = 9,
  CINTX_BACKEND_NOT_COMPILED = 10,
};
