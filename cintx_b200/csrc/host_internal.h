// Host-side internals shared by the C-ABI (host_api.cpp) and the planners (host_plan.cpp).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <string>
#include <vector>

#include "chain.cuh"
#include "common.h"

struct CINTOpt;  // the library's optimizer handle (defined below as cintx::Opt)

namespace cintx {

constexpr double kPi = 3.14159265358979323846;
constexpr int ATM_SLOTS = 6, BAS_SLOTS = 8, PTR_COORD = 1;
constexpr int ATOM_OF = 0, ANG_OF = 1, NPRIM_OF = 2, NCTR_OF = 3, PTR_EXP = 5, PTR_COEFF = 6;
constexpr int PTR_EXPCUTOFF = 0, PTR_RANGE_OMEGA = 8;

void set_error(int code, const std::string& msg);
void clear_error();

// Host-phase timer of the optimizer and plan builders: with CINTX_PLAN_LOG=1 in the environment,
// mark() prints the wall time since the previous mark (or construction) to stderr.
struct PhaseLog {
  explicit PhaseLog(const char* what);
  void mark(const char* phase);
  bool on;
  const char* what;
  double t;
};

// One contracted shell of the caller's basis.
struct ShellInfo {
  int l, nprim, nctr, atom;
  int vbase;  // first virtual shell (one per contraction)
  double r[3];
  std::vector<double> exps;
  std::vector<double> coef;      // column-major [ctr][prim] as in env
  std::vector<double> log_maxc;  // log max_ctr |c| per primitive (CINTOpt_log_max_pgto_coeff)
};

struct Basis {
  int natm = 0, nbas = 0, nvirt = 0;
  std::vector<int> atm, bas;
  std::vector<double> env;
  std::vector<ShellInfo> sh;
  std::vector<int> vshell, vctr;  // virtual shell -> (shell, contraction)
};

// Validates and copies a libcint (atm, bas, env); env length is taken from the largest
// pointer used.  Returns a status code.
int load_basis(Basis& b, const int* atm, int natm, const int* bas, int nbas, const double* env);

// Exponent cut-offs of libcint: int2e uses max(40, env[0]) + 1 (g2e.c:57-62), int3c2e and
// int2c2e use max(40, env[0]) (g3c2e.c:55-59, g2c2e.c:46-50); 60 when env[0] == 0.
double expcutoff_2e(const double* env);
double expcutoff_3c(const double* env);

// Host copy of an oriented shell pair (virtual shells a >= b in angular momentum; b < 0 is
// the unit s function used for 3- and 2-centre integrals).
struct PairHost {
  int a = -1, b = -1;
  int la = 0, lb = 0;
  double min_cce = 1e300;
  ShellPair sp{};
  std::vector<PrimPair> prims;
  std::vector<int> pa, pb;  // primitive indices (within shells a and b) of each entry of prims
};

// True when real shell sx is the recurrence centre of the pair (sx, sy): the higher l, and for
// equal l the shell whose recurrence cancels least (host_api.cpp).  Every pair the kernels see is
// oriented this way: its first shell is the centre the vertical recurrence is built on.
bool pair_base_first(const Basis& B, int sx, int sy);

// Builds the screened primitive pairs of virtual shells (a, b), in that order (b < 0: unit).
// lplus raises the pair's angular momentum in libcint's screening estimate (derivative integrals
// screen with the raised ceiling li + 1, cint2e.c CINT2e_loop_nopt -> CINTset_pairdata).
void build_pair(const Basis& B, int a, int b, double expcutoff, PairHost& out, int lplus = 0);

// Device-resident state of one CINTOpt: all unordered virtual-shell pairs (u >= v) oriented by
// angular momentum (larger l first; equal l keeps the larger index first) followed by one unit
// pair per virtual shell.
struct Opt {
  uint64_t magic;
  Basis basis;
  double build_cutoff = 0;
  int device = -1;
  int npairs = 0;             // regular pairs; unit pair of v is npairs + v
  int npv = 0;                // virtual shells u < npv have their pairs (u, v <= u) stored
  std::vector<int> pair_a, pair_b, pair_la, pair_lb, pair_nprim;
  std::vector<double> pair_min_cce;
  ShellPair* d_pairs = nullptr;
  PrimPair* d_prims = nullptr;
  int64_t nprims_total = 0;
  // host copies of the primitive pairs and their primitive indices, for the primitive
  // Schwarz pass; pair_qp[pair] = sum of the pair's q (set once prim_schwarz is true)
  std::vector<PrimPair> h_prims;
  std::vector<int> h_prim_a, h_prim_b;
  std::vector<double> pair_qp;
  // pair_amp[pair] = max over its primitive pairs of (1 + |P - C| sqrt(2 a_ab))^(la + lb), C the
  // farther of the two centres: how far the pair's recurrences can cancel below their terms
  std::vector<double> pair_amp;
  bool prim_schwarz = false;
  std::mutex mu;
  static constexpr uint64_t kMagic = 0x43494e5458423230ull;  // "CINTXB20"
};

inline int pair_index(int u, int v) {  // unordered, u >= v
  return u >= v ? u * (u + 1) / 2 + v : v * (v + 1) / 2 + u;
}

Opt* as_opt(CINTOpt* o);
// Computes every stored primitive pair's Schwarz factor q (cartesian primitive diagonals on the
// device), sorts each shell pair's primitive pairs by decreasing q and re-uploads them.
int compute_prim_schwarz(Opt* o);
// npair_shells < 0: pairs of all shells; otherwise only pairs among the first npair_shells shells
// (unit pairs are built for every shell).
int build_opt(Opt* o, const int* atm, int natm, const int* bas, int nbas, const double* env, int npair_shells = -1);

// Offsets (doubles from the start of the payload) of each order's polynomial block and
// asymptotic constants in the device layout of the Rys table, and its interval counts.
struct RysTableOffsets {
  size_t poly[CINTX_NRMAX + 1];
  size_t asym[CINTX_NRMAX + 1];
  int xmax[CINTX_NRMAX + 1];
};
// The embedded table checked against the compiled layout and transposed to the device layout
// (rys_table.cu).  Returns 0 on success.
int rys_table_image(std::vector<double>& payload, RysTableOffsets& offs);

// Per-device constants (Rys table) and per-thread scratch.
struct DeviceState {
  int dev = -1;
  void* rys_buf = nullptr;
  RysTable rys{};
};
int device_state(DeviceState** out);  // for the current device

struct ThreadScratch {
  int dev = -1;
  cudaStream_t stream = nullptr;
  void* dbuf = nullptr;
  size_t dcap = 0;
  void* hbuf = nullptr;  // pinned
  size_t hcap = 0;
  int64_t launches = 0;
};
int thread_scratch(ThreadScratch** out, size_t dbytes, size_t hbytes);

// Orientation of a requested shell tuple onto a compiled kernel class.
struct Oriented {
  int li, lj, lk, ll;       // kernel class
  int src[4];               // requested axis feeding kernel axis c
  bool swap_ab;             // kernel (ij) pair is the requested second pair
};

// Algorithmic FP64 flop count of the Rys path per primitive quartet and per contracted
// quartet (c2s) for a class.
double flops_per_prim_quartet(int li, int lj, int lk, int ll);
double flops_c2s(int li, int lj, int lk, int ll, bool sph);

bool class_needs_scratch(int li, int lj, int lk, int ll, bool sph, int variant = 0);
cudaError_t launch_class(int li, int lj, int lk, int ll, bool sph, const QuartetRec* recs, int nrec,
                         const ShellPair* pairs, const PrimPair* prims, double* out, const StrideSet& st,
                         double expcutoff, const RysTable& rys, cudaStream_t stream, bool fp32 = false,
                         double prim_eps = 0.0, int variant = 0, const double* rootbuf = nullptr,
                         const long long* rootbase = nullptr, int nsplit = 1, int chain = 0);
// Which quartets of one launch share their primitive quartets over several lane groups.  A group's
// lanes walk a quartet's primitive quartets one after another, so a launch lasts at least as long as
// its largest quartet (4096 primitive quartets of two contracted s pairs: 1.2 ms on one lane).  `work`
// is the launch's primitive quartets, `pmax` its largest quartet's: where that is over twice the
// share that a resident group (4 blocks of 128 threads per SM) has when the work is spread evenly,
// quartets of at least pmin primitive quartets run on ns groups each (ns = 1: none do; pmin = 0: the
// whole launch, which then still fits the resident groups twice).  A share under 16 primitive
// quartets on one lane (4 on a wider group) is not split further: adding up the partial blocks would
// cost as much.  One-lane classes also split quartets of 1024 and more where the launch is even: they
// are its last to end, and a warp's lanes then run the same quartet (40-atom s/p/d sweep 5.32 -> 5.06 ms
// with 8 or 32 lanes each; from 256 on 5.23, from 64 on 5.65; J/K of 120 atoms unchanged).
// Nothing is split under `least` times the even share, which is more where the split form, of the default
// shape, competes with a faster shape or adds up large blocks.  Lists of equal quartets, split over whole:
// of sliced classes (default_variant 4, 5, 7) 1.9 times the time at an even share of 1/3 of the quartet (3000
// quartets of 8 lanes), 1.3 at 1/6, 0.64 at 1/10; of split-transfer classes 1.5 at 0.42, 0.95 at 1/4 and 1/8;
// of one-lane classes of more than 10 functions 1.2 at 0.4 (30000 quartets of 81), 0.6 at 1/5.
struct PrimSplit {
  int ns = 1;
  double pmin = 0;
};
PrimSplit prim_split(int li, int lj, int lk, int ll, bool sph, double work, long long nrec, double pmax);
// The rule itself, for groups of `lanes` lanes of which `resident` fit the device and at most `most`
// share a quartet.
PrimSplit prim_split(int lanes, int most, double resident, double work, long long nrec, double pmax,
                     double least = 2);

// Learned Rys roots (rysnet.cu) of order n at count device points: out[p*2n + f], status[p]
// (0 refined, 1 table fallback, 2 closed form), asynchronous on stream.
cudaError_t rys_learned_eval(const float* d_params, const RysTable& rys, int n, const double* d_x, long long count,
                             double* d_out, int* d_status, int* d_iters, cudaStream_t stream);
// Lanes per quartet of a launch-shape variant (0 = default shape); variants that do not apply
// (cartesian or FP32 classes, unknown ids) report the default shape.
int variant_lanes(int li, int lj, int lk, int ll, bool sph, bool fp32, int variant);
// Distinct launch shape of a variant (lanes and register cap), for telling variants apart.
int variant_shape(int li, int lj, int lk, int ll, bool sph, bool fp32, int variant);
constexpr int kLaunchVariants = 12;
// The variant a spherical FP64 launch of quartets of np primitive quartets (their mean) starts with when
// nothing was tuned, by the class's size and np alone:
//   at most 48 functions         the default shape, one lane (default_acc);
//   2 lanes of 32, or else of 48 the sliced shapes with their roots unrolled (4, 5): every lane its own
//                                recurrences in registers, no barrier per primitive quartet;
//   up to 4 lanes of 48          the same with the roots rolled (7), tables of at most 72 doubles;
//   64 lanes or more, an f shell split horizontal transfers (11: 24 accumulators per lane, else 10: 12).
//                                Of (22|22), the one class without, they take 1.03 to 1.17 times the default
//                                shape's time (3000 quartets of 1, 16 and 81 primitive quartets);
//   over 40 accumulators a lane  (256 lanes, several g shells) the default shape with 255 registers (1).  With
//                                45 it pays for the primitive loop only: (42|42) and (44|22) of 1 primitive
//                                quartet 1.24 and 1.11 times the default shape's time, of 16 0.84 and 0.60;
//   the rest                     the default shape.
// All classes of a 120-atom s/p/d/f molecule, one after another: default shapes 274.7 ms, this rule
// 202.6, the fastest shape of each class as timed by the autotuner 202.1; 3-centre sweep of 40 atoms 3.84,
// 2.81 and 2.72 ms.
int default_variant(int li, int lj, int lk, int ll, double np);

}  // namespace cintx
