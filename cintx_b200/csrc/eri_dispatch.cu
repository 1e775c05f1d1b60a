// Class dispatch entry used by the host code (kept in a CUDA translation unit).
#include <algorithm>

#include "eri_launch.cuh"
#include "host_internal.h"

namespace cintx {

cudaError_t launch_class(int li, int lj, int lk, int ll, bool sph, const QuartetRec* recs, int nrec,
                         const ShellPair* pairs, const PrimPair* prims, double* out, const StrideSet& st,
                         double expcutoff, const RysTable& rys, cudaStream_t stream, bool fp32,
                         double prim_eps, int variant, const double* rootbuf, const long long* rootbase, int nsplit,
                         int chain) {
  LaunchArgs a;
  a.recs = recs;
  a.nrec = nrec;
  a.pairs = pairs;
  a.prims = prims;
  a.out = out;
  a.st = st;
  a.expcutoff = expcutoff;
  a.rys = rys;
  a.stream = stream;
  a.max_blocks = 0;
  a.fp32 = fp32;
  a.prim_eps = prim_eps;
  a.variant = variant;
  a.rootbuf = rootbuf;
  a.rootbase = rootbase;
  a.nsplit = nsplit;
  a.chain = chain;
  return dispatch_eri(li, lj, lk, ll, sph, a);
}

constexpr double kSplitLarge = 1024;

PrimSplit prim_split(int lanes, int most, double resident, double work, long long nrec, double pmax, double least) {
  PrimSplit r;
  if (most <= 1 || nrec <= 0) return r;
  const double share = std::max(work / resident, lanes == 1 ? 16.0 : 4.0);
  const double from = std::max(2 * share, least * work / resident);
  if (pmax < from) {
    if (lanes == 1 && pmax >= kSplitLarge) {
      r.ns = 8;
      r.pmin = kSplitLarge;
    }
    return r;
  }
  r.ns = 2;
  while (r.ns < most && r.ns * share < pmax) r.ns *= 2;
  if (lanes == 1 && r.ns == 64) r.ns = 32;  // one-lane teams: at most a warp, or a block
  r.pmin = (double)nrec * r.ns <= 2 * resident ? 0 : from;
  if (lanes == 1 && r.pmin > kSplitLarge) r.pmin = kSplitLarge;
  return r;
}

PrimSplit prim_split(int li, int lj, int lk, int ll, bool sph, double work, long long nrec, double pmax) {
  const int s = default_threads(li, lj, lk, ll);
  if (split_max(s) <= 1 || nrec <= 0) return PrimSplit();
  double least = 2;
  if (s == 1) {
    if (ncart(li) * ncart(lj) * ncart(lk) * ncart(ll) > 10) least = 3;
  } else if (sph) {
    const int v = default_variant(li, lj, lk, ll, work / (double)nrec);
    if (variant_sliced(v)) least = 8;
    else if (variant_splitcoop(v)) least = 3;
  }
  return prim_split(s, split_max(s), (double)device_sm_count() * 4 * (128 / s), work, nrec, pmax, least);
}

static_assert(kNumVariants == kLaunchVariants, "variant count differs between kernel and host headers");

// a split-transfer variant (10, 11) that is not compiled for the class runs the default shape
static bool splitcoop_applies(int li, int lj, int lk, int ll, int variant) {
  return variant_splitcoop(variant) && li <= CINTX_LMAX && splitcoop_dims(li, lj, lk, ll, splitcoop_acc(variant)).ok;
}

// variants that are the default shape for a class (dispatch_lij compiles only the others)
static bool is_default(int li, int lj, int lk, int ll, bool sph, bool fp32, int variant) {
  if (!sph || fp32 || variant <= 0 || variant >= kNumVariants) return true;
  if (variant_splitcoop(variant)) return !splitcoop_applies(li, lj, lk, ll, variant);
  if (variant_sliced(variant)) return !sliced_ok(li, lj, lk, ll, variant);
  // one-lane shapes take no register cap
  return default_threads(li, lj, lk, ll) == 1 &&
         (variant == 3 || pick_threads(li, lj, lk, ll, variant_acc(variant)) == 1);
}

int variant_lanes(int li, int lj, int lk, int ll, bool sph, bool fp32, int variant) {
  if (is_default(li, lj, lk, ll, sph, fp32, variant)) return default_threads(li, lj, lk, ll);
  if (variant_splitcoop(variant)) return pick_threads(li, lj, lk, ll, splitcoop_acc(variant));
  return pick_threads(li, lj, lk, ll, variant_acc(variant)) / variant_passes(variant);
}

int variant_shape(int li, int lj, int lk, int ll, bool sph, bool fp32, int variant) {
  if (is_default(li, lj, lk, ll, sph, fp32, variant)) {
    const int s = default_threads(li, lj, lk, ll);
    return s == 1 ? 1 : s * 1024 + variant_regs(0);
  }
  if (variant_splitcoop(variant))
    return (1 << 23) + pick_threads(li, lj, lk, ll, splitcoop_acc(variant)) * 1024 + kSplitCoopRegs;
  const int s = pick_threads(li, lj, lk, ll, variant_acc(variant));
  if (s == 1) return 1;
  return (variant_sliced(variant) ? 1 << 20 : 0) + (variant_roll(variant) ? 1 << 21 : 0) +
         (variant_passes(variant) > 1 ? 1 << 22 : 0) + s * 1024 +
         variant_regs(variant);
}

int default_variant(int li, int lj, int lk, int ll, double np) {
  if (li > CINTX_LMAX || !class_valid(li, lj, lk, ll) || default_threads(li, lj, lk, ll) == 1) return 0;
  auto lanes = [&](int v) { return sliced_ok(li, lj, lk, ll, v) ? pick_threads(li, lj, lk, ll, variant_acc(v)) : 0; };
  if (lanes(4) == 2) return 4;
  if (lanes(5) == 2) return 5;
  if (lanes(7) > 0) return 7;
  if (li >= 3)
    for (int v : {11, 10})
      if (splitcoop_applies(li, lj, lk, ll, v)) return v;
  // 256 lanes with more accumulators than 128 registers hold: 255 registers
  const int s = default_threads(li, lj, lk, ll), ntup = ncart(lj) * ncart(lk) * ncart(ll);
  const int acc = (ntup + s - 1) / s * ncart(li);
  return acc > 45 || (acc > 40 && np >= 2) ? 1 : 0;
}

bool class_needs_scratch(int li, int lj, int lk, int ll, bool sph, int variant) {
  LaunchArgs a{};
  a.query = 1;
  a.variant = variant;
  return dispatch_eri(li, lj, lk, ll, sph, a) == cudaErrorNotSupported;
}

}  // namespace cintx
