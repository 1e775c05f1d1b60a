// First-derivative Rys ERI kernel: (d/dx_i i j|k l) for one class (LI LJ | LK LL), the
// int2e_ip1 / int3c2e_ip1 family of libcint (autocode/grad2.c:19-88, autocode/int3c2e.c:72-88).
//
// The derivative acts on the electron coordinate of shell i.  Per primitive quartet the 2D
// integrals are built with the i ceiling raised to LI + 1 (the recurrence and horizontal transfer
// of the plain kernel on centres i and k) and the derivative of each axis is
//   D_x I(ix, ...) = ix I(ix - 1, ...) - 2 a_i I(ix + 1, ...)
// (libcint's G2E_D_I), a_i the exponent of the quartet's i primitive, which the pair tables of
// derivative launches carry in PrimPair::q as 2 a_i.  The three cartesian components share one pass
// over the primitive quartets: roots, recurrences and the columns a lane reads are the same for all
// of them, so a lane keeps all three components' accumulators (at most 9 functions, 27 doubles, per
// lane where the class has that many (j,k,l) tuples to hand out).  They are transformed to spherical
// form one after the other and written component-major: component c of element e at
// out + rec.out + c*scomp + e.
//
// Work unit: one contracted quartet per team of nsplit groups of S lanes.  The groups of a team share
// the primitive quartets (split_la) and add up their partial blocks; a group's lanes share the (axis,
// root) tables in shared memory, or with S == 1 keep them in registers.  The kernel's first pair is
// (i, j) in the requested order (no reorientation: the derivative stays on axis i); the second pair is
// oriented like the plain kernel's.
//
// All derivatives of a 4-atom s/p/d/f molecule (84 000 tuples): 140.8 ms of device time with one pass per
// component, one group per quartet and one launch after another; 3.9 ms so, launches overlapping (chain.cuh).
#pragma once
#include "eri_launch.cuh"

namespace cintx {

// Lanes per group: the fewest (a power of two, at most twice the (j,k,l) tuple count, at most 512) that
// keep a lane's functions within 9, i.e. 27 accumulators.
__host__ __device__ constexpr int ip1_threads(int li, int lj, int lk, int ll) {
  const int ntup = ncart(lj) * ncart(lk) * ncart(ll);
  const int total = ntup * ncart(li);
  int s = 1;
  while (s < 512 && (total + s - 1) / s > 9 && s * 2 <= ntup * 2) s *= 2;
  return s;
}

template <int LI, int LJ, int LK, int LL, bool SPH>
struct Ip1Shape {
  static constexpr int NR = (LI + 1 + LJ + LK + LL) / 2 + 1;
  static constexpr int NI = LI + 2, NJ = LJ + 1, NK = LK + 1, NL = LL + 1;  // i ceiling LI + 1
  static constexpr int NIJ = LI + LJ + 2, NKL = LK + LL + 1;
  static constexpr int GSZ = NI * NJ * NK * NL;
  static constexpr int NFI = ncart(LI), NFJ = ncart(LJ), NFK = ncart(LK), NFL = ncart(LL);
  static constexpr int NTUP = NFJ * NFK * NFL;
  static constexpr int S = ip1_threads(LI, LJ, LK, LL);
  static constexpr int TPT = (NTUP + S - 1) / S;
  static constexpr int MI = SPH && LI >= 2 ? 2 * LI + 1 : NFI;
  static constexpr int MJ = SPH && LJ >= 2 ? 2 * LJ + 1 : NFJ;
  static constexpr int MK = SPH && LK >= 2 ? 2 * LK + 1 : NFK;
  static constexpr int ML = SPH && LL >= 2 ? 2 * LL + 1 : NFL;
  static constexpr int NOUT = MI * MJ * MK * ML;
  static constexpr int SM_ROOTS = 2 * NR;
  static constexpr int SM_G = 3 * NR * GSZ;
  // groups of a warp or more spread the transfers of every (axis, root) over (j, l) tasks (hrr_jl) and
  // keep all 3*NR 2D tables; narrower groups run table and transfers of a task on one lane
  static constexpr bool SPLIT_H = S >= 32;
  static constexpr int NTASK_CONC = S < 3 * NR ? S : 3 * NR;
  static constexpr int SM_SCR = (SPLIT_H ? 3 * NR : NTASK_CONC) * NIJ * NKL;
  static constexpr int SM_BUFA = MI * NTUP;
  static constexpr int SM_BUFB = MI * MJ * NFK * NFL;
  static constexpr int GROUP_DOUBLES_RAW = S == 1 ? 0 : cmax(SM_ROOTS + SM_G + SM_SCR, SM_BUFA + SM_BUFB);
  static constexpr int GROUP_DOUBLES = (GROUP_DOUBLES_RAW + 1) & ~1;  // 16-byte groups
  // one-lane groups stage their root table in shared memory (as the plain kernel's one-lane classes)
  static constexpr bool STAGE_TABLE = S == 1 && NR <= 3;
  static constexpr int TABLE_DOUBLES = STAGE_TABLE ? rys_intervals(NR) * rys_stage_stride(NR) : 0;
  // groups per block: up to 128 threads, as many groups as 200 KB of shared memory holds
  static constexpr int QFIT = S == 1 ? 128 : (200 * 1024) / (GROUP_DOUBLES * 8);
  static constexpr int QWANT = S >= 128 ? 1 : 128 / S;
  static constexpr int Q = QFIT >= QWANT ? QWANT : (QFIT >= 64 ? 64 : QFIT >= 32 ? 32 : QFIT >= 16 ? 16 : QFIT >= 8 ? 8 : QFIT >= 4 ? 4 : QFIT >= 2 ? 2 : 1);
  static constexpr int BLOCK = Q * S;
  static constexpr int SMEM_BYTES = (Q * GROUP_DOUBLES + TABLE_DOUBLES) * 8;
  // most groups that can share a quartet: the block's, a warp of one-lane groups
  static constexpr int SPLIT_MAX = S == 1 ? 32 : Q;
};

// Index bounds of an ip1 shape (the kernel static_asserts it): groups fill the block, the
// primitive-loop region and the transform buffers fit the group, stages fit their buffers, the
// block's shared memory fits, named barriers (S > 32) have ids below 16, and a team of groups is a
// power of two of them inside one block.
template <class SH>
__host__ __device__ constexpr int ip1_shape_violation() {
  if (SH::S < 1 || SH::S > 512 || (SH::S & (SH::S - 1)) != 0) return 1;
  if (SH::BLOCK != SH::Q * SH::S || SH::BLOCK > 1024 || SH::Q < 1 || (SH::Q & (SH::Q - 1)) != 0) return 2;
  if (SH::TPT * SH::S < SH::NTUP) return 3;
  if (SH::S > 1 && SH::SM_ROOTS + SH::SM_G + SH::SM_SCR > SH::GROUP_DOUBLES) return 4;
  if (SH::S > 1 && SH::SM_BUFA + SH::SM_BUFB > SH::GROUP_DOUBLES) return 5;
  if (SH::MI * SH::MJ * SH::MK * SH::NFL > (SH::MJ != SH::NFJ ? SH::SM_BUFA : SH::SM_BUFB)) return 6;
  if (SH::SMEM_BYTES > 227 * 1024) return 7;
  if (SH::S > 32 && (SH::Q > 15 || SH::S % 32 != 0)) return 8;
  if (SH::S <= 32 && 32 % SH::S != 0) return 9;
  if (SH::S == 1 && (SH::TPT != SH::NTUP || SH::BLOCK != 128)) return 10;
  // the 16-byte column loads: even table sizes behind 2*NR doubles of roots in 16-byte groups
  if (SH::S > 1 && SH::NI % 2 == 0 && (SH::GSZ % 2 != 0 || SH::GROUP_DOUBLES % 2 != 0)) return 11;
  // team barriers of more than a warp and less than the block are named 1 + team: their groups have at
  // most 32 lanes (no named group barrier), and blocks of several groups have at most 128 threads, so two teams
  if (SH::S > 32 && SH::Q > 2) return 12;
  return 0;
}

// acc[c] += the three derivative products of one root for one (j,k,l) tuple from its I columns
template <int LI, int NFI>
__device__ __forceinline__ void ip1_products(double (&acc)[3][NFI], const double (&ix)[LI + 2], const double (&iy)[LI + 2],
                                             const double (&iz)[LI + 2], double ai2) {
  double dx[LI + 1], dy[LI + 1], dz[LI + 1];
  static_loop(std::make_integer_sequence<int, LI + 1>{}, [&](auto c) {
    constexpr int n = decltype(c)::value;
    dx[n] = -ai2 * ix[n + 1];
    dy[n] = -ai2 * iy[n + 1];
    dz[n] = -ai2 * iz[n + 1];
    if constexpr (n > 0) {
      dx[n] = fma((double)n, ix[n - 1], dx[n]);
      dy[n] = fma((double)n, iy[n - 1], dy[n]);
      dz[n] = fma((double)n, iz[n - 1], dz[n]);
    }
  });
  static_loop(std::make_integer_sequence<int, NFI>{}, [&](auto c) {
    constexpr int fi = decltype(c)::value;
    constexpr int cx = cart_x(LI, fi), cy = cart_y(LI, fi), cz = cart_z(LI, fi);
    acc[0][fi] = fma(dx[cx], iy[cy] * iz[cz], acc[0][fi]);
    acc[1][fi] = fma(dy[cy], ix[cx] * iz[cz], acc[1][fi]);
    acc[2][fi] = fma(dz[cz], ix[cx] * iy[cy], acc[2][fi]);
  });
}

template <int LI, int LJ, int LK, int LL, bool SPH>
__global__ void __launch_bounds__(Ip1Shape<LI, LJ, LK, LL, SPH>::BLOCK, 1)
    eri_ip1_kernel(const QuartetRec* __restrict__ recs, int nrec, const ShellPair* __restrict__ pairs,
                   const PrimPair* __restrict__ prims, double* __restrict__ out,
                   const __grid_constant__ StrideSet sts, long long scomp, double expcutoff, const __grid_constant__ RysTable rys, int nsplit,
                   int chain, int nblocks) {
  if (chain_begin(chain, nblocks)) return;
  using SH = Ip1Shape<LI, LJ, LK, LL, SPH>;
  static_assert(ip1_shape_violation<SH>() == 0, "an index of this ip1 launch shape can leave its buffer");
  constexpr int S = SH::S, NR = SH::NR, GSZ = SH::GSZ, NFI = SH::NFI, TPT = SH::TPT;
  constexpr int NI = SH::NI, NJ = SH::NJ, NK = SH::NK;
  constexpr int NIJ = SH::NIJ, NKL = SH::NKL;
  extern __shared__ __align__(16) double smem[];
  const int group = (int)threadIdx.x / S;
  const int lane = (int)threadIdx.x % S;
  double* sg = smem + SH::TABLE_DOUBLES + (size_t)group * SH::GROUP_DOUBLES;
  double* s_roots = sg;
  double* s_g = sg + SH::SM_ROOTS;
  double* s_scr = s_g + SH::SM_G;

  if constexpr (SH::STAGE_TABLE) {
    constexpr int W = NR * RYS_NC, WP = rys_stage_stride(NR) / 2;  // double2 per interval, per stride
    const double2* src = reinterpret_cast<const double2*>(rys.poly[NR]);
    double2* dst = reinterpret_cast<double2*>(smem);
    for (int i = threadIdx.x; i < rys_intervals(NR) * W; i += blockDim.x) dst[(i / W) * WP + i % W] = __ldg(src + i);
    __syncthreads();
  }

  // offsets of this lane's (fj, fk, fl) tuples into the I arrays (i ceiling LI + 1)
  int ox[TPT], oy[TPT], oz[TPT];
  if constexpr (S > 1) {
#pragma unroll
    for (int k = 0; k < TPT; ++k) {
      int t = lane + S * k;
      if (t >= SH::NTUP) t = 0;
      const int fj = t % SH::NFJ, fk = (t / SH::NFJ) % SH::NFK, fl = t / (SH::NFJ * SH::NFK);
      ox[k] = cart_x(LJ, fj) * NI + cart_x(LK, fk) * NI * NJ + cart_x(LL, fl) * NI * NJ * NK;
      oy[k] = cart_y(LJ, fj) * NI + cart_y(LK, fk) * NI * NJ + cart_y(LL, fl) * NI * NJ * NK;
      oz[k] = cart_z(LJ, fj) * NI + cart_z(LK, fk) * NI * NJ + cart_z(LL, fl) * NI * NJ * NK;
    }
  }

  const int ns = nsplit;  // groups sharing a quartet
  const int team = group / ns, sub = group % ns, per_block = SH::Q / ns;
  const int tl = sub * S + lane, tn = ns * S;  // lanes of a team
  for (int q = (int)blockIdx.x * per_block + team; q < nrec; q += nblocks * per_block) {
    const QuartetRec rec = recs[q];
    const ShellPair pij = pairs[rec.pij];
    const ShellPair pkl = pairs[rec.pkl];
    double acc[TPT][3][NFI];
#pragma unroll
    for (int k = 0; k < TPT; ++k)
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int f = 0; f < NFI; ++f) acc[k][c][f] = 0.0;
    const int da = split_la(ns, pij.nprim, pkl.nprim), db = ns / da;
    for (int b = sub / da; b < pkl.nprim; b += db) {
      const PrimPair pk = prims[pkl.prim_off + b];
      const double qcx = pk.px - pkl.ax, qcy = pk.py - pkl.ay, qcz = pk.pz - pkl.az;
      for (int a = sub % da; a < pij.nprim; a += da) {
        const PrimPair pi = prims[pij.prim_off + a];
        if (pi.cce + pk.cce > expcutoff) continue;  // CINT2e_loop eijcutoff (cint2e.c:700-712)
        const double aij = pi.aij, akl = pk.aij;
        const double pqx = pi.px - pk.px, pqy = pi.py - pk.py, pqz = pi.pz - pk.pz;
        const RysPoint pt =
            rys_point(aij * akl * (pqx * pqx + pqy * pqy + pqz * pqz), aij + akl, cintx_rys_xmax(NR));
        const double fac = pi.kab * pk.kab * pt.r;
        const double pax = pi.px - pij.ax, pay = pi.py - pij.ay, paz = pi.pz - pij.az;
        const double ai2 = pi.q;  // 2 a_i of this primitive pair's i primitive
        if constexpr (S == 1) {
          double t2[NR], w[NR];
          if constexpr (SH::STAGE_TABLE) rys_all_staged<NR>(smem, pt, t2, w);
          else rys_all_at<NR>(rys, pt, t2, w);
#pragma unroll
          for (int r = 0; r < NR; ++r) {
            double gg[3 * GSZ];
            const double rt_aa = t2[r] * pt.r2;
            const double b00 = 0.5 * rt_aa;
            const double b10 = pi.half_inv * (1.0 - rt_aa * akl);
            const double b01 = pk.half_inv * (1.0 - rt_aa * aij);
            const double ca = rt_aa * akl, cb = rt_aa * aij;
            vrr_hrr<LI + 1, LJ, LK, LL>(gg, 1.0, pax - ca * pqx, qcx + cb * pqx, b10, b01, b00, pij.abx, pkl.abx);
            vrr_hrr<LI + 1, LJ, LK, LL>(gg + GSZ, 1.0, pay - ca * pqy, qcy + cb * pqy, b10, b01, b00, pij.aby, pkl.aby);
            vrr_hrr<LI + 1, LJ, LK, LL>(gg + 2 * GSZ, w[r] * fac, paz - ca * pqz, qcz + cb * pqz, b10, b01, b00,
                                        pij.abz, pkl.abz);
            static_loop(std::make_integer_sequence<int, SH::NTUP>{}, [&](auto t) {  // registers: constant indices
              constexpr int k = decltype(t)::value;
              constexpr int fj = k % SH::NFJ, fk = (k / SH::NFJ) % SH::NFK, fl = k / (SH::NFJ * SH::NFK);
              constexpr int px = cart_x(LJ, fj) * NI + cart_x(LK, fk) * NI * NJ + cart_x(LL, fl) * NI * NJ * NK;
              constexpr int py = cart_y(LJ, fj) * NI + cart_y(LK, fk) * NI * NJ + cart_y(LL, fl) * NI * NJ * NK;
              constexpr int pz = cart_z(LJ, fj) * NI + cart_z(LK, fk) * NI * NJ + cart_z(LL, fl) * NI * NJ * NK;
              double ix[NI], iy[NI], iz[NI];
              static_loop(std::make_integer_sequence<int, NI>{}, [&](auto c) {
                constexpr int n = decltype(c)::value;
                ix[n] = gg[px + n];
                iy[n] = gg[GSZ + py + n];
                iz[n] = gg[2 * GSZ + pz + n];
              });
              ip1_products<LI, NFI>(acc[k], ix, iy, iz, ai2);
            });
          }
        } else {
          for (int f = lane; f < 2 * NR; f += S) s_roots[f] = rys_fn_at<NR>(rys, f, pt);
          group_sync<S>(group);
          for (int task = lane; task < 3 * NR; task += S) {
            const int axis = task / NR, r = task % NR;
            const double rt_aa = s_roots[r] * pt.r2;
            const double b00 = 0.5 * rt_aa;
            const double b10 = pi.half_inv * (1.0 - rt_aa * akl);
            const double b01 = pk.half_inv * (1.0 - rt_aa * aij);
            const double pa = axis == 0 ? pax : (axis == 1 ? pay : paz);
            const double qc = axis == 0 ? qcx : (axis == 1 ? qcy : qcz);
            const double pq = axis == 0 ? pqx : (axis == 1 ? pqy : pqz);
            const double g00 = axis == 2 ? s_roots[NR + r] * fac : 1.0;
            if constexpr (SH::SPLIT_H) {
              vrr_columns<NIJ, NKL, double>(s_scr + task * (NIJ * NKL), g00, pa - rt_aa * akl * pq,
                                            qc + rt_aa * aij * pq, b10, b01, b00);
            } else {
              const double ab = axis == 0 ? pij.abx : (axis == 1 ? pij.aby : pij.abz);
              const double cd = axis == 0 ? pkl.abx : (axis == 1 ? pkl.aby : pkl.abz);
              vrr_hrr_smem<LI + 1, LJ, LK, LL, double, 1>(s_g + task * GSZ, s_scr + lane * (NIJ * NKL), g00,
                                                          pa - rt_aa * akl * pq, qc + rt_aa * aij * pq, b10, b01, b00,
                                                          ab, cd, 0);
            }
          }
          group_sync<S>(group);
          if constexpr (SH::SPLIT_H) {
            for (int u = lane; u < 3 * NR * NJ * SH::NL; u += S) {
              const int task = u / (NJ * SH::NL), jl = u % (NJ * SH::NL);
              const int axis = task / NR;
              const double ab = axis == 0 ? pij.abx : (axis == 1 ? pij.aby : pij.abz);
              const double cd = axis == 0 ? pkl.abx : (axis == 1 ? pkl.aby : pkl.abz);
              hrr_jl<LI + 1, LJ, LK, LL>(s_g + task * GSZ, s_scr + task * (NIJ * NKL), jl % NJ, jl / NJ, ab, cd);
            }
            group_sync<S>(group);
          }
#pragma unroll 1
          for (int r = 0; r < NR; ++r) {
            const double* gx = s_g + (0 * NR + r) * GSZ;
            const double* gy = s_g + (1 * NR + r) * GSZ;
            const double* gz = s_g + (2 * NR + r) * GSZ;
#pragma unroll
            for (int k = 0; k < TPT; ++k) {
              double ix[NI], iy[NI], iz[NI];
              load_i_column<NI>(ix, gx + ox[k]);
              load_i_column<NI>(iy, gy + oy[k]);
              load_i_column<NI>(iz, gz + oz[k]);
              ip1_products<LI, NFI>(acc[k], ix, iy, iz, ai2);
            }
          }
          group_sync<S>(group);
        }
      }
    }
    // ---- transform each component to spherical and store ----
    double* const obase = out + rec_offset(rec);
    const OutStrides st = sts.s[rec_strides(rec)];
    if constexpr (S == 1) {
      const unsigned tmask = ns == 32 ? 0xffffffffu : (((1u << ns) - 1u) << (threadIdx.x & 31u & ~(unsigned)(ns - 1)));
      for (int o = ns >> 1; o > 0; o >>= 1) {
#pragma unroll
        for (int k = 0; k < TPT; ++k)
#pragma unroll
          for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int f = 0; f < NFI; ++f) acc[k][c][f] += __shfl_xor_sync(tmask, acc[k][c][f], o);
      }
      if (sub == 0) {
#pragma unroll
        for (int c = 0; c < 3; ++c)
          static_loop(std::make_integer_sequence<int, SH::NOUT>{}, [&](auto oc) {
            constexpr int o = decltype(oc)::value;
            constexpr int mi = o % SH::MI, mj = (o / SH::MI) % SH::MJ, mk = (o / (SH::MI * SH::MJ)) % SH::MK;
            constexpr int ml = o / (SH::MI * SH::MJ * SH::MK);
            double v = 0.0;
#pragma unroll
            for (int t = 0; t < SH::NTUP; ++t) {
              const int fj = t % SH::NFJ, fk = (t / SH::NFJ) % SH::NFK, fl = t / (SH::NFJ * SH::NFK);
              const double cj = SPH && LJ >= 2 ? c2s_coef(LJ, mj, fj) : (mj == fj ? 1.0 : 0.0);
              const double ck = SPH && LK >= 2 ? c2s_coef(LK, mk, fk) : (mk == fk ? 1.0 : 0.0);
              const double cl = SPH && LL >= 2 ? c2s_coef(LL, ml, fl) : (ml == fl ? 1.0 : 0.0);
#pragma unroll
              for (int fi = 0; fi < NFI; ++fi) {
                const double ci = SPH && LI >= 2 ? c2s_coef(LI, mi, fi) : (mi == fi ? 1.0 : 0.0);
                if (ci * cj * ck * cl != 0.0) v += ci * cj * ck * cl * acc[t][c][fi];
              }
            }
            obase[c * scomp + mi * st.s0 + mj * st.s1 + mk * st.s2 + ml * st.s3] = v;
          });
      }
    } else {
      double* bufA = sg - (size_t)sub * SH::GROUP_DOUBLES;  // the team's: its first group's region
      double* bufB = bufA + SH::SM_BUFA;
      team_sync(tn, team);  // every group's last products are read
#pragma unroll 1
      for (int comp = 0; comp < 3; ++comp) {
        double* const cbase = obase + comp * scomp;
        auto stage_i = [&](auto cc) {  // this group's partial block, its i axis transformed
          constexpr int c = decltype(cc)::value;
#pragma unroll
          for (int k = 0; k < TPT; ++k) {
            const int t = lane + S * k;
            if (t < SH::NTUP) {
#pragma unroll
              for (int mi = 0; mi < SH::MI; ++mi) {
                double v = 0.0;
#pragma unroll
                for (int fi = 0; fi < NFI; ++fi) {
                  const double f = (SPH && LI >= 2) ? c2s_coef(LI, mi, fi) : (mi == fi ? 1.0 : 0.0);
                  if (f != 0.0) v += f * acc[k][c][fi];
                }
                sg[mi + SH::MI * t] = v;
              }
            }
          }
        };
        if (comp == 0) stage_i(std::integral_constant<int, 0>{});
        else if (comp == 1) stage_i(std::integral_constant<int, 1>{});
        else stage_i(std::integral_constant<int, 2>{});
        team_sync(tn, team);
        if (ns > 1) {  // add the groups' partial blocks
          for (int e = tl; e < SH::MI * SH::NTUP; e += tn) {
            double v = bufA[e];
            for (int g = 1; g < ns; ++g) v += bufA[(size_t)g * SH::GROUP_DOUBLES + e];
            bufA[e] = v;
          }
          team_sync(tn, team);
        }
        const double* cur = bufA;
        if constexpr (SPH && LJ >= 2) {
          constexpr int n = SH::MI * SH::MJ * SH::NFK * SH::NFL;
          for (int o = tl; o < n; o += tn) {
            const int mi = o % SH::MI;
            const int mj = (o / SH::MI) % SH::MJ;
            const int rest = o / (SH::MI * SH::MJ);
            const C2SRow& row = C2S_ROWS[LJ][mj];
            double v = 0.0;
            for (int z = 0; z < row.nnz; ++z) v += row.c[z] * bufA[mi + SH::MI * (row.f[z] + SH::NFJ * rest)];
            bufB[o] = v;
          }
          team_sync(tn, team);
          cur = bufB;
        }
        if constexpr (SPH && LK >= 2) {
          double* nxt = (cur == bufA) ? bufB : bufA;
          constexpr int n = SH::MI * SH::MJ * SH::MK * SH::NFL;
          for (int o = tl; o < n; o += tn) {
            const int mij = o % (SH::MI * SH::MJ);
            const int mk = (o / (SH::MI * SH::MJ)) % SH::MK;
            const int fl = o / (SH::MI * SH::MJ * SH::MK);
            const C2SRow& row = C2S_ROWS[LK][mk];
            double v = 0.0;
            for (int z = 0; z < row.nnz; ++z) v += row.c[z] * cur[mij + SH::MI * SH::MJ * (row.f[z] + SH::NFK * fl)];
            nxt[o] = v;
          }
          team_sync(tn, team);
          cur = nxt;
        }
        {
          constexpr int n = SH::NOUT;
          constexpr int MIJK = SH::MI * SH::MJ * SH::MK;
          for (int o = tl; o < n; o += tn) {
            const int mi = o % SH::MI;
            const int mj = (o / SH::MI) % SH::MJ;
            const int mk = (o / (SH::MI * SH::MJ)) % SH::MK;
            const int ml = o / MIJK;
            const int mijk = o % MIJK;
            double v;
            if constexpr (SPH && LL >= 2) {
              const C2SRow& row = C2S_ROWS[LL][ml];
              v = 0.0;
              for (int z = 0; z < row.nnz; ++z) v += row.c[z] * cur[mijk + MIJK * row.f[z]];
            } else {
              v = cur[mijk + MIJK * ml];
            }
            cbase[mi * st.s0 + mj * st.s1 + mk * st.s2 + ml * st.s3] = v;
          }
        }
        team_sync(tn, team);
      }
    }
  }
}

struct Ip1Args {
  const QuartetRec* recs;
  int nrec;
  const ShellPair* pairs;
  const PrimPair* prims;
  double* out;
  StrideSet st;
  long long scomp;
  double expcutoff;
  RysTable rys;
  cudaStream_t stream;
  int nsplit;       // groups sharing a quartet (power of two)
  int chain;        // kChainPrev, kChainNext (chain.cuh)
  int* shape;       // not null: launch nothing, write {lanes per group, most groups per quartet}
};

template <int LI, int LJ, int LK, int LL, bool SPH>
cudaError_t launch_ip1(const Ip1Args& a) {
  using SH = Ip1Shape<LI, LJ, LK, LL, SPH>;
  if (a.shape) {
    a.shape[0] = SH::S;
    a.shape[1] = SH::SPLIT_MAX;
    return cudaSuccess;
  }
  if (a.nsplit < 1 || a.nsplit > SH::SPLIT_MAX || (a.nsplit & (a.nsplit - 1)) != 0) return cudaErrorInvalidValue;
  auto kern = eri_ip1_kernel<LI, LJ, LK, LL, SPH>;
  static int attr_done[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (SH::SMEM_BYTES > 48 * 1024 && dev < 64 && !attr_done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SH::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    attr_done[dev] = 1;
  }
  if (a.nrec <= 0) return cudaSuccess;
  const int per_block = SH::Q / a.nsplit;
  long long blocks = ((long long)a.nrec + per_block - 1) / per_block;
  const long long cap = (long long)device_sm_count() * 32;
  if (blocks > cap) blocks = cap;
  return chain_launch(kern, (unsigned)blocks, SH::BLOCK, SH::SMEM_BYTES, a.stream, a.chain, a.recs, a.nrec, a.pairs,
                      a.prims, a.out, a.st, a.scomp, a.expcutoff, a.rys, a.nsplit);
}

// Classes compiled for derivatives: the derivative pair (i, j) with li, lj <= 3 in either order,
// the second pair oriented (lk >= ll) with lk <= 3, or lk = 4 with ll = 0 (3-centre g auxiliaries).
__host__ __device__ constexpr bool ip1_class_valid(int li, int lj, int lk, int ll) {
  return li <= 3 && lj <= 3 && lk >= ll && (lk <= 3 || (lk == 4 && ll == 0));
}

template <int LI, int LJ>
cudaError_t dispatch_ip1_lij(int lk, int ll, bool sph, const Ip1Args& a) {
  cudaError_t err = cudaErrorInvalidValue;
  static_for<CINTX_LMAX + 1>([&](auto K) {
    static_for<K.value + 1>([&](auto L) {
      constexpr int k = decltype(K)::value, l = decltype(L)::value;
      if constexpr (ip1_class_valid(LI, LJ, k, l)) {
        if (lk == k && ll == l) err = sph ? launch_ip1<LI, LJ, k, l, true>(a) : launch_ip1<LI, LJ, k, l, false>(a);
      }
    });
  });
  return err;
}

}  // namespace cintx
