// The coarse end of a multigrid cycle on one thread-block cluster: every level from some level s
// down lives in the shared memory of the cluster's CTAs for the whole launch, split into x
// slabs, and the schedule (smoothing, restriction, coarsest-level relaxation, prolongation, for
// one V-cycle or for the whole FMG ramp) runs there with cluster barriers between phases.
//
// What bounds it: a phase over such a level is a chain of shared-memory loads, one SOR update
// and a barrier; no unit is near its throughput.  A launch with programmatic dependencies costs
// 2.2-2.5 us whatever the level's size; a colour sweep here 0.25 us (FP64 0.33) on an 8^3 level held
// by one CTA, 0.45 (0.5) on a 16^3 level over 16 and 0.55 on a 24x20x18 one over 12
// (bench.py --kernel-case cluster under ncu), of which a barrier alone is 0.24 us over 16 CTAs of 512 threads and
// 0.22 over one.  One CTA alone is the cheaper home only where its threads hold the level in one or
// two trips (kCtSingleCells).  Cycle counts in this file are clock64 differences inside the kernel.
//
// Layout.  As the split levels of ir_chequer.h: per colour c (cell (i,j,k) has colour (i+j+k)&1)
// one array of rows (i,j), cell k at entry m = k >> 1 -- all sizes of a level are even, since a
// level exists only where every axis halves once more.  So neighbouring lanes read neighbouring
// words, the x and y neighbours of an entry sit at the same m, and one of its two z neighbours is
// the other colour's entry m of the same row: a thread owns the pair (k = 2m, 2m+1) and keeps
// both values, their right-hand sides and diagonals in registers across the iterations of a
// smoothing call.  A rank's slab has one halo plane on each side per colour; the thread that
// updates a slab's first or last plane also stores the value into the neighbour's halo
// (st.shared::cluster), so all reads of a sweep are local.
//
// Boundary values are homogeneous on every level below 0 and are applied where a neighbour is
// read: the cell itself (Neumann), its negation (Dirichlet), zero (no condition: those ghosts
// are cleared and never written), or the wrapped cell (periodic).  These are the values the
// per-level kernels' ghost cells hold, so the reference-layout hierarchy's results are the same
// bits either way (CtPlain below); CtChq is the arithmetic of the refinement's FP32 levels.
#pragma once

#include <algorithm>
#include <array>
#include <atomic>
#include <cstring>
#include <vector>

#include "chq_device.cuh"
#include "mg_fused.h"
#include "relax_math.cuh"

namespace ocub {
namespace ct {
namespace {

using chq::FDiv;
using chq::make_fdiv;
using chq::split;

constexpr int kCtMaxLevels = 8;
constexpr int kCtThreads = 512;
constexpr size_t kCtSmemCap = 220 * 1024;
// Levels of at most this many cells are held by rank 0 alone (its 512 threads own one pair each).
constexpr long long kCtSingleCells = 1024;

template <typename T> struct BoundarySigns {
  T xn, xp, yn, yp, zn, zp;
  int px, py, pz;
};

// (an axis wraps at both ends or at neither: bc_periodic_paired)
template <typename T>
inline BoundarySigns<T> boundary_signs(const BCDev &b) {
  auto sign = [&](int f) {
    return (T)(b.type[f] == OCU_BC_NEUMANN ? 1 : b.type[f] == OCU_BC_DIRICHELET ? -1 : 0);
  };
  auto wraps = [&](int f) { return b.type[f] == OCU_BC_PERIODIC ? 1 : 0; };
  return {sign(FX_NEG), sign(FX_POS), sign(FY_NEG), sign(FY_POS), sign(FZ_NEG), sign(FZ_POS),
          wraps(FX_POS), wraps(FY_POS), wraps(FZ_POS)};
}

// Keeps a value in a register: the level records are indexed at run time, and the compiler would
// otherwise load them from the parameter bank again in every phase.
__device__ __forceinline__ void hold(int &v) { asm volatile("" : "+r"(v)); }
__device__ __forceinline__ void hold(float &v) { asm volatile("" : "+f"(v)); }
__device__ __forceinline__ void hold(double &v) { asm volatile("" : "+d"(v)); }

// ---- the two arithmetics ---------------------------------------------------------------------
// Reference-layout hierarchy: the expressions of relax_math.cuh, of the coarsest level's host
// routine (coarse_relax_block) and of prolong_cell, in their operand order.
template <typename Real>
struct CtPlain {
  using T = Real;
  struct Coef {
    RelaxCoefD<T> rc;
    ResCoefT<T> res;
  };
  struct Extra {
    CoarseCoef<T> cc;
    int unit;  // cc's fx = fy = fz = 1
    BCDev bc;  // homogeneous boundary conditions: the ghosts written back
  };
  struct Global {
    T *u, *b;
    long long xs, ys;
  };
  static constexpr bool kHostCoarse = true;
  static __device__ __forceinline__ void hold(Coef &c) {
    ct::hold(c.rc.omega), ct::hold(c.rc.hsq), ct::hold(c.rc.ld);
    ct::hold(c.rc.fx), ct::hold(c.rc.fy), ct::hold(c.rc.fz);
  }
  static __device__ __forceinline__ void hold(Extra &x) { ct::hold(x.cc.omega), ct::hold(x.cc.ld), ct::hold(x.cc.h), ct::hold(x.unit); }
  // per-cell constant of the update: the diagonal
  static __device__ __forceinline__ T diag(int i, int j, int k, int nx, int ny, int nz, const Coef &c) {
    return relax_dg<T>(i, j, k, nx, ny, nz, c.rc, nullptr);
  }
  static __device__ __forceinline__ T host_diag(int i, int j, int k, int nx, int ny, int nz, const CoarseCoef<T> &c) {
    const T xm = (i == 0) ? c.xn : (i == nx - 1) ? c.xp : (T)0;
    const T ym = (j == 0) ? c.yn : (j == ny - 1) ? c.yp : (T)0;
    const T zm = (k == 0) ? c.zn : (k == nz - 1) ? c.zp : (T)0;
    return c.ld + xm + ym + zm;
  }
  // the update's division: by the cell's diagonal, whose reciprocal is worked out once
  static __device__ __forceinline__ T reciprocal(T dg) { return (T)1 / dg; }
  // host: the coarsest level's arithmetic
  static __device__ __forceinline__ T update(T u, T b, T sx, T sy, T sz, T dg, T rdg, const Coef &c, const Extra &x,
                                             bool host) {
    const CoarseCoef<T> &h = x.cc;
    T res;
    if (host) {
      res = (-h.h * h.h * b - h.ld * u);
      if (sizeof(T) == 4 && x.unit) {
        // all factors 1: a sum of two floats rounded to double and then to float is the float sum
        // (Figueroa, "When is double rounding innocuous?", 1995: 53 >= 2 * 24 + 2)
        res = ((res + sz) + sy) + sx;
      } else {
        res = (T)((double)res + h.fz * (double)sz);
        res = (T)((double)res + h.fy * (double)sy);
        res = (T)((double)res + h.fx * (double)sx);
      }
    } else if (sizeof(T) == 4) {
      res = (-c.rc.hsq * b - c.rc.ld * u);
      res += c.rc.fz * sz;
      res += c.rc.fy * sy;
      res += c.rc.fx * sx;
    } else {
      res = -c.rc.ld * u;
      res += c.rc.fz * sz;
      res += c.rc.fy * sy;
      res += c.rc.fx * sx;
      res += c.rc.hsq * b;
    }
    return u + divide_by((host ? h.omega : c.rc.omega) * res, dg, rdg);
  }
  static __device__ __forceinline__ T residual(T u, T b, T sx, T sy, T sz, const Coef &c) {
    return b - (c.res.fzh * sz + c.res.fyh * sy + c.res.fxh * sx - c.res.dg * u);
  }
  static __device__ __forceinline__ T mean8(const T (&r)[8], int) {
    return (T)0.125 * (r[0] + r[1] + r[2] + r[3] + r[4] + r[5] + r[6] + r[7]);
  }
  static __device__ __forceinline__ T child(T f, T c, T X, T Y, T Z, T XY, T XZ, T YZ, T XYZ) {
    const T w1 = (T)0.421875, w2 = (T)0.140625, w3 = (T)0.046875, w4 = (T)0.015625;
    return f + w1 * c + w2 * (X + Y + Z) + w3 * (XY + XZ + YZ) + w4 * XYZ;
  }
  // the (-x, +y, +z) child takes its corner weight from the coarse (+1, +1, +1) neighbour
  static constexpr bool kCornerFromPlus = true;
};

// Split FP32 levels of the refinement (chq_device.cuh's s_* phases, the same expressions).
struct CtChq {
  using T = float;
  using Coef = chq::ChqK;
  struct Extra {
    float mxn, mxp, myn, myp, mzn, mzp;
  };
  struct Global {
    float *u0, *u1, *b0, *b1;
    int rz;
  };
  static constexpr bool kHostCoarse = false;
  static __device__ __forceinline__ void hold(Coef &c) {
    ct::hold(c.c0), ct::hold(c.c1), ct::hold(c.ld), ct::hold(c.hsq), ct::hold(c.fx), ct::hold(c.fy), ct::hold(c.fz);
  }
  static constexpr bool kCornerFromPlus = false;
  static __device__ __forceinline__ float reciprocal(float) { return 0.f; }  // nothing is divided
  static __device__ __forceinline__ void hold(Extra &) {}
  static __device__ __forceinline__ float update(float u, float b, float sx, float sy, float sz, float w, float,
                                                 const Coef &k, const Extra &, bool) {
    const float t = __fmaf_rn(k.fz, sz, __fmaf_rn(k.fy, sy, __fmaf_rn(k.fx, sx, -k.hsq * b)));
    return w == 0.f ? __fmaf_rn(k.c1, t, k.c0 * u) : __fmaf_rn(w, __fmaf_rn(-k.ld, u, t), u);
  }
  static __device__ __forceinline__ float residual(float u, float b, float sx, float sy, float sz, const Coef &k) {
    return chq::residual_cell(u, b, sx, sy, sz, k);
  }
  // the order of s_restrict_sum on the levels that the single-CTA tail takes, of k_chq_restrict on
  // the others
  static __device__ __forceinline__ float mean8(const float (&r)[8], int fine_cells) {
    float s = 0.f, t = 0.f;
#pragma unroll
    for (int q = 0; q < 8; q += 2) {
      s += r[q] + r[q + 1];
      t = (t + r[q]) + r[q + 1];
    }
    return 0.125f * (fine_cells <= (int)chq::kChqTailCells ? s : t);
  }
  static __device__ __forceinline__ float child(float f, float c, float X, float Y, float Z, float XY, float XZ,
                                                float YZ, float XYZ) {
    const float s1 = X + Y + Z, s2 = XY + XZ + YZ;
    return __fmaf_rn(__fmaf_rn(27.f, c, __fmaf_rn(9.f, s1, __fmaf_rn(3.f, s2, XYZ))), 0.015625f, f);
  }
};

// ---- parameters --------------------------------------------------------------------------------
template <class Op>
struct CtLevel {
  int nx, ny, nz, M;  // M = nz / 2 entries per row and colour
  int per, nact;      // planes per rank, ranks that hold planes
  FDiv fM, fY;        // division by M and ny
  int ou, us;         // u: first element of the colour-0 array (halo planes included), elements of one
  int ob, bs;         // b likewise, without halos
  typename Op::Coef k;
  typename Op::Global g;
};

// A schedule is a list of visits to levels: optionally the prolongation from the next coarser
// level, sweeps (none, nu1, nu2 or ramp_iters iterations, or the coarsest level's), optionally the
// residual's restriction into the next coarser level.
enum { CT_SWEEPS_NONE = 0, CT_SWEEPS_PRE = 1, CT_SWEEPS_POST = 2, CT_SWEEPS_COARSEST = 3, CT_SWEEPS_RAMP = 4,
       CT_SWEEPS = 7, CT_PROLONG = 8, CT_RESTRICT = 16 };

template <class Op>
struct CtParams {
  CtLevel<Op> lv[kCtMaxLevels];
  int nlev;
  int nu1, nu2, ramp_iters, post_first;  // smoothing iterations; first colour of the post-smoothing
  int coarse_iters, coarse_flip;       // RO_SYMMETRIC: iterations from coarse_flip on are black first
  int host_coarse;                     // coarsest level by the host routine's arithmetic
  int zero_u;                          // lv[0]'s u is zero and is not read
  int once, total;                     // program: [0, once) run once, [once, total) `cycles` times
  int cycles;
  unsigned char prog[256];             // visits, flags | level << 5
  int orr;                             // residual scratch (eight children per coarse cell of a rank)
  BoundarySigns<typename Op::T> sg;
  typename Op::Extra x;
};

// ---- shared::cluster access ----------------------------------------------------------------------
__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned map_rank(unsigned a, int rank) {
  unsigned d;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(rank));
  return d;
}
__device__ __forceinline__ void st_cl(unsigned a, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void st_cl(unsigned a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
// the same where `a` is not zero, as a predicated store
__device__ __forceinline__ void st_cl_if(unsigned a, unsigned off, float v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.shared::cluster.f32 [%1], %2;\n\t}" ::"r"(a), "r"(a + off), "f"(v) : "memory");
}
__device__ __forceinline__ void st_cl_if(unsigned a, unsigned off, double v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.shared::cluster.f64 [%1], %2;\n\t}" ::"r"(a), "r"(a + off), "d"(v) : "memory");
}
template <typename T> __device__ __forceinline__ T ld_cl(unsigned a);
template <> __device__ __forceinline__ float ld_cl<float>(unsigned a) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
template <> __device__ __forceinline__ double ld_cl<double>(unsigned a) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A level's record in registers.  The records are indexed at run time, and read field by field
// where they are used each read of the parameter bank is waited for on its own: here all are
// asked for at once (a prolongation phase on an 8^3 level 2780 -> 2170 cycles, the clearing of a coarse
// level 840 -> 690; 64^3 FP32 solve 470 -> 461 us).
struct LevelRegs {
  int nx, ny, nz, M, per, nact, ou, us, ob, bs;
  FDiv fM, fY;
};
template <class Op>
__device__ __forceinline__ LevelRegs level_regs(const CtLevel<Op> &R) {
  LevelRegs L{R.nx, R.ny, R.nz, R.M, R.per, R.nact, R.ou, R.us, R.ob, R.bs, R.fM, R.fY};
  asm volatile("" : "+r"(L.nx), "+r"(L.ny), "+r"(L.nz), "+r"(L.M), "+r"(L.per), "+r"(L.nact), "+r"(L.ou), "+r"(L.us),
               "+r"(L.ob), "+r"(L.bs), "+r"(L.fM.d), "+r"(L.fM.sh), "+r"(L.fM.m), "+r"(L.fM.l), "+r"(L.fY.d),
               "+r"(L.fY.sh), "+r"(L.fY.m), "+r"(L.fY.l));
  return L;
}
template <class Lv>
__device__ __forceinline__ int planes_of(const Lv &L, int r) {
  return max(0, min(L.per, L.nx - r * L.per));
}
// Barrier after a phase of a level.  A level that rank 0 holds alone is worked on by as many of
// its warps as the level has pairs for (level_threads), on a named barrier of its own; the other
// warps and ranks go on to the next visit that concerns them.
template <int NT, class Lv>
__device__ __forceinline__ int level_threads(const Lv &L) {
  return L.nact > 1 ? NT : min(NT, (L.nx * L.ny * L.M + 31) & ~31);
}
__device__ __forceinline__ void level_barrier(const LevelRegs &L, int l, int threads) {
  if (L.nact > 1) cluster_barrier();
  else if (threads == 32) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(l + 1), "r"(threads) : "memory");
}

// A thread's pair of cells (k = 2m, 2m + 1 of row (i, j)): where its neighbours are, as byte
// offsets from a colour array's start.  Bits of `self`: the neighbour is across a face, i.e. the
// sign times the cell's own value (1 x-, 2 x+, 4 y-, 8 y+, 16 z- of the even cell, 32 z+ of the
// odd one); its offset is then the pair's own, so that it can be loaded all the same.
struct Pair {
  int i, j, m;
  int id, bid;
  int xm, xp, ym, yp, zm, zp;
  int self;
  unsigned left, right;          // where a neighbour rank's halo holds the pair's colour-0 entry, or 0
};

template <class Op>
__device__ __forceinline__ Pair make_pair_at(const LevelRegs &L, const BoundarySigns<typename Op::T> &sg,
                                             unsigned ubase, int rank, int nl, int q) {
  constexpr int E = (int)sizeof(typename Op::T);
  Pair p;
  int row, pl;
  split(L.fM, q, row, p.m);
  split(L.fY, row, pl, p.j);
  p.i = rank * L.per + pl;
  const int M = L.M * E, S = L.ny * M;
  p.bid = q * E;
  p.id = p.bid + S;
  const bool x0 = p.i == 0 && !sg.px, x1 = p.i == L.nx - 1 && !sg.px;
  const bool y0 = p.j == 0, y1 = p.j == L.ny - 1, z0 = p.m == 0, z1 = p.m == L.M - 1;
  const int wy = sg.py ? S - M : 0, wz = sg.pz ? M - E : 0;  // across a y / z face: wrapped, or the pair itself
  p.xm = x0 ? p.id : p.id - S;
  p.xp = x1 ? p.id : p.id + S;
  p.ym = y0 ? p.id + wy : p.id - M;
  p.yp = y1 ? p.id - wy : p.id + M;
  p.zm = z0 ? p.id + wz : p.id - E;
  p.zp = z1 ? p.id - wz : p.id + E;
  p.self = (x0 ? 1 : 0) | (x1 ? 2 : 0) | (y0 && !sg.py ? 4 : 0) | (y1 && !sg.py ? 8 : 0) | (z0 && !sg.pz ? 16 : 0) |
           (z1 && !sg.pz ? 32 : 0);
  const int lr = rank > 0 ? rank - 1 : L.nact - 1, rr = rank + 1 < L.nact ? rank + 1 : 0;
  p.left = pl == 0 && !x0 ? map_rank(ubase + p.id + planes_of(L, lr) * S, lr) : 0u;
  p.right = pl == nl - 1 && !x1 ? map_rank(ubase + p.id - nl * S, rr) : 0u;
  return p;
}

template <class Op>
__device__ __forceinline__ typename Op::T cell_constant(const CtParams<Op> &P, const LevelRegs &L,
                                                        const typename Op::Coef &K, int i, int j, int k, bool host) {
  if constexpr (Op::kHostCoarse) {
    return host ? Op::host_diag(i, j, k, L.nx, L.ny, L.nz, P.x.cc) : Op::diag(i, j, k, L.nx, L.ny, L.nz, K);
  } else {
    float mod = 0.f;
    if (i == 0) mod += P.x.mxn;
    if (i == L.nx - 1) mod += P.x.mxp;
    if (j == 0) mod += P.x.myn;
    if (j == L.ny - 1) mod += P.x.myp;
    if (k == 0) mod += P.x.mzn;
    if (k == L.nz - 1) mod += P.x.mzp;
    return mod == 0.f ? 0.f : K.omega / (K.ld + mod);
  }
}

// Exchanges a register's two colours: m is the XOR of the values for one and the other.
__device__ __forceinline__ int flip_bits(float a, float b) { return __float_as_int(a) ^ __float_as_int(b); }
__device__ __forceinline__ long long flip_bits(double a, double b) { return __double_as_longlong(a) ^ __double_as_longlong(b); }
__device__ __forceinline__ void flip_value(float &v, int m) { v = __int_as_float(__float_as_int(v) ^ m); }
__device__ __forceinline__ void flip_value(double &v, long long m) { v = __longlong_as_double(__double_as_longlong(v) ^ m); }

// Red-black sweeps of a slab of at most NT pairs, everything a sweep needs held in registers: of the
// cell of the sweep's colour the byte addresses of its five outer neighbours (across a face its
// own, with the face's sign), its value, right-hand side and update constant, each turned into
// the other cell's by one XOR between sweeps.  A sweep costs the instructions of its busiest warp, 4
// to 5 cycles each: on a 4^3 level 520 (FP64) to 600 cycles, 580 to 680 with both colours' code and
// both arithmetics in the loop, 720 with the neighbours and the pair's cell chosen by flags, 1150
// with the loads inside branches; loads, division and remote stores are 130 of them.  One pair a
// thread: two or four in registers, or 1024 threads of 64 registers, were slower (set-up, spills).
// HOST: the coarsest level's arithmetic; SIGNED: some face is neither Neumann nor periodic, so that
// a mirrored value carries a sign.
template <class Op, int NT, bool HOST, bool SIGNED>
__device__ __forceinline__ void sweep_slab(const CtParams<Op> &P, const LevelRegs &L, int l, int nthreads, char *U,
                                           const char *B, int rank, int nl, int n, int iters, int first, int flip,
                                           const typename Op::Coef &K, const typename Op::Extra &X,
                                           const BoundarySigns<typename Op::T> &sg) {
  using T = typename Op::T;
  constexpr int E = (int)sizeof(T);
  const int us = L.us * E, bs = L.bs * E;
  int a[6] = {}, ma[6] = {};  // x-, x+, y-, y+, outer z neighbour, own
  T v = 0, w = 0, b = 0, d = 1, rd = 1, sxm = 1, sxp = 1, sym = 1, syp = 1, sz = 1;  // w: the pair's other cell
  decltype(flip_bits(T(), T())) mb = 0, md = 0, mrd = 0, msz = 0;
  unsigned left = 0, right = 0;
  const bool mine = (int)threadIdx.x < n;
  if (mine) {
    const Pair p = make_pair_at<Op>(L, sg, smem_addr(U), rank, nl, threadIdx.x);
    const int c0 = (p.i + p.j) & 1;
    left = p.left;
    right = p.right;
    if (SIGNED) {
      sxm = (p.self & 1) ? sg.xn : (T)1;
      sxp = (p.self & 2) ? sg.xp : (T)1;
      sym = (p.self & 4) ? sg.yn : (T)1;
      syp = (p.self & 8) ? sg.yp : (T)1;
    }
#pragma unroll
    for (int e = 1; e >= 0; e--) {  // e = 0: the cell of colour `first`
      const int c = first ^ e, o = c * us, q = us - o;
      const bool odd = c != c0, face = p.self & (odd ? 32 : 16);
      const int t[6] = {p.xm + ((p.self & 1) ? o : q), p.xp + ((p.self & 2) ? o : q), p.ym + ((p.self & 4) ? o : q),
                        p.yp + ((p.self & 8) ? o : q), (odd ? p.zp : p.zm) + (face ? o : q), p.id + o};
#pragma unroll
      for (int r = 0; r < 6; r++) {
        ma[r] = a[r] ^ t[r];
        a[r] = t[r];
      }
      w = v;
      v = *reinterpret_cast<const T *>(U + o + p.id);
      const T tb = *reinterpret_cast<const T *>(B + c * bs + p.bid);
      const T td = cell_constant<Op>(P, L, K, p.i, p.j, 2 * p.m + odd, HOST), tr = Op::reciprocal(td);
      const T ts = face ? (odd ? sg.zp : sg.zn) : (T)1;
      mb = flip_bits(b, tb), md = flip_bits(d, td), mrd = flip_bits(rd, tr), msz = flip_bits(sz, ts);
      b = tb, d = td, rd = tr, sz = ts;
    }
  }
  int off = first * us;  // of the sweep's colour
  auto at = [&](int o) { return *reinterpret_cast<const T *>(U + o); };
#pragma unroll 1
  for (int ph = 0; ph < 2 * iters; ph++) {
    if (ph != 0 && ph != 2 * flip) {  // the other colour, except where the order turns round
#pragma unroll
      for (int r = 0; r < 6; r++) a[r] ^= ma[r];
      flip_value(b, mb);
      flip_value(d, md);
      if (Op::kHostCoarse) flip_value(rd, mrd);
      if (SIGNED) flip_value(sz, msz);
      const T o = v;
      v = w;
      w = o;
      off = us - off;
    }
    if (mine) {
      const T ax = at(a[0]), bx = at(a[1]), ay = at(a[2]), by = at(a[3]), az = at(a[4]);
      const T sx = SIGNED ? sxm * ax + sxp * bx : ax + bx;
      const T sy = SIGNED ? sym * ay + syp * by : ay + by;
      const T sz_ = (SIGNED ? sz * az : az) + w;
      v = Op::update(v, b, sx, sy, sz_, d, rd, K, X, HOST);
      *reinterpret_cast<T *>(U + a[5]) = v;
      st_cl_if(left, off, v);
      st_cl_if(right, off, v);
    }
    level_barrier(L, l, nthreads);
  }
}

// One visit to level l.
template <class Op, int NT>
__device__ __forceinline__ void visit_level(const CtParams<Op> &P, int what, int l, typename Op::T *sm, int rank) {
  using T = typename Op::T;
  constexpr int E = (int)sizeof(T);
  const CtLevel<Op> &coarser = P.lv[min(l + 1, P.nlev - 1)];
  const LevelRegs L = level_regs(P.lv[l]);
  const int nthreads = level_threads<NT>(L);
  const int nl = planes_of(L, rank), n = nl * L.ny * L.M;
  const bool split_level = L.nact > 1, split_coarse = split_level && coarser.nact > 1;
  if ((what & CT_PROLONG) && !split_coarse) {
    level_barrier(L, l, nthreads);  // the coarser level is done
    if (split_level && rank != 0 && nl > 0) {
      // the planes of rank 0's level that this rank's cells read (halo planes included), into the
      // same place here: read one by one from every rank they cost 8000 cycles on rank 0's memory
      const LevelRegs Cl = level_regs(coarser);
      const int S = Cl.ny * Cl.M, lo = ((rank * L.per) >> 1) * S, cnt = (((nl + 1) >> 1) + 2) * S;
      for (int q = threadIdx.x; q < 2 * cnt; q += NT) {
        const int e = Cl.ou + lo + (q < cnt ? q : q - cnt + Cl.us);
        sm[e] = ld_cl<T>(map_rank(smem_addr(sm + e), 0));
      }
    }
    if (split_level) __syncthreads();
  }
  char *const U = reinterpret_cast<char *>(sm + L.ou);
  const char *const B = reinterpret_cast<const char *>(sm + L.ob);
  const unsigned ubase = smem_addr(U);
  const int us = L.us * E, bs = L.bs * E;
  const int kind = what & CT_SWEEPS;
  const bool host = Op::kHostCoarse && kind == CT_SWEEPS_COARSEST && P.host_coarse;
  const int iters = kind == CT_SWEEPS_PRE ? P.nu1 : kind == CT_SWEEPS_POST ? P.nu2 : kind == CT_SWEEPS_RAMP ? P.ramp_iters
                    : kind == CT_SWEEPS_COARSEST ? P.coarse_iters : 0;
  const int flip = kind == CT_SWEEPS_COARSEST ? P.coarse_flip : iters;
  const int first = kind == CT_SWEEPS_POST ? P.post_first : 0;
  const int most = L.per * L.ny * L.M;  // pairs of the largest slab: the same choice on every rank
  typename Op::Coef K = P.lv[l].k;
  typename Op::Extra X = P.x;
  Op::hold(X);
  BoundarySigns<T> sg = P.sg;
  Op::hold(K);
  hold(sg.xn), hold(sg.xp), hold(sg.yn), hold(sg.yp), hold(sg.zn), hold(sg.zp);
  auto at = [](const char *base, int off) { return *reinterpret_cast<const T *>(base + off); };
  if (what & CT_PROLONG) {
    const LevelRegs Cl = level_regs(coarser);
    for (int q = threadIdx.x; q < n; q += NT) {
      const Pair p = make_pair_at<Op>(L, sg, ubase, rank, nl, q);
      const int c0 = (p.i + p.j) & 1;
      T v[2];
      v[0] = at(U, c0 * us + p.id);
      v[1] = at(U, (1 - c0) * us + p.id);
      // prolongation: the four coarse rows of the pair's octant at K - 1, K, K + 1
      const int I = p.i >> 1, J = p.j >> 1, Kz = p.m, M = Cl.M * E, S = Cl.ny * M, cus = Cl.us * E;
      const bool xo = p.i & 1, yo = p.j & 1;
      // x and y of the far rows and the sign of a value there (a face rule mirrors the row itself;
      // periodic x neighbours are in the halo planes)
      const bool fx = (xo ? I == Cl.nx - 1 : I == 0) && !sg.px, fy = yo ? J == Cl.ny - 1 : J == 0;
      const int X1 = fx ? I : (xo ? I + 1 : I - 1);
      const int Y1 = fy ? (sg.py ? (yo ? 0 : Cl.ny - 1) : J) : (yo ? J + 1 : J - 1);
      const T s1 = fx ? (xo ? sg.xp : sg.xn) : (T)1, s2 = fy && !sg.py ? (yo ? sg.yp : sg.yn) : (T)1;
      const bool bz = Kz == 0, tz = Kz == Cl.nz - 1;
      const int Zm = bz ? (sg.pz ? Cl.nz - 1 : 0) : Kz - 1, Zp = tz ? (sg.pz ? 0 : Kz) : Kz + 1;
      const T szm = bz && !sg.pz ? sg.zn : (T)1, szp = tz && !sg.pz ? sg.zp : (T)1;
      const char *const cu = reinterpret_cast<const char *>(sm + Cl.ou) + (1 - (split_coarse ? rank * Cl.per : 0)) * S;
      auto val = [&](int X, int Y, int Z) {
        return at(cu, X * S + Y * M + (((X + Y + Z) & 1) ? cus : 0) + (Z >> 1) * E);
      };
      T c[4][3];  // rows (I, J), (X1, J), (I, Y1), (X1, Y1) at K, K - 1, K + 1
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const int X = (r & 1) ? X1 : I, Y = (r & 2) ? Y1 : J;
        c[r][0] = val(X, Y, Kz);
        c[r][1] = val(X, Y, Zm);
        c[r][2] = val(X, Y, Zp);
      }
      T corner = 0;
      if (Op::kCornerFromPlus) {
        // the reference kernel takes the (-x, +y, +z) child's corner from coarse (+1, +1, +1)
        const bool f2 = I == Cl.nx - 1 && !sg.px;
        corner = (f2 ? sg.xp : (T)1) * (s2 * (szp * val(f2 ? I : I + 1, Y1, Zp)));
      }
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const T s = ((r & 1) ? s1 : (T)1) * ((r & 2) ? s2 : (T)1);
        c[r][0] = s * c[r][0];
        c[r][1] = s * (szm * c[r][1]);
        c[r][2] = s * (szp * c[r][2]);
      }
      if (!(Op::kCornerFromPlus && !xo && yo)) corner = c[3][2];
      v[0] = Op::child(v[0], c[0][0], c[1][0], c[2][0], c[0][1], c[3][0], c[1][1], c[2][1], c[3][1]);
      v[1] = Op::child(v[1], c[0][0], c[1][0], c[2][0], c[0][2], c[3][0], c[1][2], c[2][2], corner);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int o = (h ^ c0) * us;
        *reinterpret_cast<T *>(U + o + p.id) = v[h];
        st_cl_if(p.left, o, v[h]);
        st_cl_if(p.right, o, v[h]);
      }
    }
    level_barrier(L, l, nthreads);
  }
  if (iters > 0) {
    const bool plus = (sg.px || (sg.xn == (T)1 && sg.xp == (T)1)) && (sg.py || (sg.yn == (T)1 && sg.yp == (T)1)) &&
                      (sg.pz || (sg.zn == (T)1 && sg.zp == (T)1));
    if (most <= NT && !host && plus) sweep_slab<Op, NT, false, false>(P, L, l, nthreads, U, B, rank, nl, n, iters, first, flip, K, X, sg);
    else if (most <= NT && !host) sweep_slab<Op, NT, false, true>(P, L, l, nthreads, U, B, rank, nl, n, iters, first, flip, K, X, sg);
    else if (Op::kHostCoarse && most <= NT && plus)
      sweep_slab<Op, NT, Op::kHostCoarse, false>(P, L, l, nthreads, U, B, rank, nl, n, iters, first, flip, K, X, sg);
    else if (Op::kHostCoarse && most <= NT)
      sweep_slab<Op, NT, Op::kHostCoarse, true>(P, L, l, nthreads, U, B, rank, nl, n, iters, first, flip, K, X, sg);
    else {  // pairs worked out again in every phase
      for (int ph = 0; ph < 2 * iters; ph++) {
        const int color = (ph & 1) ^ (ph < 2 * flip ? first : 1 - first);
        for (int q = threadIdx.x; q < n; q += NT) {
          const Pair p = make_pair_at<Op>(L, sg, ubase, rank, nl, q);
          const bool odd = ((p.i + p.j) & 1) != color;
          const char *const O = U + (1 - color) * us;
          const T u = at(U, color * us + p.id);
          const T lxm = at(O, p.xm), lxp = at(O, p.xp), lym = at(O, p.ym), lyp = at(O, p.yp), lz = at(O, odd ? p.zp : p.zm);
          const T sx = ((p.self & 1) ? sg.xn * u : lxm) + ((p.self & 2) ? sg.xp * u : lxp);
          const T sy = ((p.self & 4) ? sg.yn * u : lym) + ((p.self & 8) ? sg.yp * u : lyp);
          const T zv = (p.self & (odd ? 32 : 16)) ? (odd ? sg.zp : sg.zn) * u : lz;
          const T d = cell_constant<Op>(P, L, K, p.i, p.j, 2 * p.m + odd, host);
          const T nv = Op::update(u, at(B, color * bs + p.bid), sx, sy, zv + at(O, p.id), d, Op::reciprocal(d), K, X, host);
          *reinterpret_cast<T *>(U + color * us + p.id) = nv;
          st_cl_if(p.left, color * us, nv);
          st_cl_if(p.right, color * us, nv);
        }
        level_barrier(L, l, nthreads);
      }
    }
  }
  if (!(what & CT_RESTRICT)) return;
  const LevelRegs Cl = level_regs(coarser);
  const int stride = Cl.per * Cl.ny * Cl.nz;  // residual scratch: elements per child
  {
    for (int q = threadIdx.x; q < n; q += NT) {
      const Pair p = make_pair_at<Op>(L, sg, ubase, rank, nl, q);
      const int c0 = (p.i + p.j) & 1;
      T b[2];
      b[0] = at(B, c0 * bs + p.bid);
      b[1] = at(B, (1 - c0) * bs + p.bid);
      // residuals of both cells, stored into the scratch of the coarse cell's owner
      const char *const Oe = U + (1 - c0) * us, *const Oo = U + c0 * us;  // other colour of the even / odd cell
      const T e = at(U, c0 * us + p.id), o = at(U, (1 - c0) * us + p.id);
      const T e0 = at(Oe, p.xm), e1 = at(Oe, p.xp), e2 = at(Oe, p.ym), e3 = at(Oe, p.yp), e4 = at(Oe, p.zm);
      const T o0 = at(Oo, p.xm), o1 = at(Oo, p.xp), o2 = at(Oo, p.ym), o3 = at(Oo, p.yp), o5 = at(Oo, p.zp);
      const T exs = ((p.self & 1) ? sg.xn * e : e0) + ((p.self & 2) ? sg.xp * e : e1);
      const T oxs = ((p.self & 1) ? sg.xn * o : o0) + ((p.self & 2) ? sg.xp * o : o1);
      const T eys = ((p.self & 4) ? sg.yn * e : e2) + ((p.self & 8) ? sg.yp * e : e3);
      const T oys = ((p.self & 4) ? sg.yn * o : o2) + ((p.self & 8) ? sg.yp * o : o3);
      const T ezs = ((p.self & 16) ? sg.zn * e : e4) + o;
      const T ozs = e + ((p.self & 32) ? sg.zp * o : o5);
      const int I = (p.i >> 1) - (split_coarse ? rank * Cl.per : 0);
      const int to = P.orr + (4 * (p.i & 1) + 2 * (p.j & 1)) * stride + (I * Cl.ny + (p.j >> 1)) * Cl.nz + p.m;
      const T re = Op::residual(e, b[0], exs, eys, ezs, K), ro = Op::residual(o, b[1], oxs, oys, ozs, K);
      if (split_coarse == split_level) {  // this rank's own coarse cells
        sm[to] = re;
        sm[to + stride] = ro;
      } else {
        const unsigned far = map_rank(smem_addr(sm + to), 0);
        st_cl(far, re);
        st_cl(far + stride * E, ro);
      }
    }
    // the residuals of a split level whose coarser level is split too are read by their own rank
    if (split_coarse) __syncthreads();
    else level_barrier(L, l, nthreads);
  }
  // the coarse owner adds up each cell's eight residuals and clears u (halos included)
  const int cthreads = level_threads<NT>(Cl);
  if (Cl.nact == 1 && (rank != 0 || (int)threadIdx.x >= cthreads)) return;
  const int cl = planes_of(Cl, rank), cn = cl * Cl.ny * Cl.M, S = Cl.ny * Cl.M;
  const T *r = sm + P.orr;
  T *CU = sm + Cl.ou, *CB = sm + Cl.ob;
  for (int q = threadIdx.x; q < cn; q += cthreads) {
    int row, m, pl, j;
    split(Cl.fM, q, row, m);
    split(Cl.fY, row, pl, j);
    const int c0 = (rank * Cl.per + pl + j) & 1;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      T x[8];
#pragma unroll
      for (int e = 0; e < 8; e++) x[e] = r[e * stride + row * Cl.nz + 2 * m + h];
      CB[(h ^ c0) * Cl.bs + q] = Op::mean8(x, L.nx * L.ny * L.nz);
    }
  }
  for (int q = threadIdx.x; q < (cl + 2) * S; q += cthreads) {
    CU[q] = (T)0;
    CU[Cl.us + q] = (T)0;
  }
  level_barrier(Cl, l + 1, cthreads);
}

// The visits in order.
template <class Op, int NT>
__device__ __forceinline__ void run_schedule(const CtParams<Op> &P, typename Op::T *sm, int rank) {
  int pc = 0, left = P.cycles;
  for (;;) {
    if (pc == P.total) {
      pc = P.once;
      left--;
    }
    if (pc >= P.once && (left <= 0 || P.once == P.total)) break;
    const int step = P.prog[pc++], l = step >> 5;
    const CtLevel<Op> &L = P.lv[l];
    if (L.nact == 1 && (rank != 0 || (int)threadIdx.x >= level_threads<NT>(L))) continue;
    visit_level<Op, NT>(P, step & 31, l, sm, rank);
  }
}

// ---- loading and storing ------------------------------------------------------------------------
template <typename T, int NT>
__device__ __forceinline__ void load_top(const CtParams<CtPlain<T>> &P, T *sm, int rank) {
  const auto &L = P.lv[0];
  const int nl = planes_of(L, rank), S = L.ny * L.M;
  T *U = sm + L.ou, *B = sm + L.ob;
#pragma unroll 4
  for (int q = threadIdx.x; q < (nl + 2) * S; q += NT) {
    int row, m, pl, j;
    split(L.fM, q, row, m);
    split(L.fY, row, pl, j);
    int i = rank * L.per + pl - 1;
    T e = 0, o = 0;
    if (P.sg.px) i = i < 0 ? L.nx - 1 : i >= L.nx ? 0 : i;
    const int c0 = (i + j) & 1;
    if (nl > 0 && i >= 0 && i < L.nx) {
      const long long at = (long long)i * L.g.xs + (long long)j * L.g.ys + 2 * m;
      if (!P.zero_u) { e = L.g.u[at]; o = L.g.u[at + 1]; }
      if (pl >= 1 && pl <= nl) {
        B[c0 * L.bs + q - S] = L.g.b[at];
        B[(1 - c0) * L.bs + q - S] = L.g.b[at + 1];
      }
    }
    U[c0 * L.us + q] = e;
    U[(1 - c0) * L.us + q] = o;
  }
}

// Every level's u with its ghosts, and b below the top, as the per-level kernels leave them.  A
// cell is the source of at most one ghost per axis (GhostEmit's rule: the face's own cell, or the
// opposite face's where periodic), so a boundary pair stores itself up to four times, once per
// choice of the cell's row or its ghost along x and y, with its z ghost beside it.
template <typename T, int NT>
__device__ __forceinline__ void store_levels(const CtParams<CtPlain<T>> &P, T *sm, int rank) {
  const auto sg = P.sg;
  const int *const ty = P.x.bc.type;
  for (int l = 0; l < P.nlev; l++) {
    const auto &L = P.lv[l];
    if (L.nact == 1 && rank != 0) continue;
    const int nl = planes_of(L, rank), n = nl * L.ny * L.M, S = L.ny * L.M;
    const T *U = sm + L.ou, *B = sm + L.ob;
    T *const gu = L.g.u, *const gb = L.g.b;
    const long long xs = L.g.xs, ys = L.g.ys;
    for (int q = threadIdx.x; q < n; q += NT) {
      int row, m, pl, j;
      split(L.fM, q, row, m);
      split(L.fY, row, pl, j);
      const int i = rank * L.per + pl, c0 = (i + j) & 1;
      const long long at = (long long)i * xs + (long long)j * ys + 2 * m;
      const T e = U[c0 * L.us + q + S], o = U[(1 - c0) * L.us + q + S];
      gu[at] = e;
      gu[at + 1] = o;
      if (l > 0) {
        gb[at] = B[c0 * L.bs + q];
        gb[at + 1] = B[(1 - c0) * L.bs + q];
      }
      const bool xn = i == 0, xp = i == L.nx - 1, yn = j == 0, yp = j == L.ny - 1, zn = m == 0, zp = m == L.M - 1;
      if (!(xn || xp || yn || yp || zn || zp)) continue;
      // offsets of the ghost row along x and y (0: none), signs, and the z ghosts' places
      const long long gx = xn ? (sg.px ? L.nx * xs : ty[FX_NEG] != OCU_BC_NONE ? -xs : 0)
                         : xp ? (sg.px ? -L.nx * xs : ty[FX_POS] != OCU_BC_NONE ? xs : 0) : 0;
      const long long gy = yn ? (sg.py ? L.ny * ys : ty[FY_NEG] != OCU_BC_NONE ? -ys : 0)
                         : yp ? (sg.py ? -L.ny * ys : ty[FY_POS] != OCU_BC_NONE ? ys : 0) : 0;
      const T sx = sg.px ? (T)1 : xn ? sg.xn : sg.xp, sy = sg.py ? (T)1 : yn ? sg.yn : sg.yp;
      const T sz0 = sg.pz ? (T)1 : sg.zn, sz1 = sg.pz ? (T)1 : sg.zp;
      const int z0 = sg.pz ? L.nz : -1, z1 = sg.pz ? 1 - L.nz : 2;  // from the pair's even cell
      const bool w0 = zn && (sg.pz || ty[FZ_NEG] != OCU_BC_NONE), w1 = zp && (sg.pz || ty[FZ_POS] != OCU_BC_NONE);
#pragma unroll
      for (int a = 0; a < 4; a++) {
        if (((a & 1) && gx == 0) || ((a & 2) && gy == 0)) continue;
        const T s = ((a & 1) ? sx : (T)1) * ((a & 2) ? sy : (T)1);
        T *const g = gu + at + ((a & 1) ? gx : 0) + ((a & 2) ? gy : 0);
        if (a) {
          g[0] = s * e;
          g[1] = s * o;
        }
        if (w0) g[z0] = sz0 * (s * e);
        if (w1) g[z1] = sz1 * (s * o);
      }
    }
  }
}

template <typename, int NT>
__device__ __forceinline__ void load_top(const CtParams<CtChq> &P, float *sm, int rank) {
  const auto &L = P.lv[0];
  const int nl = planes_of(L, rank), S = L.ny * L.M;
  float *U = sm + L.ou, *B = sm + L.ob;
#pragma unroll 4
  for (int q = threadIdx.x; q < (nl + 2) * S; q += NT) {
    int row, m, pl, j;
    split(L.fM, q, row, m);
    split(L.fY, row, pl, j);
    int i = rank * L.per + pl - 1;
    float a = 0.f, b = 0.f;
    if (P.sg.px) i = i < 0 ? L.nx - 1 : i >= L.nx ? 0 : i;
    if (nl > 0 && i >= 0 && i < L.nx) {
      const long long at = ((long long)i * L.ny + j) * L.g.rz + m;
      if (!P.zero_u) { a = L.g.u0[at]; b = L.g.u1[at]; }
      if (pl >= 1 && pl <= nl) {
        B[q - S] = L.g.b0[at];
        B[L.bs + q - S] = L.g.b1[at];
      }
    }
    U[q] = a;
    U[L.us + q] = b;
  }
}

template <typename, int NT>
__device__ __forceinline__ void store_levels(const CtParams<CtChq> &P, float *sm, int rank) {
  const auto &L = P.lv[0];
  const int nl = planes_of(L, rank), n = nl * L.ny * L.M, S = L.ny * L.M;
  const float *U = sm + L.ou;
  for (int q = threadIdx.x; q < n; q += NT) {
    int row, m, pl, j;
    split(L.fM, q, row, m);
    split(L.fY, row, pl, j);
    const long long at = ((long long)(rank * L.per + pl) * L.ny + j) * L.g.rz + m;
    L.g.u0[at] = U[q + S];
    L.g.u1[at] = U[L.us + q + S];
  }
}

template <class Op, int NT>
__global__ void __launch_bounds__(NT, 1) k_cluster_tail(const __grid_constant__ CtParams<Op> P) {
  pdl_entry();
  extern __shared__ __align__(16) unsigned char ct_smem[];
  typename Op::T *sm = reinterpret_cast<typename Op::T *>(ct_smem);
  const int rank = blockIdx.x;  // one cluster is the whole grid
  load_top<typename Op::T, NT>(P, sm, rank);
  cluster_barrier();
  run_schedule<Op, NT>(P, sm, rank);
  cluster_barrier();  // no rank leaves while its shared memory may still be read or written
  store_levels<typename Op::T, NT>(P, sm, rank);
}

// ---- host side --------------------------------------------------------------------------------------
// Placement of levels s..L-1 over at most max_ranks CTAs.  Returns the shared memory in bytes.
template <class Op>
inline size_t ct_place(CtParams<Op> &P, const std::vector<std::array<int, 3>> &dims, int s, int max_ranks, int *ranks) {
  using T = typename Op::T;
  P.nlev = (int)dims.size() - s;
  // The coarsest level that is split gets as few planes per rank as max_ranks allows, and every
  // finer one twice its coarser neighbour's: a rank then owns the children of its coarse planes,
  // and transfers between split levels stay inside a rank.
  int off = 0, scratch = 0, per = 0;
  *ranks = 1;
  for (int l = P.nlev - 1; l >= 0; l--) {
    CtLevel<Op> &L = P.lv[l];
    const auto &d = dims[s + l];
    L.nx = d[0]; L.ny = d[1]; L.nz = d[2];
    L.M = d[2] / 2;
    if ((long long)d[0] * d[1] * d[2] <= kCtSingleCells && per == 0) {
      L.per = d[0];
    } else {
      per = per ? 2 * per : (d[0] + max_ranks - 1) / max_ranks;
      L.per = per;
    }
    L.nact = (d[0] + L.per - 1) / L.per;
    while (*ranks < L.nact) *ranks *= 2;
    L.fM = make_fdiv(L.M);
    L.fY = make_fdiv(L.ny);
    L.us = (L.per + 2) * L.ny * L.M;
    L.bs = L.per * L.ny * L.M;
    L.ou = off;
    off += 2 * L.us;
    L.ob = off;
    off += 2 * L.bs;
    if (l > 0) scratch = std::max(scratch, 8 * L.per * L.ny * L.nz);
  }
  P.orr = off;
  return ((size_t)off + scratch) * sizeof(T);
}

// Most cells of the finest level the cluster takes: as many as its threads own one pair each of
// (16 x 512 pairs).  Measured (us, levels from 8^3 / 16^3 / 32x32x16 / 32^3 down in the cluster): FP32
// 64^3 solve 578 / 508 / 477 / 502, 128x96x64 projection 835 / 765 / 653 / 715, 128x128x64 plain
// flow step 5356 / 4830 / 4169 / 4600; a 32^3 level costs 1.8 us a sweep here, its pairs worked out again
// in every sweep, and 2.4 us as a launch, but its visits' set-up outweighs that.
constexpr long long kCtTopCells = 2 * 16 * kCtThreads;

// First level of the cluster's part (at least `lowest`): the finest one from which all levels fit
// and whose cells number at most max_cells; -1 when not even the coarsest level fits.
template <class Op>
inline int ct_first(const std::vector<std::array<int, 3>> &dims, int lowest, long long max_cells, int max_ranks) {
  CtParams<Op> P;
  const int L = (int)dims.size();
  int s = -1;
  for (int l = L - 1; l >= lowest && L - l <= kCtMaxLevels; l--) {
    const auto &d = dims[l];
    if (d[0] % 2 || d[1] % 2 || d[2] % 2) break;
    const long long cells = (long long)d[0] * d[1] * d[2];
    if (l < L - 1 && cells > max_cells) break;
    if (cells > (1LL << 24)) break;
    int ranks;
    if (ct_place<Op>(P, dims, l, max_ranks, &ranks) > kCtSmemCap) break;
    s = l;
  }
  return s;
}

// The largest cluster of k_cluster_tail<Op> that the current device can hold (16, else 8, else 0:
// no such launch is possible), asked once per device.
template <class Op>
inline int ct_max_ranks() {
  static std::atomic<int> known[64];  // 0: not asked yet, -1: none
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::atomic<int> &k = known[dev & 63];
  if (k.load() == 0) {
    // An error that an earlier call left is for the next launch to report: the questions below would
    // clear it (cudaFuncSetAttribute does), so they are left for another time.
    if (cudaPeekAtLastError() != cudaSuccess) return 0;
    int found = -1;
    bool ok = true;
    const void *f = (const void *)k_cluster_tail<Op, kCtThreads>;
    ok = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCtSmemCap) == cudaSuccess &&
           cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    for (int c = 16; ok && found < 0 && c >= 8; c /= 2) {
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3(c);
      cfg.blockDim = dim3(kCtThreads);
      cfg.dynamicSmemBytes = kCtSmemCap;
      cudaLaunchAttribute a{};
      a.id = cudaLaunchAttributeClusterDimension;
      a.val.clusterDim.x = c;
      a.val.clusterDim.y = a.val.clusterDim.z = 1;
      cfg.attrs = &a;
      cfg.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, k_cluster_tail<Op, kCtThreads>, &cfg) == cudaSuccess && n > 0) found = c;
    }
    cudaGetLastError();  // an unsupported size leaves an error behind
    k.store(found);
  }
  return std::max(0, k.load());
}

// The schedule of one launch: the FMG ramp from lv[0]'s right-hand side if `ramp` (restriction to
// the coarsest level, then per level a prolongation and a V-cycle from it, or, on levels of more
// than vcycle_cells cells, a prolongation and ramp_iters iterations), then `cycles` V-cycles from
// lv[0].  Where lv[0] is level 0 of the whole hierarchy it has no post-smoothing and, above
// vcycle_cells, no iterations in the ramp.
template <class Op>
inline void ct_schedule(CtParams<Op> &P, bool ramp, int cycles, bool top_is_level0, long long vcycle_cells) {
  const int last = P.nlev - 1;
  int n = 0;
  // the ramp's prolongation into a level and the V-cycle that starts there are one visit
  auto visit = [&](int l, int what) { P.prog[n++] = (unsigned char)(what | l << 5); };
  auto vcycle = [&](int a, int with) {
    for (int l = a; l < last; l++) visit(l, CT_SWEEPS_PRE | CT_RESTRICT | (l == a ? with : 0));
    visit(last, CT_SWEEPS_COARSEST);
    for (int l = last - 1; l >= a; l--)
      visit(l, CT_PROLONG | (l == 0 && top_is_level0 ? CT_SWEEPS_NONE : CT_SWEEPS_POST));
  };
  if (ramp) {
    for (int l = 0; l < last; l++) visit(l, CT_SWEEPS_NONE | CT_RESTRICT);
    visit(last, CT_SWEEPS_COARSEST);
    for (int f = last - 1; f >= 0; f--) {
      if ((long long)P.lv[f].nx * P.lv[f].ny * P.lv[f].nz <= vcycle_cells) vcycle(f, CT_PROLONG);
      else visit(f, CT_PROLONG | (f == 0 && top_is_level0 ? CT_SWEEPS_NONE : CT_SWEEPS_RAMP));
    }
  }
  P.once = n;
  if (cycles > 0) vcycle(0, 0);
  P.total = n;
  P.cycles = cycles;
  P.zero_u = ramp ? 1 : 0;
}

template <class Op>
inline ocu_status ct_launch(const CtParams<Op> &P, int ranks, size_t bytes, cudaStream_t s) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(ranks);
  cfg.blockDim = dim3(kCtThreads);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = s;
  cudaLaunchAttribute a[2];
  std::memset(a, 0, sizeof(a));
  a[0].id = cudaLaunchAttributeClusterDimension;
  a[0].val.clusterDim.x = ranks;
  a[0].val.clusterDim.y = a[0].val.clusterDim.z = 1;
  a[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = a;
  cfg.numAttrs = (pdl_enabled() && !pdl_suppressed()) ? 2 : 1;
  cudaLaunchKernelEx(&cfg, k_cluster_tail<Op, kCtThreads>, P);
  return check_launch("k_cluster_tail");
}

}  // namespace
}  // namespace ct
}  // namespace ocub
