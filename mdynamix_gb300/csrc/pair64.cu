// pair64.cu -- the FP64 path's real-space sweeps: LOCALF (forces.f:813-998)
// on the short rows into H, FORCES (forces.f:1014-1202) on the long rows into
// G.  Half rows (every pair once, as in the reference list); TPO lanes walk an
// owner's row, the owner's force is summed in registers, the partner's goes
// out with FP64 atomics.
//
// GB300 issues one FP64 warp instruction per 64 cycles on each scheduler, so
// a sweep's time is its FP64 instruction count: about 84 a pair with the
// reference's expressions written out (reciprocal square root, exp, erfc
// polynomial, reciprocal).  The screened Coulomb force and energy are smooth
// functions of r^2 alone, so k_pair64t takes them from a table (PairPoly): 128
// bins an octave of r^2, each a polynomial of degree 6 in the position within
// the bin, whose four leading steps are FP64 FMAs and whose tail (2^-30 of the
// value) runs in FP32.  Its error, below 2^-54 of the value plus one
// rounding, is below that of the written-out expressions, whose roundings it
// replaces.  The bin and the position come from the bits of r^2 by integer
// operations.  A Coulomb pair then takes 19 FP64 instructions.  Pairs with an
// LJ term and the few that are not plain Ewald pairs (own molecule, 1-4,
// shifted by MDEE, r^2 outside the table) are put aside in shared memory, of
// all owners of a warp, and evaluated 32 at a time, so that no warp issues an
// expression for a few of its lanes.
//
// In a rectangular cell k_pair64x does the same in 64-bit integers, which
// leaves FP64 instructions for the LJ terms and a row's end only.
//
// Measured on a GB300 at 98,304 atoms (one warp an owner and everything
// written out; k_pair64t; k_pair64x): short rows, forces 0.526, 0.20, 0.090 ms;
// long rows with energies 4.88, 2.40, 1.15 ms, with energies by type pair
// 15.3, 3.1, 1.43 ms.  k_pair64t's FP64 pipe is 82-86 % active.  Error of the
// short rows' forces against 128 bits (200 ions; rms, of the rms force): 2.8e-15
// written out, 4e-16 in integers.
//
// k_pair64 writes the reference's expressions out for every pair: the
// reaction field (LMNBL).
#include <algorithm>
#include <cmath>
#include <cstring>

#include "mdx_internal.cuh"
#include "pair_math.cuh"
#include "px_units.h"

namespace {

// LJ tables (forces.f:838-862 / 1040-1066), by LJ type pair.
struct Lj64 {
  const double *a6lj, *b12lj, *a6lj0, *b12lj0, *a6_14, *b12_14;
};

// One bin of a tabulated function of r^2: value = c0 + t (c1 + t (c2 + t (c3 +
// t tail))), tail = c4 + t (c5 + t c6), t in [-1/2, 1/2) the position in the bin.
struct __align__(16) PairPoly {
  double c0, c1, c2, c3;
  float c4, c5, c6, pad;
};
constexpr int PT_OCT0 = -2, PT_NOCT = 12;     // r^2 from 2^-2 to 2^10 A^2
constexpr int PT_BINS = 128 * PT_NOCT;
constexpr int PT_BASE = (1023 + PT_OCT0) * 128;  // bin of r^2: its exponent and 7 leading bits
enum { PT_FORCE = 0, PT_ENER, PT_R1I, PT_R2I, PT_NFN };

// ------------------------------------------------- two-word FP64 numbers --
// Sums and products of pairs of doubles (Dekker, Numer. Math. 18, 1971): the
// table's values and coefficients, to about 100 bits.
struct dd {
  double h, l;
};
__device__ __forceinline__ dd two_sum(double a, double b) {
  const double s = a + b, t = s - a;
  return dd{s, (a - (s - t)) + (b - t)};
}
__device__ __forceinline__ dd norm(double a, double b) {
  const double s = a + b;
  return dd{s, b - (s - a)};
}
__device__ __forceinline__ dd operator+(dd a, dd b) {
  const dd s = two_sum(a.h, b.h);
  return norm(s.h, s.l + (a.l + b.l));
}
__device__ __forceinline__ dd operator-(dd a) { return dd{-a.h, -a.l}; }
__device__ __forceinline__ dd operator*(dd a, dd b) {
  const double p = a.h * b.h;
  return norm(p, fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h));
}
__device__ __forceinline__ dd D(double a) { return dd{a, 0.0}; }
__device__ dd div(dd a, dd b) {
  const double q = a.h / b.h;
  const dd r = a + -(b * D(q));
  const double q2 = r.h / b.h;
  const dd r2 = r + -(b * D(q2));
  const dd s = norm(q, q2);
  return s + D(r2.h / b.h);
}
__device__ dd sqrt_dd(double a) {
  const double s = sqrt(a);
  return norm(s, fma(-s, s, a) / (2.0 * s));
}
__device__ dd exp_neg_dd(dd y) {  // exp(-y), y >= 0; 0 beyond 600
  if (y.h > 600.0) return D(0.0);
  const double n = rint(y.h * 1.4426950408889634);
  const dd ln2{0.6931471805599453, 2.3190468138462996e-17};
  dd r = (ln2 * D(n)) + -y;  // exp(-y) = 2^-n exp(r)
  r.h *= 1.0 / 64;
  r.l *= 1.0 / 64;
  dd s = D(1.0);
  for (int k = 11; k >= 1; --k) s = D(1.0) + div(r * s, D((double)k));
  for (int k = 0; k < 6; ++k) s = s * s;
  return dd{ldexp(s.h, -(int)n), ldexp(s.l, -(int)n)};
}

// The functions at r^2 = x (exact), per unit charge product: FORCE / QIJ and
// EES / QIJ of forces.f:1149-1157 with its erfc polynomial, 1 / r^2, 1 / r.
__device__ dd pair_fn(int fn, double x, double alphad) {
  if (fn == PT_R2I) return div(D(1.0), D(x));
  const dd r = sqrt_dd(x);
  if (fn == PT_R1I) return div(D(1.0), r);
  const dd ar = D(alphad) * r;
  const dd t = div(D(1.0), D(1.0) + D(MDX_B1) * ar);
  const dd e = exp_neg_dd(D(alphad) * D(alphad) * D(x));
  dd p = D(MDX_A5) * t + D(MDX_A4);
  p = p * t + D(MDX_A3);
  p = p * t + D(MDX_A2);
  p = p * t + D(MDX_A1);
  const dd er = div(p * t * e, r);
  if (fn == PT_ENER) return er;
  return div(D(MDX_TOTPI) * D(alphad) * e + er, D(x));
}

// Coefficients of a function's polynomial in one bin: block of 32 bins x 7
// Chebyshev points.  Thread (point k, bin) forms the value at its point, its
// divided difference of each order, then coefficient k of the monomial form.
// An FP64 instruction takes a scheduler 64 cycles, so the chain of two-word
// divisions is shared by the seven, and one launch makes both sweeps' tables
// (mdx_set_params with another alpha: 400 us with one thread a bin and a launch a
// sweep, 157 now; with the same tables 15).
// Returns coefficient k = threadIdx.x / PTB, all of them left in sh.
constexpr int PN = 7, PTB = 32;
__device__ __forceinline__ double pt_node(int k) {
  return rint(0.5 * cospi((2 * k + 1) / (2.0 * PN)) * 1073741824.0) / 1073741824.0;
}
__device__ dd pt_coef(int fn, int block, int oct0, double alphad, dd (&sh)[PN][PTB]) {
  __shared__ double x[PN];
  const int b = threadIdx.x % PTB, k = threadIdx.x / PTB, bin = block * PTB + b;
  const double xk = pt_node(k);
  if (b == 0) x[k] = xk;
  dd f = pair_fn(fn, ldexp(1.0, oct0 + bin / 128) * (1.0 + ((bin % 128) + 0.5 + xk) / 128.0),
                 alphad);
  for (int o = 1; o < PN; ++o) {
    sh[k][b] = f;
    __syncthreads();
    const dd below = sh[k > 0 ? k - 1 : 0][b];
    if (k >= o) f = div(f + -below, D(xk - x[k - o]));
    __syncthreads();
  }
  // c_m = c_(m - 1) - c_m x_j, c_0 = f_j - c_0 x_j, j from the last point down
  __shared__ dd df[PN][PTB];
  df[k][b] = f;
  dd c = D(0.0);
  for (int j = PN - 1; j >= 0; --j) {
    sh[k][b] = c;
    __syncthreads();
    c = (k > 0 ? sh[k - 1][b] : df[j][b]) + -(c * D(x[j]));
    __syncthreads();
  }
  sh[k][b] = c;
  __syncthreads();
  return c;
}
__global__ void __launch_bounds__(PTB *PN) k_pair_table(double alphad, PairPoly *__restrict__ tab) {
  __shared__ dd sh[PN][PTB];
  const int bin = blockIdx.x * PTB + threadIdx.x % PTB, fn = blockIdx.y, k = threadIdx.x / PTB;
  const dd c = pt_coef(fn, blockIdx.x, PT_OCT0, alphad, sh);
  PairPoly &p = tab[(size_t)fn * PT_BINS + bin];
  const double v = c.h + c.l;
  if (k == 0) p.c0 = v;
  if (k == 1) p.c1 = v;
  if (k == 2) p.c2 = v;
  if (k == 3) p.c3 = v;
  if (k == 4) p.c4 = (float)v;
  if (k == 5) p.c5 = (float)v;
  if (k == 6) {
    p.c6 = (float)v;
    p.pad = 0.f;
  }
}

// FP32 to FP64 by the bits (a conversion instruction issues on the FP64
// pipe); a zero or denormal comes back as about 2^-127.
__device__ __forceinline__ double f2d_bits(float f) {
  const unsigned b = __float_as_uint(f);
  return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)),
                          (int)(b << 29));
}

// Bin and position of r^2.
struct PtArg {
  int bin;
  double t;
  float tf;
};
__device__ __forceinline__ PtArg pt_arg(double rr) {
  const int hi = __double2hiint(rr), lo = __double2loint(rr);
  PtArg a;
  a.bin = (hi >> 13) - PT_BASE;
  // the 45 bits below the bin's as a number in [1, 2), less 1.5
  const unsigned m = __funnelshift_l((unsigned)lo, (unsigned)hi, 7) & 0xfffffu;
  a.t = __hiloint2double((int)(0x3ff00000u | m), lo << 7) - 1.5;
  a.tf = __uint_as_float(0x3f800000u | (m << 3)) - 1.5f;
  return a;
}
__device__ __forceinline__ double pt_eval(const PairPoly *__restrict__ tab, const PtArg &a) {
  const PairPoly *p = tab + a.bin;
  const double2 c01 = __ldg(reinterpret_cast<const double2 *>(p));
  const double2 c23 = __ldg(reinterpret_cast<const double2 *>(p) + 1);
  const float4 cf = __ldg(reinterpret_cast<const float4 *>(p) + 2);
  const double q = f2d_bits(fmaf(fmaf(cf.z, a.tf, cf.y), a.tf, cf.x));
  return fma(fma(fma(fma(q, a.t, c23.y), a.t, c23.x), a.t, c01.y), a.t, c01.x);
}

// --------------------------------------------------------------- one lane --
// Sums of one lane: PELS, PE, VIR and the diagonal virial, the owner's force,
// and (SPLIT) the energies by type pair: those of one slot are kept and added
// to the block's shared sums when the slot changes (a row's partners are
// mostly of one type: an atomic per pair on a few addresses took two thirds
// of the sweep).  Slot: the type pair, or MDX_NTPP + type for the owner's
// molecule.
struct Acc64 {
  double e[6];
  double fx, fy, fz;
  int slot;
  double see, slj;
};
enum { A_EES = 0, A_ESR, A_VIR, A_VX, A_VY, A_VZ };
__device__ __forceinline__ void split_flush(Acc64 &a, double *sh) {
  if (a.slot < 0) return;
  atomicAdd(&sh[split_ee(a.slot)], a.see);
  if (a.slj != 0.0) atomicAdd(&sh[split_lj(a.slot)], a.slj);
}
__device__ __forceinline__ void split_add(Acc64 &a, int slot, double ee, double lj, double *sh) {
  if (slot != a.slot) {
    split_flush(a, sh);
    a.slot = slot;
    a.see = a.slj = 0.0;
  }
  a.see += ee;
  a.slj += lj;
}

struct Env64 {
  const dbl4 *pos;
  const int4 *ainfo;
  const double *qsite;
  Lj64 lj;
  double *fx, *fy, *fz;
  double bx, by, bz;
  long long hbxb, hbyb, hbzb;  // bits of the half boxes
  CellPbc cp;
  bool rae_on;
};

__device__ __forceinline__ Env64 env64(const dbl4 *pos, const int4 *ainfo, const double *qsite,
                                       const Lj64 &lj, double *fx, double *fy, double *fz,
                                       const CellPbc &cp, bool shrt, const PairConst &pc) {
  // ABS(D) > HBOX tests as integer compares of the magnitudes' bit patterns
  // (the same order as the FP64 compare for finite values; no FP64 issue).
  // LOCALF tests DZ against HBOXL (forces.f:871); FORCES against HBOZL
  return Env64{pos, ainfo, qsite, lj, fx, fy, fz, cp.bx, cp.by, cp.bz,
               __double_as_longlong(0.5 * cp.bx), __double_as_longlong(0.5 * cp.by),
               __double_as_longlong(shrt ? 0.5 * cp.bx : 0.5 * cp.bz), cp,
               pc.lmdee && pc.raex != 0.0};
}

// Minimum image.  CONV: the whole warp is here, and an axis is shifted behind
// a vote (the compiler turns a plain condition into an addition for every pair
// and a select; most warps have no pair across a face).
template <bool SHORT, bool CONV>
__device__ __forceinline__ void image64(const Env64 &v, double &DX, double &DY, double &DZ) {
  constexpr long long MAG = 0x7fffffffffffffffLL;
  auto some = [](bool c) { return CONV ? __any_sync(0xffffffffu, c) : c; };
  if (v.cp.icell == 0) {
    const bool cx = (__double_as_longlong(DX) & MAG) > v.hbxb,
               cz = (__double_as_longlong(DZ) & MAG) > v.hbzb,
               cy = (__double_as_longlong(DY) & MAG) > v.hbyb;
    if (some(cx) && cx) DX = DX - fsign(v.bx, DX);
    if (some(cz) && cz) DZ = DZ - fsign(v.bz, DZ);
    if (some(cy) && cy) DY = DY - fsign(v.by, DY);
  } else {  // hexagonal / truncated octahedron (forces.f:872-906, 1077-1111)
    pbc_cell(DX, DY, DZ, v.cp, SHORT ? v.cp.hbx : v.cp.hbz);
  }
}

// The pair's force onto the partner j and the owner: its register sum (i <
// 0) or atom i (pairs put aside, of any owner).
template <bool ENER>
__device__ __forceinline__ void apply64(const Env64 &v, int i, int j, double F, double DX,
                                        double DY, double DZ, bool vir, Acc64 &a) {
  // the partner's force, formed with the sign (a negation would be another
  // FP64 instruction)
  const double jx = -F * DX, jy = -F * DY, jz = -F * DZ;
  if (ENER && vir) {  // FORCE DX^2 as (FORCE DX) DX
    a.e[A_VX] = fma(-jx, DX, a.e[A_VX]);
    a.e[A_VY] = fma(-jy, DY, a.e[A_VY]);
    a.e[A_VZ] = fma(-jz, DZ, a.e[A_VZ]);
  }
  if (i < 0) {
    a.fx -= jx;
    a.fy -= jy;
    a.fz -= jz;
  } else {
    atomicAdd(&v.fx[i], F * DX);
    atomicAdd(&v.fy[i], F * DY);
    atomicAdd(&v.fz[i], F * DZ);
  }
  atomicAdd(&v.fx[j], jx);
  atomicAdd(&v.fy[j], jy);
  atomicAdd(&v.fz[j], jz);
}

__device__ __forceinline__ double ewald_erfc_poly(double ttt, double exp2a) {
  return ((((MDX_A5 * ttt + MDX_A4) * ttt + MDX_A3) * ttt + MDX_A2) * ttt + MDX_A1) * ttt * exp2a;
}

struct Pair64 {  // force / distance, the vector, whether the pair's virial counts
  double F, DX, DY, DZ;
  bool vir, skip;
};

// One listed pair, the reference's expressions written out (forces.f:868-998 /
// 1071-1198); e: the row entry (sign bit: 1-4 pair).
template <bool SHORT, bool SPLIT, bool ENER>
__device__ __forceinline__ Pair64 pair_general(const Env64 &v, int e, const dbl4 &pi,
                                               const int4 &ai, double qsi, const TypeConst &tc,
                                               const PairConst &pc, double *sh, Acc64 &a) {
  const int ti = ai.x, mi = ai.y, ni = ai.z;
  const bool is14 = SHORT && e < 0;
  const int j = e & 0x7fffffff;
  const dbl4 pj = v.pos[j];
  const int4 aj = v.ainfo[j];
  const int tj = aj.x, nj = aj.z;
  const bool same = aj.y == mi;
  double QIJ, A6, B12;
  bool rae = false;  // RAEX shifts this pair's distance (MDEE)
  const int tix = ni * pc.nnbt + nj;
  if (same) {
    if (is14) {
      QIJ = qsi * v.qsite[j] * pc.coulf * tc.c14el[ti];
      A6 = __ldg(&v.lj.a6_14[tix]) * tc.c14lj[ti];
      B12 = __ldg(&v.lj.b12_14[tix]) * tc.c14lj[ti];
    } else {
      QIJ = qsi * v.qsite[j] * pc.coulf;
      A6 = __ldg(&v.lj.a6lj0[tix]);
      B12 = __ldg(&v.lj.b12lj0[tix]);
    }
  } else {
    QIJ = pi.w * pj.w * pc.coulf;
    A6 = __ldg(&v.lj.a6lj[tix]);
    B12 = __ldg(&v.lj.b12lj[tix]);
    rae = v.rae_on && tc.iee[ti] * tc.iee[tj] == 0;
  }
  double DX = pi.x - pj.x, DY = pi.y - pj.y, DZ = pi.z - pj.z;
  image64<SHORT, false>(v, DX, DY, DZ);
  const double RR = DX * DX + DY * DY + DZ * DZ;
  if (!SHORT && __double_as_longlong(RR) > __double_as_longlong(pc.rc2))
    return Pair64{0.0, DX, DY, DZ, false, true};  // skin mode: listed beyond RCUT
  // one reciprocal square root instead of a square root and a division
  // (within an ulp of DSQRT and 1/R1)
  const double R1I = rsqrt(RR);
  const double R1 = RR * R1I;
  double R1E = R1, R1EI = R1I;
  if (rae) {
    R1E = R1 + pc.raex;
    R1EI = 1. / R1E;
  }
  double EE1, EES, FORCE, slj = 0.0;
  if (is14 || (same && tc.iee[ti] == 0)) {
    if (SHORT) {
      EE1 = QIJ * R1I;
      FORCE = tc.lmove[ti] ? EE1 * (R1I * R1I) : 0.0;
    } else {
      EE1 = QIJ / R1;
      FORCE = tc.lmove[ti] ? EE1 / (R1 * R1) : 0.0;
    }
    EES = EE1;
  } else if (pc.lmnbl) {
    EE1 = QIJ * (1.0 / R1E - 0.5 * pc.rff2 * (R1E * R1E) + pc.rff);
    EES = EE1;
    if (SHORT) {
      FORCE = QIJ * (1. / (R1E * R1E * R1E) + pc.rff2);
      if (ENER) a.e[A_VIR] += QIJ * (1.5 * pc.rff2 / (R1E * R1E) - pc.rff);
    } else {
      FORCE = QIJ * (1.0 / ((R1E * R1E) * R1) + pc.rff2);
      if (ENER) a.e[A_VIR] += QIJ * (1.5 * pc.rff2 * RR - pc.rff);
    }
  } else {
    const double ALPHAR = pc.alphad * R1;
    const double TTT = rcp_nr(1.0 + MDX_B1 * ALPHAR);
    const double EXP2A = exp_neg(ALPHAR * ALPHAR);
    const double ERFCT = ewald_erfc_poly(TTT, EXP2A);
    EE1 = QIJ * R1EI;
    EES = EE1 * ERFCT;
    FORCE = EE1 * (MDX_TOTPI * pc.alphad * EXP2A + ERFCT * R1EI) * R1I;
  }
  if (ENER) a.e[A_EES] += EES;
  if ((__double_as_longlong(B12) << 1) != 0) {  // B12 != 0
    const double R2I = R1EI * R1EI;
    const double R6I = R2I * R2I * R2I;
    double ESR = (A6 + B12 * R6I) * R6I;
    const double FSR = (6.0 * A6 + 12.0 * B12 * R6I) * R6I * R1EI;
    FORCE = FORCE + FSR * R1I;
    if (same) {
      if (SHORT) {
        if (tc.lmove[ti]) {
          slj = ESR;
          if (ENER) a.e[A_VIR] += FSR * R1;
        } else {
          ESR = 0.0;
          FORCE = 0.0;
        }
      } else {
        if (ENER && tc.lmove[ti]) a.e[A_VIR] += FSR * R1;
        slj = ESR;
      }
    } else {
      slj = ESR;
      if (ENER) a.e[A_VIR] += FSR * R1;
    }
    if (ENER) a.e[A_ESR] += ESR;
  }
  if (SPLIT) split_add(a, same ? MDX_NTPP + ti : tc.mdx[ti][tj], EE1, slj, sh);
  return Pair64{FORCE, DX, DY, DZ, SHORT || !same || tc.lmove[ti], false};
}

// The owners' forces out, by three lanes of each group of TPO.
template <int TPO>
__device__ __forceinline__ void owner_out(const Env64 &v, int i, Acc64 &a, bool any) {
  double f[4] = {a.fx, a.fy, a.fz, 0.0};
  const double s = lane_sums<4, TPO>(f);
  const int l = threadIdx.x & (TPO - 1), k = l / (TPO / 4);
  if (any && l % (TPO / 4) == 0 && k < 3)
    atomicAdd(k == 0 ? &v.fx[i] : k == 1 ? &v.fy[i] : &v.fz[i], s);
  a.fx = a.fy = a.fz = 0.0;
}

// Block end: energies and virials, energies by type pair.
template <bool SPLIT, bool ENER>
__device__ __forceinline__ void sweep_out(Acc64 &a, const Dst6 &dst, double *sh, double *split) {
  if (SPLIT) {  // one flush a warp where its lanes agree on the slot
    const int lane = threadIdx.x & 31;
    const int s0 = __reduce_max_sync(0xffffffffu, a.slot);
    if (__all_sync(0xffffffffu, a.slot == s0 || a.slot < 0)) {
      double w[2] = {a.slot < 0 ? 0.0 : a.see, a.slot < 0 ? 0.0 : a.slj};
      const double t = lane_sums<2, 32>(w);
      if (s0 >= 0 && (lane & 15) == 0 && t != 0.0)
        atomicAdd(&sh[lane == 0 ? split_ee(s0) : split_lj(s0)], t);
    } else {
      split_flush(a, sh);
    }
  }
  if (ENER) block_add<6>(a.e, dst);
  if (SPLIT) {
    __syncthreads();
    for (int k = threadIdx.x; k < SPLIT_N; k += blockDim.x)
      if (sh[k] != 0.0) atomicAdd(&split[k], sh[k]);
  }
}

__device__ __forceinline__ void acc_zero(Acc64 &a) {
#pragma unroll
  for (int k = 0; k < 6; ++k) a.e[k] = 0.0;
  a.fx = a.fy = a.fz = 0.0;
  a.slot = -1;
  a.see = a.slj = 0.0;
}

// --------------------------------------------------------------- sweeps ---
template <bool SHORT, bool SPLIT, bool ENER>
__global__ void __launch_bounds__(256) k_pair64(
    int n, const dbl4 *__restrict__ pos, const int4 *__restrict__ ainfo,
    const double *__restrict__ qsite, const int *__restrict__ cnt, const int *__restrict__ idx,
    int cap, Lj64 lj, TypeConst tc, PairConst pc, CellPbc cp, double *__restrict__ fx,
    double *__restrict__ fy, double *__restrict__ fz, Dst6 dst, double *__restrict__ split) {
  __shared__ double s_split[SPLIT ? SPLIT_N : 1];
  if (SPLIT) {
    for (int k = threadIdx.x; k < SPLIT_N; k += blockDim.x) s_split[k] = 0.0;
    __syncthreads();
  }
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const Env64 v = env64(pos, ainfo, qsite, lj, fx, fy, fz, cp, SHORT, pc);
  Acc64 a;
  acc_zero(a);
  for (int i = blockIdx.x * nw + (threadIdx.x >> 5); i < n; i += gridDim.x * nw) {
    const dbl4 pi = pos[i];
    const int4 ai = ainfo[i];
    const double qsi = qsite[i];
    const int c = cnt[i];
    const int *row = idx + (size_t)i * cap;
    for (int k = lane; k < c; k += 32) {
      const int e = row[k];
      const Pair64 p = pair_general<SHORT, SPLIT, ENER>(v, e, pi, ai, qsi, tc, pc, s_split, a);
      if (!p.skip) apply64<ENER>(v, -1, e & 0x7fffffff, p.F, p.DX, p.DY, p.DZ, p.vir, a);
    }
    __syncwarp();
    owner_out<32>(v, i, a, c > 0);
  }
  sweep_out<SPLIT, ENER>(a, dst, s_split, split);
}

constexpr int PT_WARPS = 8;
struct LjQueue {  // pairs put aside for their LJ term, per warp
  double x[64], y[64], z[64], rr[64], f[64];
  int i[64], j[64], tix[64];
};

// Ewald sweep from the tables.  eemask: bit t set for IEE(t) = 0.
template <bool SHORT, bool SPLIT, bool ENER, int TPO>
__global__ void __launch_bounds__(32 * PT_WARPS, 2) k_pair64t(
    int n, const dbl4 *__restrict__ pos, const int4 *__restrict__ ainfo,
    const double *__restrict__ qsite, const int *__restrict__ cnt, const int *__restrict__ idx,
    int cap, Lj64 lj, TypeConst tc, PairConst pc, CellPbc cp, unsigned eemask,
    const PairPoly *__restrict__ tab, double *__restrict__ fx, double *__restrict__ fy,
    double *__restrict__ fz, Dst6 dst, double *__restrict__ split) {
  __shared__ double s_split[SPLIT ? SPLIT_N : 1];
  __shared__ LjQueue s_q[PT_WARPS];
  __shared__ int2 s_slow[PT_WARPS][64];
  if (SPLIT) {
    for (int k = threadIdx.x; k < SPLIT_N; k += blockDim.x) s_split[k] = 0.0;
    __syncthreads();
  }
  constexpr int OPW = 32 / TPO;  // owners of a warp at a time
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  LjQueue &q = s_q[w];
  int2 *slow = s_slow[w];
  const Env64 v = env64(pos, ainfo, qsite, lj, fx, fy, fz, cp, SHORT, pc);
  const unsigned eem = v.rae_on ? eemask : 0u;
  const long long rc2b = __double_as_longlong(pc.rc2);
  Acc64 a;
  acc_zero(a);
  int nq = 0, nslow = 0;
  // the last m (<= 32) pairs of the LJ queue: their LJ terms, then forces
  auto lj_batch = [&](int m) {
    __syncwarp();
    if (lane < m) {
      const int e = nq - m + lane;
      const double rr = q.rr[e];
      const int tix = q.tix[e], i = q.i[e], j = q.j[e];
      const double R2I = pt_eval(tab + PT_R2I * PT_BINS, pt_arg(rr));
      const double A6 = __ldg(&lj.a6lj[tix]), B12 = __ldg(&lj.b12lj[tix]);
      const double R6I = R2I * R2I * R2I, T12 = B12 * R6I;
      const double G = fma(2.0, T12, A6) * R6I;  // FSR R1 / 6
      const double F = fma(6.0 * R2I, G, q.f[e]);
      if (ENER || SPLIT) {
        const double ESR = (A6 + T12) * R6I;
        if (ENER) {
          a.e[A_ESR] += ESR;
          a.e[A_VIR] = fma(6.0, G, a.e[A_VIR]);
        }
        if (SPLIT) split_add(a, tc.mdx[ainfo[i].x][ainfo[j].x], 0.0, ESR, s_split);
      }
      apply64<ENER>(v, i, j, F, q.x[e], q.y[e], q.z[e], true, a);
    }
    nq -= m;
    __syncwarp();
  };
  auto slow_batch = [&](int m) {
    __syncwarp();
    if (lane < m) {
      const int2 s = slow[nslow - m + lane];
      const Pair64 p = pair_general<SHORT, SPLIT, ENER>(v, s.y, pos[s.x], ainfo[s.x], qsite[s.x],
                                                        tc, pc, s_split, a);
      if (!p.skip) apply64<ENER>(v, s.x, s.y & 0x7fffffff, p.F, p.DX, p.DY, p.DZ, p.vir, a);
    }
    nslow -= m;
    __syncwarp();
  };
  for (int i0 = (blockIdx.x * PT_WARPS + w) * OPW; i0 < n; i0 += gridDim.x * PT_WARPS * OPW) {
    const int i = i0 + lane / TPO;
    const bool own = i < n;
    const dbl4 pi = pos[own ? i : 0];
    const int4 ai = ainfo[own ? i : 0];
    const double qic = pi.w * pc.coulf;
    const int c = own ? cnt[i] : 0;
    const int cmax = __reduce_max_sync(0xffffffffu, c);
    const int *row = idx + (size_t)(own ? i : 0) * cap;
    const double *b12row = lj.b12lj + ai.z * pc.nnbt;
    const bool eei = (eem >> ai.x) & 1u;
    for (int k = lane & (TPO - 1); k - (lane & (TPO - 1)) < cmax; k += TPO) {
      bool act = k < c;
      const int e = act ? row[k] : 0;
      const int j = e & 0x7fffffff;
      const dbl4 pj = pos[j];
      const int4 aj = ainfo[j];
      const bool other = (SHORT && e < 0) || aj.y == ai.y || eei || ((eem >> aj.x) & 1u);
      double DX = pi.x - pj.x, DY = pi.y - pj.y, DZ = pi.z - pj.z;
      image64<SHORT, true>(v, DX, DY, DZ);
      const double RR = DX * DX + DY * DY + DZ * DZ;
      if (!SHORT && __double_as_longlong(RR) > rc2b) act = false;  // skin mode
      PtArg p = pt_arg(RR);
      const bool sl = act && (other || (unsigned)p.bin >= (unsigned)PT_BINS);
      const bool fast = act && !sl;
      if (!fast) p.bin = 0;
      const unsigned ms = __ballot_sync(0xffffffffu, sl);
      if (ms) {
        if (sl) slow[nslow + __popc(ms & below)] = make_int2(i, e);
        nslow += __popc(ms);
        if (nslow >= 32) slow_batch(32);
      }
      const double qq = fast ? qic * pj.w : 0.0;
      const double F = qq * pt_eval(tab + PT_FORCE * PT_BINS, p);
      if (ENER) a.e[A_EES] = fma(qq, pt_eval(tab + PT_ENER * PT_BINS, p), a.e[A_EES]);
      if (SPLIT && fast)
        split_add(a, tc.mdx[ai.x][aj.x], qq * pt_eval(tab + PT_R1I * PT_BINS, p), 0.0, s_split);
      const bool lb = fast && (__double_as_longlong(__ldg(&b12row[aj.z])) << 1) != 0;  // B12 != 0
      if (fast && !lb) apply64<ENER>(v, -1, j, F, DX, DY, DZ, true, a);
      const unsigned ml = __ballot_sync(0xffffffffu, lb);
      if (ml) {
        if (lb) {
          const int s = nq + __popc(ml & below);
          q.x[s] = DX;
          q.y[s] = DY;
          q.z[s] = DZ;
          q.rr[s] = RR;
          q.f[s] = F;
          q.i[s] = i;
          q.j[s] = j;
          q.tix[s] = ai.z * pc.nnbt + aj.z;
        }
        nq += __popc(ml);
        if (nq >= 32) lj_batch(32);
      }
    }
    owner_out<TPO>(v, i, a, c > 0);
  }
  if (nq) lj_batch(nq);
  if (nslow) slow_batch(nslow);
  sweep_out<SPLIT, ENER>(a, dst, s_split, split);
}

// ------------------------------------------------- fixed-point sweeps ----
// The same sweep in 64-bit integers (rectangular cell): a multiplication of
// two 64-bit numbers is three 32 x 32 + 64 bit multiply-adds, and GB300 issues
// those 32 times as often as an FP64 instruction, so a Coulomb pair's 19 - 27
// FP64 instructions become about 200 integer ones in a quarter of the time.
// Positions are integers of 2^-px_bits A (ipos, written with the positions),
// their differences are exact, and
//   d   = difference, minimum image, shifted so that 2^rho A is 2^62
//   r2  = the upper 64 bits of d.d
//   t   = position in the bin of r2, 2^-63 units; bins as in PairPoly
//   F   = polynomial in t, 62 bits at the table's first r^2
//   G   = F q_i q_j (62 bits), fx = upper 64 bits of G dx, and so on.
// A product keeps all but its last bit, so a pair's force is good to 2^-54 of
// the force at the table's start; it is added as an integer, whatever the
// order.  The LJ term comes from a tabulated 1 / r^2 in 9 FP64 instructions
// and joins G.  Everything else goes to the FP64 expressions as before, and
// so do atoms and pairs out of the numbers' range.  The unit is one for a sweep, so
// a distant pair's force, alone, has fewer significant bits than an FP64 number;
// an atom's slow force does not show it, in a gas either, because the rounding of
// its reciprocal part is larger (two waters 10 A apart: 2.5e-13 of the force,
// written out 2.3e-13).
struct __align__(16) PxPoly {
  long long c0, c1, c2;  // c0, 2 c1, 4 c2
  int c3, sh;            // 8 c3 in units of 2^(32 - sh)
  float c4, c5, c6, pad; // 8 times, units of c3
};
struct Px {
  int s, base, nbin, rng;  // left shift of d, first bin's index, bins, range of d (upper word)
  long long lx, ly, lz, hx, hy, hz;  // box and half box (LOCALF tests DZ against HBOXL)
  unsigned long long rc2;
  double uE, uR, uV, uG, iG;  // units of energy, 1 / r, virial; of G, and 1 / that
  double du;                  // unit of d (A)
  int s2;                     // 1 / r^2 is 2^-s2 times its table's value
  const PxPoly *tab;          // PT_NFN x nbin
};

// v = h 2^32 + l, both signed (|v| < 2^63 - 2^31)
struct I2 {
  int h, l;
};
__device__ __forceinline__ I2 split2(long long v) {
  return I2{(int)((v + 0x80000000LL) >> 32), (int)v};
}
__device__ __forceinline__ long long cross2(I2 a, I2 b) {
  return (long long)a.h * b.l + (long long)a.l * b.h;
}
// upper 64 bits of a b, to the nearest (|a|, |b| <= 2^62)
__device__ __forceinline__ long long mulhi2(I2 a, I2 b) {
  return (long long)a.h * b.h + ((cross2(a, b) + 0x80000000LL) >> 32);
}
// a a / 2^62 from its crossed product c = h l + 2^28, to the nearest
__device__ __forceinline__ long long sq_cross(I2 a) {
  return (long long)a.h * a.l + 0x10000000LL;
}
__device__ __forceinline__ long long sq4(I2 a, long long c) {
  return ((long long)a.h * a.h << 2) + (c >> 29);
}
// A lane's sum of products a b / 2^64 (|a b| < 2^122), kept to 24 bits below that
// unit: the high products and the crossed ones apart.  Energies and virials are sums
// of terms that nearly cancel and one unit holds for the closest pair and the most
// distant one, so a pair's term rounded to the unit shows in the sum: 1,500 ions,
// long rows from 4.5 to 12 A, in 2^-53 of the root of the terms' squares, the virial
// 152 off rounded pair by pair, 10 so, 5 written out in FP64; the energy from 6.6 A on
// 41, 6, 3.  Costs 0.04 to 0.06 ms of the long sweep at 98,304 atoms.
struct Sum2 {
  long long h = 0, c = 0;
  __device__ __forceinline__ void add(I2 a, I2 b) {
    h += (long long)a.h * b.h;
    c += cross2(a, b) >> 8;
  }
  // whole units out, to the nearest (a floor would be the same way in every row);
  // the rest stays for the next row
  __device__ __forceinline__ double take() {
    const long long k = (c + 0x800000LL) >> 24, u = h + k;
    c -= k << 24;
    h = 0;
    return (double)u;
  }
};
struct PxArg {
  int bin;
  I2 t;
  float tf;
};
__device__ __forceinline__ PxArg px_arg(const Px &x, unsigned long long r2) {
  const int lz = __clz((int)(r2 >> 32));
  const unsigned long long m = r2 << (lz & 31);
  const unsigned mh = (unsigned)(m >> 32);
  PxArg a;
  a.bin = x.base - 128 * lz + (int)(mh >> 24);
  a.t = split2((long long)((m << 7) & 0x7fffffffffffffffull) - 0x4000000000000000LL);
  a.tf = __uint_as_float(0x3f800000u | ((mh & 0xffffffu) >> 1)) - 1.5f;
  return a;
}
__device__ __forceinline__ long long px_eval(const PxPoly *tab, const PxArg &a) {
  const PxPoly *p = tab + a.bin;
  const longlong2 c01 = *reinterpret_cast<const longlong2 *>(p);
  const int4 c23 = *(reinterpret_cast<const int4 *>(p) + 1);
  const float4 cf = *(reinterpret_cast<const float4 *>(p) + 2);
  const int s3 = c23.z + __float2int_rn(a.tf * fmaf(fmaf(cf.z, a.tf, cf.y), a.tf, cf.x));
  const long long c2 = (long long)(((unsigned long long)(unsigned)c23.y << 32) | (unsigned)c23.x);
  const long long s2 = c2 + (((long long)s3 * a.t.h) >> c23.w);
  const long long s1 = c01.y + mulhi2(split2(s2), a.t);
  return c01.x + mulhi2(split2(s1), a.t);
}

// Tables of every pair that a long sweep keeps in shared memory: F, and E with
// the energies.  32 lanes ask for 32 bins, in L1 a tag each: with the neighbours'
// records and the atomics that kept L1 88 % busy.  A third table (1 / r, force
// calls) would leave L1 too little for the records.  98,304 atoms, long rows with
// energies 1.24 ms from L1, 1.09 from shared memory; with energies by type pair
// 1.50, 1.39, with all three 2.13 (Sum2, in both since, adds 0.05).  Only where a
// warp has several owners: the copy, and the SMs' change to another split of their
// memory between two kernels of a small system, cost more (3,000 atoms, 20 steps:
// 6.64 ms without, 7.02 with; the short rows gain 4 % at 98,304 atoms and nothing at
// 21,003).
constexpr int px_tables(bool ener) { return ener ? 2 : 1; }

struct PxQueue {  // pairs put aside for their LJ term, per warp
  long long x[64], y[64], z[64], g[64];
  unsigned long long r2[64];
  int i[64], j[64], tix[64];
};

// TABSH: the tables of every pair in shared memory
template <bool SHORT, bool SPLIT, bool ENER, int TPO, bool TABSH>
__global__ void __launch_bounds__(32 * PT_WARPS, 2) k_pair64x(
    int n, const longlong4_32a *__restrict__ ipos, const dbl4 *__restrict__ pos,
    const int4 *__restrict__ ainfo, const double *__restrict__ qsite,
    const int *__restrict__ cnt, const int *__restrict__ idx, int cap, Lj64 lj, TypeConst tc,
    PairConst pc, CellPbc cp, unsigned eemask, Px px, double *__restrict__ fx,
    double *__restrict__ fy, double *__restrict__ fz, unsigned long long *__restrict__ ff,
    Dst6 dst, double *__restrict__ split) {
  extern __shared__ __align__(16) unsigned char s_tab[];
  __shared__ double s_split[SPLIT ? SPLIT_N : 1];
  __shared__ PxQueue s_q[PT_WARPS];
  __shared__ int2 s_slow[PT_WARPS][64];
  if (TABSH) {
    const int4 *src = reinterpret_cast<const int4 *>(px.tab);
    int4 *dst = reinterpret_cast<int4 *>(s_tab);
    for (int k = threadIdx.x; k < px_tables(ENER) * px.nbin * 3; k += blockDim.x)
      dst[k] = __ldg(src + k);
    __syncthreads();
  }
  const PxPoly *const tab = TABSH ? reinterpret_cast<const PxPoly *>(s_tab) : px.tab;
  if (SPLIT) {
    for (int k = threadIdx.x; k < SPLIT_N; k += blockDim.x) s_split[k] = 0.0;
    __syncthreads();
  }
  constexpr int OPW = 32 / TPO;  // owners of a warp at a time
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  PxQueue &q = s_q[w];
  int2 *slow = s_slow[w];
  const Env64 v = env64(pos, ainfo, qsite, lj, fx, fy, fz, cp, SHORT, pc);
  const unsigned eem = v.rae_on ? eemask : 0u;
  Acc64 a;
  acc_zero(a);
  Sum2 ie, ivx, ivy, ivz;  // this owner's row
  int nq = 0, nslow = 0;
  auto add = [&](int i, long long x, long long y, long long z) {
    atomicAdd(&ff[i], (unsigned long long)x);
    atomicAdd(&ff[(size_t)n + i], (unsigned long long)y);
    atomicAdd(&ff[2 * (size_t)n + i], (unsigned long long)z);
  };
  // g: to the nearest.  Forces take it floored: half a unit along each of an atom's
  // pairs cancels, in a virial it adds up.
  auto virial = [&](I2 g, I2 dx, I2 dy, I2 dz, long long cx, long long cy, long long cz) {
    ivx.add(g, split2(sq4(dx, cx)));
    ivy.add(g, split2(sq4(dy, cy)));
    ivz.add(g, split2(sq4(dz, cz)));
  };
  // the last m (<= 32) pairs of the LJ queue: their LJ terms, then forces
  auto lj_batch = [&](int m) {
    __syncwarp();
    if (lane < m) {
      const int e = nq - m + lane;
      const int tix = ENER ? q.tix[e] >> 1 : q.tix[e], i = q.i[e], j = q.j[e];
      const double r = (double)px_eval(px.tab + PT_R2I * px.nbin, px_arg(px, q.r2[e]));
      // times 2^-s2 by the exponent
      const double R2I =
          __hiloint2double(__double2hiint(r) - (px.s2 << 20), __double2loint(r));
      const double A6 = __ldg(&lj.a6lj[tix]), B12 = __ldg(&lj.b12lj[tix]);
      const double R6I = R2I * R2I * R2I, T12 = B12 * R6I;
      const double G = fma(2.0, T12, A6) * R6I;  // FSR R1 / 6
      const double FL = R2I * px.iG * G;         // in units of G
      if (ENER || SPLIT) {
        const double ESR = (A6 + T12) * R6I;
        if (ENER) {
          a.e[A_ESR] += ESR;
          a.e[A_VIR] = fma(6.0, G, a.e[A_VIR]);
        }
        if (SPLIT) split_add(a, tc.mdx[ainfo[i].x][ainfo[j].x], 0.0, ESR, s_split);
      }
      // 2^60: the sums of forces stay far below 2^63
      if ((__double_as_longlong(FL) & 0x7fffffffffffffffLL) < 0x43b0000000000000LL) {
        const long long G64 = q.g[e] + __double2ll_rn(FL);
        const I2 g = split2(G64);
        const I2 dx = split2(q.x[e]), dy = split2(q.y[e]), dz = split2(q.z[e]);
        const long long gx = mulhi2(g, dx), gy = mulhi2(g, dy), gz = mulhi2(g, dz);
        if (ENER)
          virial(split2(G64 + (q.tix[e] & 1)), dx, dy, dz, sq_cross(dx), sq_cross(dy),
                 sq_cross(dz));
        add(i, gx, gy, gz);
        add(j, -gx, -gy, -gz);
      } else {
        apply64<ENER>(v, i, j, ((double)q.g[e] + FL) * px.uG, (double)q.x[e] * px.du,
                      (double)q.y[e] * px.du, (double)q.z[e] * px.du, true, a);
      }
    }
    nq -= m;
    __syncwarp();
  };
  auto slow_batch = [&](int m) {
    __syncwarp();
    if (lane < m) {
      const int2 s = slow[nslow - m + lane];
      const Pair64 p = pair_general<SHORT, SPLIT, ENER>(v, s.y, pos[s.x], ainfo[s.x], qsite[s.x],
                                                        tc, pc, s_split, a);
      if (!p.skip) apply64<ENER>(v, s.x, s.y & 0x7fffffff, p.F, p.DX, p.DY, p.DZ, p.vir, a);
    }
    nslow -= m;
    __syncwarp();
  };
  auto image = [&](long long &d, long long h, long long l) {
    const bool c = (unsigned long long)(d + h) > 2ull * (unsigned long long)h;
    if (__any_sync(0xffffffffu, c) && c) d -= d < 0 ? -l : l;
  };
  for (int i0 = (blockIdx.x * PT_WARPS + w) * OPW; i0 < n; i0 += gridDim.x * PT_WARPS * OPW) {
    const int i = i0 + lane / TPO;
    const bool own = i < n;
    const longlong4_32a ip = ipos[own ? i : 0];
    const int4 ai = ainfo[own ? i : 0];
    const I2 qi = split2(ip.w);
    const int c = own ? cnt[i] : 0;
    const int cmax = __reduce_max_sync(0xffffffffu, c);
    const int *row = idx + (size_t)(own ? i : 0) * cap;
    const double *b12row = lj.b12lj + ai.z * pc.nnbt;
    const bool eei = ((eem >> ai.x) & 1u) || ip.w == IPOS_BAD;
    long long ax = 0, ay = 0, az = 0;
    for (int k = lane & (TPO - 1); k - (lane & (TPO - 1)) < cmax; k += TPO) {
      bool act = k < c;
      const int e = act ? row[k] : 0;
      const int j = e & 0x7fffffff;
      const longlong4_32a jp = ipos[j];
      const int4 aj = ainfo[j];
      long long DX = ip.x - jp.x, DY = ip.y - jp.y, DZ = ip.z - jp.z;
      image(DX, px.hx, px.lx);
      image(DY, px.hy, px.ly);
      image(DZ, px.hz, px.lz);
      const bool in = (unsigned)((int)(DX >> 32) + px.rng) < 2u * (unsigned)px.rng &&
                      (unsigned)((int)(DY >> 32) + px.rng) < 2u * (unsigned)px.rng &&
                      (unsigned)((int)(DZ >> 32) + px.rng) < 2u * (unsigned)px.rng;
      DX <<= px.s;
      DY <<= px.s;
      DZ <<= px.s;
      const I2 dx = split2(DX), dy = split2(DY), dz = split2(DZ);
      const long long cx = sq_cross(dx), cy = sq_cross(dy), cz = sq_cross(dz);
      const unsigned long long r2 =
          (unsigned long long)((long long)dx.h * dx.h + (long long)dy.h * dy.h +
                               (long long)dz.h * dz.h + ((cx + cy + cz + 0x10000000LL) >> 31));
      PxArg p = px_arg(px, r2);
      const bool other = (SHORT && e < 0) || aj.y == ai.y || eei || ((eem >> aj.x) & 1u) ||
                         jp.w == IPOS_BAD || !in || (unsigned)p.bin >= (unsigned)px.nbin;
      if (!SHORT && !other && r2 > px.rc2) act = false;  // skin mode
      const bool sl = act && other, fast = act && !other;
      if (!fast) p.bin = 0;
      const unsigned ms = __ballot_sync(0xffffffffu, sl);
      if (ms) {
        if (sl) slow[nslow + __popc(ms & below)] = make_int2(i, e);
        nslow += __popc(ms);
        if (nslow >= 32) slow_batch(32);
      }
      const I2 qq = split2(mulhi2(qi, split2(jp.w)));
      const I2 F = split2(px_eval(tab + PT_FORCE * px.nbin, p));
      const long long cg = cross2(F, qq);
      const long long g = (((long long)F.h * qq.h) << 4) + (cg >> 28);
      const int up = (int)(cg >> 27) & 1;  // g + up: to the nearest
      if (ENER) {
        const I2 E = split2(px_eval(tab + PT_ENER * px.nbin, p));
        if (fast) ie.add(E, qq);
      }
      if (SPLIT && fast)
        split_add(a, tc.mdx[ai.x][aj.x],
                  (double)mulhi2(split2(px_eval(px.tab + PT_R1I * px.nbin, p)), qq) * px.uR, 0.0,
                  s_split);
      const bool lb = fast && (__double_as_longlong(__ldg(&b12row[aj.z])) << 1) != 0;  // B12 != 0
      if (fast && !lb) {
        const I2 G = split2(g);
        const long long gx = mulhi2(G, dx), gy = mulhi2(G, dy), gz = mulhi2(G, dz);
        if (ENER) virial(split2(g + up), dx, dy, dz, cx, cy, cz);
        ax += gx;
        ay += gy;
        az += gz;
        add(j, -gx, -gy, -gz);
      }
      const unsigned ml = __ballot_sync(0xffffffffu, lb);
      if (ml) {
        if (lb) {
          const int s = nq + __popc(ml & below);
          q.x[s] = DX;
          q.y[s] = DY;
          q.z[s] = DZ;
          q.r2[s] = r2;
          q.g[s] = g;
          q.i[s] = i;
          q.j[s] = j;
          const int tix = ai.z * pc.nnbt + aj.z;
          q.tix[s] = ENER ? 2 * tix + up : tix;
        }
        nq += __popc(ml);
        if (nq >= 32) lj_batch(32);
      }
    }
#pragma unroll
    for (int o = 1; o < TPO; o <<= 1) {
      ax += __shfl_xor_sync(0xffffffffu, ax, o);
      ay += __shfl_xor_sync(0xffffffffu, ay, o);
      az += __shfl_xor_sync(0xffffffffu, az, o);
    }
    if (c > 0 && (lane & (TPO - 1)) < 3) {
      const int k = lane & (TPO - 1);
      atomicAdd(&ff[(size_t)k * n + i], (unsigned long long)(k == 0 ? ax : k == 1 ? ay : az));
    }
    if (ENER) {  // a row's sums stay below 2^63
      a.e[A_EES] = fma(ie.take(), px.uE, a.e[A_EES]);
      a.e[A_VX] = fma(ivx.take(), px.uV, a.e[A_VX]);
      a.e[A_VY] = fma(ivy.take(), px.uV, a.e[A_VY]);
      a.e[A_VZ] = fma(ivz.take(), px.uV, a.e[A_VZ]);
    }
  }
  if (nq) lj_batch(nq);
  if (nslow) slow_batch(nslow);
  if (ENER) {
    a.e[A_VX] = fma(ivx.take(), px.uV, a.e[A_VX]);
    a.e[A_VY] = fma(ivy.take(), px.uV, a.e[A_VY]);
    a.e[A_VZ] = fma(ivz.take(), px.uV, a.e[A_VZ]);
  }
  sweep_out<SPLIT, ENER>(a, dst, s_split, split);
}

__device__ __forceinline__ long long dd2ll(dd v, int s) {  // v 2^s to the nearest
  const double h = ldexp(v.h, s), r = rint(h);
  return (long long)r + __double2ll_rn((h - r) + ldexp(v.l, s));
}
// Block (bins of one sweep, function): the long rows' bins follow the short rows'.
__global__ void __launch_bounds__(PTB *PN) k_px_table(PxTables x, PxPoly *__restrict__ tab) {
  __shared__ dd sh[PN][PTB];
  const int nb0 = x.nbin[0] / PTB, w = (int)blockIdx.x >= nb0, block = blockIdx.x - w * nb0;
  const int b = threadIdx.x % PTB, k = threadIdx.x / PTB, fn = blockIdx.y, s = x.s[w][fn];
  const dd c = pt_coef(fn, block, x.oct0[w], x.alphad, sh);
  PxPoly &p = tab[(w ? PT_NFN * x.nbin[0] : 0) + fn * x.nbin[w] + block * PTB + b];
  const double c3 = ldexp(sh[3][b].h, s + 3);
  const int K = min(32, max(0, ilogb(fmax(fabs(c3), 1.0)) + 1 - 30));
  if (k == 0) p.c0 = dd2ll(c, s);
  if (k == 1) p.c1 = dd2ll(c, s + 1);
  if (k == 2) p.c2 = dd2ll(c, s + 2);
  if (k == 3) {
    p.c3 = (int)dd2ll(c, s + 3 - K);
    p.sh = 32 - K;
  }
  const float v = (float)ldexp(c.h, s + 3 - K);
  if (k == 4) p.c4 = v;
  if (k == 5) p.c5 = v;
  if (k == 6) {
    p.c6 = v;
    p.pad = 0.f;
  }
}

__global__ void k_ipos(int n, const dbl4 *__restrict__ pos, IPosOut o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) ipos_store(o, i, pos[i]);
}

// The sweep's constants for the current box (units of ipos as last written).
Px px_args(const mdx_ctx *ctx, bool shrt) {
  Px x{};
  if (!ctx->px_on) return x;
  const int w = shrt ? 0 : 1, rho = ctx->px_rho[w], B = ctx->px_bits;
  const int *s = ctx->px.s[w];
  auto u = [&](double a) { return std::llrint(std::ldexp(a, B)); };
  x.s = 62 - rho - B;
  x.rng = 1 << (B + rho - 32);
  x.nbin = ctx->px.nbin[w];
  // octave of r2: 2 rho + 3 - lz; the upper byte of the mantissa is 128 ..
  x.base = 128 * (2 * rho + 3 - ctx->px.oct0[w]) - 128;
  x.lx = u(ctx->boxl);
  x.ly = u(ctx->boyl);
  x.lz = u(ctx->bozl);
  x.hx = u(0.5 * ctx->boxl);
  x.hy = u(0.5 * ctx->boyl);
  x.hz = shrt ? x.hx : u(0.5 * ctx->bozl);
  x.rc2 = px_cut2(ctx->pc.rc2, rho);
  const int q2 = 2 * ctx->px_eq;
  const double cf = ctx->p.coulf;
  x.uG = std::ldexp(cf, q2 - s[PT_FORCE]);
  x.iG = 6.0 * std::ldexp(1.0 / cf, s[PT_FORCE] - q2);  // 6: FSR R1 / 6
  x.du = std::ldexp(1.0, rho - 62);
  x.uV = std::ldexp(x.uG, 2 * (rho - 62) + 126);
  x.uE = std::ldexp(cf, q2 + 4 - s[PT_ENER]);
  x.uR = std::ldexp(cf, q2 + 4 - s[PT_R1I]);
  x.s2 = s[PT_R2I];
  x.tab = reinterpret_cast<const PxPoly *>(ctx->dv.px_tab) + (shrt ? 0 : PT_NFN * ctx->px.nbin[0]);
  return x;
}

}  // namespace

// Positions beyond 2^61 units are out of range: twice the box to either side.
// At most 2^-54 A (the sweeps' shifts stay positive), which is below the last
// bit of an FP64 coordinate beyond 0.25 A.
IPosOut ipos_out(mdx_ctx *ctx) {
  if (!ctx->px_on) return IPosOut{nullptr, 0.0, 0.0};
  const double l = std::max({ctx->boxl, ctx->boyl, ctx->bozl});
  ctx->px_bits = std::min(54, 61 - (std::ilogb(2.0 * l) + 1));
  return IPosOut{reinterpret_cast<longlong2 *>(ctx->dv.ipos), std::ldexp(1.0, ctx->px_bits),
                 std::ldexp(1.0, 62 - ctx->px_eq)};
}
int launch_ipos(mdx_ctx *ctx) {
  if (!ctx->px_on) return MDX_OK;
  MDX_TIMER(ctx, MDX_T_OTHER);
  const DevData &d = ctx->dv;
  k_ipos<<<(d.n + 255) / 256, 256, 0, ctx->stream>>>(d.n, d.pos, ipos_out(ctx));
  MDX_LAUNCHED(ctx);
  return MDX_OK;
}
// force = coulf F q q d: G has 2^(s - 2 eq), d 2^(62 - rho), their product loses 64 bits
double px_force_unit(const mdx_ctx *ctx, int which) {
  if (!ctx->px_on) return 0.0;
  const int w = which == 1 ? 0 : 1;
  return std::ldexp(ctx->p.coulf, 2 * ctx->px_eq - ctx->px.s[w][PT_FORCE] + ctx->px_rho[w] + 2);
}

// The Ewald tables of the sweeps for the current parameters (FP64 path;
// set_params).  Integers where the cell is rectangular and the cut-offs and
// charges fit them: the short rows' table from r^2 = 2 A^2, the long rows'
// from the octave below (0.8 RSHORT)^2; pairs closer by go to the FP64
// expressions.  A pair's force is good to 2^-54 of the force at its table's
// start, so the short rows end at 6.6 A: a screened force is down by 2^6
// there, and the error of an atom's force stays that of its nearest
// neighbours in FP64.
int pair64_setup(mdx_ctx *ctx) {
  DevData &d = ctx->dv;
  ctx->px_on = false;
  if (ctx->mixed() || ctx->p.alphad <= 0.0 || ctx->p.lmnbl) return MDX_OK;
  double qmax = 0.0;
  for (double q : ctx->h_q) qmax = std::max(qmax, std::fabs(q));
  for (double q : ctx->h_charge) qmax = std::max(qmax, std::fabs(q));  // MDEE scales these
  const double rl = ctx->p.rcut + ctx->p.rskin;
  auto rho = [](double r) { return std::max(2, std::ilogb(r) + 1); };
  if (ctx->p.icell == 0 && ctx->p.coulf > 0.0 && qmax > 0.0 && qmax <= 4.0 && rl < 31.0 &&
      ctx->p.rshort > 2.0 && 1.2 * ctx->p.rshort < 8.0) {
    ctx->px_eq = std::ilogb(qmax) + (std::ldexp(1.0, std::ilogb(qmax)) < qmax ? 1 : 0);
    ctx->px_rho[0] = rho(1.2 * ctx->p.rshort);
    ctx->px_rho[1] = std::max(rho(rl), ctx->px_rho[0]);  // RCUT may lie below RSHORT
    PxTables x{};
    x.alphad = ctx->p.alphad;
    x.oct0[0] = 1;
    x.oct0[1] = std::max(1, std::ilogb(0.64 * ctx->p.rshort * ctx->p.rshort));
    for (int w = 0; w < 2; ++w) {
      x.nbin[w] = 128 * (2 * ctx->px_rho[w] - x.oct0[w]);
      // binary scale of each function: below 2^62 at the first r^2.  Long
      // rows, forces: 2^60, so that some hundred pairs of one sign still fit
      const double x2 = std::ldexp(1.0, x.oct0[w]), r = std::sqrt(x2);
      const double ar = ctx->p.alphad * r, t = 1.0 / (1.0 + MDX_B1 * ar), e = std::exp(-ar * ar);
      const double er =
          ((((MDX_A5 * t + MDX_A4) * t + MDX_A3) * t + MDX_A2) * t + MDX_A1) * t * e / r;
      const double f0[PT_NFN] = {(MDX_TOTPI * ctx->p.alphad * e + er) / x2, er, 1.0 / r, 1.0 / x2};
      for (int f = 0; f < PT_NFN; ++f)
        x.s[w][f] = (w && f == PT_FORCE ? 60 : 62) - 1 - std::ilogb(1.0001 * f0[f]);
    }
    // Formed again only when something they depend on has changed: a caller that
    // sets thermostats or time steps between segments keeps them.
    if (!d.px_tab) MDX_CUDA(ctx_alloc(ctx, &d.px_tab, sizeof(PxPoly) * PT_NFN * 2 * 128 * 10));
    if (std::memcmp(&ctx->px, &x, sizeof x) != 0) {
      k_px_table<<<dim3((x.nbin[0] + x.nbin[1]) / PTB, PT_NFN), PTB * PN, 0, ctx->stream>>>(
          x, reinterpret_cast<PxPoly *>(d.px_tab));
      MDX_LAUNCHED(ctx);
      ctx->px = x;
    }
    ctx->px_on = true;
    return MDX_OK;
  }
  if (d.pair_tab && ctx->pair_tab_alpha == ctx->p.alphad) return MDX_OK;
  if (!d.pair_tab)
    MDX_CUDA(ctx_alloc(ctx, &d.pair_tab, sizeof(PairPoly) * PT_NFN * PT_BINS));
  k_pair_table<<<dim3(PT_BINS / PTB, PT_NFN), PTB * PN, 0, ctx->stream>>>(
      ctx->p.alphad, reinterpret_cast<PairPoly *>(d.pair_tab));
  MDX_LAUNCHED(ctx);
  ctx->pair_tab_alpha = ctx->p.alphad;
  return MDX_OK;
}

int launch_pair64(mdx_ctx *ctx, bool shrt, bool split, bool ener, double *split_buf) {
  DevData &d = ctx->dv;
  const int T = 32 * PT_WARPS;
  const bool table = (ctx->px_on || d.pair_tab) && !ctx->p.lmnbl && ctx->p.alphad > 0.0;
  // Lanes of an owner: 32 on the long rows.  On the short rows (about 26
  // entries) fewer lanes make the owner's sums cheaper (short sweep at 98,304
  // atoms: 8 lanes 0.222 ms, 16 0.234, 32 0.257) as long as the owners still
  // fill half of the resident lanes (600 atoms: 20, 15, 13 us; 3,000: 21.2,
  // 20.7, 22.9).  The grid is the 2 resident blocks of a SM, each warp taking
  // several owners, so that the block sums at the end (a few hundred FP64
  // instructions) are formed once for all of them (long sweep at 3,000 atoms:
  // 57 us; 8 blocks a SM 69).
  int tpo = 32;
  if (shrt && table)
    while (tpo > 8 && (size_t)d.n * (tpo / 2) >= (size_t)T * ctx->nsm) tpo /= 2;
  const int per = T / tpo;  // owners of a block at a time
  const int grid = std::min((d.n + per - 1) / per, 2 * ctx->nsm);
  const int *cnt = shrt ? d.ns_cnt : d.nl_cnt;
  const int *idx = shrt ? d.ns_idx : d.nl_idx;
  const int cap = shrt ? d.cap_s : d.cap_l;
  double *fx = shrt ? d.hx : d.gx, *fy = shrt ? d.hy : d.gy, *fz = shrt ? d.hz : d.gz;
  mdx_scalars *sc = d.sc;
  const Dst6 dst =
      shrt ? dst6(ctx, grid, 6, &sc->pels2, &sc->pe2, &sc->vir2, &sc->virfx, &sc->virfy, &sc->virfz)
           : dst6(ctx, grid, 6, &sc->pels1, &sc->pe1, &sc->vir1, &sc->virx, &sc->viry, &sc->virz);
  const Lj64 lj{d.a6lj, d.b12lj, d.a6lj0, d.b12lj0, d.a6_14, d.b12_14};
  unsigned eemask = 0;
  for (int t = 0; t < ctx->d.ntypes; ++t)
    if (ctx->tc.iee[t] == 0) eemask |= 1u << t;
  const PairPoly *tab = reinterpret_cast<const PairPoly *>(d.pair_tab);
  const CellPbc cp = cell_pbc(ctx);
  const Px px = px_args(ctx, shrt);
  unsigned long long *ff = shrt ? d.hfix : d.gfix;
#define LP64T(S, P, E, K)                                                                       \
  k_pair64t<S, P, E, K><<<grid, T, 0, ctx->stream>>>(d.n, d.pos, d.ainfo, d.qsite, cnt, idx, cap, \
                                                     lj, ctx->tc, ctx->pc, cp, eemask, tab, fx, \
                                                     fy, fz, dst, split_buf)
#define LP64XT(S, P, E, K, SH)                                                                   \
  do {                                                                                           \
    const size_t sh = SH ? sizeof(PxPoly) * px_tables(E) * px.nbin : 0;                          \
    if (SH && raise_smem_limit(k_pair64x<S, P, E, K, SH>, sh) != cudaSuccess) {                  \
      ctx->err = "pair sweep: shared-memory limit";                                              \
      return MDX_ERR_CUDA;                                                                       \
    }                                                                                            \
    k_pair64x<S, P, E, K, SH><<<grid, T, sh, ctx->stream>>>(                                     \
        d.n, reinterpret_cast<longlong4_32a *>(d.ipos), d.pos, d.ainfo, d.qsite, cnt, idx, cap,  \
        lj, ctx->tc, ctx->pc, cp, eemask, px, fx, fy, fz, ff, dst, split_buf);                   \
  } while (0)
#define LP64X(S, P, E, K)                                                                        \
  do {                                                                                           \
    if (!S && d.n >= 4 * PT_WARPS * 2 * ctx->nsm) LP64XT(S, P, E, K, !S);                        \
    else LP64XT(S, P, E, K, false);                                                              \
  } while (0)
#define LP64(S, P, E)                                                                        \
  do {                                                                                       \
    if (ctx->px_on) {                                                                        \
      if (S && tpo == 8) LP64X(S, P, E, S ? 8 : 32);                                         \
      else if (S && tpo == 16) LP64X(S, P, E, S ? 16 : 32);                                  \
      else LP64X(S, P, E, 32);                                                               \
    } else if (!table)                                                                              \
      k_pair64<S, P, E><<<grid, T, 0, ctx->stream>>>(d.n, d.pos, d.ainfo, d.qsite, cnt, idx, \
                                                     cap, lj, ctx->tc, ctx->pc, cp, fx, fy,  \
                                                     fz, dst, split_buf);                    \
    else if (S && tpo == 8) LP64T(S, P, E, S ? 8 : 32);                                      \
    else if (S && tpo == 16) LP64T(S, P, E, S ? 16 : 32);                                    \
    else LP64T(S, P, E, 32);                                                                 \
  } while (0)
  // energies by type pair (force calls) come with the energies
  if (shrt) {
    if (split) LP64(true, true, true);
    else if (ener) LP64(true, false, true);
    else LP64(true, false, false);
  } else {
    if (split) LP64(false, true, true);
    else if (ener) LP64(false, false, true);
    else LP64(false, false, false);
  }
#undef LP64
#undef LP64T
#undef LP64X
#undef LP64XT
  MDX_LAUNCHED(ctx);
  return MDX_OK;
}
