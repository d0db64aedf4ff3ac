// ewald_fx.cu -- the FP64 path's reciprocal Ewald (FURIR forces.f:1286-1314)
// in fixed point, its two contractions on the tensor cores.
//
// GB300 issues one FP64 warp instruction per 64 cycles on each scheduler (1.05
// TFLOP/s), while its FP16 tensor cores do 1.9 PFLOP/s and its integer
// multiply-adds are 32 times the FP64 rate.  The quantities of this sum are
// bounded: with the tables
//   X_j(nx) = (q_j / qs) e^{i nx theta_x}, Y_j(ny), Z_j(z)   (|.| <= 1, qs a
//   power of two >= max |q|)
// everything up to the sums is a fixed-point number of known range.
//
// Both contractions are those of ewald_tc.cu,
//   S:  D[(e, c)][2z + e'] = sum_j T_j(c)_e Z_j(z)_e',  T = X Y
//   F:  D[j][4c + t]       = sum_k Z_j[k] W[4c + t][k],  k = 2z + e,
// done on integers (the splitting of Ozaki, Ogita, Oishi and Rump, Numer.
// Algorithms 59, 2012): each operand, 55 fractional bits, is cut into
// 7 signed 8-bit digits d_0 .. d_6 (base 256, d_0 the leading one), exact in
// FP16.  A product of two digits has 14 bits, so an FP32 accumulator in
// tensor memory holds the sum of up to 1024 of them exactly.  The products of
// equal weight (class s = i + j, weight 2^(-14 - 8 s)) share an accumulator;
// the 28 products with s <= 6 are kept, the rest is below 2^-53 of the
// operands' range.  F sums at most 64 (s + 1) products of a class and is exact.
// S drains its accumulators every 192 atoms, s + 1 products each: exact for s <=
// 4, and for 5 and 6 (weights 2^-54, 2^-62) unless nearly all of 192 atoms have
// digits near +-128 of one sign throughout, which then costs a few 2^-54 of one
// atom.  One MMA multiplies digit A_i with the digits B_0 .. B_(6-i) side by
// side along N: they fall on the accumulators i .. 6, which lie side by side
// too, so A_i is read once and not 7 - i times.
//
// S's accumulators are added to 64-bit integers every 192 atoms; T is formed
// in integers (complex product of two-word numbers: 12 wide multiply-adds
// and a few adds against 4 FP64 instructions of 64 cycles).  F's classes are
// put together into a 64-bit U, and Im(T U), Im(T V) weighted with nx, ny are
// again integer.  All sums are exact or rounded in one fixed order to a
// fixed unit, so the results do not depend on the order of anything else.
//
// Measured on a GB300 against the FP64-pipe passes of ewald.cu, per
// evaluation: 98,304 atoms, 16,700 k-vectors: tables 0.056 ms (0.098), S(k)
// 0.58 (7.7), forces 0.91 (12.8); 21,003 atoms, 3,576 k-vectors: S(k) 0.056
// (0.76), forces 0.113 (0.73); 609 atoms, 510 k-vectors: 0.015 (0.73), 0.025
// (0.045).  Error of the slow forces against phases and sums of more than 64
// bits, RMS relative: 5.3e-15 at 98,304 atoms (FP64 pipe: 6.8e-15), 3.6e-15
// at 3,000 (4.2e-15).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "ewald_ops.cuh"
#include "mdx_internal.cuh"
#include "tc_ptx.cuh"

namespace {

constexpr double PI_REF = 3.1415926536;  // common_inc.f:31
constexpr int FX_SL = 7;                 // digits of an operand
constexpr int FX_BITS = 8 * FX_SL - 1;   // fractional bits of an operand
constexpr int FX_ROW = 33;               // int4 per X / Y row of a 32-atom chunk (one of padding)
constexpr uint32_t FX_POLLS = 1u << 20;  // bounded mbarrier waits
constexpr size_t FX_SMEM_MAX = 227 * 1024;
// Chunks (of 32 atoms) per S accumulation: 32 x 6 x 5 products of class 4 stay
// below 2^24.  With 8 chunks they do not, and atoms of like phase lost 2^-46 of an
// atom an accumulation; with 4 every class is exact (S(k) of 98,304 atoms: 8
// chunks 0.562 ms, 6 0.576, 4 0.597).
constexpr int FX_DRAIN = 6;
constexpr int FX_TCOL = 8;               // k-columns of an F tile
constexpr int FX_TN = 4 * FX_TCOL;       // its rows (U.re, U.im, V.re, V.im)
constexpr int FX_GEN_WARPS = 16;
constexpr int FX_THREADS = 32 * (FX_GEN_WARPS + 1);
constexpr int FX_KMAX = 64;              // largest K of the F pass (2 kz rounded up to 16)

// Atoms of a 32-atom chunk are stored in the order pos(a): the 8 atoms of an
// octet, which one thread of the S pass takes, then lie 64 bytes apart and
// the four octets side by side.
__host__ __device__ __forceinline__ int fx_pos(int a) { return (a & 7) * 4 + (a >> 3); }

// A two-word number hi 2^32 + lo with lo a signed word: products need only
// signed 32 x 32 -> 64 multiply-adds.
struct W2 {
  int lo, hi;
};
__device__ __forceinline__ W2 w2(long long v) {
  W2 r;
  r.lo = (int)v;
  r.hi = (int)(v >> 32) - (r.lo >> 31);
  return r;
}
__device__ __forceinline__ long long mad(int a, int b, long long c) { return (long long)a * b + c; }
// (a b + c d) / 2^64 rounded, plus add; the low word products (below one unit)
// are left out
__device__ __forceinline__ long long dot2(W2 a, W2 b, W2 c, W2 d, long long add) {
  const long long cr =
      mad(a.hi, b.lo, mad(a.lo, b.hi, mad(c.hi, d.lo, mad(c.lo, d.hi, 1ll << 31))));
  return mad(a.hi, b.hi, mad(c.hi, d.hi, add)) + (cr >> 32);
}
__device__ __forceinline__ W2 neg(W2 a) { return W2{-a.lo, -a.hi}; }

// (a b + c d) / 2^61 for numbers of scale 2^61 (the table recurrence)
__device__ __forceinline__ long long dot61(W2 a, W2 b, W2 c, W2 d) {
  const long long cr =
      mad(a.hi, b.lo, mad(a.lo, b.hi, mad(c.hi, d.lo, mad(c.lo, d.hi, 1ll << 28))));
  return (mad(a.hi, b.hi, mad(c.hi, d.hi, 0)) << 3) + (cr >> 29);
}

// x / 2^s to the nearest, ties to even (half-up would add half a unit on
// average at s = 1, the same way in every sum: measured as a force towards
// the origin); m1 = 2^(s - 1) - 1 (0 for s = 0).
__device__ __forceinline__ long long shr_rne(long long x, int s, long long m1) {
  return (x + m1 + (s > 0 ? (x >> s) & 1 : 0)) >> s;
}
__device__ __forceinline__ long long half_m1(int s) { return s > 0 ? (1ll << (s - 1)) - 1 : 0; }

// A table entry as stored: (re.lo, re.hi, im.lo, im.hi); lo never INT_MIN, so
// that it can be negated.
__device__ __forceinline__ int4 fx_entry(long long re, long long im) {
  W2 a = w2(re), b = w2(im);
  a.lo = max(a.lo, -0x7fffffff);
  b.lo = max(b.lo, -0x7fffffff);
  return make_int4(a.lo, a.hi, b.lo, b.hi);
}

// The digits of 8 numbers v (|v| <= 2^FX_BITS; w = v + FX_BIAS) as FP16
// pairs: out[i][h] holds digit i of numbers 2h and 2h + 1.  With the bias
// every digit but the leading one is a byte of w (digit + 128) and the
// leading one the 16 bits above; 0x6400 | u is the FP16 number 1024 + u.
constexpr long long FX_BIAS = 0x80808080808080ll;
__device__ __forceinline__ unsigned fx_half2(unsigned u) {
  unsigned r;
  asm("sub.rn.f16x2 %0, %1, %2;\n" : "=r"(r) : "r"(u | 0x64006400u), "r"(0x64806480u));
  return r;
}
__device__ __forceinline__ void fx_digits(const long long (&w)[8], unsigned (&out)[FX_SL][4]) {
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    const unsigned a0 = (unsigned)w[2 * h], a1 = (unsigned)(w[2 * h] >> 32);
    const unsigned b0 = (unsigned)w[2 * h + 1], b1 = (unsigned)(w[2 * h + 1] >> 32);
#pragma unroll
    for (int b = 0; b < FX_SL - 1; ++b) {
      const int s = b & 3;
      const unsigned x = __byte_perm(b < 4 ? a0 : a1, b < 4 ? b0 : b1, s | ((4 + s) << 8));
      out[FX_SL - 1 - b][h] = fx_half2(x & 0x00ff00ffu);
    }
    out[0][h] = fx_half2(__byte_perm(a1, b1, 0x7632));
  }
}

// 1 / BOXL, 1 / BOYL, 1 / BOZL and, in the hexagonal cell, 1 / (2 BOYL) (else
// 0) with their rounding errors.
struct FxBox {
  double ib[4], ibl[4];
};
constexpr int FX_CIRCLE = 256;
constexpr double TWO_PI = 6.283185307179586;
constexpr double PI_EPS = 3.2489329648931176e-12;  // PI_REF / pi - 1

// Tables and operand images of one step; a block is one 32-atom chunk, warp a
// the axis a (lane = atom): the first phase to about 2^-59 (a table of points
// of the circle and short Taylor series: fewer FP64 instructions than the
// library's sincos, and 6 bits more), then a fixed-point recurrence (scale
// 2^61, an error below 2^-59 a step).  X (with the charge) and Y go out
// as two-word entries, X of scale 2^61, Y of 2^58 (their product / 2^64 then
// has FX_BITS fractional bits); Z goes through shared memory into the digit
// images of both passes, in the MMA's core-matrix order: zs, the S pass's B
// operand (row 7-digit major: i np + 2 z + e), zf, the F pass's A operand.
// The chunk's slice of the force accumulators is zeroed.
__global__ void __launch_bounds__(128) k_fx_tables(
    int n, const dbl4 *__restrict__ pos, FxBox box, int kx, int ky, int kz, int np, int kp, const double *__restrict__ qs, int4 *__restrict__ xy,
    unsigned char *__restrict__ zs, unsigned char *__restrict__ zf,
    unsigned long long *__restrict__ facc, int *__restrict__ bad,
    const int4 *__restrict__ circle) {
  extern __shared__ int4 sz[];  // [kz][33]
  const double *ib = box.ib, *ibl = box.ibl;
  const int lane = threadIdx.x & 31, a = threadIdx.x >> 5;
  const int c = blockIdx.x, i = c * 32 + lane;
  if (a < 3) {
    const bool live = i < n;
    dbl4 p;
    p.x = p.y = p.z = p.w = 0.0;
    if (live) p = pos[i];
    // u + ul = coordinate / box (hexagonal cell: x + y / (2 BOYL), forces.f:
    // 1402), to more than 64 bits: an error of the first phase grows n-fold
    // in entry n.  The reference's angle 2 PI u is 2 pi u (1 + PI_EPS): the
    // nearest of FX_CIRCLE points of the circle, turned by the small rest
    const double w = a == 0 ? p.x : a == 1 ? p.y : p.z;
    double u = w * ib[a];
    double ul = fma(w, ib[a], -u) + w * ibl[a];
    if (a == 0 && ib[3] != 0.0) {
      const double y = p.y * ib[3], t = u + y, bb = t - u;
      ul += (u - (t - bb)) + (y - bb) + fma(p.y, ib[3], -y) + p.y * ibl[3];
      u = t;
    }
    if (!(fabs(u) < 1e300)) {  // a non-finite position: flagged, the sums come back NaN
      *bad = 1;
      u = ul = 0.0;
    }
    const double f = u - rint(u), kd = rint(f * FX_CIRCLE);
    const double al = TWO_PI * ((f - kd * (1.0 / FX_CIRCLE)) + fma(PI_EPS, u, ul)), a2 = al * al;
    // sine and cosine - 1 of |al| <= pi / 256, Taylor (next terms below 2^-66)
    const double sn = al * fma(a2, fma(a2, fma(a2, -1.0 / 5040, 1.0 / 120), -1.0 / 6), 1.0);
    const double cm = a2 * fma(a2, fma(a2, -1.0 / 720, 1.0 / 24), -0.5);
    constexpr double ONE = 2305843009213693952.0;  // 2^61
    const int4 cc = circle[(int)kd & (FX_CIRCLE - 1)];
    const W2 cr{cc.x, cc.y}, ci{cc.z, cc.w};
    const W2 cmf = w2(__double2ll_rn(cm * ONE)), snf = w2(__double2ll_rn(sn * ONE));
    const W2 er = w2(dot61(cr, cmf, neg(ci), snf) + (((long long)cr.hi << 32) + cr.lo)),
             ei = w2(dot61(cr, snf, ci, cmf) + (((long long)ci.hi << 32) + ci.lo));
    const W2 nei = neg(ei);
    long long vr = 1ll << 61, vi = 0;
    const int len = a == 0 ? kx : a == 1 ? ky : kz;
    const W2 q = w2(live ? __double2ll_rn(p.w * qs[1] * ONE) : 0ll);
    const W2 zero{0, 0};
    int4 *dst = xy + (size_t)c * (kx + ky) * FX_ROW + fx_pos(lane);
    for (int k = 0; k < len; ++k) {
      const W2 r = w2(vr), m = w2(vi);
      if (a == 0) {
        dst[(size_t)k * FX_ROW] = fx_entry(dot61(r, q, zero, zero), dot61(m, q, zero, zero));
      } else if (a == 1) {
        dst[(size_t)(kx + k) * FX_ROW] =
            live ? fx_entry((vr + 4) >> 3, (vi + 4) >> 3) : make_int4(0, 0, 0, 0);
      } else {
        // the operands' FX_BITS bits, rounded; |.| <= 2^FX_BITS
        const long long lim = 1ll << FX_BITS;
        const long long zr = min(max((vr + 32) >> 6, -lim), lim),
                        zi = min(max((vi + 32) >> 6, -lim), lim);
        sz[k * 33 + lane] = live ? make_int4((int)zr, (int)(zr >> 32), (int)zi, (int)(zi >> 32))
                                 : make_int4(0, 0, 0, 0);
      }
      vr = dot61(r, er, m, nei);
      vi = dot61(r, ei, m, er);
    }
  } else if (i < n) {
    facc[i] = facc[n + i] = facc[2 * n + i] = 0ull;
  }
  __syncthreads();
  auto val = [&](int z, int at, int e) {
    const int4 v = sz[z * 33 + at];
    return ((long long)(e ? v.w : v.y) << 32) + (unsigned)(e ? v.z : v.x) + FX_BIAS;
  };
  const int G = FX_SL * np / 8;  // 8-row groups of the S image
  unsigned char *cs = zs + (size_t)c * FX_SL * np * 64;
  for (int t = threadIdx.x; t < kz * 8; t += blockDim.x) {  // (z, octet, re/im)
    const int o = t & 3, e = (t >> 2) & 1, z = t >> 3;
    long long w[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) w[k] = val(z, 8 * o + k, e);
    unsigned dg[FX_SL][4];
    fx_digits(w, dg);
#pragma unroll
    for (int j = 0; j < FX_SL; ++j) {
      const int r = j * np + 2 * z + e;
      *reinterpret_cast<uint4 *>(cs + ((size_t)o * G + (r >> 3)) * 128 + (r & 7) * 16) =
          make_uint4(dg[j][0], dg[j][1], dg[j][2], dg[j][3]);
    }
  }
  unsigned char *cf = zf + (size_t)(c >> 2) * (kp / 16) * FX_SL * 4096;
  for (int t = threadIdx.x; t < 4 * kp; t += blockDim.x) {  // (atom, 4 z = 8 k)
    const int at = t & 31, g = t >> 5;
    long long w[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int z = 4 * g + (k >> 1);
      w[k] = z < kz ? val(z, at, k & 1) : FX_BIAS;
    }
    unsigned dg[FX_SL][4];
    fx_digits(w, dg);
    const int r = (c & 3) * 32 + fx_pos(at);
    unsigned char *d = cf + (size_t)(g >> 1) * FX_SL * 4096 + (g & 1) * 2048 + (r >> 3) * 128 +
                       (r & 7) * 16;
#pragma unroll
    for (int j = 0; j < FX_SL; ++j)
      *reinterpret_cast<uint4 *>(d + j * 4096) =
          make_uint4(dg[j][0], dg[j][1], dg[j][2], dg[j][3]);
  }
}

// S pass: a CTA (one per SM) takes one M-tile of 64 columns (rows 0-63 T.re,
// 64-127 T.im) and a slice of atoms, 32 at a time.  Warp 16 (lane 0) brings
// in each chunk's X, Y rows and Z image (bulk copies) and issues the MMAs;
// warps 0-7 and 8-15 take turns at the chunks, forming T, its digits and the
// A operand (thread = column x octet of atoms) while the other group's chunk
// is multiplied.  Every FX_DRAIN chunks all 16 warps add the accumulators to
// 64-bit integers (unit 2^-ua); at the end those meet in integer atomics.
// Barriers: xyf[b] / zfull[b] (X, Y rows / Z image of the chunk in stage b
// landed), af[b] (A written, X, Y read: 8 arrivals), ad[b] (MMAs of that
// chunk done: A and Z free), gd (accumulators of a drain complete), rf (they
// were read: 16 arrivals).
__global__ void __launch_bounds__(FX_THREADS, 1) k_fx_sfac(
    int nchunk_all, int cps, int ncol, int np, int kx, int kxy, int ua, int ug,
    const KCol *__restrict__ cols, const int4 *__restrict__ xy,
    const unsigned char *__restrict__ zs, unsigned long long *__restrict__ acc_out,
    int *__restrict__ bad, int *__restrict__ err) {
  extern __shared__ unsigned char dsm_raw[];
  __shared__ __align__(8) unsigned long long xyf[2], zfull[2], af[2], ad[2], gd, rf;
  __shared__ uint32_t tmem_base_sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int mt = blockIdx.x;
  const int c0 = blockIdx.y * cps, nchunk = min(nchunk_all - c0, cps);
  const uint32_t raw = tc::smem_addr(dsm_raw);
  const uint32_t pad = ((raw + 1023u) & ~1023u) - raw;
  unsigned char *dsm = dsm_raw + pad;
  const uint32_t sbase = raw + pad;
  constexpr uint32_t ABYTES = FX_SL * 8192;
  const uint32_t zbytes = (uint32_t)FX_SL * np * 64, xybytes = (uint32_t)kxy * FX_ROW * 16;
  const uint32_t oZ = 2 * ABYTES, oXY = oZ + 2 * zbytes;
  if (warp == 0) {
    tc::tmem_alloc(tc::smem_addr(&tmem_base_sh), 512);
    tc::tmem_relinquish();
  }
  if (tid == 32 && blockIdx.x == 0 && blockIdx.y == 0) {  // the flag, for the kernels to come
    bad[1] = bad[0];
    bad[0] = 0;
  }
  if (tid == 0) {
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(tc::smem_addr(&xyf[b]), 1);
      tc::mbar_init(tc::smem_addr(&zfull[b]), 1);
      tc::mbar_init(tc::smem_addr(&af[b]), FX_GEN_WARPS / 2);
      tc::mbar_init(tc::smem_addr(&ad[b]), 1);
    }
    tc::mbar_init(tc::smem_addr(&gd), 1);
    tc::mbar_init(tc::smem_addr(&rf), FX_GEN_WARPS);
    tc::mbar_init_fence();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = tmem_base_sh;
  const int ndrain = (nchunk + FX_DRAIN - 1) / FX_DRAIN;
  bool ok = true;
  auto wait = [&](unsigned long long &bar, int phase) {
    if (!tc::mbar_wait(tc::smem_addr(&bar), (uint32_t)phase & 1u, FX_POLLS)) ok = false;
  };

  if (warp == FX_GEN_WARPS) {
    if (lane == 0) {
      auto copy_xy = [&](int c) {
        const uint32_t bar = tc::smem_addr(&xyf[c & 1]);
        tc::mbar_arrive_expect_tx(bar, xybytes);
        tc::bulk_g2s(sbase + oXY + (uint32_t)(c & 1) * xybytes,
                     xy + (size_t)(c0 + c) * kxy * FX_ROW, xybytes, bar);
      };
      auto copy_z = [&](int c) {
        const uint32_t bar = tc::smem_addr(&zfull[c & 1]);
        tc::mbar_arrive_expect_tx(bar, zbytes);
        tc::bulk_g2s(sbase + oZ + (uint32_t)(c & 1) * zbytes, zs + (size_t)(c0 + c) * zbytes,
                     zbytes, bar);
      };
      for (int c = 0; c < min(nchunk, 2); ++c) {
        copy_xy(c);
        copy_z(c);
      }
      const uint32_t blbo = (uint32_t)FX_SL * np * 16;  // bytes between K-adjacent core matrices
      const int q1 = 256 / np;                          // digits of B one MMA takes at most
      for (int c = 0; c < nchunk; ++c) {
        const int b = c & 1, ph = c >> 1;
        wait(af[b], ph);
        if (c + 2 < nchunk) copy_xy(c + 2);
        wait(zfull[b], ph);
        if (c % FX_DRAIN == 0 && c) wait(rf, c / FX_DRAIN - 1);
        tc::fence_after_sync();
        const uint32_t sa = sbase + (uint32_t)b * ABYTES, sz = sbase + oZ + (uint32_t)b * zbytes;
        for (int k = 0; k < 2; ++k) {
          for (int i = 0; i < FX_SL; ++i) {
            const uint64_t da = tc::sdesc(sa + (uint32_t)(i * 8192 + k * 4096), 2048, 128);
            for (int j = 0; j < FX_SL - i; j += q1) {
              const int nj = min(q1, FX_SL - i - j) * np;
              const uint64_t db = tc::sdesc(
                  sz + (uint32_t)(2 * k) * blbo + (uint32_t)(j * np) * 16, blbo, 128);
              tc::mma_f16(tbase + (uint32_t)((i + j) * np), da, db, tc::idesc_f16(128, nj),
                          (c % FX_DRAIN || k || i) ? 1u : 0u);
            }
          }
        }
        tc::mma_commit(tc::smem_addr(&ad[b]));
        if (c % FX_DRAIN == FX_DRAIN - 1 || c == nchunk - 1) tc::mma_commit(tc::smem_addr(&gd));
        // the Z image of the previous chunk is free once its MMAs are done
        if (c >= 1 && c + 1 < nchunk) {
          wait(ad[b ^ 1], (c - 1) >> 1);
          copy_z(c + 1);
        }
      }
    }
    __syncwarp();
  } else {
    const int grp = warp >> 3;
    const int o = lane >> 3, cl = (warp & 7) * 8 + (lane & 7);
    const int col = mt * 64 + cl;
    int xrow = 0, yrow = kx;
    bool have = false, yneg = false;
    if (col < ncol) {
      const KCol kc = cols[col];
      have = true;
      yneg = kc.ny < 0;
      xrow = kc.nx;
      yrow = kx + (yneg ? -kc.ny : kc.ny);
    }
    unsigned char *const arow = dsm + o * 2048 + (cl >> 3) * 128 + (cl & 7) * 16;
    long long acc[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) acc[k] = 0;
    const int qd = warp & 3, part = warp >> 2;
    const int rsh = 54 - ua;
    const long long rnd = half_m1(rsh);
    auto drain = [&](int g) {
      wait(gd, g);
      tc::fence_after_sync();
      __syncwarp();
#pragma unroll
      for (int it = 0; it < 4; ++it) {
        if (it * 16 >= np) continue;
        const uint32_t ta =
            tbase + ((uint32_t)(32 * qd) << 16) + (uint32_t)(part * (np / 4) + 4 * it);
        float v[FX_SL][4];
#pragma unroll
        for (int s = 0; s < FX_SL; ++s) tc::tmem_ld4(ta + (uint32_t)(s * np), v[s]);
        tc::tmem_ld_wait();
#pragma unroll
        for (int s = 0; s < FX_SL; ++s) tc::pin4(v[s]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          int d[FX_SL];
#pragma unroll
          for (int s = 0; s < FX_SL; ++s) d[s] = __float2int_rn(v[s][e]);
          const long long h = (long long)d[0] * 65536 + (long long)d[1] * 256 + d[2];
          const long long l = (long long)d[3] * 65536 + (long long)d[4] * 256 + d[5];
          const long long x = (h << 24) + l + ((d[6] + 128) >> 8);
          acc[4 * it + e] += shr_rne(x, rsh, rnd);
        }
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(tc::smem_addr(&rf));
    };
    int gdone = 0;
    for (int c = grp; c < nchunk; c += 2) {
      const int ph = c >> 1;
      wait(xyf[grp], ph);
      const int4 *X = reinterpret_cast<const int4 *>(dsm + oXY + (uint32_t)grp * xybytes) +
                      xrow * FX_ROW + o;
      const int4 *Y = X + (yrow - xrow) * FX_ROW;
      long long tr[8], ti[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int4 x = X[4 * k], y = Y[4 * k];
        const W2 xr{x.x, x.y}, xi{x.z, x.w}, yr{y.x, y.y};
        W2 yi{y.z, y.w}, ny = neg(yi);
        if (yneg) {
          const W2 s = yi;
          yi = ny;
          ny = s;
        }
        tr[k] = have ? dot2(xr, yr, xi, ny, FX_BIAS) : FX_BIAS;
        ti[k] = have ? dot2(xr, yi, xi, yr, FX_BIAS) : FX_BIAS;
      }
      if (c >= 2) wait(ad[grp], ph - 1);  // A buffer free
      unsigned char *da = arow + (uint32_t)grp * ABYTES;
      unsigned dg[FX_SL][4];
      fx_digits(tr, dg);
#pragma unroll
      for (int s = 0; s < FX_SL; ++s)
        *reinterpret_cast<uint4 *>(da + s * 8192) =
            make_uint4(dg[s][0], dg[s][1], dg[s][2], dg[s][3]);
      fx_digits(ti, dg);
#pragma unroll
      for (int s = 0; s < FX_SL; ++s)
        *reinterpret_cast<uint4 *>(da + s * 8192 + 1024) =
            make_uint4(dg[s][0], dg[s][1], dg[s][2], dg[s][3]);
      tc::fence_proxy_async();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(tc::smem_addr(&af[grp]));
      // the previous accumulation is read one chunk into the next
      if (gdone < c / FX_DRAIN) drain(gdone++);
    }
    while (gdone < ndrain) drain(gdone++);
    const int sh = ua - ug;
    const long long r2 = half_m1(sh);
    unsigned long long *out =
        acc_out + ((size_t)mt * np + part * (np / 4)) * 128 + 32 * qd + lane;
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      if (it * 16 >= np) continue;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        atomicAdd(out + (size_t)(4 * it + e) * 128, (unsigned long long)shr_rne(acc[4 * it + e], sh, r2));
    }
  }
  tc::fence_before_sync();
  __syncthreads();  // every MMA waited for, every tensor-memory read done
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tbase, 512);
  }
  if (!ok) atomicOr(err, DERR_TIMEOUT);
}

// S(k) of the k-vectors from the integer sums: block per column, thread per
// record p (nz = +-z).  The sums it has read are cleared for the next call.
__global__ void k_fx_form(int ncol, int np, int ug, const KCol *__restrict__ cols,
                          unsigned long long *__restrict__ acc, const double *__restrict__ qs,
                          const int *__restrict__ bad, double2 *__restrict__ sk) {
  const int c = blockIdx.x;
  if (c >= ncol) return;
  const KCol col = cols[c];
  const double scale = *bad ? __longlong_as_double(0x7ff8000000000000ll) : ldexp(qs[0], -ug);
  long long *a = reinterpret_cast<long long *>(acc) + (size_t)(c >> 6) * np * 128;
  const int r = c & 63;
  for (int p = threadIdx.x; p <= col.m; p += blockDim.x) {
    const int z = kcol_z(col, p);
    const long long A1 = a[(size_t)(2 * z) * 128 + r], A3 = a[(size_t)(2 * z + 1) * 128 + r];
    const long long A4 = a[(size_t)(2 * z) * 128 + 64 + r],
                    A2 = a[(size_t)(2 * z + 1) * 128 + 64 + r];
    a[(size_t)(2 * z) * 128 + r] = a[(size_t)(2 * z + 1) * 128 + r] = 0;
    a[(size_t)(2 * z) * 128 + 64 + r] = a[(size_t)(2 * z + 1) * 128 + 64 + r] = 0;
    const int kp = kcol_k(col, z), km = z > 0 ? kcol_k(col, -z) : -1;
    if (kp >= 0) sk[kp] = make_double2((double)(A1 - A2) * scale, (double)(A3 + A4) * scale);
    if (km >= 0) sk[km] = make_double2((double)(A1 + A2) * scale, (double)(A4 - A3) * scale);
  }
}

// F tile meta: exponents of the tile's U and V rows, left shift of T, K
// steps; bounds of the tile's sums of nx, ny weighted Im(T U) and of Im(T V).
struct FxTile {
  int eu, ev, sh, ks;
  double bu, bv;
};

__device__ __forceinline__ int exp_above(double x) {  // x < 2^e (0 for x = 0)
  return x > 0.0 ? ilogb(x) + 1 : 0;
}

// B operand of the F pass, one step, from S(k) and the per-k constants (W = 2
// AKC conj(S)), and the k-vectors' energy and virial sums: block per tile of
// FX_TCOL columns.  Row
// 4 c + t is U.re, U.im, V.re, V.im of column c (V with integer nz weights;
// 2 PI / BOZL comes with the fold), scaled to the largest U or V entry of the
// tile by a power of two, as digits in core-matrix order.
__global__ void __launch_bounds__(256) k_fx_wtiles(
    int kp, const int4 *__restrict__ slot, const int *__restrict__ scol,
    const int *__restrict__ tks, const KCol *__restrict__ cols,
    const double2 *__restrict__ sk, const double *__restrict__ kcon,
    unsigned char *__restrict__ tw, FxTile *__restrict__ meta, Dst6 dst) {
  extern __shared__ double sv[];  // [FX_TN][kp]
  __shared__ double red[2][8], rsum[FX_TN];
  __shared__ int se[2];
  const int tile = blockIdx.x, tid = threadIdx.x;
  double mx[2] = {0.0, 0.0}, acc[5] = {0, 0, 0, 0, 0};
  for (int t = tid; t < FX_TN * (kp / 2); t += blockDim.x) {
    const int z = t % (kp / 2), r = t / (kp / 2), comp = r & 3;
    const int c = scol[tile * FX_TCOL + (r >> 2)];
    double va = 0.0, vb = 0.0;
    if (c >= 0) {
      const KCol col = cols[c];
      const int kpl = kcol_k(col, z), kmi = z > 0 ? kcol_k(col, -z) : -1;
      double ar = 0.0, ai = 0.0, br = 0.0, bi = 0.0;
      auto weight = [&](int k, double &wr, double &wi) {
        const double2 S = sk[k];
        const double *c5 = kcon + 5 * (size_t)k;
        const double AK2 = 2.0 * c5[0];
        wr = AK2 * S.x;
        wi = -AK2 * S.y;
        if (comp == 0) kterm_add(acc, c5, S.y * S.y + S.x * S.x);
      };
      if (kpl >= 0) weight(kpl, ar, ai);
      if (kmi >= 0) weight(kmi, br, bi);
      if (comp >= 2) {  // nz W
        ar *= z;
        ai *= z;
        br *= -z;
        bi *= -z;
      }
      // coefficients of (Re Z, Im Z): {P.re, -M.im} and {P.im, M.re}
      va = (comp & 1) ? ai + bi : ar + br;
      vb = (comp & 1) ? ar - br : -(ai - bi);
    }
    sv[r * kp + 2 * z] = va;
    sv[r * kp + 2 * z + 1] = vb;
    const double m = fmax(fabs(va), fabs(vb));
    mx[comp >> 1] = fmax(mx[comp >> 1], m);
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx[h] = fmax(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], o));
    if ((tid & 31) == 0) red[h][tid >> 5] = mx[h];
  }
  __syncthreads();
  if (tid < 2) {
    double m = 0.0;
    for (int w = 0; w < 8; ++w) m = fmax(m, red[tid][w]);
    se[tid] = max(exp_above(m), -900);  // 2^(FX_BITS - e) stays finite
  }
  if (tid >= 32 && tid < 32 + FX_TN) {  // a row's sum of magnitudes
    double s = 0.0;
    for (int k = 0; k < kp; ++k) s += fabs(sv[(tid - 32) * kp + k]);
    rsum[tid - 32] = s;
  }
  __syncthreads();
  if (tid == 0) {
    double bx = 0.0, by = 0.0, bv = 0.0, b1 = 0.0;
    for (int c = 0; c < FX_TCOL; ++c) {
      const int4 sl = slot[tile * FX_TCOL + c];
      const double lu = rsum[4 * c] + rsum[4 * c + 1];
      bx += abs(sl.x) * lu;
      by += abs(sl.w) * lu;
      b1 = fmax(b1, lu);
      bv += rsum[4 * c + 2] + rsum[4 * c + 3];
    }
    const double bu = fmax(fmax(bx, by), b1);
    // unit of Im(T U): 2^(e - 45 - sh); sums stay below 2^62 units
    const int shu = 62 - 45 + se[0] - exp_above(bu), shv = 62 - 45 + se[1] - exp_above(bv);
    FxTile m;
    m.eu = se[0];
    m.ev = se[1];
    m.sh = max(0, min(7, min(shu, shv)));
    m.ks = tks[tile];
    m.bu = bu;
    m.bv = bv;
    meta[tile] = m;
  }
  unsigned char *out = tw + (size_t)tile * (kp / 16) * FX_SL * FX_TN * 32;
  constexpr int G = FX_SL * FX_TN / 8;
  for (int t = tid; t < FX_TN * (kp / 8); t += blockDim.x) {
    const int r = t % FX_TN, g = t / FX_TN;
    // a power of two: the product is exact
    const double up = __hiloint2double((1023 + FX_BITS - se[(r >> 1) & 1]) << 20, 0);
    long long w[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      w[k] = __double2ll_rn(sv[r * kp + 8 * g + k] * up) + FX_BIAS;
    unsigned dg[FX_SL][4];
    fx_digits(w, dg);
#pragma unroll
    for (int j = 0; j < FX_SL; ++j) {
      const int rr = j * FX_TN + r;
      *reinterpret_cast<uint4 *>(out + ((size_t)g * G + (rr >> 3)) * 128 + (rr & 7) * 16) =
          make_uint4(dg[j][0], dg[j][1], dg[j][2], dg[j][3]);
    }
  }
  acc[4] = acc[0];
  block_add<5>(acc, dst);
}

// F pass: a CTA takes 128 atoms (MMA M) and a range of tiles.  Warp 16 (lane
// 0) copies in the atoms' Z image, their X, Y rows (XYS; else the epilogue
// reads those from global memory) and the tiles' B operands (two buffers),
// and issues 7 MMAs per K step into 7 accumulators of 32 columns, two sets.
// Warps 0-15 are the epilogue: warp w takes the atoms 32 (w % 4) .. + 31 and
// the columns 2 (w / 4), + 1 of each tile.  The class sums D_s, |D_s| <= K (s
// + 1) 2^14, become integers by adding 1.5 2^23 and reading the bits, exact
// below 2^22: s <= 4 for K <= 48 (BIGK: s = 4 by a conversion instead); s = 5
// and 6, whose last bits are below U's unit, by adding 1.5 2^24.
template <bool BIGK>
__device__ __forceinline__ long long fx_join(const float (&v)[FX_SL][8], int e) {
  long long b[FX_SL];
#pragma unroll
  for (int s = 0; s < FX_SL; ++s)
    b[s] = BIGK && s == 4 ? __float2int_rn(v[s][e])
                          : __float_as_int(v[s][e] + (s < 5 ? 12582912.f : 25165824.f));
  constexpr unsigned long long C1 = 0x4B400000ull, C2 = 0x4BC00000ull;
  constexpr unsigned long long C =
      C1 * ((1ull << 40) + (1ull << 32) + (1ull << 24) + (1ull << 16) + (BIGK ? 0ull : 256ull)) +
      C2 * 2ull + (C2 >> 7);
  const long long h = b[0] * 65536 + b[1] * 256 + b[2];
  const long long l = b[3] * 65536 + b[4] * 256 + b[5] * 2 + (((int)b[6] + 64) >> 7);
  return (long long)(((unsigned long long)h << 24) + (unsigned long long)l - C);
}

template <bool XYS, bool BIGK>
__global__ void __launch_bounds__(FX_THREADS, 1) k_fx_force(
    int n, int ntile, int kp, int kxy, const int *__restrict__ parts,
    const FxTile *__restrict__ meta, const int4 *__restrict__ slot,
    const unsigned char *__restrict__ tw, const unsigned char *__restrict__ zf,
    const int4 *__restrict__ xy, unsigned long long *__restrict__ facc, int *__restrict__ gexp,
    int *__restrict__ err) {
  extern __shared__ unsigned char dsm_raw[];
  __shared__ __align__(8) unsigned long long abar, bfull[2], mdone[2], afree[2];
  __shared__ uint32_t tmem_base_sh;
  __shared__ int gsh[2];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t raw = tc::smem_addr(dsm_raw);
  const uint32_t pad = ((raw + 1023u) & ~1023u) - raw;
  unsigned char *dsm = dsm_raw + pad;
  const uint32_t sbase = raw + pad;
  const int nks = kp / 16;
  constexpr uint32_t ASTEP = FX_SL * 4096, BSTEP = FX_SL * FX_TN * 32;
  const uint32_t abytes = (uint32_t)nks * ASTEP, bbytes = (uint32_t)nks * BSTEP;
  const uint32_t xybytes = XYS ? 4u * (uint32_t)kxy * FX_ROW * 16 : 0u;
  const uint32_t oB = abytes, oXY = oB + 2 * bbytes;
  const int t0 = parts[blockIdx.y], t1 = parts[blockIdx.y + 1];
  if (warp == 0) {
    tc::tmem_alloc(tc::smem_addr(&tmem_base_sh), 512);
    tc::tmem_relinquish();
  }
  if (tid == 0) {
    tc::mbar_init(tc::smem_addr(&abar), 1);
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(tc::smem_addr(&bfull[b]), 1);
      tc::mbar_init(tc::smem_addr(&mdone[b]), 1);
      tc::mbar_init(tc::smem_addr(&afree[b]), FX_GEN_WARPS);
    }
    tc::mbar_init_fence();
  }
  if (warp == 1) {
    // the unit of the force sums, from the bounds of all tiles (the same in
    // every CTA: the same sums in the same order)
    double bu = 0.0, bv = 0.0;
    int mu = -100000, mv = -100000;
    for (int t = lane; t < ntile; t += 32) {
      const FxTile m = meta[t];
      bu += m.bu;
      bv += m.bv;
      if (m.bu > 0.0) mu = max(mu, m.eu - 45 - m.sh);
      if (m.bv > 0.0) mv = max(mv, m.ev - 45 - m.sh);
    }
    bu = warp_sum(bu);
    bv = warp_sum(bv);
    mu = __reduce_max_sync(0xffffffffu, mu);
    mv = __reduce_max_sync(0xffffffffu, mv);
    if (lane == 0) {
      gsh[0] = max(exp_above(bu) - 62, mu);
      gsh[1] = max(exp_above(bv) - 62, mv);
      if (blockIdx.x == 0 && blockIdx.y == 0) {
        gexp[0] = gsh[0];
        gexp[1] = gsh[1];
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = tmem_base_sh;
  bool ok = true;
  auto wait = [&](unsigned long long &bar, int phase) {
    if (!tc::mbar_wait(tc::smem_addr(&bar), (uint32_t)phase & 1u, FX_POLLS)) ok = false;
  };

  if (warp == FX_GEN_WARPS) {
    if (lane == 0 && t0 < t1) {
      auto copy_b = [&](int t) {  // the K steps tile t uses
        const int b = (t - t0) & 1;
        const uint32_t bar = tc::smem_addr(&bfull[b]);
        const uint32_t bytes = (uint32_t)meta[t].ks * BSTEP;
        tc::mbar_arrive_expect_tx(bar, bytes);
        tc::bulk_g2s(sbase + oB + (uint32_t)b * bbytes, tw + (size_t)t * bbytes, bytes, bar);
      };
      {
        const uint32_t bar = tc::smem_addr(&abar);
        tc::mbar_arrive_expect_tx(bar, abytes + xybytes);
        tc::bulk_g2s(sbase, zf + (size_t)blockIdx.x * abytes, abytes, bar);
        if (XYS)
          tc::bulk_g2s(sbase + oXY, xy + (size_t)blockIdx.x * 4 * kxy * FX_ROW, xybytes, bar);
      }
      copy_b(t0);
      if (t0 + 1 < t1) copy_b(t0 + 1);
      wait(abar, 0);
      for (int t = t0; t < t1; ++t) {
        const int b = (t - t0) & 1, ph = (t - t0) >> 1;
        wait(bfull[b], ph);
        if (t >= t0 + 2) wait(afree[b], ph - 1);
        tc::fence_after_sync();
        const int ks = meta[t].ks;
        const uint32_t d = tbase + (uint32_t)(b * FX_SL * FX_TN);
        const uint32_t sb = sbase + oB + (uint32_t)b * bbytes;
        for (int k = 0; k < ks; ++k)
#pragma unroll
          for (int i = 0; i < FX_SL; ++i)
            tc::mma_f16(d + (uint32_t)(i * FX_TN),
                        tc::sdesc(sbase + (uint32_t)k * ASTEP + (uint32_t)(i * 4096), 2048, 128),
                        tc::sdesc(sb + (uint32_t)k * BSTEP, BSTEP / 2, 128),
                        tc::idesc_f16(128, (FX_SL - i) * FX_TN), (k || i) ? 1u : 0u);
        tc::mma_commit(tc::smem_addr(&mdone[b]));
        if (t > t0 && t + 1 < t1) {  // buffer b ^ 1 is free once tile t - 1's MMAs are done
          wait(mdone[b ^ 1], (t - 1 - t0) >> 1);
          copy_b(t + 1);
        }
      }
    }
    __syncwarp();
  } else if (t0 < t1) {
    const int qd = warp & 3, h = warp >> 2;
    const int chunk = blockIdx.x * 4 + qd;
    const int4 *xa = XYS ? reinterpret_cast<const int4 *>(dsm + oXY) + qd * kxy * FX_ROW + lane
                         : xy + (size_t)chunk * kxy * FX_ROW + lane;
    wait(abar, 0);
    long long fx = 0, fy = 0, fz = 0;
    for (int t = t0; t < t1; ++t) {
      const int b = (t - t0) & 1;
      const FxTile m = meta[t];
      const int ru = min(63, max(0, gsh[0] - (m.eu - 45 - m.sh))),
                rv = min(63, max(0, gsh[1] - (m.ev - 45 - m.sh)));
      int4 sl[2], xe[2], ye[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        sl[c] = slot[t * FX_TCOL + 2 * h + c];  // nx, Y row, sign of ny, weight of y
        xe[c] = xa[sl[c].x * FX_ROW];
        ye[c] = xa[sl[c].y * FX_ROW];
      }
      wait(mdone[b], (t - t0) >> 1);
      tc::fence_after_sync();
      __syncwarp();
      float v[FX_SL][8];
      const uint32_t ta =
          tbase + ((uint32_t)(32 * qd) << 16) + (uint32_t)(b * FX_SL * FX_TN + 8 * h);
#pragma unroll
      for (int s = 0; s < FX_SL; ++s) tc::tmem_ld8(ta + (uint32_t)(s * FX_TN), v[s]);
      tc::tmem_ld_wait();
#pragma unroll
      for (int s = 0; s < FX_SL; ++s) tc::pin8(v[s]);
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(tc::smem_addr(&afree[b]));
      long long sx = 0, sy = 0, sz = 0;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int4 X = xe[c], Y = ye[c];
        const W2 xr{X.x, X.y}, xi{X.z, X.w}, yr{Y.x, Y.y};
        const W2 yi{sl[c].z * Y.z, sl[c].z * Y.w};
        const W2 Tr = w2(dot2(xr, yr, xi, neg(yi), 0) << m.sh),
                 Ti = w2(dot2(xr, yi, xi, yr, 0) << m.sh);
        const W2 Ur = w2(fx_join<BIGK>(v, 4 * c)), Ui = w2(fx_join<BIGK>(v, 4 * c + 1));
        const W2 Vr = w2(fx_join<BIGK>(v, 4 * c + 2)), Vi = w2(fx_join<BIGK>(v, 4 * c + 3));
        const long long tu = dot2(Tr, Ui, Ti, Ur, 0);
        sx += tu * sl[c].x;
        sy += tu * sl[c].w;
        sz += dot2(Tr, Vi, Ti, Vr, 0);
      }
      const long long hu = half_m1(ru), hv = half_m1(rv);
      fx += shr_rne(sx, ru, hu);
      fy += shr_rne(sy, ru, hu);
      fz += shr_rne(sz, rv, hv);
    }
    // row = position pos(a) of atom a = 8 (lane % 4) + lane / 4 of the chunk
    const int i = chunk * 32 + 8 * (lane & 3) + (lane >> 2);
    if (i < n) {
      atomicAdd(&facc[i], (unsigned long long)fx);
      atomicAdd(&facc[n + i], (unsigned long long)fy);
      atomicAdd(&facc[2 * n + i], (unsigned long long)fz);
    }
  }
  tc::fence_before_sync();
  __syncthreads();  // every MMA waited for, every tensor-memory read done
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tbase, 512);
  }
  if (!ok) atomicOr(err, DERR_TIMEOUT);
}

// Force sums into G: unit 2^gexp, the charge scale and 2 PI / box.
__global__ void k_fx_fold(int n, const unsigned long long *__restrict__ facc,
                          const int *__restrict__ gexp, const double *__restrict__ qs,
                          const int *__restrict__ bad, double cx, double cy, double cz,
                          double *__restrict__ gx, double *__restrict__ gy,
                          double *__restrict__ gz) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double q = *bad ? __longlong_as_double(0x7ff8000000000000ll) : qs[0];
  const double u = ldexp(q, gexp[0]), v = ldexp(q, gexp[1]);
  gx[i] += (double)(long long)facc[i] * (u * cx);
  gy[i] += (double)(long long)facc[n + i] * (u * cy);
  gz[i] += (double)(long long)facc[2 * n + i] * (v * cz);
}

size_t fx_sfac_smem(int np, int kxy) {
  return 1024 + 2 * (size_t)FX_SL * 8192 + 2 * (size_t)FX_SL * np * 64 +
         2 * (size_t)kxy * FX_ROW * 16;
}
size_t fx_force_smem(int kp, int kxy, bool xys) {
  return 1024 + (size_t)(kp / 16) * FX_SL * (4096 + 2 * FX_TN * 32) +
         (xys ? 4 * (size_t)kxy * FX_ROW * 16 : 0);
}
auto fx_force_kernel(int kp, bool xys) {
  return kp > 48 ? (xys ? k_fx_force<true, true> : k_fx_force<false, true>)
                 : (xys ? k_fx_force<true, false> : k_fx_force<false, false>);
}
// Points of the circle, scale 2^61, as two-word numbers.  Formed once: on hosts
// whose long double is done in software the 512 cosines take half a millisecond.
const std::vector<int> &circle_points() {
  static const std::vector<int> points = [] {
    std::vector<int> c(4 * FX_CIRCLE);
    for (int k = 0; k < FX_CIRCLE; ++k) {
      const long double th = 6.283185307179586476925286766559005768L * k / FX_CIRCLE;
      const long double v[2] = {std::cos(th), std::sin(th)};
      for (int e = 0; e < 2; ++e) {
        const long long x = std::llrint(v[e] * 2305843009213693952.0L);
        const int lo = std::max((int)x, -0x7fffffff);  // it can be negated
        c[4 * k + 2 * e] = lo;
        c[4 * k + 2 * e + 1] = (int)((x - lo) >> 32);
      }
    }
    return c;
  }();
  return points;
}
int ceil_log2(int n) {
  int b = 0;
  while ((1ll << b) < n) ++b;
  return b;
}

}  // namespace

// The charge scale (a power of two above every |q|) for the tables, kept on
// the device so that captured graphs see the current one: after the topology
// upload and every RECINT.
static void fx_qscale(const mdx_ctx *ctx, double (&qs)[2]) {
  double m = 0.0;
  for (double q : ctx->h_q) m = std::max(m, std::fabs(q));
  int e = 0;
  if (m > 0.0) std::frexp(m, &e);  // m < 2^e
  qs[0] = std::ldexp(1.0, e);
  qs[1] = std::ldexp(1.0, -e);
}
int fx_update_qscale(mdx_ctx *ctx) {
  if (!ctx->dv.fx_qs) return MDX_OK;
  double qs[2];
  fx_qscale(ctx, qs);
  MDX_CUDA(ctx_copy(ctx->stream, ctx->dv.fx_qs, qs, sizeof qs, cudaMemcpyHostToDevice));
  return MDX_OK;
}

void fx_release(mdx_ctx *ctx) {
  DevData &d = ctx->dv;
  ctx_free(ctx, d.fx_buf);
  d.fx_buf = nullptr;
  d.fx_qs = nullptr;
  d.fx_on = false;
}

// Sizes, tables and buffers for a k-set (INIFUR).  The passes need K = 2 kz
// <= 64 (exact class sums, tensor memory) and their operands in shared
// memory: |nz| up to 31 and about 60 X and Y rows; other k-sets keep the
// FP64-pipe passes, and so does a system whose images the device has no room for.
// Returns MDX_OK with d.fx_on telling which.
int fx_setup(mdx_ctx *ctx, const std::vector<KCol> &cols) {
  DevData &d = ctx->dv;
  fx_release(ctx);
  const int kxy = d.kx + d.ky;
  const int kp = ((2 * d.kz + 15) / 16) * 16, np = kp;
  const int ncol = (int)cols.size();
  if (ncol == 0 || kp > FX_KMAX || fx_sfac_smem(np, kxy) > FX_SMEM_MAX) return MDX_OK;
  d.fx_xys = fx_force_smem(kp, kxy, true) <= FX_SMEM_MAX;
  if (fx_force_smem(kp, kxy, d.fx_xys) > FX_SMEM_MAX) return MDX_OK;
  const int nchunk = (d.n + 31) / 32, natile = (d.n + 127) / 128;
  // S pass: one wave of CTAs, (column tile, slice of chunks)
  d.fx_ntm = (ncol + 63) / 64;
  const int ns = std::max(1, ctx->nsm / d.fx_ntm);
  d.fx_cps = (nchunk + ns - 1) / ns;
  d.fx_ns = (nchunk + d.fx_cps - 1) / d.fx_cps;
  d.fx_ua = std::min(54, 61 - ceil_log2(32 * d.fx_cps));
  d.fx_ug = std::min(d.fx_ua, 62 - ceil_log2(d.n + 1));
  // F pass: columns by falling m, FX_TCOL to a tile
  const int ntile = (ncol + FX_TCOL - 1) / FX_TCOL;
  std::vector<int> order(ncol);
  for (int c = 0; c < ncol; ++c) order[c] = c;
  auto zmax = [&](int c) { return kcol_z(cols[c], cols[c].m); };
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return zmax(a) > zmax(b); });
  std::vector<int4> slot((size_t)ntile * FX_TCOL, make_int4(0, d.kx, 1, 0));
  std::vector<int> scol((size_t)ntile * FX_TCOL, -1), ks(ntile), cum(ntile + 1, 0);
  for (int s = 0; s < ncol; ++s) {
    const KCol &c = cols[order[s]];
    scol[s] = order[s];
    slot[s] = make_int4(c.nx, d.kx + std::abs(c.ny), c.ny < 0 ? -1 : 1,
                        ctx->p.icell == 2 ? 2 * c.ny + c.nx : c.ny);
  }
  // a tile's cost: its MMAs (448 cycles a K step) or its epilogue, whichever
  // is longer, about 2.2 K steps' worth
  for (int t = 0; t < ntile; ++t) {
    ks[t] = (2 * (zmax(order[(size_t)t * FX_TCOL]) + 1) + 15) / 16;
    cum[t + 1] = cum[t] + std::max(22, 10 * ks[t]);
  }
  // tile ranges: CTAs per 128 atoms so that the grid ends close to a whole
  // wave, a CTA's start-up counted as 3 tiles
  int best = 1;
  double best_t = 1e300;
  for (int s = 1; s <= std::min(ntile, 64); ++s) {
    const double waves = std::ceil((double)natile * s / ctx->nsm);
    const double tm = waves * (cum[ntile] / (double)s + 66.0);
    if (tm < 0.98 * best_t) {
      best_t = tm;
      best = s;
    }
  }
  d.fx_nsplit = best;
  std::vector<int> parts(best + 1, ntile);
  for (int p = 0, t = 0; p < best; ++p) {
    while (t < ntile && cum[t] < (long long)cum[ntile] * p / best) ++t;
    parts[p] = t;
  }
  parts[0] = 0;
  const size_t zsb = (size_t)nchunk * FX_SL * np * 64;
  const size_t zfb = (size_t)natile * (kp / 16) * FX_SL * 4096;
  const size_t xyb = sizeof(int4) * (size_t)natile * 4 * kxy * FX_ROW;
  const size_t accb = sizeof(long long) * (size_t)d.fx_ntm * np * 128;
  // One allocation, one upload and one clearing: an INIFUR of a small box is a few
  // dozen microseconds, and each allocation or copy waits for the stream.
  size_t len = 0;
  auto part = [&](size_t bytes) {
    const size_t o = len;
    len = (len + bytes + 255) & ~(size_t)255;
    return o;
  };
  // uploaded: charge scale and circle points, column slots, columns, K steps, ranges
  const size_t oqs = part(2 * sizeof(double) + FX_CIRCLE * sizeof(int4)),
               oslot = part(sizeof(int4) * slot.size()), oscol = part(sizeof(int) * scol.size()),
               oks = part(sizeof(int) * ks.size()), oparts = part(sizeof(int) * parts.size());
  const size_t up = len;
  // cleared: the sums and the flag behind them, which k_fx_form and k_fx_sfac leave
  // cleared; chunks past the last atom (a 128-atom tile's end) and the images' rows
  // past 2 kz, which stay zero
  const size_t oacc = part(accb + 16), oxy = part(xyb), ozs = part(zsb), ozf = part(zfb);
  const size_t clear = len;
  const size_t otw = part((size_t)ntile * (kp / 16) * FX_SL * FX_TN * 32),
               ometa = part(sizeof(FxTile) * ntile),
               ofacc = part(sizeof(long long) * 3 * d.n + 16);
  if (ctx_alloc(ctx, &d.fx_buf, len) != cudaSuccess) {
    d.fx_buf = nullptr;  // no room for the images (some 2 KB an atom): the FP64-pipe passes
    return MDX_OK;
  }
  unsigned char *const buf = d.fx_buf;
  d.fx_qs = reinterpret_cast<double *>(buf + oqs);
  d.fx_slot = reinterpret_cast<int4 *>(buf + oslot);
  d.fx_scol = reinterpret_cast<int *>(buf + oscol);
  d.fx_ks = reinterpret_cast<int *>(buf + oks);
  d.fx_parts = reinterpret_cast<int *>(buf + oparts);
  d.fx_acc = reinterpret_cast<unsigned long long *>(buf + oacc);
  d.fx_xy = reinterpret_cast<int4 *>(buf + oxy);
  d.fx_zs = buf + ozs;
  d.fx_zf = buf + ozf;
  d.fx_tw = buf + otw;
  d.fx_meta = buf + ometa;
  d.fx_facc = reinterpret_cast<unsigned long long *>(buf + ofacc);
  std::vector<unsigned char> host(up);
  auto put = [&](size_t o, const void *p, size_t bytes) { std::memcpy(host.data() + o, p, bytes); };
  const std::vector<int> &circle = circle_points();
  double qs[2];
  fx_qscale(ctx, qs);
  put(oqs, qs, sizeof qs);
  put(oqs + sizeof qs, circle.data(), sizeof(int) * circle.size());
  put(oslot, slot.data(), sizeof(int4) * slot.size());
  put(oscol, scol.data(), sizeof(int) * scol.size());
  put(oks, ks.data(), sizeof(int) * ks.size());
  put(oparts, parts.data(), sizeof(int) * parts.size());
  MDX_CUDA(cudaMemsetAsync(buf + up, 0, clear - up, ctx->stream));
  MDX_CUDA(ctx_copy(ctx->stream, buf, host.data(), up, cudaMemcpyHostToDevice));
  MDX_CUDA(raise_smem_limit(k_fx_sfac, fx_sfac_smem(np, kxy)));
  const size_t fsm = fx_force_smem(kp, kxy, d.fx_xys);
  MDX_CUDA(raise_smem_limit(fx_force_kernel(kp, d.fx_xys), fsm));
  d.fx_np = np;
  d.fx_ntile = ntile;
  d.fx_on = true;
  return MDX_OK;
}

// Phase tables, operand images and S(k) of the current positions.
int fx_tables_launch(mdx_ctx *ctx) {
  DevData &d = ctx->dv;
  FxBox box{};
  const double len[4] = {ctx->boxl, ctx->boyl, ctx->bozl, 2.0 * ctx->boyl};
  for (int a = 0; a < (ctx->p.icell == 2 ? 4 : 3); ++a) {
    box.ib[a] = 1.0 / len[a];
    box.ibl[a] = std::fma(-len[a], box.ib[a], 1.0) / len[a];
  }
  const size_t accb = sizeof(long long) * (size_t)d.fx_ntm * d.fx_np * 128;
  // behind the sums, the flag of a non-finite position
  int *bad = reinterpret_cast<int *>(reinterpret_cast<unsigned char *>(d.fx_acc) + accb);
  k_fx_tables<<<(d.n + 31) / 32, 128, sizeof(int4) * 33 * d.kz, ctx->stream>>>(
      d.n, d.pos, box, d.kx, d.ky, d.kz, d.fx_np, d.fx_np, d.fx_qs, d.fx_xy, d.fx_zs, d.fx_zf, d.fx_facc, bad,
      reinterpret_cast<const int4 *>(d.fx_qs + 2));
  MDX_LAUNCHED(ctx);
  return MDX_OK;
}

int fx_sfac_launch(mdx_ctx *ctx) {
  DevData &d = ctx->dv;
  const size_t accb = sizeof(long long) * (size_t)d.fx_ntm * d.fx_np * 128;
  int *bad = reinterpret_cast<int *>(reinterpret_cast<unsigned char *>(d.fx_acc) + accb);
  const int kxy = d.kx + d.ky;
  k_fx_sfac<<<dim3(d.fx_ntm, d.fx_ns), FX_THREADS, fx_sfac_smem(d.fx_np, kxy), ctx->stream>>>(
      (d.n + 31) / 32, d.fx_cps, d.ncol, d.fx_np, d.kx, kxy, d.fx_ua, d.fx_ug, d.cols, d.fx_xy,
      d.fx_zs, d.fx_acc, bad, d.err);
  MDX_LAUNCHED(ctx);
  k_fx_form<<<d.ncol, 32, 0, ctx->stream>>>(d.ncol, d.fx_np, d.fx_ug, d.cols, d.fx_acc, d.fx_qs,
                                            bad + 1, d.sk);
  MDX_LAUNCHED(ctx);
  return MDX_OK;
}

int fx_force_launch(mdx_ctx *ctx) {
  DevData &d = ctx->dv;
  const int kp = d.fx_np, kxy = d.kx + d.ky;
  FxTile *meta = reinterpret_cast<FxTile *>(d.fx_meta);
  int *gexp = reinterpret_cast<int *>(d.fx_facc + 3 * (size_t)d.n);
  k_fx_wtiles<<<d.fx_ntile, 256, sizeof(double) * FX_TN * kp, ctx->stream>>>(
      kp, d.fx_slot, d.fx_scol, d.fx_ks, d.cols, d.sk, d.kconst, d.fx_tw, meta,
      kterm_dst(ctx, d.fx_ntile));
  MDX_LAUNCHED(ctx);
  const dim3 grid((d.n + 127) / 128, d.fx_nsplit);
  const size_t sh = fx_force_smem(kp, kxy, d.fx_xys);
  auto kern = fx_force_kernel(kp, d.fx_xys);
  kern<<<grid, FX_THREADS, sh, ctx->stream>>>(d.n, d.fx_ntile, kp, kxy, d.fx_parts, meta,
                                              d.fx_slot, d.fx_tw, d.fx_zf, d.fx_xy, d.fx_facc,
                                              gexp, d.err);
  MDX_LAUNCHED(ctx);
  return MDX_OK;
}
// The force pass's sums into G.
int fx_fold_launch(mdx_ctx *ctx) {
  DevData &d = ctx->dv;
  const size_t accb = sizeof(long long) * (size_t)d.fx_ntm * d.fx_np * 128;
  const int *bad = reinterpret_cast<int *>(reinterpret_cast<unsigned char *>(d.fx_acc) + accb) + 1;
  const int *gexp = reinterpret_cast<int *>(d.fx_facc + 3 * (size_t)d.n);
  const double two = 2.0 * PI_REF;
  k_fx_fold<<<(d.n + 255) / 256, 256, 0, ctx->stream>>>(
      d.n, d.fx_facc, gexp, d.fx_qs, bad, two / ctx->boxl,
      (ctx->p.icell == 2 ? PI_REF : two) / ctx->boyl, two / ctx->bozl, d.gx, d.gy, d.gz);
  MDX_LAUNCHED(ctx);
  return MDX_OK;
}
