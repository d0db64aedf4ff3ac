// ewald_ops.cuh -- pieces shared by the reciprocal-Ewald files.
#pragma once
#include "mdx_internal.cuh"
#include "tc_ptx.cuh"

// One k-vector's energy and virial terms (forces.f:1316-1331) from its
// constants {AKC, RXV^2 AKV, RYV^2 AKV, RZV^2 AKV, RZV} and |S|^2.  Sums: QPE,
// then the virials with QPE in them; the caller copies QPE to the fifth.
__device__ __forceinline__ void kterm_add(double (&acc)[5], const double *__restrict__ q,
                                          double S2) {
  const double Q = q[0] * S2;
  acc[0] += Q;
  acc[1] += Q - q[1] * S2;
  acc[2] += Q - q[2] * S2;
  acc[3] += Q - q[3] * S2;
}
// W = 2 AKC conj(S) and RZV W of a k-vector, its terms added to acc.
__device__ __forceinline__ dbl4 kterm(double2 S, const double *__restrict__ q,
                                      double (&acc)[5]) {
  kterm_add(acc, q, S.y * S.y + S.x * S.x);
  const double AK2 = 2.0 * q[0];
  dbl4 W;
  W.x = AK2 * S.x;
  W.y = -AK2 * S.y;
  W.z = q[4] * W.x;
  W.w = q[4] * W.y;
  return W;
}
inline Dst6 kterm_dst(const mdx_ctx *ctx, int nblocks) {
  double *k = ctx->dv.red + KT0;
  return dst6(ctx, nblocks, 5, k, k + 1, k + 2, k + 3, k + 4);
}

// Force-pass operand layout of the mixed tensor-core pass (128 rows, K-major,
// unswizzled), K-step major: the 8 K of MMA step s = k / 8 fill 8 KB, [hi | lo]
// of 4 KB each, and within a part core matrix (r / 8, k / 4) of 128 bytes sits
// at ((k / 4) % 2) 2048 + (r / 8) 128: LBO (along K) = 2048, SBO (along M/N) =
// 128.  A tile whose columns need ks steps is then its first ks x 8 KB.
constexpr uint32_t TC_STEP = 8192;  // bytes of one K step (hi and lo)
constexpr uint32_t TC_LO = 4096;    // lo part within a step
constexpr uint32_t TC_LBO = 2048, TC_SBO = 128;
__host__ __device__ __forceinline__ uint32_t core_off(int r, int k) {  // hi part
  return (uint32_t)((k >> 3) * TC_STEP + ((k >> 2) & 1) * TC_LBO + (r >> 3) * TC_SBO +
                    ((r & 7) << 4) + ((k & 3) << 2));
}
// Z(p) of atom i into the force pass's A image (per 128-atom tile kp / 8 K
// steps of [hi | lo]; entries with p >= kz stay zero, set once).
__device__ __forceinline__ void tc_zimage_store(unsigned char *__restrict__ zf, int kp, int p,
                                                int i, float2 z) {
  float ah, al, bh, bl;
  tc::tf32_split(z.x, ah, al);
  tc::tf32_split(z.y, bh, bl);
  unsigned char *base = zf + (size_t)(i >> 7) * 1024 * kp;
  const uint32_t o = core_off(i & 127, 2 * p);  // k = 2p and 2p + 1: adjacent
  *reinterpret_cast<float2 *>(base + o) = make_float2(ah, bh);
  *reinterpret_cast<float2 *>(base + TC_LO + o) = make_float2(al, bl);
}
