// Modular inversion by division steps (Bernstein and Yang, "Fast constant-time
// gcd computation and modular inversion", CHES 2019), on 30-bit signed limbs.
//
// A divstep on (delta, f, g) with f odd is
//   delta > 0, g odd:  (1 - delta, g, (g - f) / 2)
//   otherwise:         (1 + delta, f, (g + (g mod 2) f) / 2)
// and starting from (1, m, x) it ends at g = 0, f = +-1 for x coprime to m.
// Thirty steps depend only on the low 30 bits of f and g and form a 2 x 2
// integer matrix with rows of absolute sum at most 2^30; the matrix is then
// applied to the full f and g (exact division by 2^30) and to the cofactors
// d and e (f = d x and g = e x mod m, division by 2^30 mod m).
//
// Range of the cofactors: |u d + v e| <= 2^30 max(|d|, |e|), and the multiple
// of m that makes it divisible by 2^30 is at most 2^29 m in size, so a batch
// adds at most m / 2 to the largest cofactor.  The paper's bound for inputs
// below 2^256 is 741 steps, so 25 batches end every input with |d| < 14 m,
// far inside nine 30-bit limbs; no correction is needed before the end.
//
// Plain integer C++: the same code runs on the host, where a CPU test checks
// it against big-integer inverses.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define ZK_HD __host__ __device__ __forceinline__
#else
#define ZK_HD inline
#endif
#ifdef __CUDA_ARCH__
#define ZK_UNROLL _Pragma("unroll")
#else
#define ZK_UNROLL
#endif

namespace zk {

constexpr int kInvLimbs = 9;
constexpr int32_t kInvMask = (1 << 30) - 1;
constexpr int kInvBatches = 25;

ZK_HD int inv_ctz(uint32_t x) {
#ifdef __CUDA_ARCH__
  return __clz(__brev(x));
#else
  return __builtin_ctz(x);
#endif
}

// 30 divsteps on the low words of f and g; t = {u, v, q, r} with
// 2^30 (f', g') = (u f + v g, q f + r g).
ZK_HD void inv_batch(int32_t& delta, uint32_t f, uint32_t g, int32_t t[4]) {
  int32_t u = 1, v = 0, q = 0, r = 1, left = 30, dl = delta;
  for (;;) {
    // runs of even g: halve g, double f's row
    const int z = inv_ctz(g | (1u << left));
    g >>= z;
    u = (int32_t)((uint32_t)u << z);
    v = (int32_t)((uint32_t)v << z);
    dl += z;
    left -= z;
    if (left == 0) break;
    const bool swap = dl > 0;
    const uint32_t nf = swap ? g : f, ng = swap ? 0u - f : g;
    const int32_t nu = swap ? q : u, nq = swap ? -u : q;
    const int32_t nv = swap ? r : v, nr = swap ? -v : r;
    dl = swap ? -dl : dl;
    f = nf;
    u = nu;
    v = nv;
    g = ng + f;  // even; the next round halves it
    q = nq + u;
    r = nr + v;
  }
  delta = dl;
  t[0] = u;
  t[1] = v;
  t[2] = q;
  t[3] = r;
}

// (f, g) = (u f + v g, q f + r g) / 2^30, exactly
ZK_HD void inv_apply_fg(int32_t f[kInvLimbs], int32_t g[kInvLimbs], const int32_t t[4]) {
  const int64_t u = t[0], v = t[1], q = t[2], r = t[3];
  int64_t cf = u * f[0] + v * g[0], cg = q * f[0] + r * g[0];
  cf >>= 30;
  cg >>= 30;
  ZK_UNROLL
  for (int i = 1; i < kInvLimbs; i++) {
    const int32_t fi = f[i], gi = g[i];
    cf += u * fi + v * gi;
    cg += q * fi + r * gi;
    f[i - 1] = (int32_t)cf & kInvMask;
    g[i - 1] = (int32_t)cg & kInvMask;
    cf >>= 30;
    cg >>= 30;
  }
  f[kInvLimbs - 1] = (int32_t)cf;
  g[kInvLimbs - 1] = (int32_t)cg;
}

// (d, e) = (u d + v e, q d + r e) / 2^30 mod m: the multiple of m (between
// -2^29 and 2^29) that clears the low 30 bits is added first
ZK_HD void inv_apply_de(int32_t d[kInvLimbs], int32_t e[kInvLimbs], const int32_t t[4],
                        const int32_t m[kInvLimbs], uint32_t neg_inv30) {
  const int64_t u = t[0], v = t[1], q = t[2], r = t[3];
  int64_t cd = u * d[0] + v * e[0], ce = q * d[0] + r * e[0];
  // sign-extended 30-bit values of -c m^-1 mod 2^30
  const int64_t kd = (int32_t)(((uint32_t)cd * neg_inv30) << 2) >> 2;
  const int64_t ke = (int32_t)(((uint32_t)ce * neg_inv30) << 2) >> 2;
  cd = (cd + kd * m[0]) >> 30;
  ce = (ce + ke * m[0]) >> 30;
  ZK_UNROLL
  for (int i = 1; i < kInvLimbs; i++) {
    const int32_t di = d[i], ei = e[i];
    cd += u * di + v * ei + kd * m[i];
    ce += q * di + r * ei + ke * m[i];
    d[i - 1] = (int32_t)cd & kInvMask;
    e[i - 1] = (int32_t)ce & kInvMask;
    cd >>= 30;
    ce >>= 30;
  }
  d[kInvLimbs - 1] = (int32_t)cd;
  e[kInvLimbs - 1] = (int32_t)ce;
}

// limb i (30 bits) of a 256-bit value in 8 words
ZK_HD int32_t inv_limb(const uint32_t w[8], int i) {
  const int bit = 30 * i, k = bit >> 5, s = bit & 31;
  uint32_t x = w[k] >> s;
  if (s > 2 && k < 7) x |= w[k + 1] << (32 - s);
  return (int32_t)(x & (uint32_t)kInvMask);
}

// out = x^-1 mod m in [0, m) for any 256-bit x (a multiple of m gives 0), m an
// odd prime below 2^254 whose low 30 bits are neither 1 nor 2^30 - 1,
// neg_inv30 = -m^-1 mod 2^30.  Plain values, no Montgomery factor.
ZK_HD void inv_divsteps(const uint32_t x[8], const uint32_t mw[8], uint32_t neg_inv30,
                        uint32_t out[8]) {
  int32_t m[kInvLimbs], f[kInvLimbs], g[kInvLimbs], d[kInvLimbs], e[kInvLimbs];
  ZK_UNROLL
  for (int i = 0; i < kInvLimbs; i++) {
    m[i] = f[i] = inv_limb(mw, i);
    g[i] = inv_limb(x, i);
    d[i] = 0;
    e[i] = i == 0;
  }
  int32_t delta = 1;
  for (int it = 0; it < kInvBatches; it++) {
    int32_t t[4];
    const uint32_t f0 = (uint32_t)f[0] | ((uint32_t)f[1] << 30);
    const uint32_t g0 = (uint32_t)g[0] | ((uint32_t)g[1] << 30);
    inv_batch(delta, f0, g0, t);
    inv_apply_de(d, e, t, m, neg_inv30);
    inv_apply_fg(f, g, t);
    int32_t any = 0;
    ZK_UNROLL
    for (int i = 0; i < kInvLimbs; i++) any |= g[i];
    if (!any) break;
  }
  // f = +-1, or +-m for a multiple of m
  const bool unit = f[0] == 1 || f[0] == kInvMask;
  // x^-1 = sign(f) d; then into [0, m): |d| < 14 m, so d + 16 m is positive
  // and five conditional subtractions of 16 m .. m finish
  const int32_t neg = f[kInvLimbs - 1] >> 31;  // -1 when f = -1
  int64_t c = 0;
  ZK_UNROLL
  for (int i = 0; i < kInvLimbs; i++) {
    c += (int64_t)((d[i] ^ neg) - neg) + ((int64_t)m[i] << 4);
    d[i] = i < kInvLimbs - 1 ? ((int32_t)c & kInvMask) : (int32_t)c;
    c >>= 30;
  }
  ZK_UNROLL
  for (int k = 4; k >= 0; k--) {
    int32_t s[kInvLimbs];
    int64_t b = 0;
    ZK_UNROLL
    for (int i = 0; i < kInvLimbs; i++) {
      b += (int64_t)d[i] - ((int64_t)m[i] << k);
      s[i] = i < kInvLimbs - 1 ? ((int32_t)b & kInvMask) : (int32_t)b;
      b >>= 30;
    }
    const bool keep = s[kInvLimbs - 1] < 0;
    ZK_UNROLL
    for (int i = 0; i < kInvLimbs; i++) d[i] = keep ? d[i] : s[i];
  }
  ZK_UNROLL
  for (int k = 0; k < 8; k++) {
    const int bit = 32 * k, i = bit / 30, s = bit - 30 * i;
    uint64_t v = (uint64_t)(uint32_t)d[i] >> s;
    v |= (uint64_t)(uint32_t)d[i + 1] << (30 - s);
    if (i + 2 < kInvLimbs) v |= (uint64_t)(uint32_t)d[i + 2] << (60 - s);
    out[k] = unit ? (uint32_t)v : 0u;
  }
}

}  // namespace zk
