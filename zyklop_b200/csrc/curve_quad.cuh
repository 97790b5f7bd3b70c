// XYZZ group operations by a group of lanes: four lane roles hold X, Y, ZZ and
// ZZZ of a point (a quad); on G2 each role is two lanes, one per Fp component
// (eight lanes).
//
// A full addition is 14 products, which one thread runs one after the other.
// The four roles run them in four steps of one product each (14 of the 16
// role slots do useful work), with six exchanges between lanes.  That costs
// about a third more issue slots than one thread's addition and takes under a
// third of its latency, with a fraction of the point in each lane's
// registers: the right trade wherever additions form a dependent chain and
// the device is not full (bucket reductions, block trees, the later levels of
// the segmented reduction).
//
// Every lane of the warp must call these together (full-warp shuffles).
#pragma once
#include "curve.cuh"

namespace zk {

// What one lane holds of a coordinate in F.
template <class F>
struct lane_t {
  fp_t v;
};

template <class F>
constexpr int quad_shift() { return sizeof(F) == 64 ? 1 : 0; }  // log2 lanes per role
template <class F>
constexpr int quad_lanes() { return 4 << quad_shift<F>(); }
template <class F>
__device__ __forceinline__ int quad_lane() { return threadIdx.x & (quad_lanes<F>() - 1); }
template <class F>
__device__ __forceinline__ int quad_role() { return quad_lane<F>() >> quad_shift<F>(); }

// the same part of the coordinate of role (own role ^ mask) / of role `role`
template <class F>
__device__ __forceinline__ lane_t<F> quad_xor(const lane_t<F>& a, int mask) {
  lane_t<F> r;
#pragma unroll
  for (int i = 0; i < 8; i++)
    r.v.v[i] = __shfl_xor_sync(0xffffffffu, a.v.v[i], mask << quad_shift<F>());
  return r;
}
template <class F>
__device__ __forceinline__ lane_t<F> quad_get(const lane_t<F>& a, int role) {
  const int src = (role << quad_shift<F>()) | (quad_lane<F>() & (quad_shift<F>() ? 1 : 0));
  lane_t<F> r;
#pragma unroll
  for (int i = 0; i < 8; i++)
    r.v.v[i] = __shfl_sync(0xffffffffu, a.v.v[i], src, quad_lanes<F>());
  return r;
}
// whether role `role`'s coordinate is zero, in every lane of the group
template <class F>
__device__ __forceinline__ bool quad_zero(const lane_t<F>& a, int role) {
  int z = fe_is_zero(a.v);
  if (quad_shift<F>()) z &= __shfl_xor_sync(0xffffffffu, z, 1);
  return __shfl_sync(0xffffffffu, z, role << quad_shift<F>(), quad_lanes<F>()) != 0;
}

template <class F>
__device__ __forceinline__ lane_t<F> operator+(const lane_t<F>& a, const lane_t<F>& b) {
  return {a.v + b.v};
}
template <class F>
__device__ __forceinline__ lane_t<F> operator-(const lane_t<F>& a, const lane_t<F>& b) {
  return {a.v - b.v};
}
template <class F>
__device__ __forceinline__ lane_t<F> fe_dbl(const lane_t<F>& a) { return {a.v + a.v}; }
template <class F>
__device__ __forceinline__ lane_t<F> quad_sel(bool c, const lane_t<F>& a, const lane_t<F>& b) {
  lane_t<F> r;
#pragma unroll
  for (int i = 0; i < 8; i++) r.v.v[i] = c ? a.v.v[i] : b.v.v[i];
  return r;
}
template <class F>
__device__ __forceinline__ lane_t<F> quad_inf() { return {fe_zero<FpCfg>()}; }

// One component of an Fp2 product per lane of a pair: c0 = a0 b0 - a1 b1 and
// c1 = a1 b0 + a0 b1, each with one reduction.  With (a, b) the lane's parts
// and (ao, bo) its partner's, the first product is a b0 and the second
// ao b1, subtracted from p^2 for c0: both sums are below 2 p^2.
static __device__ __noinline__ fp_t fp2_lane_mul_call(fp_t a, fp_t b) {
  const bool c1 = threadIdx.x & 1;
  fp_t ao, b0, b1;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    ao.v[i] = __shfl_xor_sync(0xffffffffu, a.v[i], 1);
    const uint32_t bo = __shfl_xor_sync(0xffffffffu, b.v[i], 1);
    b0.v[i] = c1 ? bo : b.v[i];
    b1.v[i] = c1 ? b.v[i] : bo;
  }
  uint32_t x[16], w[16], y[16];
  fe_mul_wide(ao.v, b1.v, w);
  // the second term: w for c1, p^2 - w for c0
#pragma unroll
  for (int i = 0; i < 16; i++) x[i] = 0;
  add_16_psq(x, y);
  sub_16(y, w);
#pragma unroll
  for (int i = 0; i < 16; i++) x[i] = c1 ? w[i] : y[i];
  fe_mul_wide(a.v, b0.v, w);
  add_16(x, w);
  return fe_redc<FpCfg>(x);
}
__device__ __forceinline__ lane_t<fp_t> operator*(const lane_t<fp_t>& a, const lane_t<fp_t>& b) {
  return {a.v * b.v};
}
__device__ __forceinline__ lane_t<fp2_t> operator*(const lane_t<fp2_t>& a, const lane_t<fp2_t>& b) {
  return {fp2_lane_mul_call(a.v, b.v)};
}

// dbl-2008-s-1; ZZ = 0 stays 0
template <class F>
__device__ __forceinline__ lane_t<F> quad_dbl(const lane_t<F>& p) {
  const int role = quad_role<F>();
  const lane_t<F> a = quad_sel(role == 1, fe_dbl(p), p);  // X, U = 2Y, ZZ, ZZZ
  const lane_t<F> t = a * a;                              // X^2, V = U^2
  const lane_t<F> m = fe_dbl(t) + t;                      // role 0: M = 3 X^2
  const lane_t<F> s = a * quad_get(t, 1);  // S = X V, W = U V, ZZ3 = ZZ V, ZZZ V
  const lane_t<F> u = quad_get(a, 1);
  // M^2, W Y, -, ZZZ3 = ZZZ V U
  const lane_t<F> z = quad_sel(role == 0, m, s) * quad_sel(role == 0, m, quad_sel(role == 1, p, u));
  const lane_t<F> x3 = z - fe_dbl(s);
  const lane_t<F> y3 = quad_get(m * (s - x3), 0) - z;  // role 0: M (S - X3)
  return quad_sel(role == 0, x3, quad_sel(role == 1, y3, quad_sel(role == 2, s, z)));
}

// add-2008-s, with the cases of infinity and equal points.  A warp whose every
// addition has an operand at infinity skips the products: empty buckets (zero,
// few or short scalars) are most of a reduction's operands then, and their
// additions would be a product chain each.  Zero scalars, G2, 700001 points: 1.07 ms
// without the vote, 0.19 with it.
template <class F>
__device__ __forceinline__ lane_t<F> quad_add(const lane_t<F>& p, const lane_t<F>& q) {
  const int role = quad_role<F>();
  const bool lo = role < 2;
  const bool pinf = quad_zero(p, 2), qinf = quad_zero(q, 2);
  if (!__any_sync(0xffffffffu, !pinf && !qinf)) return quad_sel(pinf, q, p);
  const lane_t<F> m = p * quad_xor(q, 2);  // U1 = X1 ZZ2, S1 = Y1 ZZZ2, U2 = X2 ZZ1, S2 = Y2 ZZZ1
  const lane_t<F> n = quad_xor(m, 2);
  const lane_t<F> d = quad_sel(lo, n, m) - quad_sel(lo, m, n);  // P, R, P, R
  const bool zp = quad_zero(d, 0), zr = quad_zero(d, 1);
  const lane_t<F> t = quad_sel(lo, d, p) * quad_sel(lo, d, q);  // PP, R^2, ZZ1 ZZ2, ZZZ1 ZZZ2
  const lane_t<F> pp = quad_get(t, 0);
  const lane_t<F> e = quad_xor(d, 1);  // R, P, R, P
  // Q = U1 PP, PPP, ZZ3, PPP
  const lane_t<F> u = quad_sel(role == 0, m, quad_sel(role == 2, t, e)) * pp;
  const lane_t<F> w = quad_sel(role == 1, t - u, u);  // Q, R^2 - PPP
  const lane_t<F> x = quad_xor(w, 1);
  const lane_t<F> qq = quad_sel(role == 0, u, x);
  const lane_t<F> x3 = quad_sel(role == 0, x, w) - fe_dbl(qq);  // roles 0 and 1
  // R (Q - X3), S1 PPP, -, ZZZ3
  const lane_t<F> z =
      quad_sel(role == 0, e, quad_sel(role == 1, m, t)) * quad_sel(role == 0, qq - x3, u);
  const lane_t<F> y3 = quad_xor(z, 1) - z;
  lane_t<F> r = quad_sel(role == 0, x3, quad_sel(role == 1, y3, quad_sel(role == 2, u, z)));
  const bool same = zp && !pinf && !qinf;
  if (__any_sync(0xffffffffu, same)) {
    const lane_t<F> dbl = quad_dbl(p);
    if (same) r = quad_sel(zr, dbl, quad_inf<F>());
  }
  return quad_sel(pinf, q, quad_sel(qinf, p, r));
}

// the lane's part of a stored point (the lanes of a group read it whole)
template <class F>
__device__ __forceinline__ lane_t<F> quad_ld(const xyzz<F>* p) {
  return {ld_pod(reinterpret_cast<const fp_t*>(p) + quad_lane<F>())};
}
template <class F>
__device__ __forceinline__ void quad_st(xyzz<F>* p, const lane_t<F>& a) {
  st_pod(reinterpret_cast<fp_t*>(p) + quad_lane<F>(), a.v);
}

}  // namespace zk
