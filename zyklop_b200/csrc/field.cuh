// BN254 base field Fp and scalar field Fr on sm_100a.
//
// Elements are 8 x 32-bit little-endian limbs in Montgomery form with
// R = 2^256 — the same bytes as the reference's 4 x u64 limbs
// (include/fp_bn254.cuh:52-59, include/fr_bn254.cuh:40-49), so buffers cross
// the API unchanged.  Values are kept fully reduced in [0, m).
//
// Multiplication is separated Montgomery with 32-bit limbs: the 512-bit
// product first (schoolbook, 64 multiply pairs), then eight reduction rows
// against the modulus, whose limbs are PTX immediates, fold the low half and
// the high half is added at the end.  Every sum of limb products is kept in
// two accumulators by the parity of the limb position, so that each
// mad.lo/madc.hi pair is one aligned 64-bit multiply-add.  The unreduced
// products also enter sums of products with one reduction (Fp2 products,
// differences).  Both BN254 moduli are below 2^254, which bounds
// every intermediate (derivations at the functions).  The products are
// bit-identical to the reference's 4 x u64 CIOS fpMul / frMul
// (include/fp_bn254.cuh:187-277, include/fr_bn254.cuh:173-210): both return
// the unique a*b*R^-1 mod m in [0, m).
#pragma once
#include <cstdint>

#include "field_inv.cuh"

namespace zk {

struct FpCfg {
  static constexpr uint32_t P0 = 0xd87cfd47u, P1 = 0x3c208c16u, P2 = 0x6871ca8du, P3 = 0x97816a91u,
                            P4 = 0x8181585du, P5 = 0xb85045b6u, P6 = 0xe131a029u, P7 = 0x30644e72u;
  static constexpr uint32_t INV = 0xe4866389u;  // -p^-1 mod 2^32
  static constexpr uint32_t ONE[8] = {0xc58f0d9du, 0xd35d438du, 0xf5c70b3du, 0x0a78eb28u,
                                      0x7879462cu, 0x666ea36fu, 0x9a07df2fu, 0x0e0a77c1u};
  static constexpr uint32_t R2[8] = {0x538afa89u, 0xf32cfc5bu, 0xd44501fbu, 0xb5e71911u,
                                     0x0a417ff6u, 0x47ab1effu, 0xcab8351fu, 0x06d89f71u};
  static constexpr uint32_t R3[8] = {0xda1530dfu, 0xb1cd6dafu, 0xa7283db6u, 0x62f210e6u,
                                     0x0ada0afbu, 0xef7f0b0cu, 0x2d592544u, 0x20fd6e90u};
};

struct FrCfg {
  static constexpr uint32_t P0 = 0xf0000001u, P1 = 0x43e1f593u, P2 = 0x79b97091u, P3 = 0x2833e848u,
                            P4 = 0x8181585du, P5 = 0xb85045b6u, P6 = 0xe131a029u, P7 = 0x30644e72u;
  static constexpr uint32_t INV = 0xefffffffu;
  static constexpr uint32_t ONE[8] = {0x4ffffffbu, 0xac96341cu, 0x9f60cd29u, 0x36fc7695u,
                                      0x7879462eu, 0x666ea36fu, 0x9a07df2fu, 0x0e0a77c1u};
  static constexpr uint32_t R2[8] = {0xae216da7u, 0x1bb8e645u, 0xe35c59e3u, 0x53fe3ab1u,
                                     0x53bb8085u, 0x8c49833du, 0x7f4e44a5u, 0x0216d0b1u};
  static constexpr uint32_t R3[8] = {0xb4bf0040u, 0x5e94d8e1u, 0x1cfbb6b8u, 0x2a489cbeu,
                                     0xa19fcfedu, 0x893cc664u, 0x7fcc657cu, 0x0cf8594bu};
};

template <class C>
struct fe {
  uint32_t v[8];
};

using fp_t = fe<FpCfg>;
using fr_t = fe<FrCfg>;

// ------------------------------------------------------------------ loads
template <class C>
__device__ __forceinline__ fe<C> fe_load(const void* base, size_t idx) {
  const uint4* p = reinterpret_cast<const uint4*>(base) + 2 * idx;
  uint4 a = p[0], b = p[1];
  return fe<C>{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
}
template <class C>
__device__ __forceinline__ fe<C> fe_ldg(const void* base, size_t idx) {
  const uint4* p = reinterpret_cast<const uint4*>(base) + 2 * idx;
  uint4 a = __ldg(p), b = __ldg(p + 1);
  return fe<C>{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
}
template <class C>
__device__ __forceinline__ void fe_store(void* base, size_t idx, const fe<C>& x) {
  uint4* p = reinterpret_cast<uint4*>(base) + 2 * idx;
  p[0] = make_uint4(x.v[0], x.v[1], x.v[2], x.v[3]);
  p[1] = make_uint4(x.v[4], x.v[5], x.v[6], x.v[7]);
}

template <class C>
__device__ __forceinline__ fe<C> fe_zero() {
  return fe<C>{{0, 0, 0, 0, 0, 0, 0, 0}};
}
template <class C>
__device__ __forceinline__ fe<C> fe_one() {
  return fe<C>{{C::ONE[0], C::ONE[1], C::ONE[2], C::ONE[3], C::ONE[4], C::ONE[5], C::ONE[6], C::ONE[7]}};
}
template <class C>
__device__ __forceinline__ bool fe_is_zero(const fe<C>& a) {
  return (a.v[0] | a.v[1] | a.v[2] | a.v[3] | a.v[4] | a.v[5] | a.v[6] | a.v[7]) == 0;
}
template <class C>
__device__ __forceinline__ bool fe_eq(const fe<C>& a, const fe<C>& b) {
  uint32_t d = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) d |= a.v[i] ^ b.v[i];
  return d == 0;
}

// ------------------------------------------------------------- reduction
// r = t - m if t >= m else t  (t < 2m)
template <class C>
__device__ __forceinline__ void fe_reduce_once(uint32_t* t) {
  uint32_t s0, s1, s2, s3, s4, s5, s6, s7, bw;
  asm("sub.cc.u32  %0, %9, %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32    %8, 0, 0;"
      : "=r"(s0), "=r"(s1), "=r"(s2), "=r"(s3), "=r"(s4), "=r"(s5), "=r"(s6), "=r"(s7), "=r"(bw)
      : "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]), "r"(t[5]), "r"(t[6]), "r"(t[7]),
        "n"(C::P0), "n"(C::P1), "n"(C::P2), "n"(C::P3), "n"(C::P4), "n"(C::P5), "n"(C::P6), "n"(C::P7));
  // bw == 0xffffffff when t < m (keep t)
  t[0] = bw ? t[0] : s0;
  t[1] = bw ? t[1] : s1;
  t[2] = bw ? t[2] : s2;
  t[3] = bw ? t[3] : s3;
  t[4] = bw ? t[4] : s4;
  t[5] = bw ? t[5] : s5;
  t[6] = bw ? t[6] : s6;
  t[7] = bw ? t[7] : s7;
}

// ---------------------------------------------------------------- add/sub
template <class C>
__device__ __forceinline__ fe<C> operator+(const fe<C>& a, const fe<C>& b) {
  fe<C> r;
  asm("add.cc.u32  %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]),
        "=r"(r.v[6]), "=r"(r.v[7])
      : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]),
        "r"(a.v[7]), "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]),
        "r"(b.v[6]), "r"(b.v[7]));
  fe_reduce_once<C>(r.v);
  return r;
}

template <class C>
__device__ __forceinline__ fe<C> operator-(const fe<C>& a, const fe<C>& b) {
  fe<C> r;
  uint32_t bw;
  asm("sub.cc.u32  %0, %9, %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32    %8, 0, 0;"
      : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]),
        "=r"(r.v[6]), "=r"(r.v[7]), "=r"(bw)
      : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]),
        "r"(a.v[7]), "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]),
        "r"(b.v[6]), "r"(b.v[7]));
  // add m back when the subtraction borrowed
  asm("add.cc.u32  %0, %0, %8;\n\t"
      "addc.cc.u32 %1, %1, %9;\n\t"
      "addc.cc.u32 %2, %2, %10;\n\t"
      "addc.cc.u32 %3, %3, %11;\n\t"
      "addc.cc.u32 %4, %4, %12;\n\t"
      "addc.cc.u32 %5, %5, %13;\n\t"
      "addc.cc.u32 %6, %6, %14;\n\t"
      "addc.u32    %7, %7, %15;"
      : "+r"(r.v[0]), "+r"(r.v[1]), "+r"(r.v[2]), "+r"(r.v[3]), "+r"(r.v[4]), "+r"(r.v[5]),
        "+r"(r.v[6]), "+r"(r.v[7])
      : "r"(bw & C::P0), "r"(bw & C::P1), "r"(bw & C::P2), "r"(bw & C::P3), "r"(bw & C::P4),
        "r"(bw & C::P5), "r"(bw & C::P6), "r"(bw & C::P7));
  return r;
}

template <class C>
__device__ __forceinline__ fe<C> fe_neg(const fe<C>& a) {
  return fe_zero<C>() - a;
}

template <class C>
__device__ __forceinline__ fe<C> fe_dbl(const fe<C>& a) {
  return a + a;
}

// ------------------------------------------------------------------- mul
// Multiply-add chains on aligned word pairs.  A pair mad.lo.cc / madc.hi.cc
// on an even-odd pair of accumulator words is one 64-bit multiply-add with
// carry in the machine, at a quarter of the simple instructions' rate; pairs
// that straddle the alignment cost moves or two instructions.  So every sum
// of limb products keeps two accumulators: one for products whose position is
// even, one for odd positions (stored a word lower), and adds them up at the
// end.
//
// e[0..7] += (x0, x1, x2, x3 at words 0, 2, 4, 6) * y; the carry joins c.
__device__ __forceinline__ void mac4(uint32_t* e, uint32_t& c, uint32_t x0, uint32_t x1,
                                     uint32_t x2, uint32_t x3, uint32_t y) {
  asm("mad.lo.cc.u32  %0, %9, %13, %0;\n\t"
      "madc.hi.cc.u32 %1, %9, %13, %1;\n\t"
      "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
      "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
      "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
      "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
      "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
      "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
      "addc.u32       %8, %8, 0;"
      : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]),
        "+r"(e[7]), "+r"(c)
      : "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(y));
}
// the same where no carry can leave word 7
__device__ __forceinline__ void mac4_top(uint32_t* e, uint32_t x0, uint32_t x1, uint32_t x2,
                                         uint32_t x3, uint32_t y) {
  asm("mad.lo.cc.u32  %0, %8, %12, %0;\n\t"
      "madc.hi.cc.u32 %1, %8, %12, %1;\n\t"
      "madc.lo.cc.u32 %2, %9, %12, %2;\n\t"
      "madc.hi.cc.u32 %3, %9, %12, %3;\n\t"
      "madc.lo.cc.u32 %4, %10, %12, %4;\n\t"
      "madc.hi.cc.u32 %5, %10, %12, %5;\n\t"
      "madc.lo.cc.u32 %6, %11, %12, %6;\n\t"
      "madc.hi.u32    %7, %11, %12, %7;"
      : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]),
        "+r"(e[7])
      : "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(y));
}
// shorter rows of the same
__device__ __forceinline__ void mac3(uint32_t* e, uint32_t& c, uint32_t x0, uint32_t x1, uint32_t x2, uint32_t y) {
  asm("mad.lo.cc.u32  %0, %7, %10, %0;\n\t"
      "madc.hi.cc.u32 %1, %7, %10, %1;\n\t"
      "madc.lo.cc.u32 %2, %8, %10, %2;\n\t"
      "madc.hi.cc.u32 %3, %8, %10, %3;\n\t"
      "madc.lo.cc.u32 %4, %9, %10, %4;\n\t"
      "madc.hi.cc.u32 %5, %9, %10, %5;\n\t"
      "addc.u32       %6, %6, 0;"
      : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(c)
      : "r"(x0), "r"(x1), "r"(x2), "r"(y));
}
__device__ __forceinline__ void mac3_top(uint32_t* e, uint32_t x0, uint32_t x1, uint32_t x2, uint32_t y) {
  asm("mad.lo.cc.u32  %0, %6, %9, %0;\n\t"
      "madc.hi.cc.u32 %1, %6, %9, %1;\n\t"
      "madc.lo.cc.u32 %2, %7, %9, %2;\n\t"
      "madc.hi.cc.u32 %3, %7, %9, %3;\n\t"
      "madc.lo.cc.u32 %4, %8, %9, %4;\n\t"
      "madc.hi.u32    %5, %8, %9, %5;"
      : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5])
      : "r"(x0), "r"(x1), "r"(x2), "r"(y));
}
__device__ __forceinline__ void mac2(uint32_t* e, uint32_t& c, uint32_t x0, uint32_t x1, uint32_t y) {
  asm("mad.lo.cc.u32  %0, %5, %7, %0;\n\t"
      "madc.hi.cc.u32 %1, %5, %7, %1;\n\t"
      "madc.lo.cc.u32 %2, %6, %7, %2;\n\t"
      "madc.hi.cc.u32 %3, %6, %7, %3;\n\t"
      "addc.u32       %4, %4, 0;"
      : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(c)
      : "r"(x0), "r"(x1), "r"(y));
}
__device__ __forceinline__ void mac2_top(uint32_t* e, uint32_t x0, uint32_t x1, uint32_t y) {
  asm("mad.lo.cc.u32  %0, %4, %6, %0;\n\t"
      "madc.hi.cc.u32 %1, %4, %6, %1;\n\t"
      "madc.lo.cc.u32 %2, %5, %6, %2;\n\t"
      "madc.hi.u32    %3, %5, %6, %3;"
      : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3])
      : "r"(x0), "r"(x1), "r"(y));
}
__device__ __forceinline__ void mac1(uint32_t* e, uint32_t& c, uint32_t x0, uint32_t y) {
  asm("mad.lo.cc.u32  %0, %3, %4, %0;\n\t"
      "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
      "addc.u32       %2, %2, 0;"
      : "+r"(e[0]), "+r"(e[1]), "+r"(c)
      : "r"(x0), "r"(y));
}
__device__ __forceinline__ void mac1_top(uint32_t* e, uint32_t x0, uint32_t y) {
  asm("mad.lo.cc.u32  %0, %2, %3, %0;\n\t"
      "madc.hi.u32    %1, %2, %3, %1;"
      : "+r"(e[0]), "+r"(e[1])
      : "r"(x0), "r"(y));
}
// e[0], e[1] = x * y
__device__ __forceinline__ void mul_pair(uint32_t* e, uint32_t x, uint32_t y) {
  asm("mul.lo.u32 %0, %2, %3;\n\tmul.hi.u32 %1, %2, %3;" : "=&r"(e[0]), "=r"(e[1]) : "r"(x), "r"(y));
}

// T = E + O 2^32 (O[15] = 0; the caller's sum is below 2^512).
__device__ __forceinline__ void merge_16(const uint32_t (&E)[16], const uint32_t (&O)[16],
                                         uint32_t (&T)[16]) {
  T[0] = E[0];
  asm("add.cc.u32  %0, %15, %30;\n\t"
      "addc.cc.u32 %1, %16, %31;\n\t"
      "addc.cc.u32 %2, %17, %32;\n\t"
      "addc.cc.u32 %3, %18, %33;\n\t"
      "addc.cc.u32 %4, %19, %34;\n\t"
      "addc.cc.u32 %5, %20, %35;\n\t"
      "addc.cc.u32 %6, %21, %36;\n\t"
      "addc.cc.u32 %7, %22, %37;\n\t"
      "addc.cc.u32 %8, %23, %38;\n\t"
      "addc.cc.u32 %9, %24, %39;\n\t"
      "addc.cc.u32 %10, %25, %40;\n\t"
      "addc.cc.u32 %11, %26, %41;\n\t"
      "addc.cc.u32 %12, %27, %42;\n\t"
      "addc.cc.u32 %13, %28, %43;\n\t"
      "addc.u32    %14, %29, %44;"
      : "=r"(T[1]), "=r"(T[2]), "=r"(T[3]), "=r"(T[4]), "=r"(T[5]), "=r"(T[6]), "=r"(T[7]),
        "=r"(T[8]), "=r"(T[9]), "=r"(T[10]), "=r"(T[11]), "=r"(T[12]), "=r"(T[13]), "=r"(T[14]),
        "=r"(T[15])
      : "r"(E[1]), "r"(E[2]), "r"(E[3]), "r"(E[4]), "r"(E[5]), "r"(E[6]), "r"(E[7]), "r"(E[8]),
        "r"(E[9]), "r"(E[10]), "r"(E[11]), "r"(E[12]), "r"(E[13]), "r"(E[14]), "r"(E[15]),
        "r"(O[0]), "r"(O[1]), "r"(O[2]), "r"(O[3]), "r"(O[4]), "r"(O[5]), "r"(O[6]), "r"(O[7]),
        "r"(O[8]), "r"(O[9]), "r"(O[10]), "r"(O[11]), "r"(O[12]), "r"(O[13]), "r"(O[14]));
}

// T[0..15] = a * b for any 256-bit a and b, schoolbook by rows of b: 64
// multiply pairs.  After row j the sum of either parity is below
// 2^(32 (j + 9)), so a row's odd-limb chain (whose last pair is the first to
// reach its two words) ends without a carry and its even-limb chain carries
// into a word that only a carry has reached before.
// One Karatsuba level (48 pairs) saves a fifth of the pairs but adds ~100
// instructions in sums and moves, a third of them on the multiply pipe: 62.9
// against 61.5 G products/s at 32 warps per SM and equal at 8, with 294
// against 228 instructions a product, which the kernels that are short of
// issue slots or instruction cache pay for.
__device__ __forceinline__ void fe_mul_wide(const uint32_t (&a)[8], const uint32_t (&b)[8],
                                            uint32_t (&T)[16]) {
  uint32_t E[16], O[16];
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    mul_pair(E + i, a[i], b[0]);
    mul_pair(O + i, a[i + 1], b[0]);
  }
#pragma unroll
  for (int i = 8; i < 16; i++) E[i] = O[i] = 0;
#pragma unroll
  for (int j = 1; j < 8; j += 2) {
    mac4(O + j - 1, O[j + 7], a[0], a[2], a[4], a[6], b[j]);
    mac4_top(E + j + 1, a[1], a[3], a[5], a[7], b[j]);
    if (j < 7) {
      mac4(E + j + 1, E[j + 9], a[0], a[2], a[4], a[6], b[j + 1]);
      mac4_top(O + j + 1, a[1], a[3], a[5], a[7], b[j + 1]);
    }
  }
  merge_16(E, O, T);
}

// T[0..15] = a^2 for any 256-bit a: the 28 cross products once, in two
// accumulators by the parity of their position, doubled, and the eight squares
// as one chain of aligned pairs (36 pairs instead of 64).  A chain marked
// _top is the first to reach its last pair (beside a carry).
__device__ __forceinline__ void fe_sqr_wide(const uint32_t (&a)[8], uint32_t (&T)[16]) {
  uint32_t E[16], O[16];
  E[0] = E[1] = 0;
  mul_pair(O, a[1], a[0]);
  mul_pair(O + 2, a[3], a[0]);
  mul_pair(O + 4, a[5], a[0]);
  mul_pair(O + 6, a[7], a[0]);
  mul_pair(E + 2, a[2], a[0]);
  mul_pair(E + 4, a[4], a[0]);
  mul_pair(E + 6, a[6], a[0]);
#pragma unroll
  for (int i = 8; i < 16; i++) E[i] = O[i] = 0;
  mac3(O + 2, O[8], a[2], a[4], a[6], a[1]);
  mac3_top(E + 4, a[3], a[5], a[7], a[1]);
  mac3_top(O + 4, a[3], a[5], a[7], a[2]);
  mac2(E + 6, E[10], a[4], a[6], a[2]);
  mac2(O + 6, O[10], a[4], a[6], a[3]);
  mac2_top(E + 8, a[5], a[7], a[3]);
  mac2_top(O + 8, a[5], a[7], a[4]);
  mac1(E + 10, E[12], a[6], a[4]);
  mac1(O + 10, O[12], a[6], a[5]);
  mac1_top(E + 12, a[7], a[5]);
  mac1_top(O + 12, a[7], a[6]);
  merge_16(E, O, T);
#pragma unroll
  for (int i = 15; i > 0; i--) T[i] = __funnelshift_l(T[i - 1], T[i], 1);
  T[0] = 0;
  asm("mad.lo.cc.u32  %0, %16, %16, %0;\n\t"
      "madc.hi.cc.u32 %1, %16, %16, %1;\n\t"
      "madc.lo.cc.u32 %2, %17, %17, %2;\n\t"
      "madc.hi.cc.u32 %3, %17, %17, %3;\n\t"
      "madc.lo.cc.u32 %4, %18, %18, %4;\n\t"
      "madc.hi.cc.u32 %5, %18, %18, %5;\n\t"
      "madc.lo.cc.u32 %6, %19, %19, %6;\n\t"
      "madc.hi.cc.u32 %7, %19, %19, %7;\n\t"
      "madc.lo.cc.u32 %8, %20, %20, %8;\n\t"
      "madc.hi.cc.u32 %9, %20, %20, %9;\n\t"
      "madc.lo.cc.u32 %10, %21, %21, %10;\n\t"
      "madc.hi.cc.u32 %11, %21, %21, %11;\n\t"
      "madc.lo.cc.u32 %12, %22, %22, %12;\n\t"
      "madc.hi.cc.u32 %13, %22, %22, %13;\n\t"
      "madc.lo.cc.u32 %14, %23, %23, %14;\n\t"
      "madc.hi.u32    %15, %23, %23, %15;"
      : "+r"(T[0]), "+r"(T[1]), "+r"(T[2]), "+r"(T[3]), "+r"(T[4]), "+r"(T[5]), "+r"(T[6]),
        "+r"(T[7]), "+r"(T[8]), "+r"(T[9]), "+r"(T[10]), "+r"(T[11]), "+r"(T[12]), "+r"(T[13]),
        "+r"(T[14]), "+r"(T[15])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]));
}

// One row of the reduction.  s: accumulator whose pairs start at the row's
// position, o: the other one, whose pairs start a word later.  The row's word
// is s[0] + o_low (the high half of o's previous pair); its carry enters the
// odd-limb chain.  q m clears the word, so the row leaves s[0] = 0 and the
// next row's word is s[1] + o[0].
template <class C>
__device__ __forceinline__ void redc_row(uint32_t* s, uint32_t* o, uint32_t o_low) {
  uint32_t q;
  asm("add.cc.u32     %0, %0, %18;\n\t"
      "mul.lo.u32     %17, %0, %19;\n\t"
      "madc.lo.cc.u32 %9, %17, %21, %9;\n\t"
      "madc.hi.cc.u32 %10, %17, %21, %10;\n\t"
      "madc.lo.cc.u32 %11, %17, %23, %11;\n\t"
      "madc.hi.cc.u32 %12, %17, %23, %12;\n\t"
      "madc.lo.cc.u32 %13, %17, %25, %13;\n\t"
      "madc.hi.cc.u32 %14, %17, %25, %14;\n\t"
      "madc.lo.cc.u32 %15, %17, %27, %15;\n\t"
      "madc.hi.u32    %16, %17, %27, %16;\n\t"
      "mad.lo.cc.u32  %0, %17, %20, %0;\n\t"
      "madc.hi.cc.u32 %1, %17, %20, %1;\n\t"
      "madc.lo.cc.u32 %2, %17, %22, %2;\n\t"
      "madc.hi.cc.u32 %3, %17, %22, %3;\n\t"
      "madc.lo.cc.u32 %4, %17, %24, %4;\n\t"
      "madc.hi.cc.u32 %5, %17, %24, %5;\n\t"
      "madc.lo.cc.u32 %6, %17, %26, %6;\n\t"
      "madc.hi.cc.u32 %7, %17, %26, %7;\n\t"
      "addc.u32       %8, %8, 0;"
      : "+r"(s[0]), "+r"(s[1]), "+r"(s[2]), "+r"(s[3]), "+r"(s[4]), "+r"(s[5]), "+r"(s[6]),
        "+r"(s[7]), "+r"(s[8]), "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]),
        "+r"(o[5]), "+r"(o[6]), "+r"(o[7]), "=&r"(q)
      : "r"(o_low), "n"(C::INV), "n"(C::P0), "n"(C::P1), "n"(C::P2), "n"(C::P3), "n"(C::P4),
        "n"(C::P5), "n"(C::P6), "n"(C::P7));
}

// Montgomery reduction T * 2^-256 mod m, below m + T / 2^256 (below 2m for
// T < 2^256 m; the result always fits 256 bits when T_hi <= 2^256 - m).
// Eight rows fold the low half: row i adds q_i m 2^(32 i) with q_i = t_i
// (-m^-1) mod 2^32, where t_i is the sum's word i, so after it
// T_lo + sum q_j m 2^(32 j) is a multiple of 2^(32 (i + 1)) below
// 2^(32 (i + 9)): the odd-limb chain's last pair (m's top word is below 2^30)
// carries nothing out, and the even-limb chain's carry is the first thing in
// its word.  The two accumulators, with pairs at even (A) and odd (B)
// positions, trade places in every row.  T_hi is added at the end.
template <class C>
__device__ __forceinline__ fe<C> fe_redc_lazy(const uint32_t (&T)[16]) {
  uint32_t A[16], B[16];  // word k of B is position k; B[0] is unused
#pragma unroll
  for (int i = 0; i < 8; i++) A[i] = T[i];
#pragma unroll
  for (int i = 8; i < 16; i++) A[i] = 0;
#pragma unroll
  for (int i = 0; i < 16; i++) B[i] = 0;
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    redc_row<C>(A + i, B + i + 1, B[i]);
    redc_row<C>(B + i + 1, A + i + 2, A[i + 1]);
  }
  fe<C> r;
  asm("add.cc.u32  %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]),
        "=r"(r.v[6]), "=r"(r.v[7])
      : "r"(A[8]), "r"(A[9]), "r"(A[10]), "r"(A[11]), "r"(A[12]), "r"(A[13]), "r"(A[14]),
        "r"(A[15]), "r"(B[8]), "r"(B[9]), "r"(B[10]), "r"(B[11]), "r"(B[12]), "r"(B[13]),
        "r"(B[14]), "r"(B[15]));
  asm("add.cc.u32  %0, %0, %8;\n\t"
      "addc.cc.u32 %1, %1, %9;\n\t"
      "addc.cc.u32 %2, %2, %10;\n\t"
      "addc.cc.u32 %3, %3, %11;\n\t"
      "addc.cc.u32 %4, %4, %12;\n\t"
      "addc.cc.u32 %5, %5, %13;\n\t"
      "addc.cc.u32 %6, %6, %14;\n\t"
      "addc.u32    %7, %7, %15;"
      : "+r"(r.v[0]), "+r"(r.v[1]), "+r"(r.v[2]), "+r"(r.v[3]), "+r"(r.v[4]), "+r"(r.v[5]),
        "+r"(r.v[6]), "+r"(r.v[7])
      : "r"(T[8]), "r"(T[9]), "r"(T[10]), "r"(T[11]), "r"(T[12]), "r"(T[13]), "r"(T[14]),
        "r"(T[15]));
  return r;
}
// fully reduced, for T < 2^256 m
template <class C>
__device__ __forceinline__ fe<C> fe_redc(const uint32_t (&T)[16]) {
  fe<C> r = fe_redc_lazy<C>(T);
  fe_reduce_once<C>(r.v);
  return r;
}

// Full product: a, b < m give T < m^2 < 2^256 * m / 4.
template <class C>
__device__ __forceinline__ fe<C> fe_mul_inline(const fe<C>& a, const fe<C>& b) {
  uint32_t T[16];
  fe_mul_wide(a.v, b.v, T);
  return fe_redc<C>(T);
}

// Out-of-line product (arguments and result travel in registers).  Curve
// formulas use it through operator*: inlining every product of a mixed add,
// doubling and full add made the MSM kernels several times larger than the
// instruction cache (ncu: warps stalled on instruction fetch); one shared
// body per kernel keeps the hot loop resident.
template <class C>
__device__ __noinline__ fe<C> fe_mul_call(fe<C> a, fe<C> b) {
  return fe_mul_inline(a, b);
}

template <class C>
__device__ __forceinline__ fe<C> operator*(const fe<C>& a, const fe<C>& b) {
  return fe_mul_call<C>(a, b);
}

// Out-of-line square.
template <class C>
__device__ __noinline__ fe<C> fe_sqr_call(fe<C> a) {
  uint32_t T[16];
  fe_sqr_wide(a.v, T);
  return fe_redc<C>(T);
}

template <class C>
__device__ __forceinline__ fe<C> fe_sqr(const fe<C>& a) {
  return fe_sqr_call<C>(a);
}

// Montgomery encode / decode
template <class C>
__device__ __forceinline__ fe<C> fe_to_mont(const fe<C>& a) {
  const fe<C> r2{{C::R2[0], C::R2[1], C::R2[2], C::R2[3], C::R2[4], C::R2[5], C::R2[6], C::R2[7]}};
  return a * r2;
}
// a R^-1: the reduction alone
template <class C>
__device__ __forceinline__ fe<C> fe_from_mont(const fe<C>& a) {
  uint32_t T[16];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    T[i] = a.v[i];
    T[8 + i] = 0;
  }
  return fe_redc<C>(T);
}

// Inverse by division steps (field_inv.cuh); inv(0) = 0 like the reference's
// Bernstein-Yang inversion (include/fp_bn254.cuh:720-773).  For a = x R the
// division steps give x^-1 R^-1, and one product by R^3 makes it x^-1 R.
// About 15 K instructions against ~100 K for a^(m-2).
template <class C>
__device__ __noinline__ fe<C> fe_inv_call(fe<C> a) {
  const uint32_t m[8] = {C::P0, C::P1, C::P2, C::P3, C::P4, C::P5, C::P6, C::P7};
  const fe<C> r3{{C::R3[0], C::R3[1], C::R3[2], C::R3[3], C::R3[4], C::R3[5], C::R3[6], C::R3[7]}};
  fe<C> t;
  inv_divsteps(a.v, m, C::INV & (uint32_t)kInvMask, t.v);
  return t * r3;
}
template <class C>
__device__ __forceinline__ fe<C> fe_inv(const fe<C>& a) {
  return fe_inv_call<C>(a);
}

// ------------------------------------------------------------------- Fp2
// Fp2 = Fp[u]/(u^2 + 1): c0 + c1 u, stored [c0, c1] like the reference
// (include/fp2_bn254.cuh:96-180).
struct fp2_t {
  fp_t c0, c1;
};

__device__ __forceinline__ fp2_t operator+(const fp2_t& a, const fp2_t& b) { return {a.c0 + b.c0, a.c1 + b.c1}; }
__device__ __forceinline__ fp2_t operator-(const fp2_t& a, const fp2_t& b) { return {a.c0 - b.c0, a.c1 - b.c1}; }

// x[0..15] -= y[0..15]; the caller guarantees x >= y.
__device__ __forceinline__ void sub_16(uint32_t (&x)[16], const uint32_t (&y)[16]) {
  asm("sub.cc.u32  %0, %0, %16;\n\t"
      "subc.cc.u32 %1, %1, %17;\n\t"
      "subc.cc.u32 %2, %2, %18;\n\t"
      "subc.cc.u32 %3, %3, %19;\n\t"
      "subc.cc.u32 %4, %4, %20;\n\t"
      "subc.cc.u32 %5, %5, %21;\n\t"
      "subc.cc.u32 %6, %6, %22;\n\t"
      "subc.cc.u32 %7, %7, %23;\n\t"
      "subc.cc.u32 %8, %8, %24;\n\t"
      "subc.cc.u32 %9, %9, %25;\n\t"
      "subc.cc.u32 %10, %10, %26;\n\t"
      "subc.cc.u32 %11, %11, %27;\n\t"
      "subc.cc.u32 %12, %12, %28;\n\t"
      "subc.cc.u32 %13, %13, %29;\n\t"
      "subc.cc.u32 %14, %14, %30;\n\t"
      "subc.u32    %15, %15, %31;"
      : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3]), "+r"(x[4]), "+r"(x[5]), "+r"(x[6]),
        "+r"(x[7]), "+r"(x[8]), "+r"(x[9]), "+r"(x[10]), "+r"(x[11]), "+r"(x[12]), "+r"(x[13]),
        "+r"(x[14]), "+r"(x[15])
      : "r"(y[0]), "r"(y[1]), "r"(y[2]), "r"(y[3]), "r"(y[4]), "r"(y[5]), "r"(y[6]), "r"(y[7]),
        "r"(y[8]), "r"(y[9]), "r"(y[10]), "r"(y[11]), "r"(y[12]), "r"(y[13]), "r"(y[14]),
        "r"(y[15]));
}

// x[0..15] += y[0..15]; the caller guarantees x + y < 2^512.
__device__ __forceinline__ void add_16(uint32_t (&x)[16], const uint32_t (&y)[16]) {
  asm("add.cc.u32  %0, %0, %16;\n\t"
      "addc.cc.u32 %1, %1, %17;\n\t"
      "addc.cc.u32 %2, %2, %18;\n\t"
      "addc.cc.u32 %3, %3, %19;\n\t"
      "addc.cc.u32 %4, %4, %20;\n\t"
      "addc.cc.u32 %5, %5, %21;\n\t"
      "addc.cc.u32 %6, %6, %22;\n\t"
      "addc.cc.u32 %7, %7, %23;\n\t"
      "addc.cc.u32 %8, %8, %24;\n\t"
      "addc.cc.u32 %9, %9, %25;\n\t"
      "addc.cc.u32 %10, %10, %26;\n\t"
      "addc.cc.u32 %11, %11, %27;\n\t"
      "addc.cc.u32 %12, %12, %28;\n\t"
      "addc.cc.u32 %13, %13, %29;\n\t"
      "addc.cc.u32 %14, %14, %30;\n\t"
      "addc.u32    %15, %15, %31;"
      : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3]), "+r"(x[4]), "+r"(x[5]), "+r"(x[6]),
        "+r"(x[7]), "+r"(x[8]), "+r"(x[9]), "+r"(x[10]), "+r"(x[11]), "+r"(x[12]), "+r"(x[13]),
        "+r"(x[14]), "+r"(x[15])
      : "r"(y[0]), "r"(y[1]), "r"(y[2]), "r"(y[3]), "r"(y[4]), "r"(y[5]), "r"(y[6]), "r"(y[7]),
        "r"(y[8]), "r"(y[9]), "r"(y[10]), "r"(y[11]), "r"(y[12]), "r"(y[13]), "r"(y[14]),
        "r"(y[15]));
}

// y = x + p^2 (p the base-field modulus; every caller's x + p^2 < 2^512).
__device__ __forceinline__ void add_16_psq(const uint32_t (&x)[16], uint32_t (&y)[16]) {
  asm("add.cc.u32  %0, %16, 0x275d69b1;\n\t"
      "addc.cc.u32 %1, %17, 0x3b5458a2;\n\t"
      "addc.cc.u32 %2, %18, 0x09eac101;\n\t"
      "addc.cc.u32 %3, %19, 0xa602072d;\n\t"
      "addc.cc.u32 %4, %20, 0x6d96cadc;\n\t"
      "addc.cc.u32 %5, %21, 0x4a50189c;\n\t"
      "addc.cc.u32 %6, %22, 0x7a1242c8;\n\t"
      "addc.cc.u32 %7, %23, 0x04689e95;\n\t"
      "addc.cc.u32 %8, %24, 0x34c6b38d;\n\t"
      "addc.cc.u32 %9, %25, 0x26edfa5c;\n\t"
      "addc.cc.u32 %10, %26, 0x16375606;\n\t"
      "addc.cc.u32 %11, %27, 0xb00b8551;\n\t"
      "addc.cc.u32 %12, %28, 0x0348d21c;\n\t"
      "addc.cc.u32 %13, %29, 0x599a6f7c;\n\t"
      "addc.cc.u32 %14, %30, 0x763cbf9c;\n\t"
      "addc.u32    %15, %31, 0x0925c4b8;"
      : "=r"(y[0]), "=r"(y[1]), "=r"(y[2]), "=r"(y[3]), "=r"(y[4]), "=r"(y[5]), "=r"(y[6]),
        "=r"(y[7]), "=r"(y[8]), "=r"(y[9]), "=r"(y[10]), "=r"(y[11]), "=r"(y[12]), "=r"(y[13]),
        "=r"(y[14]), "=r"(y[15])
      : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]),
        "r"(x[8]), "r"(x[9]), "r"(x[10]), "r"(x[11]), "r"(x[12]), "r"(x[13]), "r"(x[14]),
        "r"(x[15]));
}

// s = a + b without reduction (a, b < p give s < 2p < 2^255).
__device__ __forceinline__ void add_raw(const uint32_t (&a)[8], const uint32_t (&b)[8],
                                        uint32_t (&s)[8]) {
  asm("add.cc.u32  %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]),
        "=r"(s[7])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]),
        "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]));
}

// (a0 + a1 u)(b0 + b1 u) with two reductions instead of three (Karatsuba over
// Fp2 on unreduced 512-bit products):
//   c0 = REDC(a0 b0 - a1 b1 + p^2),  c1 = REDC((a0 + a1)(b0 + b1) - a0 b0 - a1 b1).
// Both REDC arguments lie in [0, 2 p^2), below the 2^256 p / 2 that fe_redc
// needs (p < 2^254); adding p^2 changes nothing mod p.  Same result as three
// reduced products (the reference's fp2Mul, include/fp2_bn254.cuh:96-180).
// Out of line like fe_mul_call, so the curve formulas share one body.
static __device__ __noinline__ fp2_t fp2_mul_call(fp2_t a, fp2_t b) {
  uint32_t s[8], t[8], x[16], y[16], w[16];
  add_raw(a.c0.v, a.c1.v, s);
  add_raw(b.c0.v, b.c1.v, t);
  fe_mul_wide(s, t, x);
  fe_mul_wide(a.c0.v, b.c0.v, w);
  sub_16(x, w);
  add_16_psq(w, y);
  fe_mul_wide(a.c1.v, b.c1.v, w);
  sub_16(x, w);
  sub_16(y, w);
  return {fe_redc<FpCfg>(y), fe_redc<FpCfg>(x)};
}

__device__ __forceinline__ fp2_t operator*(const fp2_t& a, const fp2_t& b) {
  return fp2_mul_call(a, b);
}

// a b - c d in Fp with one reduction: REDC(a b + p^2 - c d), whose argument
// lies in (0, 2 p^2).  The Y coordinate of every XYZZ addition and doubling
// has this shape (Y3 = R (Q - X3) - Y1 PPP).
static __device__ __noinline__ fp_t fp_mul_sub_call(fp_t a, fp_t b, fp_t c, fp_t d) {
  uint32_t x[16], w[16];
  fe_mul_wide(a.v, b.v, w);
  add_16_psq(w, x);
  fe_mul_wide(c.v, d.v, w);
  sub_16(x, w);
  return fe_redc<FpCfg>(x);
}

__device__ __forceinline__ fp_t fe_mul_sub(const fp_t& a, const fp_t& b, const fp_t& c,
                                           const fp_t& d) {
  return fp_mul_sub_call(a, b, c, d);
}

// In Fp2 the same sharing (two reductions instead of four) keeps three
// 512-bit accumulators beside four Fp2 operands; the G2 kernels spilled and
// ran slower, so the Fp2 form stays two products and a subtraction.
__device__ __forceinline__ fp2_t fe_mul_sub(const fp2_t& a, const fp2_t& b, const fp2_t& c,
                                            const fp2_t& d) {
  return a * b - c * d;
}

__device__ __forceinline__ fp2_t fe_sqr(const fp2_t& a) {
  // (c0 + c1)(c0 - c1) + 2 c0 c1 u: 2 multiplications
  fp_t t = a.c0 * a.c1;
  return {(a.c0 + a.c1) * (a.c0 - a.c1), t + t};
}
__device__ __forceinline__ fp2_t fe_dbl(const fp2_t& a) { return {a.c0 + a.c0, a.c1 + a.c1}; }
__device__ __forceinline__ bool fe_is_zero(const fp2_t& a) { return fe_is_zero(a.c0) && fe_is_zero(a.c1); }
__device__ __forceinline__ fp2_t fe_neg(const fp2_t& a) { return {fe_neg(a.c0), fe_neg(a.c1)}; }
// Norm to Fp and the inverse from the inverse norm: 1/a = conj(a) / N(a) with
// N(a) = c0^2 + c1^2 (nonzero for a nonzero, as -1 is not a square mod p).
// The sum of the two unreduced squares is below 2 p^2, one reduction.  In Fp
// the norm is the element itself, so code written over norms shares
// inversions in Fp for both groups.
static __device__ __noinline__ fp_t fp2_norm_call(fp2_t a) {
  uint32_t x[16], w[16];
  fe_sqr_wide(a.c0.v, x);
  fe_sqr_wide(a.c1.v, w);
  add_16(x, w);
  return fe_redc<FpCfg>(x);
}
__device__ __forceinline__ fp_t fe_norm(const fp_t& a) { return a; }
__device__ __forceinline__ fp_t fe_norm(const fp2_t& a) { return fp2_norm_call(a); }
__device__ __forceinline__ fp_t fe_inv_of(const fp_t&, const fp_t& ni) { return ni; }
__device__ __forceinline__ fp2_t fe_inv_of(const fp2_t& a, const fp_t& ni) {
  return {a.c0 * ni, fe_neg(a.c1 * ni)};
}
__device__ __forceinline__ fp2_t fe_inv(const fp2_t& a) { return fe_inv_of(a, fe_inv(fe_norm(a))); }
__device__ __forceinline__ bool fe_eq(const fp2_t& a, const fp2_t& b) {
  return fe_eq(a.c0, b.c0) && fe_eq(a.c1, b.c1);
}

template <class T>
__device__ __forceinline__ T fe_zero_of();
template <>
__device__ __forceinline__ fp_t fe_zero_of<fp_t>() { return fe_zero<FpCfg>(); }
template <>
__device__ __forceinline__ fp2_t fe_zero_of<fp2_t>() { return {fe_zero<FpCfg>(), fe_zero<FpCfg>()}; }
template <class T>
__device__ __forceinline__ T fe_one_of();
template <>
__device__ __forceinline__ fp_t fe_one_of<fp_t>() { return fe_one<FpCfg>(); }
template <>
__device__ __forceinline__ fp2_t fe_one_of<fp2_t>() { return {fe_one<FpCfg>(), fe_zero<FpCfg>()}; }

}  // namespace zk
