// field.cuh -- 256-bit Montgomery arithmetic for BN254 on sm_100a.
//
// Elements are 8 little-endian 32-bit limbs held in registers, Montgomery form
// x * 2^256 mod p, always fully reduced to [0, p) at the boundary of every operation, so
// results are word-for-word the values the reference's host code produces
// (src/cuda/ff.cpp montmult_h / addm_h / subm_h, same layout as src/cuda/types.h
// NWORDS_256BIT).  Products are Montgomery products on 32x32->64 multiply-adds with carry,
// one row of a*b and one of m*p per limb of b; BN254 moduli are below 2^254, so the running
// value fits nine limbs and a single conditional subtraction finishes every product.
#pragma once
#include <cstdint>

#include "modinv.cuh"

namespace csb {

#define CSB_DEV __device__ __forceinline__

// ---------------------------------------------------------------- moduli ------------
struct ModQ {  // base field q (the reference's MOD_GROUP, pidx 0)
  static constexpr uint32_t P0 = 0xd87cfd47u, P1 = 0x3c208c16u, P2 = 0x6871ca8du, P3 = 0x97816a91u,
                            P4 = 0x8181585du, P5 = 0xb85045b6u, P6 = 0xe131a029u, P7 = 0x30644e72u;
  static constexpr uint32_t NP0 = 0xe4866389u;  // -q^-1 mod 2^32
  static constexpr uint32_t ONE0 = 0xc58f0d9du, ONE1 = 0xd35d438du, ONE2 = 0xf5c70b3du, ONE3 = 0x0a78eb28u,
                            ONE4 = 0x7879462cu, ONE5 = 0x666ea36fu, ONE6 = 0x9a07df2fu, ONE7 = 0x0e0a77c1u;
  static constexpr uint32_t R20 = 0x538afa89u, R21 = 0xf32cfc5bu, R22 = 0xd44501fbu, R23 = 0xb5e71911u,
                            R24 = 0x0a417ff6u, R25 = 0x47ab1effu, R26 = 0xcab8351fu, R27 = 0x06d89f71u;
  static constexpr uint32_t R30 = 0xda1530dfu, R31 = 0xb1cd6dafu, R32 = 0xa7283db6u, R33 = 0x62f210e6u,
                            R34 = 0x0ada0afbu, R35 = 0xef7f0b0cu, R36 = 0x2d592544u, R37 = 0x20fd6e90u;
};
struct ModR {  // scalar field r (the reference's MOD_FIELD, pidx 1)
  static constexpr uint32_t P0 = 0xf0000001u, P1 = 0x43e1f593u, P2 = 0x79b97091u, P3 = 0x2833e848u,
                            P4 = 0x8181585du, P5 = 0xb85045b6u, P6 = 0xe131a029u, P7 = 0x30644e72u;
  static constexpr uint32_t NP0 = 0xefffffffu;  // -r^-1 mod 2^32
  static constexpr uint32_t ONE0 = 0x4ffffffbu, ONE1 = 0xac96341cu, ONE2 = 0x9f60cd29u, ONE3 = 0x36fc7695u,
                            ONE4 = 0x7879462eu, ONE5 = 0x666ea36fu, ONE6 = 0x9a07df2fu, ONE7 = 0x0e0a77c1u;
  static constexpr uint32_t R20 = 0xae216da7u, R21 = 0x1bb8e645u, R22 = 0xe35c59e3u, R23 = 0x53fe3ab1u,
                            R24 = 0x53bb8085u, R25 = 0x8c49833du, R26 = 0x7f4e44a5u, R27 = 0x0216d0b1u;
  static constexpr uint32_t R30 = 0xb4bf0040u, R31 = 0x5e94d8e1u, R32 = 0x1cfbb6b8u, R33 = 0x2a489cbeu,
                            R34 = 0xa19fcfedu, R35 = 0x893cc664u, R36 = 0x7fcc657cu, R37 = 0x0cf8594bu;
};

// ------------------------------------------------------------ carry-chain helpers ----
// Each helper is one PTX instruction; `volatile` keeps the carry flag sequence in program
// order.  So every statement that writes or reads the flag is volatile, the rows of products below
// too: one that was not could be placed between the instructions of a chain.  (Each chain as one
// statement, none volatile: 0.2-1 % slower, H step on the coset 2^15 84.5 against 85.3 us.)
// An output that a statement writes before it has read its last input is early-clobbered (&):
// otherwise an input of the same value as another operand may be given the output's register.
#define ADD_CC(d, a, b)     asm volatile("add.cc.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b))
#define ADDC_CC(d, a, b)    asm volatile("addc.cc.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b))
#define ADDC(d, a, b)       asm volatile("addc.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b))
#define SUB_CC(d, a, b)     asm volatile("sub.cc.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b))
#define SUBC_CC(d, a, b)    asm volatile("subc.cc.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b))
#define SUBC(d, a, b)       asm volatile("subc.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b))

// Montgomery products accumulate in two sets of columns, the partial products sorted by the
// alignment of their limbs (as Emmart, Luitjens, Weems and Woolley do for half-word products,
// "Optimizing modular multiplication for NVIDIA's Maxwell GPUs", ARITH 2016): e holds columns
// 0..7 as the 64-bit pairs (0,1) (2,3) (4,5) (6,7), o columns 1..8 as (1,2) (3,4) (5,6) (7,8), and
// the value is e + 2^32 o.  A limb's products with the even limbs of the other operand tile e's pairs and
// those with its odd limbs tile o's, so every 32x32->64 product is one multiply-add with
// carry in and out (a mad.lo.cc / madc.hi.cc pair on one aligned pair issues as one wide
// multiply-add) and no separate additions fold it in.  Shifting the value down one limb
// swaps the roles: o's pairs become the new even ones and e's the new odd ones, one column
// lower, with e's second limb left over.  Every value below stays under 2^288 (9 limbs)
// while a + c + p < 2^256, so o never carries out.
// B200: a wide multiply-add with carry holds the multiply pipe for 4 cycles a warp, so a
// product (128 of them and 8 low products) takes at least 528; measured 545 (68 G products/s
// over the GPU) against 807 for wide products folded by add-with-carry chains (46 G/s) and
// 651 for a radix-2^52 product on the FP64 pipe (57 G/s).  Warps of both kinds side by side
// gain nothing over this one alone, nor does a Karatsuba a*b (112 multiply-adds, 577 cycles:
// its additions cost what it saves).

// e, o = a * b
CSB_DEV void eo_mul(uint32_t (&e)[8], uint32_t (&o)[8], const uint32_t (&a)[8], uint32_t b) {
#pragma unroll
  for (int k = 0; k < 8; k += 2) {
    asm("mul.lo.u32 %0, %2, %3;\n\tmul.hi.u32 %1, %2, %3;" : "=&r"(e[k]), "=&r"(e[k + 1]) : "r"(a[k]), "r"(b));
    asm("mul.lo.u32 %0, %2, %3;\n\tmul.hi.u32 %1, %2, %3;" : "=&r"(o[k]), "=&r"(o[k + 1]) : "r"(a[k + 1]), "r"(b));
  }
}
// e, o += a * b
CSB_DEV void eo_mad(uint32_t (&e)[8], uint32_t (&o)[8], const uint32_t (&a)[8], uint32_t b) {
  asm volatile(
      "{\n\t"
      "mad.lo.cc.u32 %8, %17, %24, %8;\n\tmadc.hi.cc.u32 %9, %17, %24, %9;\n\t"
      "madc.lo.cc.u32 %10, %19, %24, %10;\n\tmadc.hi.cc.u32 %11, %19, %24, %11;\n\t"
      "madc.lo.cc.u32 %12, %21, %24, %12;\n\tmadc.hi.cc.u32 %13, %21, %24, %13;\n\t"
      "madc.lo.cc.u32 %14, %23, %24, %14;\n\tmadc.hi.u32 %15, %23, %24, %15;\n\t"
      "mad.lo.cc.u32 %0, %16, %24, %0;\n\tmadc.hi.cc.u32 %1, %16, %24, %1;\n\t"
      "madc.lo.cc.u32 %2, %18, %24, %2;\n\tmadc.hi.cc.u32 %3, %18, %24, %3;\n\t"
      "madc.lo.cc.u32 %4, %20, %24, %4;\n\tmadc.hi.cc.u32 %5, %20, %24, %5;\n\t"
      "madc.lo.cc.u32 %6, %22, %24, %6;\n\tmadc.hi.cc.u32 %7, %22, %24, %7;\n\t"
      "addc.u32 %15, %15, 0;\n\t}"
      : "+&r"(e[0]), "+&r"(e[1]), "+&r"(e[2]), "+&r"(e[3]), "+&r"(e[4]), "+&r"(e[5]), "+&r"(e[6]), "+&r"(e[7]), "+&r"(o[0]),
        "+&r"(o[1]), "+&r"(o[2]), "+&r"(o[3]), "+&r"(o[4]), "+&r"(o[5]), "+&r"(o[6]), "+&r"(o[7])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(b));
}
// (e, o) <- ((e, o) >> 32) + a * b, for e[0] = 0.  The left-over limb e[1] goes into the new
// column 0 first; its carry (column 1) enters the odd chain, which starts there.
CSB_DEV void eo_shift_mad(uint32_t (&e)[8], uint32_t (&o)[8], const uint32_t (&a)[8], uint32_t b) {
  uint32_t n0, n1, n2, n3, n4, n5, n6, n7;
  asm volatile(
      "{\n\t"
      "add.cc.u32 %0, %0, %16;\n\t"
      "madc.lo.cc.u32 %8, %24, %31, %17;\n\tmadc.hi.cc.u32 %9, %24, %31, %18;\n\t"
      "madc.lo.cc.u32 %10, %26, %31, %19;\n\tmadc.hi.cc.u32 %11, %26, %31, %20;\n\t"
      "madc.lo.cc.u32 %12, %28, %31, %21;\n\tmadc.hi.cc.u32 %13, %28, %31, %22;\n\t"
      "madc.lo.cc.u32 %14, %30, %31, 0;\n\tmadc.hi.u32 %15, %30, %31, 0;\n\t"
      "mad.lo.cc.u32 %0, %23, %31, %0;\n\tmadc.hi.cc.u32 %1, %23, %31, %1;\n\t"
      "madc.lo.cc.u32 %2, %25, %31, %2;\n\tmadc.hi.cc.u32 %3, %25, %31, %3;\n\t"
      "madc.lo.cc.u32 %4, %27, %31, %4;\n\tmadc.hi.cc.u32 %5, %27, %31, %5;\n\t"
      "madc.lo.cc.u32 %6, %29, %31, %6;\n\tmadc.hi.cc.u32 %7, %29, %31, %7;\n\t"
      "addc.u32 %15, %15, 0;\n\t}"
      : "+&r"(o[0]), "+&r"(o[1]), "+&r"(o[2]), "+&r"(o[3]), "+&r"(o[4]), "+&r"(o[5]), "+&r"(o[6]), "+&r"(o[7]), "=&r"(n0),
        "=&r"(n1), "=&r"(n2), "=&r"(n3), "=&r"(n4), "=&r"(n5), "=&r"(n6), "=&r"(n7)
      : "r"(e[1]), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(a[0]), "r"(a[1]), "r"(a[2]),
        "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(b));
#pragma unroll
  for (int k = 0; k < 8; k++) e[k] = o[k];
  o[0] = n0; o[1] = n1; o[2] = n2; o[3] = n3; o[4] = n4; o[5] = n5; o[6] = n6; o[7] = n7;
}
// r = (e + 2^32 o) >> 32, for e[0] = 0 and a value below 2^288
CSB_DEV void eo_join(uint32_t (&r)[8], const uint32_t (&e)[8], const uint32_t (&o)[8]) {
  ADD_CC(r[0], o[0], e[1]);  ADDC_CC(r[1], o[1], e[2]); ADDC_CC(r[2], o[2], e[3]); ADDC_CC(r[3], o[3], e[4]);
  ADDC_CC(r[4], o[4], e[5]); ADDC_CC(r[5], o[5], e[6]); ADDC_CC(r[6], o[6], e[7]); ADDC(r[7], o[7], 0u);
}

// t += x * b over adjacent 64-bit pairs (x: every second limb of an operand), carry into c
template <int N>
CSB_DEV void pair_chain(uint32_t* t, uint32_t& c, const uint32_t* x, uint32_t b) {
  if constexpr (N == 1)
    asm volatile(
        "mad.lo.cc.u32 %0, %3, %4, %0;\n\tmadc.hi.cc.u32 %1, %3, %4, %1;\n\taddc.u32 %2, %2, 0;"
        : "+&r"(t[0]), "+&r"(t[1]), "+&r"(c) : "r"(x[0]), "r"(b));
  if constexpr (N == 2)
    asm volatile(
        "mad.lo.cc.u32 %0, %5, %7, %0;\n\tmadc.hi.cc.u32 %1, %5, %7, %1;\n\t"
        "madc.lo.cc.u32 %2, %6, %7, %2;\n\tmadc.hi.cc.u32 %3, %6, %7, %3;\n\taddc.u32 %4, %4, 0;"
        : "+&r"(t[0]), "+&r"(t[1]), "+&r"(t[2]), "+&r"(t[3]), "+&r"(c) : "r"(x[0]), "r"(x[2]), "r"(b));
  if constexpr (N == 3)
    asm volatile(
        "mad.lo.cc.u32 %0, %7, %10, %0;\n\tmadc.hi.cc.u32 %1, %7, %10, %1;\n\t"
        "madc.lo.cc.u32 %2, %8, %10, %2;\n\tmadc.hi.cc.u32 %3, %8, %10, %3;\n\t"
        "madc.lo.cc.u32 %4, %9, %10, %4;\n\tmadc.hi.cc.u32 %5, %9, %10, %5;\n\taddc.u32 %6, %6, 0;"
        : "+&r"(t[0]), "+&r"(t[1]), "+&r"(t[2]), "+&r"(t[3]), "+&r"(t[4]), "+&r"(t[5]), "+&r"(c)
        : "r"(x[0]), "r"(x[2]), "r"(x[4]), "r"(b));
  if constexpr (N == 4)
    asm volatile(
        "mad.lo.cc.u32 %0, %9, %13, %0;\n\tmadc.hi.cc.u32 %1, %9, %13, %1;\n\t"
        "madc.lo.cc.u32 %2, %10, %13, %2;\n\tmadc.hi.cc.u32 %3, %10, %13, %3;\n\t"
        "madc.lo.cc.u32 %4, %11, %13, %4;\n\tmadc.hi.cc.u32 %5, %11, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, %12, %13, %6;\n\tmadc.hi.cc.u32 %7, %12, %13, %7;\n\taddc.u32 %8, %8, 0;"
        : "+&r"(t[0]), "+&r"(t[1]), "+&r"(t[2]), "+&r"(t[3]), "+&r"(t[4]), "+&r"(t[5]), "+&r"(t[6]), "+&r"(t[7]), "+&r"(c)
        : "r"(x[0]), "r"(x[2]), "r"(x[4]), "r"(x[6]), "r"(b));
}
// lo, hi = a * b
CSB_DEV void wide_mul(uint32_t& lo, uint32_t& hi, uint32_t a, uint32_t b) {
  asm("mul.lo.u32 %0, %2, %3;\n\tmul.hi.u32 %1, %2, %3;" : "=&r"(lo), "=&r"(hi) : "r"(a), "r"(b));
}
// t = a b
CSB_DEV void mul_wide(uint32_t (&t)[16], const uint32_t (&a)[8], const uint32_t (&b)[8]) {
  uint32_t e[17], o[16];  // e[k]: column k, o[k]: column k + 1
#pragma unroll
  for (int k = 8; k < 16; k++) e[k] = o[k] = 0;
  e[16] = 0;
#pragma unroll
  for (int k = 0; k < 8; k += 2) {
    wide_mul(e[k], e[k + 1], a[k], b[0]);
    wide_mul(o[k], o[k + 1], a[k + 1], b[0]);
  }
#pragma unroll
  for (int i = 1; i < 8; i++) {
    if (i & 1) {
      pair_chain<4>(e + i + 1, e[i + 9], a + 1, b[i]);
      pair_chain<4>(o + i - 1, o[i + 7], a, b[i]);
    } else {
      pair_chain<4>(e + i, e[i + 8], a, b[i]);
      pair_chain<4>(o + i, o[i + 8], a + 1, b[i]);
    }
  }
  t[0] = e[0];
  ADD_CC(t[1], e[1], o[0]);
#pragma unroll
  for (int k = 2; k < 15; k++) ADDC_CC(t[k], e[k], o[k - 1]);
  ADDC(t[15], e[15], o[14]);
}
// t = a^2: the 28 products of distinct limbs once, in even (e[k]: column k) and odd (o[k]:
// column k + 1) pairs, doubled, and the 8 squares added in one chain over the even pairs.
CSB_DEV void sqr_wide(uint32_t (&t)[16], const uint32_t (&a)[8]) {
  uint32_t e[16], o[16];
#pragma unroll
  for (int k = 0; k < 16; k++) e[k] = o[k] = 0;
  wide_mul(o[0], o[1], a[1], a[0]); wide_mul(o[2], o[3], a[3], a[0]);
  wide_mul(o[4], o[5], a[5], a[0]); wide_mul(o[6], o[7], a[7], a[0]);
  wide_mul(e[2], e[3], a[2], a[0]); wide_mul(e[4], e[5], a[4], a[0]); wide_mul(e[6], e[7], a[6], a[0]);
  pair_chain<3>(o + 2, o[8], a + 2, a[1]);   pair_chain<3>(e + 4, e[10], a + 3, a[1]);
  pair_chain<3>(o + 4, o[10], a + 3, a[2]);  pair_chain<2>(e + 6, e[10], a + 4, a[2]);
  pair_chain<2>(o + 6, o[10], a + 4, a[3]);  pair_chain<2>(e + 8, e[12], a + 5, a[3]);
  pair_chain<2>(o + 8, o[12], a + 5, a[4]);  pair_chain<1>(e + 10, e[12], a + 6, a[4]);
  pair_chain<1>(o + 10, o[12], a + 6, a[5]); pair_chain<1>(e + 12, e[14], a + 7, a[5]);
  pair_chain<1>(o + 12, o[14], a + 7, a[6]);
  t[0] = 0; t[1] = o[0];
  ADD_CC(t[2], e[2], o[1]);
#pragma unroll
  for (int k = 3; k < 15; k++) ADDC_CC(t[k], e[k], o[k - 1]);
  ADDC(t[15], o[14], 0u);
  ADD_CC(t[1], t[1], t[1]);
#pragma unroll
  for (int k = 2; k < 15; k++) ADDC_CC(t[k], t[k], t[k]);
  ADDC(t[15], t[15], t[15]);
  asm volatile(
      "mad.lo.cc.u32 %0, %16, %16, %0;\n\tmadc.hi.cc.u32 %1, %16, %16, %1;\n\t"
      "madc.lo.cc.u32 %2, %17, %17, %2;\n\tmadc.hi.cc.u32 %3, %17, %17, %3;\n\t"
      "madc.lo.cc.u32 %4, %18, %18, %4;\n\tmadc.hi.cc.u32 %5, %18, %18, %5;\n\t"
      "madc.lo.cc.u32 %6, %19, %19, %6;\n\tmadc.hi.cc.u32 %7, %19, %19, %7;\n\t"
      "madc.lo.cc.u32 %8, %20, %20, %8;\n\tmadc.hi.cc.u32 %9, %20, %20, %9;\n\t"
      "madc.lo.cc.u32 %10, %21, %21, %10;\n\tmadc.hi.cc.u32 %11, %21, %21, %11;\n\t"
      "madc.lo.cc.u32 %12, %22, %22, %12;\n\tmadc.hi.cc.u32 %13, %22, %22, %13;\n\t"
      "madc.lo.cc.u32 %14, %23, %23, %14;\n\tmadc.hi.u32 %15, %23, %23, %15;"
      : "+&r"(t[0]), "+&r"(t[1]), "+&r"(t[2]), "+&r"(t[3]), "+&r"(t[4]), "+&r"(t[5]), "+&r"(t[6]), "+&r"(t[7]), "+&r"(t[8]),
        "+&r"(t[9]), "+&r"(t[10]), "+&r"(t[11]), "+&r"(t[12]), "+&r"(t[13]), "+&r"(t[14]), "+&r"(t[15])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]));
}
// (e, o) <- ((e, o) >> 32) + p * m with m = -(column 0) / p mod 2^32, for e[0] = 0: one
// reduction row of a value that has no further products to add.  Column 0 becomes 0.
template <class M>
CSB_DEV void eo_shift_reduce(uint32_t (&e)[8], uint32_t (&o)[8]) {
  const uint32_t P[8] = {M::P0, M::P1, M::P2, M::P3, M::P4, M::P5, M::P6, M::P7};
  uint32_t n0, n1, n2, n3, n4, n5, n6, n7, m;
  asm volatile(
      "add.cc.u32 %0, %0, %10;\n\t"
      "mul.lo.u32 %9, %0, %17;\n\t"
      "madc.lo.cc.u32 %1, %18, %9, %11;\n\tmadc.hi.cc.u32 %2, %18, %9, %12;\n\t"
      "madc.lo.cc.u32 %3, %19, %9, %13;\n\tmadc.hi.cc.u32 %4, %19, %9, %14;\n\t"
      "madc.lo.cc.u32 %5, %20, %9, %15;\n\tmadc.hi.cc.u32 %6, %20, %9, %16;\n\t"
      "madc.lo.cc.u32 %7, %21, %9, 0;\n\tmadc.hi.u32 %8, %21, %9, 0;"
      : "+&r"(o[0]), "=&r"(n0), "=&r"(n1), "=&r"(n2), "=&r"(n3), "=&r"(n4), "=&r"(n5), "=&r"(n6), "=&r"(n7), "=&r"(m)
      : "r"(e[1]), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(M::NP0), "r"(P[1]), "r"(P[3]),
        "r"(P[5]), "r"(P[7]));
#pragma unroll
  for (int k = 0; k < 8; k++) e[k] = o[k];
  o[0] = n0; o[1] = n1; o[2] = n2; o[3] = n3; o[4] = n4; o[5] = n5; o[6] = n6; o[7] = n7;
  pair_chain<4>(e, o[7], P, m);
}

template <class M>
struct Fp;
// Out-of-line Montgomery product (arguments and result in registers): keeps loop bodies
// that chain many products small enough for the instruction cache.
template <class M>
__device__ __noinline__ Fp<M> fp_mul_call(Fp<M> a, Fp<M> b);

template <class M>
struct Fp {
  uint32_t v[8];

  static CSB_DEV Fp zero() { Fp r; for (int i = 0; i < 8; i++) r.v[i] = 0; return r; }
  static CSB_DEV Fp one() {
    return Fp{{M::ONE0, M::ONE1, M::ONE2, M::ONE3, M::ONE4, M::ONE5, M::ONE6, M::ONE7}};
  }
  static CSB_DEV Fp r2() { return Fp{{M::R20, M::R21, M::R22, M::R23, M::R24, M::R25, M::R26, M::R27}}; }
  static CSB_DEV Fp r3() { return Fp{{M::R30, M::R31, M::R32, M::R33, M::R34, M::R35, M::R36, M::R37}}; }

  CSB_DEV bool is_zero() const {
    return (v[0] | v[1] | v[2] | v[3] | v[4] | v[5] | v[6] | v[7]) == 0;
  }
  CSB_DEV bool operator==(const Fp& o) const {
    return ((v[0] ^ o.v[0]) | (v[1] ^ o.v[1]) | (v[2] ^ o.v[2]) | (v[3] ^ o.v[3]) |
            (v[4] ^ o.v[4]) | (v[5] ^ o.v[5]) | (v[6] ^ o.v[6]) | (v[7] ^ o.v[7])) == 0;
  }

  // r = t - p if t >= p else t, for t < 2p (t given in 8 limbs).
  static CSB_DEV void reduce_once(uint32_t (&t)[8]) {
    uint32_t u[8], br;
    SUB_CC(u[0], t[0], M::P0); SUBC_CC(u[1], t[1], M::P1); SUBC_CC(u[2], t[2], M::P2);
    SUBC_CC(u[3], t[3], M::P3); SUBC_CC(u[4], t[4], M::P4); SUBC_CC(u[5], t[5], M::P5);
    SUBC_CC(u[6], t[6], M::P6); SUBC_CC(u[7], t[7], M::P7); SUBC(br, 0u, 0u);
    // br = 0xffffffff if t < p (borrow), 0 otherwise
#pragma unroll
    for (int i = 0; i < 8; i++) t[i] = (t[i] & br) | (u[i] & ~br);
  }

  friend CSB_DEV Fp operator+(const Fp& a, const Fp& b) {
    uint32_t t[8];
    ADD_CC(t[0], a.v[0], b.v[0]);  ADDC_CC(t[1], a.v[1], b.v[1]); ADDC_CC(t[2], a.v[2], b.v[2]);
    ADDC_CC(t[3], a.v[3], b.v[3]); ADDC_CC(t[4], a.v[4], b.v[4]); ADDC_CC(t[5], a.v[5], b.v[5]);
    ADDC_CC(t[6], a.v[6], b.v[6]); ADDC(t[7], a.v[7], b.v[7]);
    reduce_once(t);
    Fp r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = t[i];
    return r;
  }
  friend CSB_DEV Fp operator-(const Fp& a, const Fp& b) {
    uint32_t t[8], br;
    SUB_CC(t[0], a.v[0], b.v[0]);  SUBC_CC(t[1], a.v[1], b.v[1]); SUBC_CC(t[2], a.v[2], b.v[2]);
    SUBC_CC(t[3], a.v[3], b.v[3]); SUBC_CC(t[4], a.v[4], b.v[4]); SUBC_CC(t[5], a.v[5], b.v[5]);
    SUBC_CC(t[6], a.v[6], b.v[6]); SUBC_CC(t[7], a.v[7], b.v[7]); SUBC(br, 0u, 0u);
    // add p back if the subtraction borrowed
    const uint32_t p0 = M::P0 & br, p1 = M::P1 & br, p2 = M::P2 & br, p3 = M::P3 & br;
    const uint32_t p4 = M::P4 & br, p5 = M::P5 & br, p6 = M::P6 & br, p7 = M::P7 & br;
    Fp r;
    ADD_CC(r.v[0], t[0], p0);  ADDC_CC(r.v[1], t[1], p1); ADDC_CC(r.v[2], t[2], p2);
    ADDC_CC(r.v[3], t[3], p3); ADDC_CC(r.v[4], t[4], p4); ADDC_CC(r.v[5], t[5], p5);
    ADDC_CC(r.v[6], t[6], p6); ADDC(r.v[7], t[7], p7);
    return r;
  }
  CSB_DEV Fp neg() const { return zero() - *this; }
  CSB_DEV Fp dbl() const { return *this + *this; }

  // Montgomery product without the final conditional subtraction: below (a b + m p) / 2^256,
  // that is (1 + 0.19 i j) p for a <= i p, b <= j p (p = 0.189 * 2^256).  Needs a + p below
  // 2^256; b may be any 256-bit value.
  static CSB_DEV Fp mul_raw(const Fp& a, const Fp& b) {
    const uint32_t P[8] = {M::P0, M::P1, M::P2, M::P3, M::P4, M::P5, M::P6, M::P7};
    uint32_t e[8], o[8];
    eo_mul(e, o, a.v, b.v[0]);
    eo_mad(e, o, P, e[0] * M::NP0);
#pragma unroll
    for (int i = 1; i < 8; i++) {
      eo_shift_mad(e, o, a.v, b.v[i]);
      eo_mad(e, o, P, e[0] * M::NP0);
    }
    Fp r;
    eo_join(r.v, e, o);
    return r;
  }

  // t / 2^256 mod p: the low half reduced alone (at most p), the high half added
  static CSB_DEV Fp redc_wide(const uint32_t (&t)[16]) {
    const uint32_t P[8] = {M::P0, M::P1, M::P2, M::P3, M::P4, M::P5, M::P6, M::P7};
    uint32_t e[8], o[8];
#pragma unroll
    for (int k = 0; k < 8; k++) e[k] = t[k];
    const uint32_t m = e[0] * M::NP0;
#pragma unroll
    for (int k = 0; k < 8; k += 2) wide_mul(o[k], o[k + 1], P[k + 1], m);
    pair_chain<4>(e, o[7], P, m);
#pragma unroll
    for (int i = 1; i < 8; i++) eo_shift_reduce<M>(e, o);
    Fp r;
    eo_join(r.v, e, o);
    ADD_CC(r.v[0], r.v[0], t[8]);   ADDC_CC(r.v[1], r.v[1], t[9]);  ADDC_CC(r.v[2], r.v[2], t[10]);
    ADDC_CC(r.v[3], r.v[3], t[11]); ADDC_CC(r.v[4], r.v[4], t[12]); ADDC_CC(r.v[5], r.v[5], t[13]);
    ADDC_CC(r.v[6], r.v[6], t[14]); ADDC(r.v[7], r.v[7], t[15]);
    return r;
  }
  // Montgomery square, same bound: 36 multiply-adds for a^2 instead of 64 (467 cycles a warp
  // against 545 of mul_raw)
  static CSB_DEV Fp sqr_raw(const Fp& a) {
    uint32_t t[16];
    sqr_wide(t, a.v);
    return redc_wide(t);
  }
  // a + b without reduction (sums below 2^256)
  static CSB_DEV Fp add_raw(const Fp& a, const Fp& b) {
    Fp r;
    ADD_CC(r.v[0], a.v[0], b.v[0]);  ADDC_CC(r.v[1], a.v[1], b.v[1]); ADDC_CC(r.v[2], a.v[2], b.v[2]);
    ADDC_CC(r.v[3], a.v[3], b.v[3]); ADDC_CC(r.v[4], a.v[4], b.v[4]); ADDC_CC(r.v[5], a.v[5], b.v[5]);
    ADDC_CC(r.v[6], a.v[6], b.v[6]); ADDC(r.v[7], a.v[7], b.v[7]);
    return r;
  }
  // a + p - b for b <= p, not reduced
  static CSB_DEV Fp sub_raw(const Fp& a, const Fp& b) {
    uint32_t t[8];
    SUB_CC(t[0], M::P0, b.v[0]);  SUBC_CC(t[1], M::P1, b.v[1]); SUBC_CC(t[2], M::P2, b.v[2]);
    SUBC_CC(t[3], M::P3, b.v[3]); SUBC_CC(t[4], M::P4, b.v[4]); SUBC_CC(t[5], M::P5, b.v[5]);
    SUBC_CC(t[6], M::P6, b.v[6]); SUBC(t[7], M::P7, b.v[7]);
    Fp r;
    ADD_CC(r.v[0], a.v[0], t[0]);  ADDC_CC(r.v[1], a.v[1], t[1]); ADDC_CC(r.v[2], a.v[2], t[2]);
    ADDC_CC(r.v[3], a.v[3], t[3]); ADDC_CC(r.v[4], a.v[4], t[4]); ADDC_CC(r.v[5], a.v[5], t[5]);
    ADDC_CC(r.v[6], a.v[6], t[6]); ADDC(r.v[7], a.v[7], t[7]);
    return r;
  }
  // a b + c d with one reduction (200 multiply-adds instead of 256): below
  // (a b + c d) / 2^256 + p, for a + c + p < 2^256 (BN254: a, c <= 2p).
  static CSB_DEV Fp mul2_raw(const Fp& a, const Fp& b, const Fp& c, const Fp& d) {
    const uint32_t P[8] = {M::P0, M::P1, M::P2, M::P3, M::P4, M::P5, M::P6, M::P7};
    uint32_t e[8], o[8];
    eo_mul(e, o, a.v, b.v[0]);
    eo_mad(e, o, c.v, d.v[0]);
    eo_mad(e, o, P, e[0] * M::NP0);
#pragma unroll
    for (int i = 1; i < 8; i++) {
      eo_shift_mad(e, o, a.v, b.v[i]);
      eo_mad(e, o, c.v, d.v[i]);
      eo_mad(e, o, P, e[0] * M::NP0);
    }
    Fp r;
    eo_join(r.v, e, o);
    return r;
  }

  // ---- lazily reduced values in [0, 2p) (BN254: 4p < 2^256): products of two such values
  // are below 2p without the final subtraction (1.76 p)

  // 2p, limb i
  static CSB_DEV uint32_t p2(int i) {
    const uint32_t P[8] = {M::P0, M::P1, M::P2, M::P3, M::P4, M::P5, M::P6, M::P7};
    return (P[i] << 1) | (i > 0 ? P[i - 1] >> 31 : 0u);
  }
  // a + b for a, b < 2p, result < 2p
  static CSB_DEV Fp add_lazy(const Fp& a, const Fp& b) {
    uint32_t t[8], u[8], br;
    ADD_CC(t[0], a.v[0], b.v[0]);  ADDC_CC(t[1], a.v[1], b.v[1]); ADDC_CC(t[2], a.v[2], b.v[2]);
    ADDC_CC(t[3], a.v[3], b.v[3]); ADDC_CC(t[4], a.v[4], b.v[4]); ADDC_CC(t[5], a.v[5], b.v[5]);
    ADDC_CC(t[6], a.v[6], b.v[6]); ADDC(t[7], a.v[7], b.v[7]);
    SUB_CC(u[0], t[0], p2(0)); SUBC_CC(u[1], t[1], p2(1)); SUBC_CC(u[2], t[2], p2(2));
    SUBC_CC(u[3], t[3], p2(3)); SUBC_CC(u[4], t[4], p2(4)); SUBC_CC(u[5], t[5], p2(5));
    SUBC_CC(u[6], t[6], p2(6)); SUBC_CC(u[7], t[7], p2(7)); SUBC(br, 0u, 0u);
    Fp r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = (t[i] & br) | (u[i] & ~br);
    return r;
  }
  // a - b for a, b < 2p, result < 2p
  static CSB_DEV Fp sub_lazy(const Fp& a, const Fp& b) {
    uint32_t t[8], br;
    SUB_CC(t[0], a.v[0], b.v[0]);  SUBC_CC(t[1], a.v[1], b.v[1]); SUBC_CC(t[2], a.v[2], b.v[2]);
    SUBC_CC(t[3], a.v[3], b.v[3]); SUBC_CC(t[4], a.v[4], b.v[4]); SUBC_CC(t[5], a.v[5], b.v[5]);
    SUBC_CC(t[6], a.v[6], b.v[6]); SUBC_CC(t[7], a.v[7], b.v[7]); SUBC(br, 0u, 0u);
    Fp r;
    ADD_CC(r.v[0], t[0], p2(0) & br);  ADDC_CC(r.v[1], t[1], p2(1) & br); ADDC_CC(r.v[2], t[2], p2(2) & br);
    ADDC_CC(r.v[3], t[3], p2(3) & br); ADDC_CC(r.v[4], t[4], p2(4) & br); ADDC_CC(r.v[5], t[5], p2(5) & br);
    ADDC_CC(r.v[6], t[6], p2(6) & br); ADDC(r.v[7], t[7], p2(7) & br);
    return r;
  }
  // 2p - a for a < 2p, in (0, 2p]
  static CSB_DEV Fp neg_lazy(const Fp& a) {
    Fp r;
    SUB_CC(r.v[0], p2(0), a.v[0]);  SUBC_CC(r.v[1], p2(1), a.v[1]); SUBC_CC(r.v[2], p2(2), a.v[2]);
    SUBC_CC(r.v[3], p2(3), a.v[3]); SUBC_CC(r.v[4], p2(4), a.v[4]); SUBC_CC(r.v[5], p2(5), a.v[5]);
    SUBC_CC(r.v[6], p2(6), a.v[6]); SUBC(r.v[7], p2(7), a.v[7]);
    return r;
  }
  // a or a - 2p, below 2p, for a < 4p
  static CSB_DEV Fp reduce_2p(const Fp& a) {
    uint32_t u[8], br;
    SUB_CC(u[0], a.v[0], p2(0)); SUBC_CC(u[1], a.v[1], p2(1)); SUBC_CC(u[2], a.v[2], p2(2));
    SUBC_CC(u[3], a.v[3], p2(3)); SUBC_CC(u[4], a.v[4], p2(4)); SUBC_CC(u[5], a.v[5], p2(5));
    SUBC_CC(u[6], a.v[6], p2(6)); SUBC_CC(u[7], a.v[7], p2(7)); SUBC(br, 0u, 0u);
    Fp r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = (a.v[i] & br) | (u[i] & ~br);
    return r;
  }
  // k a mod p, below 2p, for a < 2p and k <= 1024: the 9-limb product less q p, with q from its
  // top bits (2^238 and up) times 2^270 / p, at most one below the true quotient
  static CSB_DEV Fp mul_small(const Fp& a, uint32_t k) {
    constexpr uint32_t kInv = 0x15291u;  // floor(2^270 / p), the same for both moduli
    const uint32_t P[8] = {M::P0, M::P1, M::P2, M::P3, M::P4, M::P5, M::P6, M::P7};
    uint32_t e[8], o[8], t[9];
    eo_mul(e, o, a.v, k);
    t[0] = e[0];
    ADD_CC(t[1], e[1], o[0]);  ADDC_CC(t[2], e[2], o[1]); ADDC_CC(t[3], e[3], o[2]); ADDC_CC(t[4], e[4], o[3]);
    ADDC_CC(t[5], e[5], o[4]); ADDC_CC(t[6], e[6], o[5]); ADDC_CC(t[7], e[7], o[6]); ADDC(t[8], o[7], 0u);
    const uint32_t q = __umulhi((t[8] << 18) | (t[7] >> 14), kInv);
    eo_mul(e, o, P, q);
    Fp r;
    SUB_CC(r.v[0], t[0], e[0]);  SUBC_CC(r.v[1], t[1], e[1]); SUBC_CC(r.v[2], t[2], e[2]); SUBC_CC(r.v[3], t[3], e[3]);
    SUBC_CC(r.v[4], t[4], e[4]); SUBC_CC(r.v[5], t[5], e[5]); SUBC_CC(r.v[6], t[6], e[6]); SUBC(r.v[7], t[7], e[7]);
    SUB_CC(r.v[1], r.v[1], o[0]);  SUBC_CC(r.v[2], r.v[2], o[1]); SUBC_CC(r.v[3], r.v[3], o[2]);
    SUBC_CC(r.v[4], r.v[4], o[3]); SUBC_CC(r.v[5], r.v[5], o[4]); SUBC_CC(r.v[6], r.v[6], o[5]); SUBC(r.v[7], r.v[7], o[6]);
    return r;
  }
  // zero mod p for a value < 2p: 0 or p
  CSB_DEV bool is_zero_lazy() const {
    const uint32_t z = v[0] | v[1] | v[2] | v[3] | v[4] | v[5] | v[6] | v[7];
    const uint32_t e = (v[0] ^ M::P0) | (v[1] ^ M::P1) | (v[2] ^ M::P2) | (v[3] ^ M::P3) | (v[4] ^ M::P4) |
                       (v[5] ^ M::P5) | (v[6] ^ M::P6) | (v[7] ^ M::P7);
    return z == 0 || e == 0;
  }
  // the canonical representative in [0, p) of a value < 2p
  CSB_DEV Fp canon() const {
    uint32_t t[8];
#pragma unroll
    for (int i = 0; i < 8; i++) t[i] = v[i];
    reduce_once(t);
    Fp r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = t[i];
    return r;
  }

  friend CSB_DEV Fp operator*(const Fp& a, const Fp& b) {
#if defined(CSB_MUL_NOINLINE)
    return fp_mul_call<M>(a, b);
#else
    return mul_raw(a, b).canon();
#endif
  }

  CSB_DEV Fp sqr() const;

  // x -> x * R mod p (normal form to Montgomery); any 256-bit x is accepted: the product
  // with r2 < p on the left is below 2p.
  CSB_DEV Fp to_mont() const { return r2() * (*this); }
  CSB_DEV Fp from_mont() const {
    Fp o = zero();
    o.v[0] = 1;
    return (*this) * o;
  }

  // Montgomery inverse (aR -> a^-1 R; 0 -> 0): the GCD on the integer x = aR gives
  // x^-1 = a^-1 R^-1, one Montgomery product by R^3 restores a^-1 R.
  CSB_DEV Fp inv() const;
};

using Fq = Fp<ModQ>;
using Fr = Fp<ModR>;

template <class M>
__device__ __noinline__ Fp<M> fp_mul_call(Fp<M> a, Fp<M> b) {
  return Fp<M>::mul_raw(a, b).canon();
}

template <class M>
__device__ __noinline__ Fp<M> fp_sqr_call(Fp<M> a) {
  return Fp<M>::sqr_raw(a).canon();
}

template <class M>
__device__ __noinline__ Fp<M> fp_inv_call(Fp<M> a) {
  const uint32_t P[8] = {M::P0, M::P1, M::P2, M::P3, M::P4, M::P5, M::P6, M::P7};
  Fp<M> r;
  modinv(a.v, P, M::NP0, r.v);
  return Fp<M>::mul_raw(Fp<M>::r3(), r).canon();
}
template <class M>
CSB_DEV Fp<M> Fp<M>::inv() const { return fp_inv_call<M>(*this); }

// Out of line (CSB_MUL_NOINLINE units) or inlined
#if defined(CSB_MUL_NOINLINE)
template <class M>
CSB_DEV Fp<M> Fp<M>::sqr() const { return fp_sqr_call<M>(*this); }
#else
template <class M>
CSB_DEV Fp<M> Fp<M>::sqr() const { return sqr_raw(*this).canon(); }
#endif

// ------------------------------------------------------------ Fq2 = Fq[u]/(u^2+1) ----
struct Fq2 {
  Fq c0, c1;
  static CSB_DEV Fq2 zero() { return {Fq::zero(), Fq::zero()}; }
  static CSB_DEV Fq2 one() { return {Fq::one(), Fq::zero()}; }
  CSB_DEV bool is_zero() const { return c0.is_zero() && c1.is_zero(); }
  CSB_DEV bool operator==(const Fq2& o) const { return c0 == o.c0 && c1 == o.c1; }
  friend CSB_DEV Fq2 operator+(const Fq2& a, const Fq2& b) { return {a.c0 + b.c0, a.c1 + b.c1}; }
  friend CSB_DEV Fq2 operator-(const Fq2& a, const Fq2& b) { return {a.c0 - b.c0, a.c1 - b.c1}; }
  // Karatsuba on unreduced products (src/cuda/ff.cpp montmult_ext_h: same non-residue -1):
  // three 512-bit products, combined before two reductions instead of reduced one by one (336
  // multiply-adds instead of 408, and 16-limb subtractions instead of five modular ones).
  static CSB_DEV Fq2 mul_kar(const Fq2& a, const Fq2& b) {
    uint32_t t0[16], t1[16], s[16], br;
    const Fq sa = Fq::add_raw(a.c0, a.c1), sb = Fq::add_raw(b.c0, b.c1);  // < 2q
    csb::mul_wide(t0, a.c0.v, b.c0.v);
    csb::mul_wide(t1, a.c1.v, b.c1.v);
    csb::mul_wide(s, sa.v, sb.v);
    // s - t0 - t1 = a0 b1 + a1 b0 < 2q^2
    SUB_CC(s[0], s[0], t0[0]);
#pragma unroll
    for (int k = 1; k < 15; k++) SUBC_CC(s[k], s[k], t0[k]);
    SUBC(s[15], s[15], t0[15]);
    SUB_CC(s[0], s[0], t1[0]);
#pragma unroll
    for (int k = 1; k < 15; k++) SUBC_CC(s[k], s[k], t1[k]);
    SUBC(s[15], s[15], t1[15]);
    // t0 - t1, plus q 2^256 where negative: below q 2^256
    SUB_CC(t0[0], t0[0], t1[0]);
#pragma unroll
    for (int k = 1; k < 16; k++) SUBC_CC(t0[k], t0[k], t1[k]);
    SUBC(br, 0u, 0u);
    ADD_CC(t0[8], t0[8], ModQ::P0 & br);    ADDC_CC(t0[9], t0[9], ModQ::P1 & br);
    ADDC_CC(t0[10], t0[10], ModQ::P2 & br); ADDC_CC(t0[11], t0[11], ModQ::P3 & br);
    ADDC_CC(t0[12], t0[12], ModQ::P4 & br); ADDC_CC(t0[13], t0[13], ModQ::P5 & br);
    ADDC_CC(t0[14], t0[14], ModQ::P6 & br); ADDC(t0[15], t0[15], ModQ::P7 & br);
    return {Fq::redc_wide(t0).canon(), Fq::redc_wide(s).canon()};
  }
  // (a0 + a1 u)^2 = (a0 + a1)(a0 - a1) + 2 a0 a1 u, the factors below 2q
  static CSB_DEV Fq2 sqr_two(const Fq2& a) {
    const Fq r0 = Fq::mul_raw(Fq::add_raw(a.c0, a.c1), Fq::sub_raw(a.c0, a.c1));
    return {r0.canon(), Fq::mul_raw(Fq::add_raw(a.c0, a.c0), a.c1).canon()};
  }
  friend CSB_DEV Fq2 operator*(const Fq2& a, const Fq2& b);
  CSB_DEV Fq2 sqr() const;
  CSB_DEV Fq2 neg() const { return {c0.neg(), c1.neg()}; }
  CSB_DEV Fq2 dbl() const { return {c0.dbl(), c1.dbl()}; }
  CSB_DEV Fq2 inv() const {
    const Fq d = (c0.sqr() + c1.sqr()).inv();
    return {c0 * d, (c1 * d).neg()};
  }
};

static __device__ __noinline__ Fq2 fq2_mul_call(Fq2 a, Fq2 b) { return Fq2::mul_kar(a, b); }
static __device__ __noinline__ Fq2 fq2_sqr_call(Fq2 a) { return Fq2::sqr_two(a); }
#if defined(CSB_MUL_NOINLINE)
CSB_DEV Fq2 operator*(const Fq2& a, const Fq2& b) { return fq2_mul_call(a, b); }
CSB_DEV Fq2 Fq2::sqr() const { return fq2_sqr_call(*this); }
#else
CSB_DEV Fq2 operator*(const Fq2& a, const Fq2& b) { return Fq2::mul_kar(a, b); }
CSB_DEV Fq2 Fq2::sqr() const { return Fq2::sqr_two(*this); }
#endif

}  // namespace csb
