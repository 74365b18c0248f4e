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
// Each helper is one PTX instruction; `volatile` keeps the carry flag sequence in
// program order.
#define ADD_CC(d, a, b)     asm volatile("add.cc.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b))
#define ADDC_CC(d, a, b)    asm volatile("addc.cc.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b))
#define ADDC(d, a, b)       asm volatile("addc.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b))
#define SUB_CC(d, a, b)     asm volatile("sub.cc.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b))
#define SUBC_CC(d, a, b)    asm volatile("subc.cc.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b))
#define SUBC(d, a, b)       asm volatile("subc.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b))

// Montgomery products accumulate in two sets of columns: e holds columns 0..7 as the 64-bit
// pairs (0,1) (2,3) (4,5) (6,7), o columns 1..8 as (1,2) (3,4) (5,6) (7,8), and the value is
// e + 2^32 o.  A limb's products with the even limbs of the other operand tile e's pairs and
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
  asm("{\n\t"
      "mad.lo.cc.u32 %8, %17, %24, %8;\n\tmadc.hi.cc.u32 %9, %17, %24, %9;\n\t"
      "madc.lo.cc.u32 %10, %19, %24, %10;\n\tmadc.hi.cc.u32 %11, %19, %24, %11;\n\t"
      "madc.lo.cc.u32 %12, %21, %24, %12;\n\tmadc.hi.cc.u32 %13, %21, %24, %13;\n\t"
      "madc.lo.cc.u32 %14, %23, %24, %14;\n\tmadc.hi.u32 %15, %23, %24, %15;\n\t"
      "mad.lo.cc.u32 %0, %16, %24, %0;\n\tmadc.hi.cc.u32 %1, %16, %24, %1;\n\t"
      "madc.lo.cc.u32 %2, %18, %24, %2;\n\tmadc.hi.cc.u32 %3, %18, %24, %3;\n\t"
      "madc.lo.cc.u32 %4, %20, %24, %4;\n\tmadc.hi.cc.u32 %5, %20, %24, %5;\n\t"
      "madc.lo.cc.u32 %6, %22, %24, %6;\n\tmadc.hi.cc.u32 %7, %22, %24, %7;\n\t"
      "addc.u32 %15, %15, 0;\n\t}"
      : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]), "+r"(o[0]),
        "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(b));
}
// (e, o) <- ((e, o) >> 32) + a * b, for e[0] = 0.  The left-over limb e[1] goes into the new
// column 0 first; its carry (column 1) enters the odd chain, which starts there.
CSB_DEV void eo_shift_mad(uint32_t (&e)[8], uint32_t (&o)[8], const uint32_t (&a)[8], uint32_t b) {
  uint32_t n0, n1, n2, n3, n4, n5, n6, n7;
  asm("{\n\t"
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
      : "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7]), "=&r"(n0),
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
  CSB_DEV bool is_one() const { return *this == one(); }

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

  // ---- lazily reduced values in [0, 2p) (BN254: 4p < 2^256): products of two such values
  // are below 2p without the final subtraction (1.76 p)
  static CSB_DEV Fp mul_lazy(const Fp& a, const Fp& b);
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

  CSB_DEV Fp sqr() const { return (*this) * (*this); }

  // x -> x * R mod p (normal form to Montgomery); any 256-bit x is accepted: the product
  // with r2 < p on the left is below 2p.
  CSB_DEV Fp to_mont() const { return r2() * (*this); }
  CSB_DEV Fp from_mont() const {
    Fp o = zero();
    o.v[0] = 1;
    return (*this) * o;
  }

  // Montgomery inverse (aR -> a^-1 R; 0 -> 0).  Binary extended Euclid on the integer
  // x = aR gives x^-1 = a^-1 R^-1; one Montgomery product by R^3 restores a^-1 R.  Used
  // for the few final affine conversions, where a single thread's latency is what counts.
  CSB_DEV Fp inv() const {
    if (is_zero()) return zero();
    const uint32_t P[8] = {M::P0, M::P1, M::P2, M::P3, M::P4, M::P5, M::P6, M::P7};
    uint32_t u[8], v[8], x1[8], x2[8];
#pragma unroll
    for (int i = 0; i < 8; i++) { u[i] = this->v[i]; v[i] = P[i]; x1[i] = 0; x2[i] = 0; }
    x1[0] = 1;
#pragma unroll 1
    for (int guard = 0; guard < 2048; guard++) {
      const bool u1 = (u[0] == 1) && ((u[1] | u[2] | u[3] | u[4] | u[5] | u[6] | u[7]) == 0);
      const bool v1 = (v[0] == 1) && ((v[1] | v[2] | v[3] | v[4] | v[5] | v[6] | v[7]) == 0);
      if (u1 || v1) break;
      // (a zero u or v only arises from an unreduced input; the bounded loops end anyway)
#pragma unroll 1
      for (int k = 0; k < 256 && (u[0] & 1u) == 0; k++) { shr1(u); half_mod(x1, P); }
#pragma unroll 1
      for (int k = 0; k < 256 && (v[0] & 1u) == 0; k++) { shr1(v); half_mod(x2, P); }
      if (geq(u, v)) { sub8(u, v); sub_mod(x1, x2, P); }
      else { sub8(v, u); sub_mod(x2, x1, P); }
    }
    const bool u1 = (u[0] == 1) && ((u[1] | u[2] | u[3] | u[4] | u[5] | u[6] | u[7]) == 0);
    Fp r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = u1 ? x1[i] : x2[i];
    return r * r3();
  }

 private:
  static CSB_DEV void shr1(uint32_t (&a)[8]) {
#pragma unroll
    for (int i = 0; i < 7; i++) a[i] = (a[i] >> 1) | (a[i + 1] << 31);
    a[7] >>= 1;
  }
  static CSB_DEV bool geq(const uint32_t (&a)[8], const uint32_t (&b)[8]) {
#pragma unroll
    for (int i = 7; i >= 0; i--) {
      if (a[i] != b[i]) return a[i] > b[i];
    }
    return true;
  }
  static CSB_DEV void sub8(uint32_t (&a)[8], const uint32_t (&b)[8]) {
    SUB_CC(a[0], a[0], b[0]); SUBC_CC(a[1], a[1], b[1]); SUBC_CC(a[2], a[2], b[2]);
    SUBC_CC(a[3], a[3], b[3]); SUBC_CC(a[4], a[4], b[4]); SUBC_CC(a[5], a[5], b[5]);
    SUBC_CC(a[6], a[6], b[6]); SUBC(a[7], a[7], b[7]);
  }
  // x <- x/2 mod p for x < p
  static CSB_DEV void half_mod(uint32_t (&x)[8], const uint32_t (&P)[8]) {
    if (x[0] & 1u) {
      uint32_t c;
      ADD_CC(x[0], x[0], P[0]); ADDC_CC(x[1], x[1], P[1]); ADDC_CC(x[2], x[2], P[2]);
      ADDC_CC(x[3], x[3], P[3]); ADDC_CC(x[4], x[4], P[4]); ADDC_CC(x[5], x[5], P[5]);
      ADDC_CC(x[6], x[6], P[6]); ADDC_CC(x[7], x[7], P[7]); ADDC(c, 0u, 0u);
      shr1(x);
      x[7] |= c << 31;
    } else {
      shr1(x);
    }
  }
  // x <- x - y mod p for x, y < p
  static CSB_DEV void sub_mod(uint32_t (&x)[8], const uint32_t (&y)[8], const uint32_t (&P)[8]) {
    uint32_t br;
    SUB_CC(x[0], x[0], y[0]); SUBC_CC(x[1], x[1], y[1]); SUBC_CC(x[2], x[2], y[2]);
    SUBC_CC(x[3], x[3], y[3]); SUBC_CC(x[4], x[4], y[4]); SUBC_CC(x[5], x[5], y[5]);
    SUBC_CC(x[6], x[6], y[6]); SUBC_CC(x[7], x[7], y[7]); SUBC(br, 0u, 0u);
    if (br) {
      ADD_CC(x[0], x[0], P[0]); ADDC_CC(x[1], x[1], P[1]); ADDC_CC(x[2], x[2], P[2]);
      ADDC_CC(x[3], x[3], P[3]); ADDC_CC(x[4], x[4], P[4]); ADDC_CC(x[5], x[5], P[5]);
      ADDC_CC(x[6], x[6], P[6]); ADDC(x[7], x[7], P[7]);
    }
  }

 public:
};

using Fq = Fp<ModQ>;
using Fr = Fp<ModR>;

template <class M>
__device__ __noinline__ Fp<M> fp_mul_call(Fp<M> a, Fp<M> b) {
  return Fp<M>::mul_raw(a, b).canon();
}

template <class M>
__device__ __noinline__ Fp<M> fp_mul_lazy_call(Fp<M> a, Fp<M> b) {
  return Fp<M>::mul_raw(a, b);
}

template <class M>
CSB_DEV Fp<M> Fp<M>::mul_lazy(const Fp<M>& a, const Fp<M>& b) {
#if defined(CSB_MUL_NOINLINE)
  return fp_mul_lazy_call<M>(a, b);
#else
  return mul_raw(a, b);
#endif
}

// ------------------------------------------------------------ Fq2 = Fq[u]/(u^2+1) ----
struct Fq2 {
  Fq c0, c1;
  static CSB_DEV Fq2 zero() { return {Fq::zero(), Fq::zero()}; }
  static CSB_DEV Fq2 one() { return {Fq::one(), Fq::zero()}; }
  CSB_DEV bool is_zero() const { return c0.is_zero() && c1.is_zero(); }
  CSB_DEV bool operator==(const Fq2& o) const { return c0 == o.c0 && c1 == o.c1; }
  friend CSB_DEV Fq2 operator+(const Fq2& a, const Fq2& b) { return {a.c0 + b.c0, a.c1 + b.c1}; }
  friend CSB_DEV Fq2 operator-(const Fq2& a, const Fq2& b) { return {a.c0 - b.c0, a.c1 - b.c1}; }
  // Karatsuba, 3 products (src/cuda/ff.cpp montmult_ext_h: same non-residue -1)
  friend CSB_DEV Fq2 operator*(const Fq2& a, const Fq2& b) {
    const Fq v0 = a.c0 * b.c0;
    const Fq v1 = a.c1 * b.c1;
    const Fq s = (a.c0 + a.c1) * (b.c0 + b.c1);
    return {v0 - v1, s - v0 - v1};
  }
  // (a0 + a1 u)^2 = (a0 + a1)(a0 - a1) + 2 a0 a1 u
  CSB_DEV Fq2 sqr() const {
    const Fq p = c0 * c1;
    return {(c0 + c1) * (c0 - c1), p + p};
  }
  CSB_DEV Fq2 neg() const { return {c0.neg(), c1.neg()}; }
  CSB_DEV Fq2 dbl() const { return {c0.dbl(), c1.dbl()}; }
  CSB_DEV Fq2 inv() const {
    const Fq d = (c0.sqr() + c1.sqr()).inv();
    return {c0 * d, (c1 * d).neg()};
  }
};

}  // namespace csb
