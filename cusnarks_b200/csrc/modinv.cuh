// modinv.cuh -- inverse mod an odd 254-bit modulus (host and device).
//
// Binary GCD on word-sized approximations (Pornin, "Optimized binary GCD for modular
// inversion", 2020): 30 division steps at a time run on 62-bit approximations of a and b
// (their low 30 and their top 32 bits), collecting a 2x2 matrix of 31-bit factors that is
// then applied to the full a, b and to the cofactors u, v.  17 rounds reach gcd 1 for any
// 254-bit operand, with no data-dependent branch, so lanes of a warp stay together.  One
// thread's chain: about 500 dependent steps of a few instructions on one word pair instead of
// about 500 steps on eight limbs each.
#pragma once
#include <cstdint>

namespace csb {

namespace modinv_detail {
// r = |x f + y g| / 2^30 for an exact division; returns all ones where x f + y g < 0
__host__ __device__ inline uint32_t update_ab(const uint32_t* x, const uint32_t* y, int32_t f, int32_t g, uint32_t* r) {
  int64_t c = 0;
  uint32_t t[9];
  for (int i = 0; i < 8; i++) {
    c += (int64_t)((uint64_t)x[i]) * f + (int64_t)((uint64_t)y[i]) * g;
    t[i] = (uint32_t)c;
    c >>= 32;
  }
  t[8] = (uint32_t)c;
  const uint32_t neg = (uint32_t)(c >> 63);
  uint32_t carry = neg & 1u;
  for (int i = 0; i < 8; i++) {
    const uint32_t w = (t[i] >> 30) | (t[i + 1] << 2);
    const uint64_t s = (uint64_t)(w ^ neg) + carry;
    r[i] = (uint32_t)s;
    carry = (uint32_t)(s >> 32);
  }
  return neg;
}
// r = (x f + y g) / 2^30 mod p for x, y < p; np = -1/p mod 2^32
__host__ __device__ inline void update_uv(const uint32_t* x, const uint32_t* y, int32_t f, int32_t g, const uint32_t* p,
                                          uint32_t np, uint32_t* r) {
  // add the multiple of p that makes the sum divisible by 2^30
  const uint32_t q = ((x[0] * (uint32_t)f + y[0] * (uint32_t)g) * np) & 0x3fffffffu;
  int64_t c = 0;
  uint32_t t[9];
  for (int i = 0; i < 8; i++) {
    c += (int64_t)((uint64_t)x[i]) * f + (int64_t)((uint64_t)y[i]) * g;
    // the running sum stays below 2^63: |f| + |g| <= 2^30 and q < 2^30
    c += (int64_t)((uint64_t)p[i] * q);
    t[i] = (uint32_t)c;
    c >>= 32;
  }
  t[8] = (uint32_t)c;
  // (-p, 2p) -> [0, p)
  const uint32_t neg = (uint32_t)(c >> 63);
  uint32_t carry = 0;
  for (int i = 0; i < 8; i++) {
    const uint32_t w = (t[i] >> 30) | (t[i + 1] << 2);
    const uint64_t s = (uint64_t)w + (p[i] & neg) + carry;
    r[i] = (uint32_t)s;
    carry = (uint32_t)(s >> 32);
  }
  uint32_t u[8], borrow = 0;
  for (int i = 0; i < 8; i++) {
    const uint64_t s = (uint64_t)r[i] - p[i] - borrow;
    u[i] = (uint32_t)s;
    borrow = (uint32_t)(s >> 63);
  }
  for (int i = 0; i < 8; i++) r[i] = borrow ? r[i] : u[i];
}
}  // namespace modinv_detail

// out = x^-1 mod p for 0 < x < p (0 for x = 0); np = -1/p mod 2^32
__host__ __device__ inline void modinv(const uint32_t* x, const uint32_t* p, uint32_t np, uint32_t* out) {
  using namespace modinv_detail;
  uint32_t a[8], b[8], u[8], v[8], ra[8], rb[8];
  for (int i = 0; i < 8; i++) { a[i] = x[i]; b[i] = p[i]; u[i] = i == 0; v[i] = 0; }
#pragma unroll 1
  for (int round = 0; round < 17; round++) {
    // the two limbs from the longer operand's highest nonzero one down, of which the top 32 bits
    // are taken; operands that fit 62 bits are taken whole
    uint32_t a2 = a[1], a1 = a[0], b2 = b[1], b1 = b[0];
    for (int i = 2; i < 8; i++) {
      const bool nz = (a[i] | b[i]) != 0;
      a2 = nz ? a[i] : a2; a1 = nz ? a[i - 1] : a1;
      b2 = nz ? b[i] : b2; b1 = nz ? b[i - 1] : b1;
    }
    const bool big = (a[2] | a[3] | a[4] | a[5] | a[6] | a[7] | b[2] | b[3] | b[4] | b[5] | b[6] | b[7]) != 0;
    const uint32_t top = a2 | b2;
#ifdef __CUDA_ARCH__
    int lz = __clz((int)top);
#else
    int lz = top ? __builtin_clz(top) : 32;
#endif
    const bool whole = !big && lz >= 2;
    lz &= 31;
    // top 32 bits of the two limbs
    const uint32_t ta = (uint32_t)((((uint64_t)a2 << 32 | a1) << lz) >> 32);
    const uint32_t tb = (uint32_t)((((uint64_t)b2 << 32 | b1) << lz) >> 32);
    uint64_t xa = (uint64_t)ta << 30 | (a[0] & 0x3fffffffu), xb = (uint64_t)tb << 30 | (b[0] & 0x3fffffffu);
    if (whole) {
      xa = (uint64_t)a[1] << 32 | a[0];
      xb = (uint64_t)b[1] << 32 | b[0];
    }
    int32_t f0 = 1, g0 = 0, f1 = 0, g1 = 1;
#pragma unroll 5
    for (int k = 0; k < 30; k++) {
      const bool odd = (xa & 1u) != 0;
      const bool swap = odd && xa < xb;
      const uint64_t ya = swap ? xb : xa, yb = swap ? xa : xb;
      const int32_t p0 = swap ? f1 : f0, p1 = swap ? f0 : f1, q0 = swap ? g1 : g0, q1 = swap ? g0 : g1;
      xa = (ya - (odd ? yb : 0)) >> 1;
      xb = yb;
      f0 = p0 - (odd ? p1 : 0);
      g0 = q0 - (odd ? q1 : 0);
      f1 = p1 * 2;
      g1 = q1 * 2;
    }
    const uint32_t na = update_ab(a, b, f0, g0, ra), nb = update_ab(a, b, f1, g1, rb);
    for (int i = 0; i < 8; i++) { a[i] = ra[i]; b[i] = rb[i]; }
    if (na) { f0 = -f0; g0 = -g0; }
    if (nb) { f1 = -f1; g1 = -g1; }
    update_uv(u, v, f0, g0, p, np, ra);
    update_uv(u, v, f1, g1, p, np, rb);
    for (int i = 0; i < 8; i++) { u[i] = ra[i]; v[i] = rb[i]; }
  }
  for (int i = 0; i < 8; i++) out[i] = v[i];
}

}  // namespace csb
