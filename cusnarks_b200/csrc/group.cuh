// group.cuh -- point operations spread over a group of lanes, operands in shared memory.
//
// For points whose chain of operations runs alone (a window's Horner steps, a scalar
// multiplication) or among too few others to fill the schedulers (the buckets and the bucket
// reduction of a small MSM): the independent products of each dependency level are computed by
// the lanes of a group, one base-field product a lane, so an addition costs 4 product latencies
// instead of 14 and a doubling 3 instead of 9.  A group is 4 lanes over Fq (a level's products)
// and 16 over Fq2 (the four products of base-field coordinates that make each Fq2 product).
// Points and products live in shared memory (lazily reduced, below 2q) and a lane reads the
// operands of its own product only: holding whole points in every lane instead, with shuffles,
// took 255 registers and 2 KB of spills a thread over Fq2.
// Every lane of a warp calls these together (warp barriers between the levels); groups of one
// warp may hold different points.
#pragma once
#include "curve.cuh"

namespace csb {

CSB_DEV Fq lds_fq(const uint32_t* p) {
  const uint4 a = reinterpret_cast<const uint4*>(p)[0], b = reinterpret_cast<const uint4*>(p)[1];
  return Fq{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
}
CSB_DEV void sts_fq(uint32_t* p, const Fq& x) { st_limbs8(p, x.v); }
CSB_DEV Fq select_fq(bool c, const Fq& a, const Fq& b) {
  Fq r;
#pragma unroll
  for (int i = 0; i < 8; i++) r.v[i] = c ? a.v[i] : b.v[i];
  return r;
}

// Equal or opposite points (rare): one lane, canonical arithmetic.  Both points are read 16 bytes
// at a time.
template <class F>
__device__ __noinline__ void group_add_slow(const uint32_t* p, const uint32_t* q, bool q_affine, bool neg,
                                            uint32_t* out) {
  constexpr int FW = FieldWords<F>::value;
  XYZZ<F> a, b = XYZZ<F>::from_affine(Affine<F>{F::zero(), F::one()});
  uint32_t* aw = reinterpret_cast<uint32_t*>(&a);
  uint32_t* bw = reinterpret_cast<uint32_t*>(&b);
  for (int k = 0; k < FW / 2; k++) {  // coordinates of Fq
    Fq x = lds_fq(p + 8 * k).canon();
    for (int i = 0; i < 8; i++) aw[8 * k + i] = x.v[i];
    if (q_affine && k >= FW / 4) continue;
    x = lds_fq(q + 8 * k).canon();
    for (int i = 0; i < 8; i++) bw[8 * k + i] = x.v[i];
  }
  if (neg) b.Y = b.Y.neg();
  const XYZZ<F> r = xyzz_add(a, b);
  const uint32_t* rw = reinterpret_cast<const uint32_t*>(&r);
  for (int k = 0; k < 4 * FW; k++) out[k] = rw[k];
}

template <class F>
struct Group {
  static constexpr int C = FieldWords<F>::value / 8;   // base-field coordinates of an element
  static constexpr int G = C == 1 ? 4 : 16;            // lanes
  static constexpr int PW = 32 * C;                    // words of a point (X, Y, ZZ, ZZZ)
  static constexpr int kScratch = 4 * G * 8;           // words: four levels of products

  int l, j, a, b;  // lane; its product of a level, and the coordinates of the factors it takes
  uint32_t* scr;

  CSB_DEV explicit Group(uint32_t* scratch) : scr(scratch) {
    l = threadIdx.x & (G - 1);
    if (C == 1) { j = l; a = b = 0; }
    else { j = l >> 2; a = (l >> 1) & 1; b = l & 1; }
  }
  static CSB_DEV const uint32_t* at(const uint32_t* pt, int coord, int c) { return pt + (coord * C + c) * 8; }
  // coordinate c of product k of a level
  CSB_DEV Fq val(int level, int k, int c) const {
    return lds_fq(scr + (level * G + C * k + c) * 8);
  }
  // This lane's product of the level.  Over Fq2 eight lanes then join the four products of
  // coordinates of each element (c = 0: p00 - p11, c = 1: p01 + p10) in place, once for all
  // readers (joined by every reader instead, 254 doublings and the inversion of a window sum
  // took 650 us, now 629, and the bit trees and window sums of a small MSM 8-9 % more).
  CSB_DEV void put(int level, const Fq& x, const Fq& y) const {
    uint32_t* s = scr + level * G * 8;
    sts_fq(s + l * 8, Fq::mul_raw(x, y));
    __syncwarp();
    if (C == 2) {
      Fq r;
      if (l < 8) {
        const int k = l >> 1, c = l & 1;
        const Fq u = lds_fq(s + (4 * k + c) * 8), v = lds_fq(s + (4 * k + 3 - c) * 8);
        r = Fq::add_lazy(u, select_fq(c != 0, v, Fq::neg_lazy(v)));
      }
      __syncwarp();
      if (l < 8) sts_fq(s + l * 8, r);
      __syncwarp();
    }
  }
  static CSB_DEV bool zero_coord(const uint32_t* pt, int coord) {
    bool z = lds_fq(at(pt, coord, 0)).is_zero_lazy();
    if (C == 2) z = z && lds_fq(at(pt, coord, 1)).is_zero_lazy();
    return z;
  }
  // whether the element whose coordinate a is held by the lanes of product k is zero
  CSB_DEV bool element_zero(bool z, int k) const {
    const uint32_t m = __ballot_sync(0xffffffffu, z) >> ((threadIdx.x & 31) & ~(G - 1));
    return C == 1 ? ((m >> k) & 1u) != 0 : ((m >> (4 * k)) & 5u) == 5u;
  }
  // dst = p + q (add-2008-s), unless !live; points in shared memory (dst may be p or q), q also
  // in global memory
  CSB_DEV void add(uint32_t* dst, const uint32_t* p, const uint32_t* q, bool live = true) const {
    const bool inf1 = zero_coord(p, 2), inf2 = zero_coord(q, 2);
    // level 1: U1 = X1 ZZ2, U2 = X2 ZZ1, S1 = Y1 ZZZ2, S2 = Y2 ZZZ1
    {
      const int xy = j >> 1;
      const uint32_t *f = (j & 1) ? q : p, *g = (j & 1) ? p : q;
      put(0, lds_fq(at(f, xy, a)), lds_fq(at(g, 2 + xy, b)));
    }
    // level 2: PP = P^2, RR = R^2, Z2 = ZZ1 ZZ2, Z3 = ZZZ1 ZZZ2, with P = U2 - U1, R = S2 - S1
    const int k = 2 * (j & 1);
    const Fq pr = Fq::sub_lazy(val(0, k + 1, a), val(0, k, a));
    const bool same = element_zero(pr.is_zero_lazy(), 0) && !inf1 && !inf2 && live;
    {
      const int zc = 2 + (j & 1);
      const Fq prb = C == 1 ? pr : Fq::sub_lazy(val(0, k + 1, b), val(0, k, b));
      const bool z = j >= 2;
      put(1, select_fq(z, lds_fq(at(p, zc, a)), pr), select_fq(z, lds_fq(at(q, zc, b)), prb));
    }
    // level 3: PPP = P PP, Q = U1 PP, ZZ3 = Z2 PP
    {
      const Fq v = val(j == 1 ? 0 : 1, j == 1 ? 0 : 2, a);
      put(2, select_fq(j == 0, pr, v), val(1, 0, b));
    }
    // level 4: S1 PPP, R (Q - X3), ZZZ3 = Z3 PPP, with X3 = RR - PPP - 2 Q
    const Fq s1 = val(j == 0 ? 0 : 1, j == 0 ? 2 : 3, a);
    if (__any_sync(0xffffffffu, same)) {
      __syncwarp();  // a vote orders no memory accesses: s1 has been read before level 1 is written over
      if (same && l == 0) group_add_slow<F>(p, q, false, false, scr);
    }
    finish(dst, p, inf1, inf2, same, live, pr, s1, q, q + 16 * C, false, false);
  }

  // dst = p + (qx, +-qy) (madd-2008-s), affine and canonical, unless !live
  CSB_DEV void madd(uint32_t* dst, const uint32_t* p, const uint32_t* qx, const uint32_t* qy, bool neg, bool live) const {
    const bool inf1 = zero_coord(p, 2);
    Fq y2 = lds_fq(qy + 8 * a);
    {
      Fq n = Fq::zero() - y2;
      y2 = select_fq(neg, n, y2);
    }
    // level 1: U2 = X2 ZZ1, S2 = Y2 ZZZ1
    put(0, select_fq((j & 1) != 0, y2, lds_fq(qx + 8 * a)), lds_fq(at(p, 2 + (j & 1), b)));
    // level 2: PP, RR
    const Fq pr = Fq::sub_lazy(val(0, j & 1, a), lds_fq(at(p, j & 1, a)));
    const bool same = element_zero(pr.is_zero_lazy(), 0) && !inf1 && live;
    {
      const Fq prb = C == 1 ? pr : Fq::sub_lazy(val(0, j & 1, b), lds_fq(at(p, j & 1, b)));
      put(1, pr, prb);
    }
    // level 3: PPP = P PP, Q = X1 PP, ZZ3 = ZZ1 PP
    put(2, select_fq(j == 0, pr, lds_fq(at(p, j == 1 ? 0 : 2, a))), val(1, 0, b));
    // level 4: Y1 PPP, R (Q - X3), ZZZ1 PPP
    const Fq s1 = lds_fq(at(p, j == 0 ? 1 : 3, a));
    // level 1 of the scratch was last read before level 2's barriers
    if (__any_sync(0xffffffffu, same) && same && l == 0) {
      __align__(16) uint32_t q[PW / 2];  // read as uint4
      for (int i = 0; i < PW / 4; i++) { q[i] = qx[i]; q[PW / 4 + i] = qy[i]; }
      group_add_slow<F>(p, q, true, neg, scr);
    }
    finish(dst, p, inf1, false, same, live, pr, s1, qx, qy, true, neg);
  }

  // Level 4 of both additions -- s1 PPP, R (Q - X3), and the ZZZ product (s1 of those lanes times
  // PPP), with X3 = RR - PPP - 2 Q and pr = R in the lanes of product 1 -- and the result: the sum,
  // or what stands in the scratch (same), q where p is infinity, p where q is.  qx, q2: q's first
  // two coordinates and the other two, or x and y where it is affine.
  CSB_DEV void finish(uint32_t* dst, const uint32_t* p, bool inf1, bool inf2, bool same, bool live, const Fq& pr,
                      const Fq& s1, const uint32_t* qx, const uint32_t* q2, bool q_affine, bool neg) const {
    const Fq ppp = val(2, 0, b), qq = val(2, 1, b);
    const Fq x3 = Fq::sub_lazy(Fq::sub_lazy(val(1, 1, b), ppp), Fq::add_lazy(qq, qq));
    put(3, select_fq(j == 1, pr, s1), select_fq(j == 1, Fq::sub_lazy(qq, x3), ppp));
    if (l < 4 * C && live) {
      const int coord = l / C, c = l % C;  // c = b: x3 is this lane's
      const Fq v = val(coord == 2 ? 2 : 3, coord == 2 ? 2 : coord == 1 ? 1 : 2, c);
      Fq r = select_fq(coord == 0, x3, select_fq(coord == 1, Fq::sub_lazy(v, val(3, 0, c)), v));
      if (same) r = lds_fq(scr + 8 * l);
      if (inf2) {
        r = lds_fq(p + 8 * l);
      } else if (inf1) {
        if (!q_affine) {
          r = coord < 2 ? lds_fq(qx + 8 * l) : lds_fq(q2 + 8 * (l - 2 * C));
        } else if (coord < 2) {
          r = lds_fq((coord == 0 ? qx : q2) + 8 * c);
          if (coord == 1 && neg) r = r.neg();
        } else {
          r = c == 0 ? Fq::one() : Fq::zero();
        }
      }
      sts_fq(dst + 8 * l, r);
    }
    __syncwarp();
  }

  // dst = 2 p (dbl-2008-s-1), unless !live; infinity stays infinity (ZZ = 0)
  CSB_DEV void dbl(uint32_t* dst, const uint32_t* p, bool live = true) const {
    // level 1: V = U^2, XX = X^2 with U = 2 Y
    const int c0 = (j & 1) ? 0 : 1;
    const Fq v0 = lds_fq(at(p, c0, a)), w0 = lds_fq(at(p, c0, b));
    const Fq u = select_fq(c0 == 1, Fq::add_lazy(v0, v0), v0);  // U (product 0) or X (product 1)
    put(0, u, select_fq(c0 == 1, Fq::add_lazy(w0, w0), w0));
    // level 2: W = U V, S = X V, MM = M^2, ZZ3 = V ZZ with M = 3 XX
    const Fq xa = val(0, 1, a), xb = val(0, 1, b);
    const Fq ma = Fq::add_lazy(Fq::add_lazy(xa, xa), xa), mb = Fq::add_lazy(Fq::add_lazy(xb, xb), xb);
    put(1, select_fq(j < 2, u, select_fq(j == 2, ma, lds_fq(at(p, 2, a)))), select_fq(j == 2, mb, val(0, 0, b)));
    // level 3: W Y, M (S - X3), ZZZ3 = W ZZZ with X3 = MM - 2 S
    const Fq s = val(1, 1, b);
    const Fq x3 = Fq::sub_lazy(val(1, 2, b), Fq::add_lazy(s, s));
    put(2, select_fq(j == 1, ma, val(1, 0, a)),
        select_fq(j == 1, Fq::sub_lazy(s, x3), lds_fq(at(p, j == 0 ? 1 : 3, b))));
    if (l < 4 * C && live) {
      const int coord = l / C, c = l % C;
      const Fq v = val(coord == 2 ? 1 : 2, coord == 2 ? 3 : coord == 1 ? 1 : 2, c);
      sts_fq(dst + 8 * l, select_fq(coord == 0, x3, select_fq(coord == 1, Fq::sub_lazy(v, val(2, 0, c)), v)));
    }
    __syncwarp();
  }

  // shared <- canonical point in global memory where have, else infinity
  CSB_DEV void load(uint32_t* dst, const uint32_t* src, bool have = true) const {
    if (l < 4 * C) {
      Fq x = l == C ? Fq::one() : Fq::zero();
      if (have) x = lds_fq(src + 8 * l);
      sts_fq(dst + 8 * l, x);
    }
    __syncwarp();
  }
  CSB_DEV void store(uint32_t* dst, const uint32_t* src) const {
    if (l < 4 * C) sts_fq(dst + 8 * l, lds_fq(src + 8 * l).canon());
  }
  // one lane: the point in shared memory to an affine one in global memory
  static CSB_DEV void store_affine(uint32_t* dst, const uint32_t* src) {
    XYZZ<F> r;
    uint32_t* w = reinterpret_cast<uint32_t*>(&r);
    for (int k = 0; k < 4 * C; k++) {
      const Fq x = lds_fq(src + 8 * k).canon();
      for (int i = 0; i < 8; i++) w[8 * k + i] = x.v[i];
    }
    st_affine<F>(dst, xyzz_to_affine(r));
  }
};

// A run of doublings over Fq in two product levels each instead of three, from the curve equation
// y^2 = x^3 + 3 (X^3 = Y^2 - C with C = 3 ZZZ^2): with B = Y^2,
//   X' = X (B - 9 C),  Y' = (B + 9 C)^2 - 108 C^2,  ZZZ' = 8 B (Y ZZZ),  ZZ' = 4 B ZZ,
// the first level B, ZZZ^2, Y ZZZ and the previous step's ZZ', the second the other products;
// small multiples cost a twentieth of a product (Fp::mul_small).  1.28 us a doubling against
// 1.7 of Group::dbl.  (Over Fq2 the curve constant is a full element, which takes a fifth
// product and all 32 lanes: no faster than Group::dbl, 651 and 637 us for 252 doublings.)
// Points must lie on the curve, as an MSM's inputs do.
// pt <- 2^d pt (shared memory); with steps given, the points 2^i pt go to steps + 32 i
// (i = 1..d, and ZZ of i = 0) and pt stays.  Nothing is written where !live.
CSB_DEV void doubling_run(uint32_t* scr, uint32_t* pt, int d, uint32_t* steps = nullptr, bool live = true) {
  if (d <= 0) return;
  const int j = threadIdx.x & 3;
  auto val = [&](int level, int k) { return lds_fq(scr + (level * 4 + k) * 8); };
  auto put = [&](int level, const Fq& x, const Fq& y) {
    sts_fq(scr + (level * 4 + j) * 8, Fq::mul_raw(x, y));
    __syncwarp();
  };
  Fq X = lds_fq(pt), Y = lds_fq(pt + 8), ZZ = lds_fq(pt + 16), Z3 = lds_fq(pt + 24), b4 = Fq::one();
  __syncwarp();
#pragma unroll 1
  for (int i = 1; i <= d; i++) {
    // Y Y, ZZZ ZZZ, Y ZZZ, ZZ (4 B) of the step before
    put(0, select_fq(j == 3, ZZ, select_fq(j == 1, Z3, Y)), select_fq(j == 0, Y, select_fq(j == 3, b4, Z3)));
    const Fq B = val(0, 0), S = val(0, 1);  // S = C / 3
    ZZ = val(0, 3);
    if (steps && live && j == 2) sts_fq(steps + (size_t)(i - 1) * 32 + 16, ZZ);
    // X (B - 27 S), (B + 27 S)^2, S (972 S), (Y ZZZ) (8 B)
    const Fq m = Fq::mul_small(select_fq(j == 3, B, S), j == 3 ? 8u : j == 2 ? 972u : 27u);
    put(1, select_fq(j == 0, X, select_fq(j == 1, Fq::add_lazy(B, m), select_fq(j == 2, S, val(0, 2)))),
        select_fq(j == 0, Fq::sub_lazy(B, m), select_fq(j == 1, Fq::add_lazy(B, m), m)));
    X = val(1, 0);
    Y = Fq::sub_lazy(val(1, 1), val(1, 2));
    Z3 = val(1, 3);
    b4 = Fq::add_lazy(B, B);
    b4 = Fq::add_lazy(b4, b4);
    if (steps && live && i < d && j != 2)
      sts_fq(steps + (size_t)i * 32 + 8 * j, select_fq(j == 0, X, select_fq(j == 1, Y, Z3)));
  }
  ZZ = Fq::mul_raw(ZZ, b4);
  if (live)
    sts_fq((steps ? steps + (size_t)d * 32 : pt) + 8 * j,
           select_fq(j == 0, X, select_fq(j == 1, Y, select_fq(j == 2, ZZ, Z3))));
  __syncwarp();
}
// pt <- 2^d pt for a group's point
template <class F>
CSB_DEV void double_times(const Group<F>& grp, uint32_t* pt, int d, bool live = true) {
  if constexpr (Group<F>::C == 1) {
    doubling_run(grp.scr, pt, d, nullptr, live);
  } else {
#pragma unroll 1
    for (int i = 0; i < d; i++) grp.dbl(pt, pt, live);
  }
}

}  // namespace csb
