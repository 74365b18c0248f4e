// msm_impl.cuh -- kernels and launch sequence of the Pippenger MSM (pipeline in msm.cuh),
// instantiated for G1 in msm_g1.cu and for G2 in msm_g2.cu.
#pragma once
#include <algorithm>
#include <atomic>
#include "msm.cuh"
#include "curve.cuh"
#include "glv.cuh"
#include "group.cuh"
#include "scan.cuh"
#include "runtime.cuh"

namespace csb {
namespace msm_detail {

constexpr int SCALAR_BITS = 254;  // scalars are reduced below r < 2^254 first
constexpr uint32_t NEG_BIT = 0x80000000u;
// Generic G1 MSMs with the GLV split: an entry of the k2 half reads phi(P_i) = (beta x_i, y_i)
// (terms below 2^30).
constexpr uint32_t PHI_BIT = 0x40000000u;
constexpr uint32_t kMinTask = 32;  // workspace bounds assume tasks of at least this size
// ... except for smaller MSMs: their bounds assume tasks of layout_min_task(entries), down to 8
// entries, so the bound stays near 65,536 tasks.  The latency form splits buckets of MSMs of
// at most kSmallEntries entries in tasks of 16 (2^12 fixed-base G1 MSM 0.469 -> 0.445 ms, 2^12
// proof 1.586 -> 1.533 ms against 32; 8 is slower: more partial sums).
constexpr size_t kSmallEntries = 1u << 19;
constexpr uint32_t kLatMinTask = 16;
inline uint32_t layout_min_task(uint64_t entries) {
  return (uint32_t)std::min<uint64_t>(kMinTask, std::max<uint64_t>(8, entries / 65536));
}

__host__ __device__ inline int num_windows(int c) { return SCALAR_BITS / c + 1; }
// Windows of a GLV half-scalar (|k1|, |k2| < 2^127): c W >= 128 leaves the top digit at most
// 2^(c-1) after the signed recoding's carry, so no further window is needed.
__host__ __device__ inline int glv_windows(int c) { return (128 + c - 1) / c; }
// Window count of an MSM: generic G1 MSMs split their scalars by the endomorphism (glv).
__host__ __device__ inline int msm_windows(int c, bool glv) { return glv ? glv_windows(c) : num_windows(c); }

// k <- k mod r for any 256-bit k (at most 5 subtractions since 2^256 / r < 6)
CSB_DEV void scalar_reduce(uint32_t (&k)[8]) {
#pragma unroll 1
  for (int it = 0; it < 6; it++) {
    uint32_t u[8], br;
    SUB_CC(u[0], k[0], ModR::P0); SUBC_CC(u[1], k[1], ModR::P1); SUBC_CC(u[2], k[2], ModR::P2);
    SUBC_CC(u[3], k[3], ModR::P3); SUBC_CC(u[4], k[4], ModR::P4); SUBC_CC(u[5], k[5], ModR::P5);
    SUBC_CC(u[6], k[6], ModR::P6); SUBC_CC(u[7], k[7], ModR::P7); SUBC(br, 0u, 0u);
    if (br) break;
#pragma unroll
    for (int i = 0; i < 8; i++) k[i] = u[i];
  }
}

CSB_DEV uint32_t scalar_bits(const uint32_t (&k)[8], int off, int c) {
  const int w = off >> 5, sh = off & 31;
  if (w >= 8) return 0;
  uint32_t v = k[w] >> sh;
  if (sh + c > 32 && w + 1 < 8) v |= k[w + 1] << (32 - sh);
  return v & ((1u << c) - 1u);
}

// Signed recoding: digit j in (-2^(c-1), 2^(c-1)].  Calls f(j, |d|, negative) for
// every nonzero digit.
template <class Fn>
CSB_DEV void for_each_digit(const uint32_t (&k)[8], int c, int W, Fn f) {
  const uint32_t half = 1u << (c - 1);
  const uint32_t full = 1u << c;
  uint32_t carry = 0;
  for (int j = 0; j < W; j++) {
    const uint32_t raw = scalar_bits(k, j * c, c) + carry;
    if (raw > half) {
      carry = 1;
      const uint32_t mag = full - raw;
      if (mag) f(j, mag, true);
    } else {
      carry = 0;
      if (raw) f(j, raw, false);
    }
  }
}

template <class F>
CSB_DEV bool point_is_inf(const uint32_t* p) {
  constexpr int W = FieldWords<F>::value;
  // reference encoding: X == 0 and Y == 1_mont (Y.c1 == 0 for G2)
  for (int i = 0; i < W; i++)
    if (p[i]) return false;
  const Fq one = Fq::one();
  for (int i = 0; i < 8; i++)
    if (p[W + i] != one.v[i]) return false;
  for (int i = 8; i < W; i++)
    if (p[W + i]) return false;
  return true;
}

template <class F>
CSB_DEV bool load_scalar(const uint32_t* scalars, const uint32_t* points, uint32_t i,
                         uint32_t (&k)[8]) {
  ld_limbs8(k, scalars + (size_t)i * 8);
  scalar_reduce(k);
  if ((k[0] | k[1] | k[2] | k[3] | k[4] | k[5] | k[6] | k[7]) == 0) return false;
  constexpr int PW = 2 * FieldWords<F>::value;
  return !point_is_inf<F>(points + (size_t)i * PW);
}

// Claims a place in bucket b: its old count or cursor plus this lane's rank among the converged
// lanes that claim in the same bucket, with one atomic for all of them.  Used for the lowest
// window only: a witness's bits and small values crowd into a few of its buckets, where atomics
// to one address run one after another (100,003 terms, half of them 0 or 1: see k_count).
CSB_DEV uint32_t claim_shared(uint32_t* slots, size_t b) {
  const uint32_t act = __activemask(), lane = threadIdx.x & 31;
  const uint32_t peers = __match_any_sync(act, (unsigned long long)b);
  uint32_t base = 0;
  const int leader = __ffs((int)peers) - 1;
  if ((int)lane == leader) base = atomicAdd(&slots[b], (uint32_t)__popc(peers));
  base = __shfl_sync(peers, base, leader);
  return base + __popc(peers & ((1u << lane) - 1u));
}

// Entry placement.  Generic: bucket (window j, |d|-1) of W*B, entry = point index i.
// Fixed-base (tables T[j*n + i] = 2^(c j) P_i): one set of B buckets, bucket |d|-1,
// entry = table index j*n + i, so no per-window sums and no Horner step remain.
template <class F, bool FIXED>
__global__ void k_count(const uint32_t* __restrict__ scalars, const uint32_t* __restrict__ points,
                        uint32_t n, int c, int W, uint32_t* __restrict__ counts) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t k[8];
  if (!load_scalar<F>(scalars, points, i, k)) return;
  const uint32_t B = 1u << (c - 1);
  for_each_digit(k, c, W, [&](int j, uint32_t mag, bool) {
    const size_t b = (FIXED ? 0 : (size_t)j * B) + (mag - 1);
    if (j == 0) claim_shared(counts, b); else atomicAdd(&counts[b], 1u);
  });
}

// Writes entry(j, negative) of every nonzero digit into a place of bucket(j, |d|), four
// windows' atomics in flight at a time: one after another they cost about 1 us each (21 us for
// the 20 windows of 4096 terms).
template <class BucketFn, class EntryFn>
CSB_DEV void scatter_digits(const uint32_t (&k)[8], int c, int W, uint32_t* cursor, uint32_t* entries, BucketFn bucket,
                            EntryFn entry) {
  const uint32_t half = 1u << (c - 1), full = 1u << c;
  uint32_t carry = 0;
#pragma unroll 1
  for (int j0 = 0; j0 < W; j0 += 4) {
    uint32_t mag[4], neg[4], pos[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const uint32_t raw = j0 + q < W ? scalar_bits(k, (j0 + q) * c, c) + carry : 0u;
      neg[q] = raw > half;
      carry = neg[q];
      mag[q] = neg[q] ? full - raw : raw;
    }
    if (j0 == 0 && mag[0]) pos[0] = claim_shared(cursor, bucket(0, mag[0]));
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (mag[q] && j0 + q > 0) pos[q] = atomicAdd(&cursor[bucket(j0 + q, mag[q])], 1u);
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (mag[q]) entries[pos[q]] = entry(j0 + q, neg[q] != 0);
  }
}

template <class F, bool FIXED>
__global__ void k_scatter(const uint32_t* __restrict__ scalars, const uint32_t* __restrict__ points,
                          uint32_t n, int c, int W, uint32_t* __restrict__ cursor,
                          uint32_t* __restrict__ entries) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t k[8];
  if (!load_scalar<F>(scalars, points, i, k)) return;
  const uint32_t B = 1u << (c - 1);
  scatter_digits(k, c, W, cursor, entries,
                 [&](int j, uint32_t mag) { return (FIXED ? 0 : (size_t)j * B) + (mag - 1); },
                 [&](int j, bool neg) { return (FIXED ? (uint32_t)j * n + i : i) | (neg ? NEG_BIT : 0u); });
}

// GLV split of a generic G1 MSM: k_i P_i = k1 P_i + k2 phi(P_i) with k_i = k1 + k2 lambda
// (mod r), |k1|, |k2| < 2^127, so the pipeline sorts 2n half-size scalars: half the windows,
// half the bucket sets to reduce and half the window Horner.  k_glv_prep writes, per term,
// s2[i] = |k1| (words 0-3) and |k2| (words 4-7) with each half's sign in bit 31 of its top
// word (zero halves for a zero scalar or a point at infinity), and phix[i] = beta x_i.  The
// points themselves are not copied: an entry of the k2 half carries PHI_BIT and reads x from
// phix and y from P_i, so the gathered set stays the n input points plus n x-coordinates.
template <class F>
CSB_DEV void glv_prep_term(const uint32_t* scalar, const uint32_t* P, uint32_t* s2, uint32_t* phix) {
  uint32_t k[8];
  ld_limbs8(k, scalar);
  scalar_reduce(k);
  uint32_t k1[4] = {0, 0, 0, 0}, k2[4] = {0, 0, 0, 0}, neg1 = 0, neg2 = 0;
  const bool zero = (k[0] | k[1] | k[2] | k[3] | k[4] | k[5] | k[6] | k[7]) == 0;
  if (!zero && !point_is_inf<F>(P)) {
    const uint64_t kk[4] = {k[0] | (uint64_t)k[1] << 32, k[2] | (uint64_t)k[3] << 32, k[4] | (uint64_t)k[5] << 32,
                            k[6] | (uint64_t)k[7] << 32};
    glv::split_reduced(kk, k1, &neg1, k2, &neg2);
  }
  uint4* o = reinterpret_cast<uint4*>(s2);
  o[0] = make_uint4(k1[0], k1[1], k1[2], k1[3] | (neg1 << 31));
  o[1] = make_uint4(k2[0], k2[1], k2[2], k2[3] | (neg2 << 31));
  F x, beta;
  ld_field(x, P);
  glv::beta_mont(beta.v);
  st_field(phix, x * beta);
}
template <class F>
__global__ void k_glv_prep(const uint32_t* __restrict__ scalars, const uint32_t* __restrict__ points, uint32_t n,
                           uint32_t* __restrict__ s2, uint32_t* __restrict__ phix) {
  constexpr int PW = 2 * FieldWords<F>::value;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  glv_prep_term<F>(scalars + (size_t)i * 8, points + (size_t)i * PW, s2 + (size_t)i * 8, phix + (size_t)i * 8);
}

// Digits of both halves of a split term: f(half, window, |d|, negative), the half's sign
// folded into the digit's.
template <class Fn>
CSB_DEV void for_each_glv_digit(const uint32_t (&t)[8], int c, int W, Fn f) {
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const uint32_t k[8] = {t[4 * h], t[4 * h + 1], t[4 * h + 2], t[4 * h + 3] & 0x7fffffffu, 0u, 0u, 0u, 0u};
    const bool sgn = (t[4 * h + 3] >> 31) != 0;
    for_each_digit(k, c, W, [&](int j, uint32_t mag, bool neg) { f(h, j, mag, neg != sgn); });
  }
}

// Places a split term's entries; its buckets start at bucket0.
CSB_DEV void scatter_glv_term(const uint32_t (&t)[8], uint32_t i, int c, int W, uint32_t bucket0, uint32_t* cursor,
                              uint32_t* entries) {
  const uint32_t B = 1u << (c - 1);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const uint32_t k[8] = {t[4 * h], t[4 * h + 1], t[4 * h + 2], t[4 * h + 3] & 0x7fffffffu, 0u, 0u, 0u, 0u};
    const bool sgn = (t[4 * h + 3] >> 31) != 0;
    scatter_digits(k, c, W, cursor, entries, [&](int j, uint32_t mag) { return bucket0 + (size_t)j * B + (mag - 1); },
                   [&](int, bool neg) { return i | (h ? PHI_BIT : 0u) | (neg != sgn ? NEG_BIT : 0u); });
  }
}

template <class F>
__global__ void k_count_glv(const uint32_t* __restrict__ s2, uint32_t n, int c, int W, uint32_t* __restrict__ counts) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t t[8];
  ld_limbs8(t, s2 + (size_t)i * 8);
  const uint32_t B = 1u << (c - 1);
  for_each_glv_digit(t, c, W, [&](int, int j, uint32_t mag, bool) {
    const size_t b = (size_t)j * B + (mag - 1);
    if (j == 0) claim_shared(counts, b); else atomicAdd(&counts[b], 1u);
  });
}

template <class F>
__global__ void k_scatter_glv(const uint32_t* __restrict__ s2, uint32_t n, int c, int W, uint32_t* __restrict__ cursor,
                              uint32_t* __restrict__ entries) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t t[8];
  ld_limbs8(t, s2 + (size_t)i * 8);
  scatter_glv_term(t, i, c, W, 0, cursor, entries);
}

// The base of an entry: P_i, or phi(P_i) = (phix[i], y_i) for a GLV k2 entry (phix given).
// One load path either way (the x address is selected), so lanes of a warp that read P and
// phi(P) do not diverge.
template <class F>
CSB_DEV Affine<F> ld_entry_point(const uint32_t* base, const uint32_t* phix, uint32_t ent) {
  constexpr int FW = FieldWords<F>::value;
  constexpr int PW = 2 * FW;
  if constexpr (FW == 8) {
    const bool phi = phix != nullptr && (ent & PHI_BIT) != 0;
    const uint32_t i = ent & ~(NEG_BIT | (phix ? PHI_BIT : 0u));
    const uint32_t* xp = phi ? phix + (size_t)i * 8 : base + (size_t)i * PW;
    Affine<F> p;
    ld_field(p.x, xp);
    ld_field(p.y, base + (size_t)i * PW + FW);
    return p;
  } else {
    return ld_affine<F>(base + (size_t)(ent & ~NEG_BIT) * PW);
  }
}

// A batch's side array of beta x holds its terms' in order (unused where an instance is not split).
CSB_DEV const uint32_t* job_phix(const BatchJob& jb, const uint32_t* phix) {
  return jb.glv ? phix + (size_t)jb.term0 * 8 : nullptr;
}

// Task record: entries [start, start+len) summed into dst.  dst < nb: bucket index;
// dst >= nb: partial slot (dst - nb).  job: the instance whose bases the entries index (a
// batch of MSMs shares one task list; 0 for a single MSM).
struct Task {
  uint32_t start, len, dst, job;
};

// Index of the job whose bucket range holds bucket b (bucket0 ascending, bucket0[0] = 0).
CSB_DEV uint32_t job_of_bucket(const BatchJob* jobs, uint32_t njobs, uint32_t b) {
  uint32_t lo = 0, hi = njobs;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (jobs[mid].bucket0 <= b) lo = mid; else hi = mid;
  }
  return lo;
}
// Partial sums to add up: `count` of them from slot pbase on, `stride` slots apart, into dst (as a
// task's).  A bucket of up to kCombineSerial partial sums is one such sum; one of more has each
// run of kCombineSerial summed into the run's first slot and then, in a second pass, those
// (stride kCombineSerial), so no thread adds up more than a few of a crowded bucket's thousands.
struct Multi {
  uint32_t dst, pbase, count, stride;
};
constexpr uint32_t kCombineSerial = 8;

// Task lengths are in [1, TASK]; tasks are emitted in descending length (a counting sort
// over TASK+1 bins) so the 32 lanes of a warp walk buckets of nearly equal size.
constexpr int kMaxTask = 96;

// Pass 1: per bucket, histogram of its task lengths; empty buckets become infinity.
template <class F>
__global__ void k_task_hist(const uint32_t* __restrict__ offsets, uint32_t nb, uint32_t task_len,
                            uint32_t* __restrict__ hist, uint32_t* __restrict__ buckets) {
  __shared__ uint32_t sh[kMaxTask + 1];
  for (int i = threadIdx.x; i <= kMaxTask; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < nb) {
    const uint32_t cnt = offsets[b + 1] - offsets[b];
    if (cnt == 0) {
      constexpr int XW = 4 * FieldWords<F>::value;
      st_xyzz<F>(buckets + (size_t)b * XW, XYZZ<F>::inf());
    } else {
      const uint32_t nfull = (cnt - 1) / task_len;
      if (nfull) atomicAdd(&sh[task_len], nfull);
      atomicAdd(&sh[cnt - nfull * task_len], 1u);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i <= kMaxTask; i += blockDim.x)
    if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

// Pass 2: emit task records at their sorted positions (longest first).  Each block works out
// where the length bins start, reserves a range per bin with one global atomic and ranks its
// tasks inside it.  counters[0] = number of tasks.
template <class F>
__global__ void k_task_emit(const uint32_t* __restrict__ offsets, uint32_t nb, uint32_t task_len,
                            const uint32_t* __restrict__ hist, uint32_t* __restrict__ cursor, Task* __restrict__ tasks,
                            uint32_t* __restrict__ counters, Multi* __restrict__ multi,
                            const BatchJob* __restrict__ jobs = nullptr, uint32_t njobs = 0) {
  __shared__ uint32_t cnt_s[kMaxTask + 1], base_s[kMaxTask + 1], first_s[kMaxTask + 1];
  for (int i = threadIdx.x; i <= kMaxTask; i += blockDim.x) cnt_s[i] = 0;
  if (threadIdx.x < 32) {  // bin l starts after the tasks longer than l
    constexpr int per = (kMaxTask + 32) / 32;  // bins a lane, from kMaxTask down
    const int top = kMaxTask - per * (int)threadIdx.x;
    uint32_t v[per], sum = 0;
#pragma unroll
    for (int q = 0; q < per; q++) {
      v[q] = top - q >= 1 ? hist[top - q] : 0u;
      sum += v[q];
    }
    uint32_t incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
      if ((int)threadIdx.x >= d) incl += t;
    }
    uint32_t run = incl - sum;
#pragma unroll
    for (int q = 0; q < per; q++) {
      if (top - q >= 0) first_s[top - q] = run;
      run += v[q];
    }
    if (blockIdx.x == 0 && threadIdx.x == 31) counters[0] = incl;
  }
  __syncthreads();
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t start = 0, cnt = 0, nfull = 0, last = 0;
  if (b < nb) {
    start = offsets[b];
    cnt = offsets[b + 1] - start;
    if (cnt) {
      nfull = (cnt - 1) / task_len;
      last = cnt - nfull * task_len;
      if (nfull) atomicAdd(&cnt_s[task_len], nfull);
      atomicAdd(&cnt_s[last], 1u);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i <= kMaxTask; i += blockDim.x)
    base_s[i] = cnt_s[i] ? first_s[i] + atomicAdd(&cursor[i], cnt_s[i]) : 0u;
  __syncthreads();
  for (int i = threadIdx.x; i <= kMaxTask; i += blockDim.x) cnt_s[i] = 0;
  __syncthreads();
  const uint32_t nt = cnt ? nfull + 1 : 0u;
  const uint32_t job = jobs && cnt ? job_of_bucket(jobs, njobs, b) : 0u;
  uint32_t pbase = 0, mslot = 0;
  if (nt > 1) {
    pbase = atomicAdd(&counters[1], nt);
    mslot = atomicAdd(&counters[2], nt > kCombineSerial ? 1 + (nt + kCombineSerial - 1) / kCombineSerial : 1u);
    multi[mslot] = nt > kCombineSerial ? Multi{b, pbase, (nt + kCombineSerial - 1) / kCombineSerial, kCombineSerial}
                                       : Multi{b, pbase, nt, 1u};
  }
  // a crowded bucket's records are written by the whole warp
  constexpr uint32_t kAlone = 16;
  const uint32_t lane = threadIdx.x & 31;
  for (uint32_t big = __ballot_sync(0xffffffffu, nt > kAlone); big; big &= big - 1) {
    const int src = __ffs((int)big) - 1;
    const uint32_t o_nt = __shfl_sync(0xffffffffu, nt, src), o_start = __shfl_sync(0xffffffffu, start, src);
    const uint32_t o_last = __shfl_sync(0xffffffffu, last, src), o_pbase = __shfl_sync(0xffffffffu, pbase, src);
    const uint32_t o_mslot = __shfl_sync(0xffffffffu, mslot, src), o_job = __shfl_sync(0xffffffffu, job, src);
    uint32_t at = 0;
    if ((int)lane == src) at = base_s[task_len] + atomicAdd(&cnt_s[task_len], o_nt - 1);
    at = __shfl_sync(0xffffffffu, at, src);
    for (uint32_t t = lane; t < o_nt - 1; t += 32)
      tasks[at + t] = {o_start + t * task_len, task_len, nb + o_pbase + t, o_job};
    if ((int)lane == src) {
      const uint32_t slot = base_s[o_last] + atomicAdd(&cnt_s[o_last], 1u);
      tasks[slot] = {o_start + (o_nt - 1) * task_len, o_last, nb + o_pbase + o_nt - 1, o_job};
    }
    for (uint32_t q = lane; q * kCombineSerial < o_nt; q += 32)
      multi[o_mslot + 1 + q] = {nb + o_pbase + q * kCombineSerial, o_pbase + q * kCombineSerial,
                                min(kCombineSerial, o_nt - q * kCombineSerial), 1u};
  }
  if (nt == 0 || nt > kAlone) return;
#pragma unroll 1
  for (uint32_t t = 0; t < nt; t++) {
    const uint32_t len = t < nfull ? task_len : last;
    const uint32_t slot = base_s[len] + atomicAdd(&cnt_s[len], 1u);
    tasks[slot] = {start + t * task_len, len, nt == 1 ? b : nb + pbase + t, job};
  }
  if (nt > kCombineSerial)
    for (uint32_t q = 0; q * kCombineSerial < nt; q++)
      multi[mslot + 1 + q] = {nb + pbase + q * kCombineSerial, pbase + q * kCombineSerial,
                              min(kCombineSerial, nt - q * kCombineSerial), 1u};
}

// Minimum resident blocks per SM asked of the compiler for the accumulation kernel: G1 at 4
// (128 registers, what its inlined addition takes), G2 at 3 (168 registers: 12 warps per SM
// instead of 8, measured faster).
// The G1 accumulation is bound by its multiply-adds (the products of xyzz_madd_lazy): 2^20
// fixed-base terms 2.18 ms, 5950 cycles per 32 additions and scheduler, against 2.44 ms with
// the products called out of line and one reduction each; 3 and 5 blocks 2.18 and 2.15 ms (but
// 2.79 against 2.71 ms over the GLV split's points), loading the next point ahead 2.18-2.25 ms.
template <class F> struct AccMinBlocks { static constexpr int value = 4; };
template <> struct AccMinBlocks<Fq2> { static constexpr int value = 3; };

// The accumulation's mixed addition: over Fq with lazily reduced coordinates (no final
// conditional subtraction per product; the bucket is canonicalised when stored), over Fq2
// the canonical one.
CSB_DEV XYZZ<Fq> madd_acc(const XYZZ<Fq>& acc, const Affine<Fq>& p) { return xyzz_madd_lazy(acc, p); }
CSB_DEV XYZZ<Fq2> madd_acc(const XYZZ<Fq2>& acc, const Affine<Fq2>& p) { return xyzz_madd(acc, p); }
CSB_DEV XYZZ<Fq> canon_acc(const XYZZ<Fq>& a) { return xyzz_canon(a); }
CSB_DEV XYZZ<Fq2> canon_acc(const XYZZ<Fq2>& a) { return a; }

template <class F>
__global__ void __launch_bounds__(128, AccMinBlocks<F>::value) k_accumulate(const Task* __restrict__ tasks,
                                                    const uint32_t* __restrict__ counters,
                                                    const uint32_t* __restrict__ entries,
                                                    const uint32_t* __restrict__ points, uint32_t nb,
                                                    uint32_t* __restrict__ buckets,
                                                    uint32_t* __restrict__ partials,
                                                    const BatchJob* __restrict__ jobs = nullptr,
                                                    const uint32_t* __restrict__ phix = nullptr) {
  constexpr int PW = 2 * FieldWords<F>::value;
  constexpr int XW = 4 * FieldWords<F>::value;
  const uint32_t ntasks = counters[0];
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < ntasks; t += gridDim.x * blockDim.x) {
    const Task tk = tasks[t];
    const uint32_t* base = jobs ? jobs[tk.job].points : points;
    const uint32_t* px = jobs ? job_phix(jobs[tk.job], phix) : phix;
    XYZZ<F> acc = XYZZ<F>::inf();
    if (entries) {
#pragma unroll 1
      for (uint32_t e = 0; e < tk.len; e++) {
        const uint32_t ent = entries[tk.start + e];
        Affine<F> p = ld_entry_point<F>(base, px, ent);
        if (ent & NEG_BIT) p.y = p.y.neg();
        acc = madd_acc(acc, p);
      }
    } else {  // after batch-affine rounds: points in bucket order, (0, 0) = infinity
#pragma unroll 1
      for (uint32_t e = 0; e < tk.len; e++) {
        const Affine<F> p = ld_affine<F>(base + (size_t)(tk.start + e) * PW);
        if (!(p.x.is_zero() && p.y.is_zero())) acc = madd_acc(acc, p);
      }
    }
    uint32_t* dst = tk.dst < nb ? buckets + (size_t)tk.dst * XW : partials + (size_t)(tk.dst - nb) * XW;
    st_xyzz<F>(dst, canon_acc(acc));
  }
}

// Latency form of k_accumulate for an MSM too small to fill the GPU: one group of lanes per
// task (group.cuh; 4 product latencies per addition instead of 10).  Same tasks, same results.
// The groups of a warp step together: each walks the longest of the warp's tasks and leaves
// its sum alone past its own task's end (tasks are emitted longest first, so neighbours are
// about as long).
template <class F>
__global__ void __launch_bounds__(128, 4) k_accumulate_group(
    const Task* __restrict__ tasks, const uint32_t* __restrict__ counters, const uint32_t* __restrict__ entries,
    const uint32_t* __restrict__ points, uint32_t nb, uint32_t* __restrict__ buckets,
    uint32_t* __restrict__ partials, const BatchJob* __restrict__ jobs = nullptr,
    const uint32_t* __restrict__ phix = nullptr) {
  using Gr = Group<F>;
  constexpr int FW = FieldWords<F>::value, PW = 2 * FW, XW = 4 * FW;
  constexpr uint32_t G = Gr::G, GPW = 32 / G, NG = 128 / G;
  __shared__ __align__(16) uint32_t scr[NG][Gr::kScratch], accs[NG][XW];
  const Gr grp(scr[threadIdx.x / G]);
  uint32_t* acc = accs[threadIdx.x / G];
  const uint32_t ntasks = counters[0];
  const uint32_t warp0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  const uint32_t gw = (threadIdx.x & 31) / G;  // group within the warp
  for (uint32_t first = warp0 * GPW; first < ntasks; first += nwarps * GPW) {  // warp-uniform
    const uint32_t t = first + gw;
    const bool valid = t < ntasks;
    const Task tk = valid ? tasks[t] : Task{0, 0, 0, 0};
    const uint32_t* pts = jobs && valid ? jobs[tk.job].points : points;  // read only where live
    const uint32_t* px = jobs ? (valid ? job_phix(jobs[tk.job], phix) : nullptr) : phix;
    const uint32_t steps = __reduce_max_sync(0xffffffffu, tk.len);
    grp.load(acc, nullptr, false);
#pragma unroll 1
    for (uint32_t e = 0; e < steps; e++) {
      const bool live = e < tk.len;
      const uint32_t *qx = acc, *qy = acc;  // past the task's end: any readable address
      bool neg = false;
      if (live) {
        const uint32_t ent = entries[tk.start + e];
        const uint32_t i = ent & ~(NEG_BIT | (px ? PHI_BIT : 0u));
        qy = pts + (size_t)i * PW + FW;
        qx = FW == 8 && px && (ent & PHI_BIT) ? px + (size_t)i * FW : pts + (size_t)i * PW;
        neg = (ent & NEG_BIT) != 0;
      }
      grp.madd(acc, acc, qx, qy, neg, live);
    }
    if (valid) {
      uint32_t* dst = tk.dst < nb ? buckets + (size_t)tk.dst * XW : partials + (size_t)(tk.dst - nb) * XW;
      grp.store(dst, acc);
    }
    __syncwarp();
  }
}

// buckets[b] += add[b] (XYZZ, canonical): folds another fixed-base MSM's buckets (same window)
// into this one's before the reduction.
template <class F>
__global__ void __launch_bounds__(128) k_add_buckets(uint32_t* __restrict__ buckets, const uint32_t* __restrict__ add,
                                                     uint32_t nb) {
  constexpr int XW = 4 * FieldWords<F>::value;
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nb) return;
  const XYZZ<F> x = ld_xyzz<F>(buckets + (size_t)b * XW), y = ld_xyzz<F>(add + (size_t)b * XW);
  st_xyzz<F>(buckets + (size_t)b * XW, xyzz_add(x, y));
}

// First pass: one group of lanes per sum of at most kCombineSerial neighbouring partial sums
// (few of them, and a chain each: one thread per sum took 131 us over Fq2 where a group takes
// 20).  The top window of a scalar has fewer bits, so its digits crowd into fewer buckets and
// many of those split.
template <class F>
__global__ void __launch_bounds__(128, 4) k_combine_small(const Multi* __restrict__ multi,
                                                          const uint32_t* __restrict__ counters, uint32_t nb,
                                                          uint32_t* partials, uint32_t* __restrict__ buckets) {
  using Gr = Group<F>;
  constexpr int XW = 4 * FieldWords<F>::value;
  constexpr uint32_t G = Gr::G, GPW = 32 / G, NG = 128 / G;
  __shared__ __align__(16) uint32_t scr[NG][Gr::kScratch], accs[NG][XW];
  const Gr grp(scr[threadIdx.x / G]);
  uint32_t* acc = accs[threadIdx.x / G];
  const uint32_t nm = counters[2];
  const uint32_t warp0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t first = warp0 * GPW; first < nm; first += nwarps * GPW) {  // warp-uniform
    const uint32_t m = first + (threadIdx.x & 31) / G;
    Multi mu = m < nm ? multi[m] : Multi{0, 0, 0, 0};
    if (mu.stride != 1) mu.count = 0;  // k_combine
    const uint32_t steps = __reduce_max_sync(0xffffffffu, mu.count);
    grp.load(acc, partials + (size_t)mu.pbase * XW, mu.count != 0);
#pragma unroll 1
    for (uint32_t i = 1; i < steps; i++) {
      const bool live = i < mu.count;
      grp.add(acc, acc, live ? partials + (size_t)(mu.pbase + i) * XW : acc, live);
    }
    if (mu.count)
      grp.store(mu.dst < nb ? buckets + (size_t)mu.dst * XW : partials + (size_t)(mu.dst - nb) * XW, acc);
    __syncwarp();
  }
}

// Second pass: the runs of a bucket with more partial sums, one block each: every group adds up
// its share, then a tree over the groups.
template <class F>
__global__ void __launch_bounds__(128, 4) k_combine(const Multi* __restrict__ multi,
                                                    const uint32_t* __restrict__ counters,
                                                    const uint32_t* __restrict__ partials,
                                                    uint32_t* __restrict__ buckets) {
  using Gr = Group<F>;
  constexpr int XW = 4 * FieldWords<F>::value;
  constexpr uint32_t G = Gr::G, NG = 128 / G;
  __shared__ __align__(16) uint32_t scr[NG][Gr::kScratch], accs[NG][XW];
  const uint32_t g = threadIdx.x / G;
  const Gr grp(scr[g]);
  uint32_t* acc = accs[g];
  const uint32_t nm = counters[2];
  for (uint32_t m = blockIdx.x; m < nm; m += gridDim.x) {
    const Multi mu = multi[m];
    if (mu.stride == 1) continue;  // first pass (the whole block leaves together)
    auto at = [&](uint32_t i) { return partials + (size_t)(mu.pbase + i * mu.stride) * XW; };
    grp.load(acc, at(g), g < mu.count);
#pragma unroll 1
    for (uint32_t i = NG; i < mu.count; i += NG) grp.add(acc, acc, i + g < mu.count ? at(i + g) : acc, i + g < mu.count);
    __syncthreads();
#pragma unroll 1
    for (uint32_t d = NG / 2; d >= 1; d >>= 1) {
      grp.add(acc, acc, accs[(g + d) & (NG - 1)], g < d);
      __syncthreads();
    }
    if (g == 0) grp.store(buckets + (size_t)mu.dst * XW, acc);
    __syncthreads();
  }
}

// Level k of the bucket reduction.  y: W sequences of n XYZZ points (stride n); z: the
// weighted carry from the previous level (null at level 0).  Thread (j, t) handles
// y[j][8t .. 8t+8):
//   acc = sum_i y_i,  s = sum_i i*y_i,  z'[j][t] = sum_i z[j][8t+i] + 8^k * s,
//   y'[j][t] = acc.
template <class F>
__global__ void __launch_bounds__(128) k_reduce_level(const uint32_t* __restrict__ y,
                                                      const uint32_t* __restrict__ z, uint32_t n,
                                                      uint32_t nout, int W, int level,
                                                      uint32_t* __restrict__ yout,
                                                      uint32_t* __restrict__ zout) {
  constexpr int XW = 4 * FieldWords<F>::value;
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= (uint32_t)W * nout) return;
  const uint32_t j = g / nout, t = g % nout;
  const uint32_t* yj = y + (size_t)j * n * XW;
  XYZZ<F> acc = XYZZ<F>::inf(), s = XYZZ<F>::inf();
#pragma unroll 1
  for (int i = 7; i >= 1; i--) {
    const uint32_t idx = 8 * t + i;
    if (idx < n) acc = xyzz_add(acc, ld_xyzz<F>(yj + (size_t)idx * XW));
    s = xyzz_add(s, acc);
  }
  if (8 * t < n) acc = xyzz_add(acc, ld_xyzz<F>(yj + (size_t)(8 * t) * XW));
#pragma unroll 1
  for (int d = 0; d < 3 * level; d++) s = xyzz_dbl(s);
  if (z) {
    const uint32_t* zj = z + (size_t)j * n * XW;
#pragma unroll 1
    for (int i = 0; i < 8; i++) {
      const uint32_t idx = 8 * t + i;
      if (idx < n) s = xyzz_add(s, ld_xyzz<F>(zj + (size_t)idx * XW));
    }
  }
  st_xyzz<F>(yout + ((size_t)j * nout + t) * XW, acc);
  st_xyzz<F>(zout + ((size_t)j * nout + t) * XW, s);
}


// Bucket reduction of few buckets, by bits: with S_b the n = 2^k values of a window (n values of
// the last level), sum_b b S_b = sum_j 2^j T_j, T_j the sum of the S_b whose index has bit j set.
// A binary tree gives all T_j at once: joining the left and right halves of a node adds their
// totals and their T_j pairwise, and the right half's total is the node's new T_j, so 2n
// additions in all and a chain of k of them, where running sums over segments of eight take
// about as many additions but chains of 13 a level and a scan over the segments left.
// One block joins 2^lg <= 64 values in shared memory: node i of level q starts at slot i 2^q and
// its T_j lies in slot i 2^q + 2^j, where the right half's total already is.  It writes its total
// and T_j back to the same places, so a later stage finds the earlier bits' partial sums at the
// same offsets of every 64 slots and adds them up (blockIdx.x: bucket sets and their segments;
// blockIdx.y: 0 the totals, which give the next bits; 1..bits the T_j; then z, whose plain sum is
// needed); after the last stage a set has its total in slot 0 and T_j in slot 2^j.
// The sets of all windows, and of all window widths of a batch, go through one launch a stage.
struct BitTree {
  uint32_t *y, *z;         // windows * 2^k values each (z may be null)
  uint32_t k, windows;     // bits of a set's index, sets
  uint32_t shift;          // weight of a value: 2^shift times its index
  uint32_t block0, wsum0;  // first block of a launch, first window sum
};
constexpr int kMaxTrees = 24;  // widths 4..24
struct BitTrees {
  BitTree t[kMaxTrees];
  int count;
};
CSB_DEV const BitTree& tree_of_block(const BitTrees& T) {
  int i = 0;
  while (i + 1 < T.count && T.t[i + 1].block0 <= blockIdx.x) i++;
  return T.t[i];
}
template <class F> struct TreeGroups { static constexpr int value = 32; };
template <> struct TreeGroups<Fq2> { static constexpr int value = 16; };  // 48 KB of shared memory

template <class F>
__global__ void __launch_bounds__(Group<F>::G* TreeGroups<F>::value, 512 / (Group<F>::G * TreeGroups<F>::value))
    k_bit_tree(const __grid_constant__ BitTrees trees, int bits) {
  using Gr = Group<F>;
  constexpr int XW = 4 * FieldWords<F>::value;
  constexpr uint32_t NG = TreeGroups<F>::value, G = Gr::G;
  __shared__ __align__(16) uint32_t scr[NG][Gr::kScratch], node[64][XW];
  const BitTree& tr = tree_of_block(trees);
  uint32_t *y = tr.y, *z = tr.z;
  const int lg = min(6, (int)tr.k - bits);
  const uint32_t n = 1u << tr.k, block = blockIdx.x - tr.block0;
  if ((int)blockIdx.y > bits && !z) return;
  const Gr grp(scr[threadIdx.x / G]);
  const uint32_t g = threadIdx.x / G, g0 = (threadIdx.x & ~31u) / G;  // this group, the warp's first
  const int role = blockIdx.y;
  const uint32_t segs = n >> (bits + lg), seg = block % segs;
  uint32_t* arr = (role <= bits ? y : z) + (size_t)(block / segs) * n * XW;
  const uint32_t off = role >= 1 && role <= bits ? 1u << (role - 1) : 0u;
  auto at = [&](uint32_t i) { return arr + ((size_t)((((seg << lg) + i) << bits) + off)) * XW; };
  for (uint32_t w = threadIdx.x; w < (XW / 4u) << lg; w += blockDim.x) {
    const uint32_t i = w / (XW / 4), q = w % (XW / 4);
    reinterpret_cast<uint4*>(node[i])[q] = reinterpret_cast<const uint4*>(at(i))[q];
  }
  __syncthreads();
  for (int q = 1; q <= lg; q++) {
    const uint32_t half = 1u << (q - 1), per = role == 0 ? (uint32_t)q : 1u;
    const uint32_t ops = (1u << (lg - q)) * per;
    for (uint32_t o0 = 0; o0 + g0 < ops; o0 += NG) {  // warp-uniform
      const uint32_t o = o0 + g;
      const bool live = o < ops;
      const uint32_t i = live ? o / per : 0u, k = live ? o % per : 0u;  // k: 0 the total, k - 1 the bit
      const uint32_t dst = (i << q) + (k ? 1u << (k - 1) : 0u);
      grp.add(node[dst], node[dst], node[dst + half], live);
    }
    __syncthreads();
  }
  const uint32_t outs = role == 0 ? (uint32_t)lg + 1 : 1u;
  for (uint32_t o = g; o < outs; o += NG) {
    const uint32_t i = o ? 1u << (o - 1) : 0u;
    grp.store(at(i), node[i]);
  }
}

// One warp per bucket set: Z + Y + 2^shift sum_j 2^j T_j from the places k_bit_tree left them in
// (no Z where z is null), the bits in two halves at once: the upper half's Horner chain, doubled
// over the lower bits, joins the lower's.  out: the affine result (one set), else wsum.
template <class F>
__global__ void __launch_bounds__(32) k_window_horner(const __grid_constant__ BitTrees trees,
                                                      uint32_t* __restrict__ wsum, uint32_t* __restrict__ out) {
  using Gr = Group<F>;
  constexpr int XW = 4 * FieldWords<F>::value;
  constexpr uint32_t G = Gr::G, NG = 32 / G;
  __shared__ __align__(16) uint32_t scr[NG][Gr::kScratch], accs[NG][XW];
  const BitTree& tr = tree_of_block(trees);
  const uint32_t *y = tr.y, *z = tr.z, n = 1u << tr.k, window = blockIdx.x - tr.block0;
  const int bits = (int)tr.k, shift = (int)tr.shift;
  const Gr grp(scr[threadIdx.x / G]);
  uint32_t* acc = accs[threadIdx.x / G];
  const bool upper = ((threadIdx.x / G) & 1) != 0;
  const uint32_t* yw = y + (size_t)window * n * XW;
  const int s = (bits + 1) / 2, lo = upper ? s : 0;
  auto has = [&](int i) { return lo + i < bits; };
  auto T = [&](int i) { return yw + ((size_t)1 << (lo + i)) * XW; };
  grp.load(acc, s > 0 ? T(s - 1) : yw, s > 0 && has(s - 1));
#pragma unroll 1
  for (int i = s - 2; i >= 0; i--) {
    grp.dbl(acc, acc);
    grp.add(acc, acc, has(i) ? T(i) : acc, has(i));
  }
  uint32_t* a0 = accs[0];
  double_times<F>(grp, acc, s, upper);
  grp.add(acc, acc, accs[(threadIdx.x / G) | 1], !upper);
  double_times<F>(grp, acc, shift);
  grp.add(acc, acc, yw, !upper);
  if (z) grp.add(acc, acc, z + (size_t)window * n * XW, !upper);
  if (threadIdx.x >= G) return;
  if (out) {
    if (threadIdx.x == 0) Gr::store_affine(out, a0);
  } else {
    grp.store(wsum + (size_t)(tr.wsum0 + window) * XW, a0);
  }
}

// sum_j 2^(c j) S_j (Horner over the windows) and the affine result.
template <class F>
CSB_DEV void windows_horner(const uint32_t* wsum, int W, int c, uint32_t* out, uint32_t* xyzz_out) {
  // one warp; its groups compute the same
  using Gr = Group<F>;
  constexpr int XW = 4 * FieldWords<F>::value;
  constexpr uint32_t G = Gr::G, NG = 32 / G;
  __shared__ __align__(16) uint32_t scr[NG][Gr::kScratch], accs[NG][XW];
  const Gr grp(scr[(threadIdx.x & 31) / G]);
  uint32_t* acc = accs[(threadIdx.x & 31) / G];
  grp.load(acc, wsum + (size_t)(W - 1) * XW);
#pragma unroll 1
  for (int j = W - 2; j >= 0; j--) {
    double_times<F>(grp, acc, c);
    grp.add(acc, acc, wsum + (size_t)j * XW);
  }
  if (xyzz_out) {
    if ((threadIdx.x & 31) < G) grp.store(xyzz_out, acc);
  } else if ((threadIdx.x & 31) == 0) {
    Gr::store_affine(out, acc);
  }
}
template <class F>
__global__ void __launch_bounds__(32) k_finish(const uint32_t* __restrict__ wsum, int W, int c,
                                               uint32_t* __restrict__ out, uint32_t* __restrict__ xyzz_out) {
  windows_horner<F>(wsum, W, c, out, xyzz_out);
}

template <class F>
__global__ void k_store_inf(uint32_t* out) {
  if (threadIdx.x == 0) st_affine<F>(out, Affine<F>{F::zero(), F::one()});
}

// ---------------------------------------------------------- batch-affine rounds ----
// Before the XYZZ accumulation, buckets are halved R times by adding their points in pairs
// in affine coordinates: lambda = (y2 - y1) / (x2 - x1) (or 3 x^2 / 2y for equal points),
// x3 = lambda^2 - x1 - x2, y3 = lambda (x1 - x3) - y1.  The divisions of kAffK consecutive
// pairs share one inversion (Montgomery's simultaneous inversion: prefix products, one
// inverse, back substitution), so an addition costs about 6 products instead of the
// 10 of an XYZZ + affine addition.  Round r maps bucket b's c_b points at in_off[b] to
// ceil(c_b / 2) points at out_off[b]; an odd last point is copied.  Points at infinity
// inside the rounds are (0, 0), which is on neither curve.
constexpr uint32_t kAffK = 64;  // 32 and 128 measured slower (G2 fixed-base 2^20)

template <class F>
CSB_DEV bool aff_zero(const Affine<F>& a) { return a.x.is_zero() && a.y.is_zero(); }

// Pair of round-r inputs for output slot s of bucket b.  FIRST: round 0 reads the bases
// through the sorted entries (sign bit -> negated y); later rounds read the previous round.
template <class F, bool FIRST>
CSB_DEV void aff_pair(const uint32_t* in_off, const uint32_t* out_off, uint32_t b, uint32_t s,
                      const uint32_t* entries, const uint32_t* src, Affine<F>& p, Affine<F>& q, bool& has_q) {
  constexpr int PW = 2 * FieldWords<F>::value;
  const uint32_t j = s - out_off[b];
  const uint32_t i0 = in_off[b] + 2 * j;
  has_q = i0 + 1 < in_off[b + 1];
  if (FIRST) {
    const uint32_t e0 = entries[i0];
    p = ld_affine<F>(src + (size_t)(e0 & ~NEG_BIT) * PW);
    if (e0 & NEG_BIT) p.y = p.y.neg();
    if (has_q) {
      const uint32_t e1 = entries[i0 + 1];
      q = ld_affine<F>(src + (size_t)(e1 & ~NEG_BIT) * PW);
      if (e1 & NEG_BIT) q.y = q.y.neg();
    }
  } else {
    p = ld_affine<F>(src + (size_t)i0 * PW);
    if (has_q) q = ld_affine<F>(src + (size_t)(i0 + 1) * PW);
  }
}

// Denominator of a pair and its kind: 0 add, 1 double, 2 result p, 3 result q, 4 infinity.
template <class F>
CSB_DEV int aff_kind(const Affine<F>& p, const Affine<F>& q, bool has_q, F& d) {
  d = F::one();
  if (!has_q || aff_zero(q)) return 2;
  if (aff_zero(p)) return 3;
  if (!(p.x == q.x)) {
    d = q.x - p.x;
    return 0;
  }
  if (p.y == q.y) {
    d = p.y.dbl();
    return 1;
  }
  return 4;
}

// The denominator of slot s from the two x coordinates alone (half the bytes of the pair);
// the y coordinates are read only where the kind depends on them (a zero x: a point at
// infinity or x = 0; equal x: doubling or opposite points).
template <class F, bool FIRST>
CSB_DEV F aff_denominator(const uint32_t* in_off, const uint32_t* out_off, uint32_t b, uint32_t s,
                          const uint32_t* entries, const uint32_t* src) {
  constexpr int PW = 2 * FieldWords<F>::value;
  const uint32_t i0 = in_off[b] + 2 * (s - out_off[b]);
  if (i0 + 1 >= in_off[b + 1]) return F::one();  // odd last point: copied
  const uint32_t a0 = FIRST ? (entries[i0] & ~NEG_BIT) : i0;
  const uint32_t a1 = FIRST ? (entries[i0 + 1] & ~NEG_BIT) : i0 + 1;
  F px, qx;
  ld_field(px, src + (size_t)a0 * PW);
  ld_field(qx, src + (size_t)a1 * PW);
  if (!px.is_zero() && !qx.is_zero() && !(px == qx)) return qx - px;
  Affine<F> p, q;
  bool has_q;
  aff_pair<F, FIRST>(in_off, out_off, b, s, entries, src, p, q, has_q);
  F d;
  aff_kind(p, q, has_q, d);
  return d;
}

template <class F>
CSB_DEV uint32_t bucket_of_slot(const uint32_t* off, uint32_t nb, uint32_t s) {
  uint32_t lo = 0, hi = nb;  // largest b with off[b] <= s (empty buckets share offsets)
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (off[mid] <= s) lo = mid; else hi = mid;
  }
  return lo;
}

// At least 3 blocks a SM asked for: over Fq2 the products take 198 registers uncapped, two
// blocks (2^20 fixed-base G2 MSM 8.50 ms); at 168 registers, three blocks, 7.48 ms.
template <class F, bool FIRST>
__global__ void __launch_bounds__(128, 3) k_affine_round(const uint32_t* __restrict__ in_off,
                                                      const uint32_t* __restrict__ out_off, uint32_t nb,
                                                      const uint32_t* __restrict__ entries,
                                                      const uint32_t* __restrict__ src, uint32_t* __restrict__ dst,
                                                      uint32_t* __restrict__ pref) {
  constexpr int FW = FieldWords<F>::value;
  constexpr int PW = 2 * FW;
  const uint32_t total = out_off[nb];
  const uint32_t s0 = (blockIdx.x * blockDim.x + threadIdx.x) * kAffK;
  if (s0 >= total) return;
  const uint32_t s1 = min(total, s0 + kAffK);
  const uint32_t b0 = bucket_of_slot<F>(out_off, nb, s0);
  // phase 1: prefix products of the denominators
  F acc = F::one();
  uint32_t b = b0;
  for (uint32_t s = s0; s < s1; s++) {
    while (out_off[b + 1] <= s) b++;
    acc = acc * aff_denominator<F, FIRST>(in_off, out_off, b, s, entries, src);
    st_field(pref + (size_t)s * FW, acc);
  }
  F inv = acc.inv();
  // phase 2: back substitution and the additions, last slot first
  for (uint32_t s = s1; s-- > s0;) {
    while (out_off[b] > s) b--;
    Affine<F> p, q;
    bool has_q;
    aff_pair<F, FIRST>(in_off, out_off, b, s, entries, src, p, q, has_q);
    F d;
    const int kind = aff_kind(p, q, has_q, d);
    F before = F::one();
    if (s > s0) {  // written above by this thread: a plain (coherent) load, not __ldg
      uint32_t* bw = reinterpret_cast<uint32_t*>(&before);
      const uint4* pv = reinterpret_cast<const uint4*>(pref + (size_t)(s - 1) * FW);
#pragma unroll
      for (int k = 0; k < FW / 4; k++) {
        const uint4 v = pv[k];
        bw[4 * k] = v.x; bw[4 * k + 1] = v.y; bw[4 * k + 2] = v.z; bw[4 * k + 3] = v.w;
      }
    }
    const F id = inv * before;  // 1 / d
    inv = inv * d;
    Affine<F> r;
    if (kind == 0 || kind == 1) {
      const F lam = kind == 0 ? (q.y - p.y) * id : (p.x.sqr() * (F::one() + F::one() + F::one())) * id;
      const F x3 = lam.sqr() - p.x - q.x;
      r.x = x3;
      r.y = lam * (p.x - x3) - p.y;
    } else if (kind == 2) {
      r = p;
    } else if (kind == 3) {
      r = q;
    } else {
      r.x = F::zero();
      r.y = F::zero();
    }
    st_affine<F>(dst + (size_t)s * PW, r);
  }
}

// out[b] = ceil(in[b] / 2) for the next round's counts (written into a count array that the
// scan turns into offsets; out[nb] = 0 so the scan's last element is the total).
static __global__ void k_half_counts(const uint32_t* __restrict__ off, uint32_t nb, uint32_t* __restrict__ out) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < nb) out[b] = (off[b + 1] - off[b] + 1) >> 1;
  if (b == nb) out[b] = 0;
}

// --------------------------------------------------------------- workspace layout ----
// counters block: [0] tasks, [1] partial slots, [2] split buckets; hist at +16 and
// bin cursors at +128 (kMaxTask + 1 words each).
constexpr int kCtrHist = 16, kCtrCursor = 128, kCtrWords = 256;
static_assert(kCtrHist + kMaxTask + 1 <= kCtrCursor && kCtrCursor + kMaxTask + 1 <= kCtrWords,
              "task-length bins must not overlap");

struct Layout {
  size_t counts, offsets, entries, tasks, multi, partials, buckets, lv_y, lv_z, lv_y2, lv_z2, wsum,
      counters, off2, pa, pb, pref, glv_s, glv_p, total;
  bool affine, glv;
};

static inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// task_len: the shortest task the MSM will run (0: automatic, layout_min_task of its entries).
inline Layout make_layout(uint32_t n, int c, int xyzz_bytes, uint32_t task_len, bool fixed = false,
                          bool affine = true, bool glv = false) {
  const int W = msm_windows(c, glv);
  const size_t nt = glv ? 2 * (size_t)n : n;  // terms the pipeline sorts (GLV: k1 P_i and k2 phi(P_i))
  const size_t nb = fixed ? ((size_t)1 << (c - 1)) : (size_t)W << (c - 1);
  const int WR = fixed ? 1 : W;  // bucket sets reduced
  const size_t ne = nt * W;
  if (task_len == 0) task_len = layout_min_task(ne);
  const size_t max_tasks = nb + ne / task_len + 1;
  const size_t max_partials = 2 * (ne / task_len) + 1;
  const size_t n1 = ((size_t)1 << (c - 1)) / 8 + 1;
  const size_t n2 = (size_t)WR * (n1 / 8 + 1);
  Layout L{};
  size_t o = 0;
  L.counters = o; o = align256(o + kCtrWords * sizeof(uint32_t));
  L.counts = o;   o = align256(o + (nb + 1) * sizeof(uint32_t));
  L.offsets = o;  o = align256(o + (nb + 1) * sizeof(uint32_t));
  L.entries = o;  o = align256(o + ne * sizeof(uint32_t));
  L.tasks = o;    o = align256(o + max_tasks * sizeof(Task));
  L.multi = o;    o = align256(o + (ne / (task_len + 1) + 1) * sizeof(Multi));
  L.partials = o; o = align256(o + max_partials * (size_t)xyzz_bytes);
  L.buckets = o;  o = align256(o + nb * (size_t)xyzz_bytes);
  L.lv_y = o;     o = align256(o + (size_t)WR * n1 * xyzz_bytes);
  L.lv_z = o;     o = align256(o + (size_t)WR * n1 * xyzz_bytes);
  L.lv_y2 = o;    o = align256(o + n2 * xyzz_bytes);
  L.lv_z2 = o;    o = align256(o + n2 * xyzz_bytes);
  L.wsum = o;     o = align256(o + (size_t)WR * xyzz_bytes);
  L.glv = glv;
  if (glv) {  // per term: both split halves (8 words) and beta x_i (8 words)
    L.glv_s = o;  o = align256(o + (size_t)n * 32);
    L.glv_p = o;  o = align256(o + (size_t)n * 32);
  }
  L.affine = affine;
  if (affine) {  // batch-affine rounds: offsets ping-pong, two point arrays, prefix products
    const size_t pb = (size_t)xyzz_bytes / 2, fb = (size_t)xyzz_bytes / 4;
    L.off2 = o;   o = align256(o + (nb + 1) * sizeof(uint32_t));
    L.pa = o;     o = align256(o + (ne / 2 + 2 * nb + 1) * pb);
    L.pb = o;     o = align256(o + (ne / 4 + 2 * nb + 1) * pb);
    L.pref = o;   o = align256(o + (ne / 2 + 2 * nb + 1) * fb);
  }
  L.total = o + scan_workspace_bytes(nb + 1);
  return L;
}

// Batch-affine rounds before the XYZZ accumulation (the expected bucket size is N W /
// buckets; a round needs about 8 points per bucket to pay).  Measured at 2^20: G1 is
// fastest without rounds (its XYZZ addition, 10 products, outruns the affine round, which
// waits on its gathers), G2 with two (Fq2 products are 3 Fq products, so the 6-vs-10 product
// saving outweighs the extra traffic).
inline int auto_affine_rounds_rt(bool ec2, uint32_t n, int W, size_t nb) {
  // a round runs kAffK pairs per thread in sequence around one inversion: it needs enough
  // pairs (>= 2^22, i.e. N W >= 2^23 entries) to fill the GPU, or its chain sets the latency
  // (2 rounds cost 2.5 ms in a 2^12-term G2 MSM)
  if ((uint64_t)n * W < (1ull << 23)) return 0;
  // G1: the 2^20 fixed-base MSM takes 3.03 ms without rounds, 3.50 with one, 3.72 with two.
  // (L2 prefetching the round's gathers a few slots ahead did not help G2 either.)
  const int cap = ec2 ? 2 : 0;
  const double avg = (double)n * W / (double)nb;
  int r = 0;
  while (r < cap && avg >= (double)(8u << r)) r++;
  return r;
}
template <class F>
inline int auto_affine_rounds(uint32_t n, int W, size_t nb) {
  return auto_affine_rounds_rt(FieldWords<F>::value == 16, n, W, nb);
}
// Whether an MSM reserves the round buffers: affine_mode -1 auto, 0 never, > 0 that many rounds.
inline bool layout_affine(bool ec2, int affine_mode, uint32_t n, int c, bool fixed, bool glv = false) {
  if (affine_mode >= 0) return affine_mode > 0;
  const int W = msm_windows(c, glv);
  const size_t nb = fixed ? ((size_t)1 << (c - 1)) : (size_t)W << (c - 1);
  return auto_affine_rounds_rt(ec2, glv ? 2 * n : n, W, nb) > 0;
}
// Whether an MSM splits its scalars by the GLV endomorphism: generic G1 MSMs unless turned off.
// Batch-affine rounds (asked for explicitly; G1 runs none by default) read plain point indices,
// so they turn the split off.
inline bool use_glv(bool ec2, bool fixed, int glv_mode, int affine_mode, uint32_t n) {
  return !ec2 && !fixed && glv_mode != 0 && affine_mode <= 0 && n < PHI_BIT;
}

// Resident blocks of k_accumulate per SM, cached per device (callers on several threads and
// devices: server slots, the allocation-free entry point).
template <class F>
int accumulate_grid(int dev, int sms) {
  static std::atomic<int> blocks_per_sm[64];
  const int slot = dev >= 0 && dev < 64 ? dev : 0;
  int b = blocks_per_sm[slot].load(std::memory_order_relaxed);
  if (b == 0) {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_accumulate<F>, 128, 0) != cudaSuccess || b < 1)
      b = 1;
    blocks_per_sm[slot].store(b, std::memory_order_relaxed);
  }
  return b * sms;
}

// The bucket sums of WR sets of B = 2^(c-1) buckets each (overwritten) as a tree to join: levels
// of eight buckets per thread (least work, and what fills the GPU best) come first while the
// values would fill the resident threads' groups many times over.
// Measured (us): 22 sets of 2048 over Fq2, levels 252 + 61, tree 172; 2^19 buckets over Fq, levels
// 268 + 97, tree alone 500.
template <class F> struct TreeFill { static constexpr uint64_t value = 16; };
template <> struct TreeFill<Fq2> { static constexpr uint64_t value = 32; };
template <class F>
bool reduce_needs_levels(uint32_t n, uint32_t WR, uint64_t resident) {
  return n >= 8 && (uint64_t)n * WR * Group<F>::G > TreeFill<F>::value * resident;
}
template <class F>
BitTree reduce_levels(uint32_t* buckets, uint32_t B, uint32_t WR, uint32_t* lv_y, uint32_t* lv_z, uint32_t* lv_y2,
                      uint32_t* lv_z2, uint64_t resident, cudaStream_t st) {
  BitTree t{buckets, nullptr, 0, WR, 0, 0, 0};
  uint32_t n = B;
  int level = 0;
  for (; reduce_needs_levels<F>(n, WR, resident); level++) {
    const uint32_t nout = n / 8;
    uint32_t *yo = level % 2 ? lv_y2 : lv_y, *zo = level % 2 ? lv_z2 : lv_z;
    k_reduce_level<F><<<(uint32_t)(((uint64_t)WR * nout + 127) / 128), 128, 0, st>>>(t.y, t.z, n, nout, (int)WR, level, yo,
                                                                                      zo);
    note_launch();
    t.y = yo;
    t.z = zo;
    n = nout;
  }
  t.shift = 3 * level;
  while ((1u << t.k) < n) t.k++;
  return t;
}
// Joins the trees: their window sums to wsum, or the affine result of a single set to out.
template <class F>
void join_trees(BitTrees& T, uint32_t* wsum, uint32_t* out, cudaStream_t st) {
  uint32_t kmax = 0;
  bool any_z = false;
  for (int i = 0; i < T.count; i++) {
    kmax = std::max(kmax, T.t[i].k);
    any_z |= T.t[i].z != nullptr;
  }
  for (uint32_t bits = 0; bits < kmax; bits += 6) {
    BitTrees S{};  // the trees that still have bits to join
    uint32_t blocks = 0;
    for (int i = 0; i < T.count; i++) {
      if (T.t[i].k <= bits) continue;
      BitTree& t = S.t[S.count++] = T.t[i];
      t.block0 = blocks;
      blocks += t.windows << (t.k - bits - std::min(6u, t.k - bits));
    }
    k_bit_tree<F><<<dim3(blocks, 1 + bits + (any_z ? 1 : 0)), Group<F>::G * TreeGroups<F>::value, 0, st>>>(S, (int)bits);
    note_launch();
  }
  uint32_t blocks = 0;
  for (int i = 0; i < T.count; i++) {
    T.t[i].block0 = blocks;
    blocks += T.t[i].windows;
  }
  k_window_horner<F><<<blocks, 32, 0, st>>>(T, wsum, out);
  note_launch();
}

// One MSM.  Generic: d_points holds n points.  FIXED: d_points is a table of W*n points,
// T[j*n + i] = 2^(c j) P_i, built with the same c (fixed_table_impl).
template <class F, bool FIXED>
cudaError_t msm_impl(const uint32_t* d_scalars, const uint32_t* d_points, uint32_t n_in,
                     uint32_t* d_out, void* d_work, size_t work_bytes, const MsmConfig& cfg,
                     cudaStream_t st) {
  constexpr bool EC2 = FieldWords<F>::value == 16;
  constexpr int XB = 4 * FieldWords<F>::value * 4;  // bytes per XYZZ point
  if (cfg.xyzz_out && n_in == 0) return cudaErrorInvalidValue;
  // shared buckets: fixed-base MSMs (one bucket set) with terms (the accumulation is what
  // writes every bucket of the array)
  if ((cfg.bucket_out || cfg.bucket_add) && (!FIXED || n_in == 0)) return cudaErrorInvalidValue;
  if (cfg.bucket_out && cfg.bucket_add) return cudaErrorInvalidValue;
  if (n_in == 0) {
    k_store_inf<F><<<1, 32, 0, st>>>(d_out);
    note_launch();
    return cudaGetLastError();
  }
  if (FIXED && cfg.c <= 0) return cudaErrorInvalidValue;  // the table fixes the window
  const int c = cfg.c > 0 ? cfg.c : msm_default_window(n_in, EC2);
  if (c < 4 || c > 24) return cudaErrorInvalidValue;
  const bool glv = use_glv(EC2, FIXED, cfg.glv, cfg.affine, n_in);
  const int W = msm_windows(c, glv);
  // entry positions are uint32 and fixed-base entries carry a table index below the sign bit
  if ((uint64_t)W * n_in * (glv ? 2 : 1) >= (uint64_t)NEG_BIT) return cudaErrorInvalidValue;
  const uint32_t n = glv ? 2 * n_in : n_in;  // terms sorted into buckets
  const uint32_t nb = FIXED ? (1u << (c - 1)) : (uint32_t)W << (c - 1);
  const int rounds_req = cfg.affine < 0 ? auto_affine_rounds<F>(n, W, nb) : cfg.affine;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // Threads the accumulation keeps resident: an MSM whose tasks (an upper bound, at 32 entries)
  // fit kRoom times over runs in latency form (one group of lanes per task, shortest tasks).  A
  // group spends 16 lane products on a G1 addition where a thread spends 10 (64 and about 27 over
  // G2), so the line lies where the idle lanes run out: over tables, where tiles rather than buckets
  // make the tasks, twice as early, because the groups' tiles of 16 are twice as many.  Measured (us,
  // groups / threads; in brackets how many times the tasks fit):
  //   generic G2  1,000 terms (11.2) 881 / 910, 2,000 (9.3) 931 / 934, 4,000 (5.1) 1024 / 990
  //   fixed G2    1,000 (32) 311 / 343, 2,000 (16.6) 363 / 365, 8,000 (6.2) 534 / 455
  //   generic G1  1,000 (25) 395 / 392, 4,000 (7.6) 430 / 436, 8,000 (4.1) 500 / 467, 12,000 (3.6)
  //               531 / 507
  //   fixed G1    1,000 (43) 247 / 233, 4,000 (11.5) 248 / 251, 8,000 (8.3) 297 / 277, 16,000 (3.0)
  //               322 / 299
  // (over Fq the two are within 7 % of each other up to the line).
  const uint64_t resident = (uint64_t)accumulate_grid<F>(dev, sms) * 128;
  constexpr uint64_t kRoom = (EC2 ? 8 : 4) * (FIXED ? 2 : 1);
  const bool latency_mode = rounds_req == 0 && ((uint64_t)nb + (uint64_t)n * W / kMinTask + 1) * kRoom <= resident;
  // Automatic tile: about one task per resident thread, so a mid-size MSM (too many tasks for
  // the latency form, too few to fill the GPU at 64 entries a task) still keeps every thread
  // busy; 64 entries at most, or 96 where buckets average 48 or more (a GLV-split 2^20 MSM
  // averages 64: tiles of 64 split half its buckets and the partial sums cost a combine pass;
  // 2^20 5.16 -> 5.07 ms, 2^22 17.8 -> 17.3 ms); the latency form the shortest.
  const uint64_t ne = (uint64_t)n * W;
  const uint32_t tmin = cfg.min_task > 0 ? (uint32_t)cfg.min_task : layout_min_task(ne);  // the layout's bound
  uint32_t task_len;
  if (cfg.task > 0) {
    task_len = (uint32_t)cfg.task;
  } else {
    const uint64_t room = resident > nb / 2 + 1024 ? resident - nb / 2 : resident / 2;  // split buckets
    task_len = (uint32_t)std::min<uint64_t>(64, (ne + room - 1) / room);
    if (task_len == 64 && ne >= 48ull * nb) task_len = 96;
  }
  if (latency_mode) task_len = ne <= kSmallEntries ? kLatMinTask : kMinTask;
  task_len = std::max(task_len, tmin);  // the workspace is sized for tasks of at least tmin entries
  if (task_len > (uint32_t)kMaxTask) task_len = kMaxTask;
  const Layout L = make_layout(n_in, c, XB, cfg.min_task > 0 ? (uint32_t)cfg.min_task : 0u, FIXED,
                               layout_affine(EC2, cfg.affine, n_in, c, FIXED, glv), glv);
  if (work_bytes < L.total || d_work == nullptr) return cudaErrorInvalidValue;
  char* base = static_cast<char*>(d_work);
  uint32_t* counters = reinterpret_cast<uint32_t*>(base + L.counters);
  uint32_t* counts = reinterpret_cast<uint32_t*>(base + L.counts);
  uint32_t* offsets = reinterpret_cast<uint32_t*>(base + L.offsets);
  uint32_t* entries = reinterpret_cast<uint32_t*>(base + L.entries);
  Task* tasks = reinterpret_cast<Task*>(base + L.tasks);
  Multi* multi = reinterpret_cast<Multi*>(base + L.multi);
  uint32_t* partials = reinterpret_cast<uint32_t*>(base + L.partials);
  uint32_t* buckets = cfg.bucket_out ? cfg.bucket_out : reinterpret_cast<uint32_t*>(base + L.buckets);
  uint32_t* lv_y = reinterpret_cast<uint32_t*>(base + L.lv_y);
  uint32_t* lv_z = reinterpret_cast<uint32_t*>(base + L.lv_z);
  uint32_t* lv_y2 = reinterpret_cast<uint32_t*>(base + L.lv_y2);
  uint32_t* lv_z2 = reinterpret_cast<uint32_t*>(base + L.lv_z2);
  uint32_t* wsum = reinterpret_cast<uint32_t*>(base + L.wsum);
  void* scan_tmp = base + (L.total - scan_workspace_bytes(nb + 1));

  cudaError_t e;
  const int T = 256;
  uint32_t* glv_s = glv ? reinterpret_cast<uint32_t*>(base + L.glv_s) : nullptr;
  const uint32_t* phix = glv ? reinterpret_cast<uint32_t*>(base + L.glv_p) : nullptr;
  if constexpr (!EC2 && !FIXED) {
    if (glv) {
      k_glv_prep<F><<<(n_in + T - 1) / T, T, 0, st>>>(d_scalars, d_points, n_in, glv_s, const_cast<uint32_t*>(phix));
      note_launch();
    }
  }
  // counters and counts are neighbours
  if ((e = cudaMemsetAsync(counters, 0, L.counts - L.counters + ((size_t)nb + 1) * sizeof(uint32_t), st)) != cudaSuccess)
    return e;
  if (glv)
    k_count_glv<F><<<(n_in + T - 1) / T, T, 0, st>>>(glv_s, n_in, c, W, counts);
  else
    k_count<F, FIXED><<<(n + T - 1) / T, T, 0, st>>>(d_scalars, d_points, n, c, W, counts);
  note_launch();
  // counts becomes the scatter cursor
  if ((e = scan_exclusive_u32(counts, offsets, (size_t)nb + 1, scan_tmp, st, counts)) != cudaSuccess) return e;
  if (glv)
    k_scatter_glv<F><<<(n_in + T - 1) / T, T, 0, st>>>(glv_s, n_in, c, W, counts, entries);
  else
    k_scatter<F, FIXED><<<(n + T - 1) / T, T, 0, st>>>(d_scalars, d_points, n, c, W, counts, entries);
  note_launch();
  // batch-affine halving rounds (counts is free again and holds the halved counts)
  const uint32_t* acc_entries = entries;
  const uint32_t* acc_points = d_points;
  uint32_t* acc_off = offsets;
  const int rounds = L.affine ? std::min(rounds_req, 6) : 0;
  if (rounds > 0) {
    uint32_t* off_in = offsets;
    uint32_t* off_out = reinterpret_cast<uint32_t*>(base + L.off2);
    uint32_t* pa = reinterpret_cast<uint32_t*>(base + L.pa);
    uint32_t* pb = reinterpret_cast<uint32_t*>(base + L.pb);
    uint32_t* pref = reinterpret_cast<uint32_t*>(base + L.pref);
    const uint32_t* src = d_points;
    uint32_t* dst = pa;
    size_t max_slots = (size_t)n * W / 2 + 2 * (size_t)nb + 1;
    for (int r = 0; r < rounds; r++) {
      k_half_counts<<<(nb + 1 + T - 1) / T, T, 0, st>>>(off_in, nb, counts);
      if ((e = scan_exclusive_u32(counts, off_out, nb + 1, scan_tmp, st)) != cudaSuccess) return e;
      const size_t threads = (max_slots + kAffK - 1) / kAffK;
      const unsigned blocks = (unsigned)((threads + 127) / 128);
      if (r == 0)
        k_affine_round<F, true><<<blocks, 128, 0, st>>>(off_in, off_out, nb, entries, d_points, dst, pref);
      else
        k_affine_round<F, false><<<blocks, 128, 0, st>>>(off_in, off_out, nb, nullptr, src, dst, pref);
      note_launch(2);
      src = dst;
      dst = dst == pa ? pb : pa;
      uint32_t* t = off_in; off_in = off_out; off_out = t;
      max_slots = max_slots / 2 + 2 * (size_t)nb + 1;
    }
    acc_entries = nullptr;
    acc_points = src;
    acc_off = off_in;
  }
  k_task_hist<F><<<(nb + T - 1) / T, T, 0, st>>>(acc_off, nb, task_len, counters + kCtrHist, buckets);
  note_launch();
  k_task_emit<F><<<(nb + T - 1) / T, T, 0, st>>>(acc_off, nb, task_len, counters + kCtrHist, counters + kCtrCursor,
                                                  tasks, counters, multi);
  note_launch();
  if (cfg.acc_start) cudaEventRecord(cfg.acc_start, st);
  if (latency_mode)
    k_accumulate_group<F><<<sms * 8, 128, 0, st>>>(tasks, counters, acc_entries, acc_points, nb, buckets, partials,
                                                    nullptr, phix);
  else
    k_accumulate<F><<<accumulate_grid<F>(dev, sms), 128, 0, st>>>(tasks, counters, acc_entries, acc_points, nb,
                                                             buckets, partials, nullptr, phix);
  note_launch();
  k_combine_small<F><<<sms * 4, 128, 0, st>>>(multi, counters, nb, partials, buckets);
  k_combine<F><<<sms * 4, 128, 0, st>>>(multi, counters, partials, buckets);
  note_launch(2);
  if (cfg.acc_stop) cudaEventRecord(cfg.acc_stop, st);
  const int WR = FIXED ? 1 : W;
  const uint32_t B = 1u << (c - 1);
  if (cfg.bucket_out) {  // buckets handed on: this MSM's own result is the point at infinity
    k_store_inf<F><<<1, 32, 0, st>>>(d_out);
    note_launch();
    return cudaGetLastError();
  }
  if (cfg.bucket_add) {
    if (cfg.bucket_ready) cudaStreamWaitEvent(st, cfg.bucket_ready, 0);
    k_add_buckets<F><<<(B + 127) / 128, 128, 0, st>>>(buckets, cfg.bucket_add, B);
    note_launch();
  }
  BitTrees trees{};
  trees.t[trees.count++] = reduce_levels<F>(buckets, B, (uint32_t)WR, lv_y, lv_z, lv_y2, lv_z2, resident, st);
  join_trees<F>(trees, cfg.xyzz_out && WR == 1 ? cfg.xyzz_out : wsum, WR == 1 && !cfg.xyzz_out ? d_out : nullptr, st);
  if (WR > 1) {
    k_finish<F><<<1, 32, 0, st>>>(wsum, WR, c, d_out, cfg.xyzz_out);
    note_launch();
  }
  return cudaGetLastError();
}

// Fixed-base tables.  table[0..n) = points; table[j n + i] = 2^c table[(j-1) n + i],
// computed in XYZZ and brought back to affine with one inversion per run of kAffRun
// points (Montgomery's simultaneous inversion).  Points at infinity stay infinity.
constexpr int kAffRun = 16;

template <class F>
__global__ void __launch_bounds__(128) k_table_double(const uint32_t* __restrict__ src, uint32_t n, int c,
                                                      uint32_t* __restrict__ xyzz) {
  constexpr int XW = 4 * FieldWords<F>::value;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Affine<F> p = ld_affine<F>(src + (size_t)i * 2 * FieldWords<F>::value);
  XYZZ<F> r = XYZZ<F>::inf();
  if (!affine_is_inf(p)) {
    r = xyzz_mdbl(p);
#pragma unroll 1
    for (int d = 1; d < c; d++) r = xyzz_dbl(r);
  }
  st_xyzz<F>(xyzz + (size_t)i * XW, r);
}

// Thread t converts points [t R, t R + R): prefix products of ZZ*ZZZ, one inverse, and
// the back substitution; `pref` holds the prefix products (n field elements).
template <class F>
__global__ void __launch_bounds__(128) k_batch_affine(const uint32_t* __restrict__ xyzz, uint32_t n,
                                                      uint32_t* __restrict__ pref, uint32_t* __restrict__ dst) {
  constexpr int FW = FieldWords<F>::value;
  constexpr int XW = 4 * FW;
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t lo = t * kAffRun;
  if (lo >= n) return;
  const uint32_t hi = min(n, lo + kAffRun);
  F acc = F::one();
  for (uint32_t i = lo; i < hi; i++) {
    const XYZZ<F> p = ld_xyzz<F>(xyzz + (size_t)i * XW);
    if (!p.is_inf()) acc = acc * (p.ZZ * p.ZZZ);
    st_field(pref + (size_t)i * FW, acc);
  }
  F inv = acc.inv();
  for (uint32_t i = hi; i-- > lo;) {
    const XYZZ<F> p = ld_xyzz<F>(xyzz + (size_t)i * XW);
    uint32_t* o = dst + (size_t)i * 2 * FW;
    if (p.is_inf()) {
      st_affine<F>(o, Affine<F>{F::zero(), F::one()});
      continue;
    }
    F before = F::one();
    if (i > lo) {  // written above by this thread: a plain (coherent) load, not __ldg
      uint32_t* bw = reinterpret_cast<uint32_t*>(&before);
      const uint4* src = reinterpret_cast<const uint4*>(pref + (size_t)(i - 1) * FW);
#pragma unroll
      for (int q = 0; q < FW / 4; q++) {
        const uint4 v = src[q];
        bw[4 * q] = v.x; bw[4 * q + 1] = v.y; bw[4 * q + 2] = v.z; bw[4 * q + 3] = v.w;
      }
    }
    const F ip = inv * before;          // 1 / (ZZ ZZZ)
    inv = inv * (p.ZZ * p.ZZZ);
    st_affine<F>(o, Affine<F>{p.X * (p.ZZZ * ip), p.Y * (p.ZZ * ip)});
  }
}

inline size_t fixed_table_work_bytes(uint32_t n, int xyzz_bytes, int field_bytes) {
  return align256((size_t)n * xyzz_bytes) + align256((size_t)n * field_bytes);
}

template <class F>
cudaError_t fixed_table_impl(const uint32_t* d_points, uint32_t n, int c, uint32_t* d_table, void* d_work,
                             size_t work_bytes, cudaStream_t st) {
  constexpr int FW = FieldWords<F>::value;
  constexpr int XB = 16 * FW, PB = 8 * FW;
  if (c < 4 || c > 24) return cudaErrorInvalidValue;
  if (n == 0) return cudaSuccess;
  if (!d_work || work_bytes < fixed_table_work_bytes(n, XB, 4 * FW)) return cudaErrorInvalidValue;
  uint32_t* xyzz = static_cast<uint32_t*>(d_work);
  uint32_t* pref = reinterpret_cast<uint32_t*>(static_cast<char*>(d_work) + align256((size_t)n * XB));
  const int W = num_windows(c);
  cudaError_t e = cudaMemcpyAsync(d_table, d_points, (size_t)n * PB, cudaMemcpyDeviceToDevice, st);
  if (e != cudaSuccess) return e;
  const uint32_t runs = (n + kAffRun - 1) / kAffRun;
  for (int j = 1; j < W; j++) {
    const uint32_t* src = d_table + (size_t)(j - 1) * n * 2 * FW;
    uint32_t* dst = d_table + (size_t)j * n * 2 * FW;
    k_table_double<F><<<(n + 127) / 128, 128, 0, st>>>(src, n, c, xyzz);
    k_batch_affine<F><<<(runs + 127) / 128, 128, 0, st>>>(xyzz, n, pref, dst);
    note_launch(2);
  }
  return cudaGetLastError();
}

}  // namespace msm_detail
}  // namespace csb
