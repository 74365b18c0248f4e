// msm_batch.cuh -- many MSM instances of uneven size in one pass (instantiated for G1 in
// msm_batch_g1.cu and for G2 in msm_batch_g2.cu).
//
// The reference runs one GPU multi-exp call per instance (src/python/cuda_wrapper.py:216
// ec_mad_cuda2, batches dispatched one by one by groth_prover.py:1563).  Here all instances of
// one group share one digit sort and ONE accumulation launch:
//   * k_bcount / k_bscatter: one thread per term of any instance (binary search of the
//     instance's first term), digits with the instance's own window, buckets in one bucket
//     space (instance after instance, ordered by window);
//   * the task pipeline of the single MSM over all buckets, each task tagged with its
//     instance, and one persistent k_accumulate over the union of tasks, longest first --
//     the work is split by bucket size, not by instance, so a 2^10 instance next to a 2^20
//     one costs its share and no launch;
//   * reduction of all window groups' trees together (instances with equal c are contiguous),
//     and k_bfinish: one warp per instance for the window Horner and the affine result.
// Fixed-base instances (resident tables T[j n + i] = 2^(c j) P_i, the proof's MSMs) put every
// digit into one bucket set and need no window Horner.
// The sequence contains no allocation and no host synchronisation, so it can be captured in a
// CUDA graph once and replayed (cs_msm_batch_run).
#pragma once
#include "msm_impl.cuh"

namespace csb {
namespace msm_detail {

// Index of the job whose term range holds global term t (term0 ascending; empty jobs share
// their successor's term0 and are skipped by taking the last job with term0 <= t).
CSB_DEV uint32_t job_of_term(const BatchJob* jobs, uint32_t njobs, uint32_t t) {
  uint32_t lo = 0, hi = njobs;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (jobs[mid].term0 <= t) lo = mid; else hi = mid;
  }
  return lo;
}

// Splits the terms of the split instances: halves to s2, beta x to phix, at the global term.
template <class F>
__global__ void k_bprep(const BatchJob* __restrict__ jobs, uint32_t njobs, uint32_t terms, uint32_t* __restrict__ s2,
                        uint32_t* __restrict__ phix) {
  constexpr int PW = 2 * FieldWords<F>::value;
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= terms) return;
  const BatchJob jb = jobs[job_of_term(jobs, njobs, t)];
  if (!jb.glv) return;
  const uint32_t i = t - jb.term0;
  glv_prep_term<F>(jb.scalars + (size_t)i * 8, jb.points + (size_t)i * PW, s2 + (size_t)t * 8, phix + (size_t)t * 8);
}

template <class F>
__global__ void k_bcount(const BatchJob* __restrict__ jobs, uint32_t njobs, uint32_t terms,
                         const uint32_t* __restrict__ s2, uint32_t* __restrict__ counts) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= terms) return;
  const BatchJob jb = jobs[job_of_term(jobs, njobs, t)];
  const uint32_t i = t - jb.term0;
  uint32_t k[8];
  const uint32_t B = 1u << (jb.c - 1);
  if (jb.glv) {
    ld_limbs8(k, s2 + (size_t)t * 8);
    for_each_glv_digit(k, (int)jb.c, (int)jb.W, [&](int, int j, uint32_t mag, bool) {
      const size_t b = jb.bucket0 + (size_t)j * B + (mag - 1);
      if (j == 0) claim_shared(counts, b); else atomicAdd(&counts[b], 1u);
    });
    return;
  }
  if (!load_scalar<F>(jb.scalars, jb.points, i, k)) return;
  for_each_digit(k, (int)jb.c, (int)jb.W, [&](int j, uint32_t mag, bool) {
    const size_t b = jb.bucket0 + (jb.fixed ? 0 : (size_t)j * B) + (mag - 1);
    if (j == 0) claim_shared(counts, b); else atomicAdd(&counts[b], 1u);
  });
}

template <class F>
__global__ void k_bscatter(const BatchJob* __restrict__ jobs, uint32_t njobs, uint32_t terms,
                           const uint32_t* __restrict__ s2, uint32_t* __restrict__ cursor,
                           uint32_t* __restrict__ entries) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= terms) return;
  const BatchJob jb = jobs[job_of_term(jobs, njobs, t)];
  const uint32_t i = t - jb.term0;
  uint32_t k[8];
  if (jb.glv) {
    ld_limbs8(k, s2 + (size_t)t * 8);
    scatter_glv_term(k, i, (int)jb.c, (int)jb.W, jb.bucket0, cursor, entries);
    return;
  }
  if (!load_scalar<F>(jb.scalars, jb.points, i, k)) return;
  const uint32_t B = 1u << (jb.c - 1);
  scatter_digits(k, (int)jb.c, (int)jb.W, cursor, entries,
                 [&](int j, uint32_t mag) { return jb.bucket0 + (jb.fixed ? 0 : (size_t)j * B) + (mag - 1); },
                 [&](int j, bool neg) { return (jb.fixed ? (uint32_t)j * jb.n + i : i) | (neg ? NEG_BIT : 0u); });
}

// One warp per instance (block i: instance i):
// sum_j 2^(c j) S_j over its bucket sets (a fixed-base instance has one), affine result.
template <class F>
__global__ void __launch_bounds__(32) k_bfinish(const BatchJob* __restrict__ jobs, const uint32_t* __restrict__ wsum) {
  const BatchJob jb = jobs[blockIdx.x];
  windows_horner<F>(wsum + (size_t)jb.window0 * 4 * FieldWords<F>::value, (int)jb.sets, (int)jb.c, jb.out, nullptr);
}

struct BatchLayout {
  size_t counters, counts, offsets, entries, tasks, multi, partials, buckets, lv_y, lv_z, lv_y2, lv_z2, wsum,
      glv_s, glv_p, scan, total;
};

inline BatchLayout batch_layout(const MsmBatch& b, int xyzz_bytes) {
  const size_t nb = b.nbuckets, ne = b.nentries;
  const size_t tl = (size_t)std::max(kBatchMinTask, std::min(b.task, kMaxTask));
  const size_t lv = b.lv_points, lv2 = b.lv2_points;
  BatchLayout L{};
  size_t o = 0;
  L.counters = o; o = align256(o + kCtrWords * sizeof(uint32_t));
  L.counts = o;   o = align256(o + (nb + 1) * sizeof(uint32_t));
  L.offsets = o;  o = align256(o + (nb + 1) * sizeof(uint32_t));
  L.entries = o;  o = align256(o + ne * sizeof(uint32_t));
  L.tasks = o;    o = align256(o + (nb + ne / tl + 1) * sizeof(Task));
  L.multi = o;    o = align256(o + (ne / (tl + 1) + 1) * sizeof(Multi));
  L.partials = o; o = align256(o + (2 * (ne / tl) + 1) * (size_t)xyzz_bytes);
  L.buckets = o;  o = align256(o + nb * (size_t)xyzz_bytes);
  L.lv_y = o;     o = align256(o + lv * xyzz_bytes);
  L.lv_z = o;     o = align256(o + lv * xyzz_bytes);
  L.lv_y2 = o;    o = align256(o + lv2 * xyzz_bytes);
  L.lv_z2 = o;    o = align256(o + lv2 * xyzz_bytes);
  L.wsum = o;     o = align256(o + (size_t)b.nwindows * xyzz_bytes);
  L.glv_s = L.glv_p = o;
  if (b.glv) {
    o = align256(o + (size_t)b.terms * 32);
    L.glv_p = o;
    o = align256(o + (size_t)b.terms * 32);
  }
  L.scan = o;
  L.total = o + scan_workspace_bytes(nb + 1);
  return L;
}

template <class F>
cudaError_t batch_impl(const MsmBatch& b, void* d_work, size_t work_bytes, cudaStream_t st) {
  constexpr int XB = 4 * FieldWords<F>::value * 4;
  constexpr int XWD = XB / 4;
  if (b.njobs == 0) return cudaSuccess;
  const BatchLayout L = batch_layout(b, XB);
  if (!d_work || work_bytes < L.total || b.nentries >= (uint64_t)0xffffffffu) return cudaErrorInvalidValue;
  char* base = static_cast<char*>(d_work);
  auto at = [&](size_t off) { return reinterpret_cast<uint32_t*>(base + off); };
  uint32_t *counters = at(L.counters), *counts = at(L.counts), *offsets = at(L.offsets);
  uint32_t *entries = at(L.entries), *partials = at(L.partials), *buckets = at(L.buckets);
  uint32_t *lv_y = at(L.lv_y), *lv_z = at(L.lv_z), *lv_y2 = at(L.lv_y2), *lv_z2 = at(L.lv_z2), *wsum = at(L.wsum);
  Task* tasks = reinterpret_cast<Task*>(base + L.tasks);
  Multi* multi = reinterpret_cast<Multi*>(base + L.multi);
  const uint32_t nb = b.nbuckets;
  const uint32_t task_len = (uint32_t)std::max(kBatchMinTask, std::min(b.task, kMaxTask));  // as the layout
  cudaError_t e;
  // counters and counts are neighbours
  if ((e = cudaMemsetAsync(counters, 0, L.counts - L.counters + ((size_t)nb + 1) * sizeof(uint32_t), st)) != cudaSuccess)
    return e;
  const int T = 256;
  uint32_t *glv_s = at(L.glv_s), *phix = b.glv ? at(L.glv_p) : nullptr;
  if constexpr (FieldWords<F>::value == 8) {
    if (b.glv && b.terms) {
      k_bprep<F><<<(b.terms + T - 1) / T, T, 0, st>>>(b.d_jobs, b.njobs, b.terms, glv_s, phix);
      note_launch();
    }
  }
  if (b.terms) {
    k_bcount<F><<<(b.terms + T - 1) / T, T, 0, st>>>(b.d_jobs, b.njobs, b.terms, glv_s, counts);
    note_launch();
  }
  // counts becomes the scatter cursor
  if ((e = scan_exclusive_u32(counts, offsets, (size_t)nb + 1, base + L.scan, st, counts)) != cudaSuccess) return e;
  if (b.terms) {
    k_bscatter<F><<<(b.terms + T - 1) / T, T, 0, st>>>(b.d_jobs, b.njobs, b.terms, glv_s, counts, entries);
    note_launch();
  }
  k_task_hist<F><<<(nb + T - 1) / T, T, 0, st>>>(offsets, nb, task_len, counters + kCtrHist, buckets);
  k_task_emit<F><<<(nb + T - 1) / T, T, 0, st>>>(offsets, nb, task_len, counters + kCtrHist, counters + kCtrCursor,
                                                  tasks, counters, multi, b.d_jobs, b.njobs);
  note_launch(2);
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // Latency form (one group of lanes per task) while the resident threads would fit the tasks (an
  // upper bound: every bucket and every full tile) this many times: 4, or 16 over tables,
  // where a batch of proofs runs three batches of MSMs side by side.
  // Measured (us, groups / threads; in brackets how many times the tasks fit): G1 instances of
  // 1,351 terms together (8.0) 363 / 368, of 2,791 (3.9) 390 / 380; G2 of 1,351 (5.2) 908 / 924, of
  // 2,791 (2.5) 1004 / 955; two proofs of 2^7 (17-53) 444 / 447, of 2^8 (9-28) 457 / 455, of 2^9
  // (6-17) 521 / 490, four of 2^10 (1.5-4.6) 736 / 585.
  const uint64_t resident = (uint64_t)accumulate_grid<F>(dev, sms) * 128;
  const uint64_t room = b.fixed ? 16 : 4;
  const bool latency_mode = ((uint64_t)nb + b.nentries / task_len + 1) * room <= resident;
  if (latency_mode)
    k_accumulate_group<F><<<sms * 8, 128, 0, st>>>(tasks, counters, entries, nullptr, nb, buckets, partials, b.d_jobs,
                                                    phix);
  else
    k_accumulate<F><<<accumulate_grid<F>(dev, sms), 128, 0, st>>>(tasks, counters, entries, nullptr, nb, buckets,
                                                             partials, b.d_jobs, phix);
  k_combine_small<F><<<sms * 4, 128, 0, st>>>(multi, counters, nb, partials, buckets);
  k_combine<F><<<sms * 4, 128, 0, st>>>(multi, counters, partials, buckets);
  note_launch(3);
  // reduction: the groups that need levels of eight (and their buffers) one by one, the others'
  // trees together (24 instances of six widths 3098 -> 2850 us, where each width took a chain of
  // three launches)
  BitTrees trees{};
  for (uint32_t g = 0; g < b.ngroups; g++) {
    const BatchGroup& G = b.groups[g];
    const uint32_t B = 1u << (G.c - 1);
    BitTrees one{};
    const bool levels = reduce_needs_levels<F>(B, G.windows, resident);
    BitTree t = reduce_levels<F>(buckets + (size_t)G.bucket0 * XWD, B, G.windows, lv_y, lv_z, lv_y2, lv_z2, resident, st);
    t.wsum0 = G.window0;
    BitTrees& T = levels ? one : trees;
    T.t[T.count++] = t;
    if (levels || trees.count == kMaxTrees) {
      join_trees<F>(T, wsum, nullptr, st);
      T.count = 0;
    }
  }
  if (trees.count) join_trees<F>(trees, wsum, nullptr, st);
  k_bfinish<F><<<b.njobs, 32, 0, st>>>(b.d_jobs, wsum);
  note_launch();
  return cudaGetLastError();
}

}  // namespace msm_detail
}  // namespace csb
