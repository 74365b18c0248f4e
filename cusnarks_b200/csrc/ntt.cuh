// ntt.cuh -- number-theoretic transforms over Fr on sm_100a and the QAP H step.
//
// Transform: X_k = sum_j x_j w^(jk) in natural order (the reference's ntt_h / intt_h,
// src/cuda/ntt.cpp:453 / :583: bit-reverse, then radix-2 decimation in time).  A
// transform of 2^L points runs as ceil(L/11) passes; each pass keeps 2^S elements of one
// sub-transform in registers and shared memory, the first pass gathers in bit-reversed
// order (and can form its input from products of other arrays) and the last pass can
// multiply every output by a per-element table or one scalar (used for 1/n scaling, coset
// shifts and leaving Montgomery form).
//
// Twiddles: W[j] = w^j (Montgomery), j < n_tab/2, for a table built for 2^L_tab points;
// a transform of 2^L <= 2^L_tab points reads W with stride 2^(L_tab - L).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace csb {

// What the first pass reads as element i of the logical input.
enum class NttLoad {
  kPlain,        // in[i]
  kInterleaved,  // i even: in[i/2] * mul[i/2];  i odd: odd[i/2] * odd_mul[i/2] * scalar
  kQuotient,     // (in[i] * mul[i] - sub[i]) * scalar
};

struct NttArgs {
  // up to three transforms of one size and table side by side (arrays at unrelated
  // addresses): transform z reads in[z] and writes out + z * out_step words
  const uint32_t* in[3] = {nullptr, nullptr, nullptr};
  uint32_t count = 1;
  uint32_t* out = nullptr;          // natural-order output; may lie over in[] where tmp is given
  size_t out_step = 0;
  uint32_t* tmp = nullptr;          // scratch, laid out as out, when out overlaps the input
  uint32_t log_n = 0;
  const uint32_t* W = nullptr;      // twiddles for direction of this transform
  uint32_t log_tab = 0;             // W is a table for 2^log_tab points
  NttLoad load = NttLoad::kPlain;
  const uint32_t *mul = nullptr, *odd = nullptr, *odd_mul = nullptr, *sub = nullptr, *scalar = nullptr;
  const uint32_t* post_tab = nullptr;     // out[i] *= post_tab[i] (Montgomery product)
  const uint32_t* post_scalar = nullptr;  // out[i] *= *post_scalar (Montgomery product)
  bool lazy_out = false;            // leave the outputs below 4r instead of below r
  // batch instances of the transforms: instance y reads and writes the input arrays, out and
  // tmp offset by y * stride words (W, post_tab and the scalars are shared)
  uint32_t batch = 1;
  size_t stride = 0;
};

cudaError_t ntt_run(const NttArgs& a, cudaStream_t st);
// Whether arrays of nx and ny elements overlap.
inline bool ntt_overlap(const uint32_t* x, size_t nx, const uint32_t* y, size_t ny) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(x), b = reinterpret_cast<uintptr_t>(y);
  return a < b + ny * 32 && b < a + nx * 32;
}

// W[j] = root^j for j < count (root: one Montgomery element in device memory).
cudaError_t ntt_powers(uint32_t* d_out, const uint32_t* d_root, uint32_t count, cudaStream_t st);
// d_out[j] = table[(stride * idx(j)) mod (stride * n)] with idx(j) = j (dir +1) or
// (n - j) mod n (dir -1), j < count: the reference's root indexing for one direction.
cudaError_t ntt_gather_roots(uint32_t* d_out, const uint32_t* d_table, uint64_t stride, uint32_t n,
                             int dir, uint32_t count, cudaStream_t st);

}  // namespace csb
