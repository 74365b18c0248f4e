// ntt.cu -- radix-2 NTT passes in shared memory and Fr elementwise helpers (ntt.cuh).
#include <algorithm>

#include "ntt.cuh"
#include "curve.cuh"
#include "runtime.cuh"

namespace csb {

namespace {

constexpr int kMaxStages = 11;  // 2^11 elements x 32 B = 64 KB of shared memory per block
constexpr int kThreads = 256;
// One thread per butterfly (k_ntt_pass2) up to this many warps a scheduler, beyond it a thread
// per four elements (us, at 1 / 4 / 8: H step of 2^15 97 / 79 / 79, of 2^16 123.6 / 116.5 / 116.4,
// of 2^17 196.0 / 196.1 / 199.1; NTT 2^18 66.8 / 66.8 / 70.4).
constexpr uint64_t kLatencyWarps = 4;

// One pass: stages s0 .. s0+S-1 of a radix-2 DIT transform of 2^L points.  Block q owns
// the 2^S elements base + (i << s0), base = ((q >> s0) << (s0 + S)) + (q & (2^s0 - 1)).
// blockIdx.y: the instance of a batch, its arrays `stride` words after the previous one's;
// blockIdx.z: the transform (NttArgs::count).
struct Pass {
  const uint32_t* in[3];
  uint32_t* out;
  const uint32_t *mul, *odd, *odd_mul, *sub, *scalar;
  const uint32_t *W, *post_tab, *post_scalar;
  size_t stride, in_step, out_step;  // in_step: offset of in[0] per transform where in[1] is null
  uint32_t L, s0, S, wshift;
  int bitrev, load, canon;
};

// Element g of the pass's input, below 4r.
CSB_DEV Fr pass_load(const Pass& a, const uint32_t* in, size_t inst, uint32_t g) {
  if (!a.bitrev) return ld_fp<ModR>(in + (size_t)g * 8);
  const uint32_t i = __brev(g) >> (32 - a.L);
  if (a.load == (int)NttLoad::kPlain) return ld_fp<ModR>(in + (size_t)i * 8);
  if (a.load == (int)NttLoad::kInterleaved) {
    const size_t o = inst + (size_t)(i >> 1) * 8;
    if ((i & 1) == 0) return Fr::mul_raw(ld_fp<ModR>(in + (size_t)(i >> 1) * 8), ld_fp<ModR>(a.mul + o));
    return Fr::mul_raw(Fr::mul_raw(ld_fp<ModR>(a.odd + o), ld_fp<ModR>(a.odd_mul + o)), ld_fp<ModR>(a.scalar));
  }
  const size_t o = inst + (size_t)i * 8;
  const Fr ab = Fr::mul_raw(ld_fp<ModR>(in + (size_t)i * 8), ld_fp<ModR>(a.mul + o));  // < 1.2r
  return Fr::mul_raw(Fr::sub_lazy(ab, ld_fp<ModR>(a.sub + o)), ld_fp<ModR>(a.scalar));
}
// Element g of the pass's output from x < 4r.
CSB_DEV void pass_store(const Pass& a, uint32_t* out, uint32_t g, Fr x) {
  if (a.post_scalar) x = Fr::mul_raw(x, ld_fp<ModR>(a.post_scalar));
  if (a.post_tab) x = Fr::mul_raw(x, ld_fp<ModR>(a.post_tab + (size_t)g * 8));
  if (a.canon) x = Fr::reduce_2p(x).canon();
  st_fp<ModR>(out + (size_t)g * 8, x);
}
// Butterfly on values below 4r (4r < 2^256): x, y -> x + t, x - t with t = w y < 2r, both
// below 4r again: one conditional subtraction of 2r instead of three reductions to [0, r).
CSB_DEV void butterfly(Fr& x, Fr& y, const Fr& t) {
  const Fr u = Fr::reduce_2p(x);
  x = Fr::add_raw(u, t);
  y = Fr::add_raw(u, Fr::neg_lazy(t));
}

// Elements as two arrays of 16-byte halves: lanes read consecutive 16-byte words, where
// whole 32-byte elements would meet in half the banks.
struct Tile {
  uint4 *lo, *hi;
  CSB_DEV Fr get(uint32_t i) const {
    const uint4 a = lo[i], b = hi[i];
    return Fr{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
  }
  CSB_DEV void put(uint32_t i, const Fr& x) const {
    lo[i] = make_uint4(x.v[0], x.v[1], x.v[2], x.v[3]);
    hi[i] = make_uint4(x.v[4], x.v[5], x.v[6], x.v[7]);
  }
};

struct Block {
  const uint32_t* in;
  uint32_t* out;
  size_t inst;
  uint32_t r, base;
};
CSB_DEV Block pass_block(const Pass& a) {
  Block b;
  b.inst = (size_t)blockIdx.y * a.stride;
  const uint32_t z = blockIdx.z;
  b.in = (a.in[1] ? a.in[z] : a.in[0] + z * a.in_step) + b.inst;
  b.out = a.out + b.inst + z * a.out_step;
  uint32_t q = blockIdx.x;
  // the first pass's gather leaves a block's neighbours in memory to blocks 2^(L-S-1) and
  // 2^(L-S-2) further on: four consecutive blocks share their 128-byte lines this way
  if (a.bitrev && a.L - a.S >= 2) q = (q >> 2) | ((q & 3u) << (a.L - a.S - 2));
  const uint32_t rmask = (1u << a.s0) - 1u;
  b.r = q & rmask;
  b.base = ((q >> a.s0) << (a.s0 + a.S)) + b.r;
  return b;
}

// Throughput form (2^22 points 0.87 ms, bound by the products: 0.68 ms at the GPU's rate; 1.05 ms
// with one stage a barrier and values reduced below r after each): a thread takes four elements
// through two stages at a time, so a pass crosses shared memory and the barrier (S - 1) / 2 times;
// the first stages read from and the last write to global memory directly.  An odd S starts with
// one single stage.  BLOCKS resident blocks a SM: three (80 registers) from 2^20 elements in all
// transforms of the launch on, where there are blocks enough to keep them full, two below (us, two /
// three: NTT 2^19 117 / 122, 2^20 220 / 215, 2^22 896 / 872; H step of 2^18 346 / 371, of 2^19, two
// transforms side by side, 669 / 648; on the coset, three of them, 2^18 404 / 402, 2^19 774 / 756).
template <int BLOCKS>
__global__ void __launch_bounds__(kThreads, BLOCKS) k_ntt_pass4(const Pass a) {
  extern __shared__ uint4 sm[];
  const uint32_t cnt = 1u << a.S, s0 = a.s0;
  const Tile tile{sm, sm + cnt};
  const Block b = pass_block(a);
  uint32_t t = 0;
  if (a.S & 1) {
    const Fr w = ld_fp<ModR>(a.W + ((size_t)b.r << (a.L - s0 - 1 + a.wshift)) * 8);
#pragma unroll 1
    for (uint32_t j = threadIdx.x; j < cnt / 2; j += blockDim.x) {
      Fr x = pass_load(a, b.in, b.inst, b.base + ((2 * j) << s0));
      Fr y = pass_load(a, b.in, b.inst, b.base + ((2 * j + 1) << s0));
      butterfly(x, y, s0 == 0 ? Fr::reduce_2p(y) : Fr::mul_raw(y, w));
      tile.put(2 * j, x);
      tile.put(2 * j + 1, y);
    }
    t = 1;
    __syncthreads();
  }
#pragma unroll 1
  for (; t < a.S; t += 2) {
    const bool first = t == 0, last = t + 2 == a.S;
    const uint32_t sh = a.L - (s0 + t) - 2 + a.wshift;  // of the second stage's twiddles
#pragma unroll 1
    for (uint32_t j = threadIdx.x; j < cnt / 4; j += blockDim.x) {
      const uint32_t low = j & ((1u << t) - 1u);
      const uint32_t i0 = ((j >> t) << (t + 2)) | low;
      const uint32_t k = b.r + (low << s0);
      Fr x[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const uint32_t i = i0 + ((uint32_t)q << t);
        x[q] = first ? pass_load(a, b.in, b.inst, b.base + (i << s0)) : tile.get(i);
      }
      if (first && s0 == 0) {  // twiddles 1, 1 and 1, w^(n/4)
        butterfly(x[0], x[1], Fr::reduce_2p(x[1]));
        butterfly(x[2], x[3], Fr::reduce_2p(x[3]));
        butterfly(x[0], x[2], Fr::reduce_2p(x[2]));
      } else {
        const Fr w1 = ld_fp<ModR>(a.W + ((size_t)k << (sh + 1)) * 8);
        butterfly(x[0], x[1], Fr::mul_raw(x[1], w1));
        butterfly(x[2], x[3], Fr::mul_raw(x[3], w1));
        butterfly(x[0], x[2], Fr::mul_raw(x[2], ld_fp<ModR>(a.W + ((size_t)k << sh) * 8)));
      }
      butterfly(x[1], x[3], Fr::mul_raw(x[3], ld_fp<ModR>(a.W + ((size_t)(k + (1u << (s0 + t))) << sh) * 8)));
      if (first && last) __syncthreads();  // one round: every element read before any is written
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const uint32_t i = i0 + ((uint32_t)q << t);
        if (last) pass_store(a, b.out, b.base + (i << s0), x[q]);
        else tile.put(i, x[q]);
      }
    }
    __syncthreads();
  }
}

// Latency form, for transforms that leave schedulers idle: a thread per butterfly, one stage
// at a time (a stage is one product deep), the next stage's twiddle loaded ahead.
__global__ void __launch_bounds__(1024) k_ntt_pass2(const Pass a) {
  extern __shared__ uint4 sm[];
  const uint32_t cnt = 1u << a.S, s0 = a.s0, j = threadIdx.x;
  const Tile tile{sm, sm + cnt};
  const Block b = pass_block(a);
  auto twiddle = [&](uint32_t t) {
    const uint32_t k = b.r + ((j & ((1u << t) - 1u)) << s0);
    return ld_fp<ModR>(a.W + ((size_t)k << (a.L - (s0 + t) - 1 + a.wshift)) * 8);
  };
  Fr w = twiddle(0);
  Fr x = pass_load(a, b.in, b.inst, b.base + ((2 * j) << s0));
  Fr y = pass_load(a, b.in, b.inst, b.base + ((2 * j + 1) << s0));
#pragma unroll 1
  for (uint32_t t = 0;; t++) {
    const uint32_t i = ((j >> t) << (t + 1)) | (j & ((1u << t) - 1u));
    const Fr wn = t + 1 < a.S ? twiddle(t + 1) : w;
    if (t) {
      x = tile.get(i);
      y = tile.get(i + (1u << t));
    }
    butterfly(x, y, Fr::mul_raw(y, w));
    w = wn;
    if (t + 1 == a.S) {
      if (t == 0) __syncthreads();  // one stage: every element read before any is written
      pass_store(a, b.out, b.base + (i << s0), x);
      pass_store(a, b.out, b.base + ((i + (1u << t)) << s0), y);
      return;
    }
    tile.put(i, x);
    tile.put(i + (1u << t), y);
    __syncthreads();
  }
}

// W[j] = root^j: each thread raises root to its first index, then steps.
__global__ void k_powers(uint32_t* __restrict__ out, const uint32_t* __restrict__ root, uint32_t count,
                         uint32_t per_thread) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t first = (uint64_t)t * per_thread;
  if (first >= count) return;
  const Fr w = ld_fp<ModR>(root);
  Fr acc = Fr::one(), base = w;
  uint64_t e = first;
  while (e) {
    if (e & 1) acc = acc * base;
    base = base.sqr();
    e >>= 1;
  }
  for (uint32_t j = 0; j < per_thread && first + j < count; j++) {
    st_fp<ModR>(out + (first + j) * 8, acc);
    acc = acc * w;
  }
}

__global__ void k_gather_roots(uint32_t* __restrict__ out, const uint32_t* __restrict__ table,
                               uint64_t stride, uint32_t n, int dir, uint32_t count) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= count) return;
  const uint64_t idx = dir > 0 ? j : (uint64_t)((n - j) & (n - 1));
  const uint64_t src = (stride * idx) & (stride * (uint64_t)n - 1);
  const uint4* s = reinterpret_cast<const uint4*>(table + src * 8);
  uint4* d = reinterpret_cast<uint4*>(out + (uint64_t)j * 8);
  d[0] = s[0];
  d[1] = s[1];
}

// Stages per pass.  At least two passes from 2^9 points on: one block would run alone on its
// SM otherwise (2^11 points 50 us in one pass, 17 in two).
void plan_passes(uint32_t L, uint32_t* sizes, int* np) {
  const int n = std::max((int)((L + kMaxStages - 1) / kMaxStages), L >= 9 ? 2 : 1);
  int k = 0;
  uint32_t left = L;
  for (int p = 0; p < n; p++) {
    const uint32_t sz = (left + (n - p) - 1) / (n - p);  // even split, larger first
    sizes[k++] = sz;
    left -= sz;
  }
  *np = k;
}

}  // namespace

cudaError_t ntt_run(const NttArgs& a, cudaStream_t st) {
  const uint32_t L = a.log_n;
  if (L == 0 || L > 28 || a.log_tab < L || !a.W || !a.in[0] || !a.out || a.batch == 0 || a.batch > 65535 ||
      a.count == 0 || a.count > 3)
    return cudaErrorInvalidValue;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  uint32_t sizes[8];
  int np = 0;
  plan_passes(L, sizes, &np);
  uint32_t* work = a.out;
  if (np > 1) {
    // the first pass must not write where other blocks still read
    const size_t n = (size_t)1 << L, n_in = a.load == NttLoad::kInterleaved ? n / 2 : n;
    bool over = false;
    for (uint32_t z = 0; z < a.count; z++)
      for (uint32_t y = 0; y < a.count; y++) over |= ntt_overlap(a.in[z], n_in, a.out + y * a.out_step, n);
    if (over) {
      if (!a.tmp) return cudaErrorInvalidValue;
      work = a.tmp;
    }
  }
  // one thread per butterfly while that leaves at most kLatencyWarps warps a scheduler
  const uint64_t elements = (uint64_t)a.count * a.batch << L;
  const bool latency = elements / 2 <= (uint64_t)sms * 4 * 32 * kLatencyWarps;
  uint32_t s0 = 0;
  for (int p = 0; p < np; p++) {
    const uint32_t S = sizes[p];
    const bool first = (p == 0), last = (p == np - 1);
    Pass q{};
    for (int z = 0; z < 3; z++) q.in[z] = first ? (z < (int)a.count ? a.in[z] : nullptr) : nullptr;
    if (!first) q.in[0] = work;
    q.in_step = a.out_step;
    q.out = last ? a.out : work;
    q.out_step = a.out_step;
    q.stride = a.stride;
    q.mul = a.mul; q.odd = a.odd; q.odd_mul = a.odd_mul; q.sub = a.sub; q.scalar = a.scalar;
    q.W = a.W;
    q.post_tab = last ? a.post_tab : nullptr;
    q.post_scalar = last ? a.post_scalar : nullptr;
    q.L = L; q.s0 = s0; q.S = S; q.wshift = a.log_tab - L;
    q.bitrev = first ? 1 : 0;
    q.load = (int)a.load;
    q.canon = last && !a.lazy_out;
    const dim3 grid(1u << (L - S), a.batch, a.count);
    auto* pass4 = elements >= 1u << 20 ? k_ntt_pass4<3> : k_ntt_pass4<2>;
    if ((32u << S) > 48u * 1024) {  // above the default limit of a block's shared memory
      const cudaError_t e = cudaFuncSetAttribute(latency ? (const void*)k_ntt_pass2 : (const void*)pass4,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, 32 << S);
      if (e != cudaSuccess) return e;
    }
    if (latency || S == 1) {
      k_ntt_pass2<<<grid, 1u << (S - 1), (1u << S) * 32, st>>>(q);
    } else {
      const unsigned threads = (1u << (S - 2)) < (unsigned)kThreads ? (1u << (S - 2)) : (unsigned)kThreads;
      pass4<<<grid, threads, (1u << S) * 32, st>>>(q);
    }
    note_launch();
    s0 += S;
  }
  return cudaGetLastError();
}

cudaError_t ntt_powers(uint32_t* d_out, const uint32_t* d_root, uint32_t count, cudaStream_t st) {
  if (count == 0) return cudaSuccess;
  const uint32_t per = 64;
  const uint32_t threads = (count + per - 1) / per;
  k_powers<<<(threads + 127) / 128, 128, 0, st>>>(d_out, d_root, count, per);
  note_launch();
  return cudaGetLastError();
}

cudaError_t ntt_gather_roots(uint32_t* d_out, const uint32_t* d_table, uint64_t stride, uint32_t n,
                             int dir, uint32_t count, cudaStream_t st) {
  if (count == 0) return cudaSuccess;
  k_gather_roots<<<(count + 255) / 256, 256, 0, st>>>(d_out, d_table, stride, n, dir, count);
  note_launch();
  return cudaGetLastError();
}

}  // namespace csb
