// Measurement sampling on the device: shots drawn from the state's outcome distribution without
// downloading it, by the inverse-CDF rule of qsv's cdf_sample (crates/qsv-core/src/sample.rs:163-172).
//
// Shot k takes the k-th `unit()` value of SplitMix64(seed) (crates/qsv-core/src/circuits.rs:22-46),
// u_k in [0, 1), scales it by the total probability, x_k = u_k * total, and returns the first
// outcome i whose cumulative probability CDF(i) >= x_k (cdf_sample's `partition_point(|&c| c < u)`,
// a lower bound; the last outcome if rounding leaves none). The probabilities are |amp|^2 computed
// as the trait's `probabilities` does, in the state's precision (re*re + im*im, no fused
// multiply-add), and accumulated in FP64; the device sums them in another order than the
// reference's chunked scan, so a draw can differ only where x_k lies within rounding of a CDF value.
// Steps: the FP64 total of each 8192-amplitude block; an exclusive scan of those; the scaled
// uniforms sorted with their shot numbers; the first shot of each block; then one pass over the
// blocks: block b takes the sorted values x with CDFstart(b) < x <= CDFstart(b + 1) (block 0 also
// x = 0), builds its inclusive prefix in shared memory and places each shot by binary search, writing
// the outcome at the shot's original position.

#include <cuda_runtime.h>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <vector>

#include "qsvb_internal.h"

namespace qsvb {
namespace {

constexpr int kBlockBits = 13;
constexpr int kSampleThreads = 512;

// Device scratch of one call, carved out of one block: the context keeps a block of up to
// kSampleKeep bytes for the next call (allocating and freeing eight buffers a call took longer than
// the kernels on small states); a larger one is freed when the call returns.
constexpr size_t kSampleKeep = size_t(64) << 20;
struct Scratch {
  qsvb_ctx* c;
  char* p = nullptr;
  bool keep = false;
  Scratch(qsvb_ctx* ctx, size_t bytes) : c(ctx), keep(bytes <= kSampleKeep) {
    if (!keep) {
      device_malloc(c, reinterpret_cast<void**>(&p), bytes);
      return;
    }
    if (c->sample_cap < bytes) {
      QSVB_CK(cudaStreamSynchronize(c->stream));
      if (c->d_sample) QSVB_CK(cudaFree(c->d_sample));
      c->d_sample = nullptr;
      c->sample_cap = 0;
      device_malloc(c, reinterpret_cast<void**>(&c->d_sample), bytes);
      c->sample_cap = bytes;
    }
    p = c->d_sample;
  }
  ~Scratch() {
    if (!keep) cudaFree(p);  // (waits for the stream's work)
  }
  Scratch(const Scratch&) = delete;
  Scratch& operator=(const Scratch&) = delete;
};

// |amp|^2 rounded as StateVector::probabilities computes it in the state's precision
// (crates/qsv-core/src/state/mod.rs:130-134: re*re + im*im with separate roundings), widened to FP64.
__device__ __forceinline__ double prob_of(float x, float y) {
  return double(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)));
}
__device__ __forceinline__ double prob_of(double x, double y) { return __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)); }

__device__ __forceinline__ uint64_t mix64s(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// FP64 sum of |amp|^2 over each block of 2^bb amplitudes (one block per CTA iteration). A thread's 16
// amplitudes of a full block are all requested before the first is used: one at a time, the loop ran at
// the latency of its loads (a call for 1000 shots, where this pass is nearly all of it, 27 qubits
// complex128: 0.80 -> 0.43 ms; one read of the state takes 0.33). The order of the sums is part of the
// result (draws compare against them), so it stays one amplitude every 512.
template <class R>
__global__ void __launch_bounds__(kSampleThreads) k_block_sums(const R* __restrict__ re, const R* __restrict__ im,
                                                               uint32_t bb, uint64_t nblocks,
                                                               double* __restrict__ bsum) {
  __shared__ double s_red[2][kSampleThreads / 32];
  const uint32_t B = 1u << bb;
  int half = 0;
  for (uint64_t b = blockIdx.x; b < nblocks; b += gridDim.x, half ^= 1) {
    double acc = 0.0;
    if (bb == uint32_t(kBlockBits)) {
      constexpr int PER = (1 << kBlockBits) / kSampleThreads;
      R x[PER], y[PER];
#pragma unroll
      for (int u = 0; u < PER; ++u) {
        const uint64_t a = (b << bb) + u * kSampleThreads + threadIdx.x;
        x[u] = re[a];
        y[u] = im[a];
      }
#pragma unroll
      for (int u = 0; u < PER; ++u) acc += prob_of(x[u], y[u]);
    } else {
      for (uint32_t i = threadIdx.x; i < B; i += kSampleThreads) {
        const uint64_t a = (b << bb) + i;
        acc += prob_of(re[a], im[a]);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) s_red[half][threadIdx.x >> 5] = acc;
    __syncthreads();  // (the other half's sums are read before the barrier of the next iteration)
    if (threadIdx.x == 0) {
      double s = 0.0;
      for (int w = 0; w < kSampleThreads / 32; ++w) s += s_red[half][w];
      bsum[b] = s;
    }
  }
}

// Scaled uniforms as sortable keys (non-negative doubles order like their bit patterns).
__global__ void k_uniforms(uint64_t shots, uint64_t seed, const double* __restrict__ bcdf,
                           const double* __restrict__ bsum, uint64_t nblocks, uint64_t* __restrict__ keys,
                           uint64_t* __restrict__ vals) {
  const double total = bcdf[nblocks - 1] + bsum[nblocks - 1];
  const uint64_t G = 0x9E3779B97F4A7C15ull;
  for (uint64_t k = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; k < shots; k += uint64_t(gridDim.x) * blockDim.x) {
    const double u = double(mix64s(seed + (k + 1) * G) >> 11) * 0x1.0p-53;
    keys[k] = __double_as_longlong(u * total);
    vals[k] = k;
  }
}

// First index of the sorted keys whose value is > x.
__device__ __forceinline__ uint64_t upper_bound_keys(const uint64_t* __restrict__ keys, uint64_t n, double x) {
  uint64_t lo = 0, hi = n;
  while (lo < hi) {
    const uint64_t mid = (lo + hi) >> 1;
    if (__longlong_as_double(keys[mid]) <= x) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// First sorted shot of each block: block b holds shots range[b] .. range[b + 1] - 1, the scaled uniforms
// in (bcdf[b], bcdf[b + 1]] (block 0 from 0 inclusive). One thread a block; searched by one thread of each
// block of k_assign, the two chains of dependent loads stood in front of every block's own work.
__global__ void k_ranges(const double* __restrict__ bcdf, uint64_t nblocks, const uint64_t* __restrict__ keys,
                         uint64_t shots, uint64_t* __restrict__ range) {
  for (uint64_t b = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; b <= nblocks; b += uint64_t(gridDim.x) * blockDim.x)
    range[b] = b == 0 ? 0 : b == nblocks ? shots : upper_bound_keys(keys, shots, bcdf[b]);
}

// Each block that holds shots scans its probabilities (FP64, inclusive) and places them. The amplitudes
// are read in rows of the block and turned into each thread's run of consecutive ones through shared
// memory (one pad word every 16, so that neither side meets bank conflicts); read as runs, a warp's load
// touched 32 lines. A call with k_ranges and the new loads, 27 qubits complex128: 3.24 -> 0.87 ms for
// 20,000 shots (70 % of the blocks hold one), 8.5 -> 2.2 ms for 10^6.
__host__ __device__ __forceinline__ uint32_t pad16(uint32_t i) { return i + (i >> 4); }

template <class R>
__global__ void __launch_bounds__(kSampleThreads) k_assign(const R* __restrict__ re, const R* __restrict__ im,
                                                           uint32_t bb, uint64_t nblocks,
                                                           const double* __restrict__ bcdf,
                                                           const uint64_t* __restrict__ range,
                                                           const uint64_t* __restrict__ keys,
                                                           const uint64_t* __restrict__ vals,
                                                           uint64_t* __restrict__ out) {
  extern __shared__ double s_pre[];  // 2^bb inclusive prefix sums, padded
  __shared__ double s_warp[kSampleThreads / 32];
  constexpr int PER = (1 << kBlockBits) / kSampleThreads;
  const uint32_t B = 1u << bb;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (uint64_t b = blockIdx.x; b < nblocks; b += gridDim.x) {
    const uint64_t j0 = range[b], j1 = range[b + 1];
    if (j1 == j0) continue;  // (the same for the whole block)
    if (bb == uint32_t(kBlockBits)) {
      R x[PER], y[PER];
#pragma unroll
      for (int u = 0; u < PER; ++u) {
        const uint64_t a = (b << bb) + u * kSampleThreads + tid;
        x[u] = re[a];
        y[u] = im[a];
      }
#pragma unroll
      for (int u = 0; u < PER; ++u) s_pre[pad16(u * kSampleThreads + tid)] = prob_of(x[u], y[u]);
    } else {
      for (uint32_t i = tid; i < B; i += kSampleThreads) s_pre[pad16(i)] = prob_of(re[(b << bb) + i], im[(b << bb) + i]);
    }
    __syncthreads();
    // this thread's run of consecutive amplitudes (B / threads of them, or one when B is small)
    const uint32_t per = B >= uint32_t(kSampleThreads) ? B / kSampleThreads : 1u;
    const uint32_t first = uint32_t(tid) * per;
    double run = 0.0;
    if (first < B)
      for (uint32_t e = 0; e < per; ++e) {
        run += s_pre[pad16(first + e)];
        s_pre[pad16(first + e)] = run;
      }
    // exclusive scan of the run totals across the block
    double incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      double w = lane < kSampleThreads / 32 ? s_warp[lane] : 0.0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += v;
      }
      if (lane < kSampleThreads / 32) s_warp[lane] = w;
    }
    __syncthreads();
    const double off = (incl - run) + (warp > 0 ? s_warp[warp - 1] : 0.0);
    if (first < B)
      for (uint32_t e = 0; e < per; ++e) s_pre[pad16(first + e)] += off;
    __syncthreads();
    const double base = bcdf[b];
    for (uint64_t j = j0 + tid; j < j1; j += kSampleThreads) {
      const double x = __longlong_as_double(keys[j]);
      // the first index whose cumulative probability base + prefix is >= x (the block's last
      // one if none: rounding can leave x just above the block's own total)
      uint32_t lo = 0, hi = B - 1;
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__dadd_rn(base, s_pre[pad16(mid)]) >= x) hi = mid;
        else lo = mid + 1;
      }
      // in that clamped case, step back over trailing zero probabilities
      if (__dadd_rn(base, s_pre[pad16(lo)]) < x)
        while (lo > 0 && s_pre[pad16(lo)] == s_pre[pad16(lo - 1)]) --lo;
      out[vals[j]] = (b << bb) + lo;
    }
    __syncthreads();
  }
}

template <class R>
void sample_impl(qsvb_ctx* c, const qsvb_state* st, uint64_t shots, uint64_t seed, uint64_t* out_host) {
  const uint32_t n = st->n_qubits;
  const uint32_t bb = std::min<uint32_t>(n, kBlockBits);
  const uint64_t nblocks = uint64_t(1) << (n - bb);
  const R* re = static_cast<const R*>(st->re);
  const R* im = static_cast<const R*>(st->im);
  cudaStream_t s = c->stream;
  size_t tb_scan = 0, tb_sort = 0;
  QSVB_CK(cub::DeviceScan::ExclusiveSum(nullptr, tb_scan, (double*)nullptr, (double*)nullptr, nblocks, s));
  QSVB_CK(cub::DeviceRadixSort::SortPairs(nullptr, tb_sort, (uint64_t*)nullptr, (uint64_t*)nullptr,
                                          (uint64_t*)nullptr, (uint64_t*)nullptr, shots, 0, 64, s));
  size_t need = 0;
  auto take = [&](size_t bytes) {
    const size_t at = need;
    need += (bytes + 255) & ~size_t(255);
    return at;
  };
  const size_t o_bsum = take(8 * nblocks), o_bcdf = take(8 * nblocks), o_range = take(8 * (nblocks + 1));
  const size_t o_keys = take(8 * shots), o_vals = take(8 * shots), o_keys2 = take(8 * shots), o_vals2 = take(8 * shots);
  const size_t o_out = take(8 * shots), o_temp = take(std::max(tb_scan, tb_sort));
  Scratch scratch(c, need);
  double* bsum = reinterpret_cast<double*>(scratch.p + o_bsum);
  double* bcdf = reinterpret_cast<double*>(scratch.p + o_bcdf);
  uint64_t* range = reinterpret_cast<uint64_t*>(scratch.p + o_range);
  uint64_t* keys = reinterpret_cast<uint64_t*>(scratch.p + o_keys);
  uint64_t* vals = reinterpret_cast<uint64_t*>(scratch.p + o_vals);
  uint64_t* keys2 = reinterpret_cast<uint64_t*>(scratch.p + o_keys2);
  uint64_t* vals2 = reinterpret_cast<uint64_t*>(scratch.p + o_vals2);
  uint64_t* out = reinterpret_cast<uint64_t*>(scratch.p + o_out);
  char* temp = scratch.p + o_temp;
  const int grid = int(std::min<uint64_t>(nblocks, uint64_t(c->num_sms) * 4));
  k_block_sums<R><<<grid, kSampleThreads, 0, s>>>(re, im, bb, nblocks, bsum);
  QSVB_CK(cudaGetLastError());
  QSVB_CK(cub::DeviceScan::ExclusiveSum(temp, tb_scan, bsum, bcdf, nblocks, s));
  const int small = int(std::min<uint64_t>((shots + 255) / 256, uint64_t(c->num_sms) * 8));
  k_uniforms<<<small, 256, 0, s>>>(shots, seed, bcdf, bsum, nblocks, keys, vals);
  QSVB_CK(cudaGetLastError());
  QSVB_CK(cub::DeviceRadixSort::SortPairs(temp, tb_sort, keys, keys2, vals, vals2, shots, 0, 64, s));
  const int edges = int(std::min<uint64_t>(nblocks / 256 + 1, uint64_t(c->num_sms) * 8));
  k_ranges<<<edges, 256, 0, s>>>(bcdf, nblocks, keys2, shots, range);
  QSVB_CK(cudaGetLastError());
  const size_t smem = sizeof(double) * (pad16((uint32_t(1) << bb) - 1) + 1);
  QSVB_CK(cudaFuncSetAttribute(k_assign<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  k_assign<R><<<grid, kSampleThreads, smem, s>>>(re, im, bb, nblocks, bcdf, range, keys2, vals2, out);
  QSVB_CK(cudaGetLastError());
  d2h_staged(c, out_host, out, shots * sizeof(uint64_t));
}

}  // namespace

void sample_shots(qsvb_ctx* c, const qsvb_state* st, uint64_t shots, uint64_t seed, uint64_t* out) {
  QSVB_REQUIRE(out != nullptr, "null output");
  QSVB_REQUIRE(shots >= 1 && shots <= (uint64_t(1) << 30), "shots must be 1..2^30");
  if (st->dtype == QSVB_C128) sample_impl<double>(c, st, shots, seed, out);
  else sample_impl<float>(c, st, shots, seed, out);
}

}  // namespace qsvb
