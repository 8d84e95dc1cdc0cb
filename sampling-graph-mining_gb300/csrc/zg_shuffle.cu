// zg_shuffle.cu — the seeded edge permutation of a graph build (the counterpart of the Fisher-Yates
// shuffle at src/Graph.cpp:218-231): edge i gets the 64-bit Philox key of (seed, shuffle stream, i),
// and the edges go in the order of (key, i).
//
// The keys are uniform, so the order is one scatter and one small sort per bucket instead of eight
// radix passes over 16-byte pairs: the key's top bits pick one of 2^k buckets of at most 2 048
// expected edges (the key is computed where it is scattered, never stored for its own sake), and
// one block per bucket orders its edges in shared memory, by the next 11 bits and then, among the
// one or two edges of a bin, by comparison.  The edges are fetched in that order straight into the
// output.  Bound by the scatter's atomics and partial sectors on graphs that fit L2, by the random
// reads of the fetch beyond.  The atomics of one 128-byte line run one after another (about 2 ns
// each), so the buckets' counters lie a line apart while that takes no more than 4 MB: 308 k edges
// in 256 buckets 71 us with the counters side by side, 10 us so spread.  1.5 M edges (R-MAT scale 20,
// ef 3, half kept): 430 us of radix passes and a 24 us gather before, 67 us now.
#include <cub/device/device_scan.cuh>

#include <math.h>

#include "zg_scratch.cuh"

namespace {

constexpr int kT = 512;
constexpr uint32_t kMean = 2048, kCap = 2560, kBins = 2048;  // 39 KB a block: five blocks a SM

__global__ void __launch_bounds__(256) k_shuffle_scatter(uint64_t m, uint64_t seed, uint32_t bits, uint32_t cap,
                                                         uint32_t spread,
                                                         uint32_t* __restrict__ cursor,
                                                         unsigned long long* __restrict__ keys,
                                                         uint32_t* __restrict__ ids, uint32_t* __restrict__ full) {
  const uint64_t stride = (uint64_t)gridDim.x * 256;
  for (uint64_t i0 = blockIdx.x * 256ull + threadIdx.x; i0 < m; i0 += 4 * stride) {
    unsigned long long key[4];
    uint32_t b[4], at[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint64_t i = i0 + j * stride;
      key[j] = zg_draw_word(seed, ZG_STREAM_SHUFFLE, i, 0);
      b[j] = bits ? (uint32_t)(key[j] >> (64 - bits)) : 0u;
      at[j] = i < m ? atomicAdd(&cursor[(uint64_t)b[j] << spread], 1u) : cap;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint64_t i = i0 + j * stride;
      if (at[j] < cap) {
        const uint64_t to = (uint64_t)b[j] * cap + at[j];
        keys[to] = key[j];
        ids[to] = (uint32_t)i;
      } else if (i < m) {
        *full = 1u;
      }
    }
  }
}

__global__ void k_shuffle_counts(uint64_t buckets, uint32_t spread, const uint32_t* __restrict__ cursor,
                                 uint32_t* __restrict__ counts) {
  const uint64_t b = blockIdx.x * 256ull + threadIdx.x;
  if (b < buckets) counts[b] = cursor[b << spread];
}

// Block b puts bucket b in order and fetches its edges.
__global__ void __launch_bounds__(kT) k_shuffle_bucket(uint32_t bits, uint32_t cap, const uint32_t* __restrict__ counts,
                                                       const uint32_t* __restrict__ base,
                                                       const unsigned long long* __restrict__ keys,
                                                       const uint32_t* __restrict__ ids, const uint2* __restrict__ coo,
                                                       const uint32_t* __restrict__ w,
                                                       const unsigned long long* __restrict__ parent,
                                                       uint2* __restrict__ coo_out, uint32_t* __restrict__ w_out,
                                                       unsigned long long* __restrict__ parent_out) {
  __shared__ unsigned long long s_key[kCap];
  __shared__ uint32_t s_id[kCap], s_bin[kBins + 1], s_warp[kT / 32];
  constexpr int kPer = kCap / kT, kOwn = kBins / kT;
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  const uint32_t n = min(counts[blockIdx.x], cap);
  const uint64_t from = (uint64_t)blockIdx.x * cap;
#pragma unroll
  for (int i = 0; i < kOwn; ++i) s_bin[tid + i * kT] = 0;
  __syncthreads();
  unsigned long long key[kPer];
  uint32_t id[kPer], nth[kPer];
  auto bin_of = [&](unsigned long long k) { return (uint32_t)((k << bits) >> 53); };
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const uint32_t t = i * kT + tid;
    if (t < n) {
      key[i] = keys[from + t];
      id[i] = ids[from + t];
      nth[i] = atomicAdd(&s_bin[bin_of(key[i])], 1u);
    }
  }
  __syncthreads();
  // exclusive scan of the bins, kOwn neighbouring ones per thread
  uint32_t own[kOwn], sum = 0;
#pragma unroll
  for (int i = 0; i < kOwn; ++i) {
    own[i] = sum;
    sum += s_bin[tid * kOwn + i];
  }
  uint32_t incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= (uint32_t)o) incl += v;
  }
  if (lane == 31) s_warp[tid / 32] = incl;
  __syncthreads();
  uint32_t before = incl - sum;
  for (uint32_t i = 0; i < tid / 32; ++i) before += s_warp[i];
#pragma unroll
  for (int i = 0; i < kOwn; ++i) s_bin[tid * kOwn + i] = before + own[i];
  if (tid == 0) s_bin[kBins] = n;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kPer; ++i)
    if ((uint32_t)i * kT + tid < n) {
      const uint32_t at = s_bin[bin_of(key[i])] + nth[i];
      s_key[at] = key[i];
      s_id[at] = id[i];
    }
  __syncthreads();
  const uint64_t to = base[blockIdx.x];
  for (uint32_t t = tid; t < n; t += kT) {
    const unsigned long long k = s_key[t];
    const uint32_t e = s_id[t], b = bin_of(k), lo = s_bin[b], hi = s_bin[b + 1];
    uint32_t r = lo;
    for (uint32_t x = lo; x < hi; ++x) r += s_key[x] < k || (s_key[x] == k && s_id[x] < e);
    coo_out[to + r] = coo[e];
    if (w) w_out[to + r] = w[e];
    parent_out[to + r] = parent ? parent[e] : e;
  }
}

}  // namespace

// (coo, w, parent)[perm] into the *_out arrays (m >= 1 entries each; w and parent may be null, a null
// parent counting the input positions).  m < 2^32.
int zg_shuffle_edges(const uint2* coo, const uint32_t* w, const unsigned long long* parent, uint64_t m, uint64_t seed,
                     cudaStream_t s, uint2* coo_out, uint32_t* w_out, unsigned long long* parent_out) {
  uint32_t bits = 0;
  while ((m >> bits) > kMean || ((m >> bits) == kMean && (m & ((1ull << bits) - 1)))) ++bits;
  // Buckets hold mean + 10 standard deviations; one that overflows all the same (a chance below
  // 1e-20) sends the call around again with twice the buckets.
  for (int attempt = 0; attempt < 4; ++attempt, ++bits) {
    const uint64_t buckets = 1ull << bits;
    const double mean = (double)m / (double)buckets;
    const uint32_t cap = (uint32_t)(mean + 10 * sqrt(mean) + 32);
    ZgCarve c;
    size_t tb = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tb, (uint32_t*)nullptr, (uint32_t*)nullptr, (int64_t)buckets, s);
    const uint32_t spread = bits <= 15 ? 5 : bits <= 20 ? 20 - bits : 0;
    const size_t o_cur = c.take((4 * buckets) << spread), o_full = c.take(4), o_cnt = c.take(4 * buckets),
                 o_base = c.take(4 * buckets), o_tmp = c.take(tb), o_key = c.take(8 * buckets * cap), o_id = c.take(4 * buckets * cap);
    ZgScratch x(s);
    if (int rc = x.alloc(c.at)) return rc;
    uint32_t *cursor = x.as<uint32_t>(o_cur), *full = x.as<uint32_t>(o_full), *counts = x.as<uint32_t>(o_cnt),
             *base = x.as<uint32_t>(o_base);
    cudaMemsetAsync(cursor, 0, o_cnt - o_cur, s);
    const uint64_t blocks = (m + 1023) / 1024, most = (uint64_t)zg_num_sms() * 16;
    k_shuffle_scatter<<<(int)(blocks < most ? blocks : most), 256, 0, s>>>(m, seed, bits, cap, spread, cursor,
                                                                          x.as<unsigned long long>(o_key),
                                                                          x.as<uint32_t>(o_id), full);
    k_shuffle_counts<<<(int)((buckets + 255) / 256), 256, 0, s>>>(buckets, spread, cursor, counts);
    cub::DeviceScan::ExclusiveSum(x.as<char>(o_tmp), tb, counts, base, (int64_t)buckets, s);
    k_shuffle_bucket<<<(int)buckets, kT, 0, s>>>(bits, cap, counts, base, x.as<unsigned long long>(o_key),
                                                 x.as<uint32_t>(o_id), coo, w, parent, coo_out, w_out, parent_out);
    uint32_t overflow = 0;
    cudaError_t e = cudaMemcpyAsync(&overflow, full, 4, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return zg_check_cuda(e, "edge shuffle");
    if (!overflow) return ZG_OK;
  }
  return zg_set_error(ZG_ERR_CUDA, "edge shuffle: a bucket overflowed"), ZG_ERR_CUDA;
}
