// zg_graph.cu — device graph store: the GB300 counterpart of Graph<E> + CSRConstructor
// (include/Graph.hpp:148-210, src/Graph.cpp:215-377), GraphFilter (src/GraphFilters.cpp:17-177)
// and GraphSampler (src/Graph.cpp:629-780).
//
// Build:
//   1. half-edges (v, nbr, eid) in edge-id order, sorted stably by v (CUB) -> adj_e: each list is
//      in edge-id order exactly as the reference's outgoing_adj_list.  The sort carries the end of
//      the edge in the edge id's top bit, so one pass over its result tells every edge both its
//      places (one 4-byte store each) and every vertex its degree;
//   2. adj_e read in order is sorted by neighbour, so a second stable sort by the other end gives
//      adj_n (ties keep edge-id order) on a 32-bit key;
//   3. one pass per edge writes its record in its final layout from the two places and the offsets;
//   4. the cuckoo table.
// The graph's arrays are one allocation, whose last-written part the sorts use before; other scratch comes
// from the library's pool.  R-MAT scale 20, ef 3 (3.1 M edges) from a host list, shuffled, with a first
// estimate: 4.6 ms with ten more allocations, a degree count in 64-bit atomics, wide records scattered per
// half-edge and then narrowed, and 7-pass sorts of 64-bit keys; 1.7 ms now, of which the device works 1.2,
// copies from and to the host included.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>

#include "zg_programs.cuh"
#include "zg_scratch.cuh"

int zg_shuffle_edges(const uint2* coo, const uint32_t* w, const unsigned long long* parent, uint64_t m, uint64_t seed,
                     cudaStream_t s, uint2* coo_out, uint32_t* w_out, unsigned long long* parent_out);

namespace {

template <typename T>
int dev_alloc(T** p, size_t count, cudaStream_t s) {
  const size_t bytes = sizeof(T) * (count ? count : 1);
  cudaError_t e = cudaMalloc((void**)p, bytes);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    zg_trim_pool(s);
    e = cudaMalloc((void**)p, bytes);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    zg_set_error(ZG_ERR_OOM, "cudaMalloc(%zu bytes) failed: %s", bytes, cudaGetErrorString(e));
    return ZG_ERR_OOM;
  }
  return ZG_OK;
}

int grid_for(uint64_t n, int block) {
  uint64_t g = (n + block - 1) / block;
  uint64_t cap = (uint64_t)zg_num_sms() * 32;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

int bits_for(uint64_t maxval) {
  int b = 1;
  while (b < 64 && (maxval >> b)) ++b;
  return b;
}

constexpr uint32_t kDstSide = 0x80000000u;  // in an edge id while building: this is the edge's dst end

struct BuildFlags {
  uint32_t bad, dup, max_degree;
  // of the table, in one copy
  struct Table {
    uint32_t fail, open_triangle, open_clique;
  } table;
};

// Validates the COO (src/Graph.cpp:454 asserts src != dst) and emits the half-edges.
__global__ void __launch_bounds__(256) k_half_edges(const uint2* __restrict__ coo, uint64_t m, uint32_t nv,
                                                    uint2* __restrict__ keys, ulonglong2* __restrict__ vals,
                                                    BuildFlags* __restrict__ flags) {
  for (uint64_t e = blockIdx.x * 256ull + threadIdx.x; e < m; e += (uint64_t)gridDim.x * 256) {
    uint2 c = coo[e];
    if (c.x >= nv || c.y >= nv || c.x == c.y) {
      flags->bad = 1u;
      c = make_uint2(0u, 0u);  // stays in range until the flag is read
    }
    keys[e] = c;
    vals[e] = make_ulonglong2((unsigned long long)c.y | (e << 32), (unsigned long long)c.x | ((e | kDstSide) << 32));
  }
}

// Position g of the sorted half-edges: the entry without its side, the edge's place, the vertex's
// degree (its last position less its first), and the (neighbour, (v, eid)) pair of the second sort.
__global__ void __launch_bounds__(256) k_place(const uint32_t* __restrict__ vkeys, uint2* __restrict__ adj_e, uint64_t n2,
                                               uint32_t* __restrict__ places, uint32_t* __restrict__ deg,
                                               uint32_t* __restrict__ nkeys, uint2* __restrict__ nvals) {
  for (uint64_t g = blockIdx.x * 256ull + threadIdx.x; g < n2; g += (uint64_t)gridDim.x * 256) {
    const uint32_t v = vkeys[g];
    uint2 a = adj_e[g];
    const uint32_t side = a.y >> 31;
    a.y &= ~kDstSide;
    adj_e[g] = a;
    places[2ull * a.y + side] = (uint32_t)g;
    if (g == 0 || vkeys[g - 1] != v) atomicSub(&deg[v], (uint32_t)g);
    if (g + 1 == n2 || vkeys[g + 1] != v) atomicAdd(&deg[v], (uint32_t)g + 1);
    if (nkeys) {
      nkeys[g] = a.x;
      nvals[g] = make_uint2(v, a.y);
    }
  }
}

// The 64-bit offsets and the largest degree (src/Graph.cpp:467-474).
__global__ void __launch_bounds__(256) k_offsets(const uint32_t* __restrict__ off32, uint64_t nv,
                                                 int64_t* __restrict__ off, BuildFlags* __restrict__ flags) {
  uint32_t most = 0;
  for (uint64_t v = blockIdx.x * 256ull + threadIdx.x; v <= nv; v += (uint64_t)gridDim.x * 256) {
    const uint32_t o = off32[v];
    off[v] = o;
    if (v < nv) most = max(most, off32[v + 1] - o);
  }
  __shared__ uint32_t s_most;  // one atomic a block: those on one address run one after another
  if (threadIdx.x == 0) s_most = 0;
  __syncthreads();
  atomicMax(&s_most, __reduce_max_sync(0xffffffffu, most));
  __syncthreads();
  if (threadIdx.x == 0 && s_most) atomicMax(&flags->max_degree, s_most);
}

// The same neighbour twice in a vertex's sorted list.
__global__ void __launch_bounds__(256) k_duplicates(const uint32_t* __restrict__ vkeys, const uint2* __restrict__ adj_n,
                                                    uint64_t n2, BuildFlags* __restrict__ flags) {
  for (uint64_t g = blockIdx.x * 256ull + threadIdx.x + 1; g < n2; g += (uint64_t)gridDim.x * 256)
    if (vkeys[g] == vkeys[g - 1] && adj_n[g].x == adj_n[g - 1].x) flags->dup = 1u;
}

// Every edge's record in the graph's layout, from its places and its ends' offsets.
__global__ void __launch_bounds__(256) k_records(const uint2* __restrict__ coo, uint64_t m, const uint2* __restrict__ places,
                                                 const uint32_t* __restrict__ off32, void* __restrict__ rec, uint32_t wide,
                                                 uint32_t packed, uint32_t vb, uint32_t sb, uint32_t pb) {
  for (uint64_t e = blockIdx.x * 256ull + threadIdx.x; e < m; e += (uint64_t)gridDim.x * 256) {
    const uint2 c = coo[e], p = places[e];
    const uint32_t ss = off32[c.x + 1] - 1 - p.x, sd = off32[c.y + 1] - 1 - p.y;  // entries after the edge
    if (wide) {
      ((ZgRec*)rec)[e].e = make_uint4(c.x, c.y, ss, sd);
      ((ZgRec*)rec)[e].p = make_uint4(p.x, p.y, p.x - off32[c.x], p.y - off32[c.y]);
    } else if (packed) {
      const uint64_t w0 = (uint64_t)c.x | ((uint64_t)c.y << vb) | ((uint64_t)ss << (2 * vb));
      const uint64_t w1 = (uint64_t)sd | ((uint64_t)p.x << sb) | ((uint64_t)p.y << (sb + pb));
      ((uint4*)rec)[e] = make_uint4((uint32_t)w0, (uint32_t)(w0 >> 32), (uint32_t)w1, (uint32_t)(w1 >> 32));
    } else {
      ((uint4*)rec)[e] = make_uint4(c.x, c.y, ss, sd);
    }
  }
}

// Bucketed two-choice cuckoo insertion of every edge's entry (fingerprint << 32 | edge id).  A
// thread claims an empty slot of either bucket with atomicCAS; when both are full it swaps its
// entry into slot 1..3 of one (atomicExch) and carries the evicted entry to that entry's other
// bucket (its key is rebuilt from the edge list).  Whenever an entry goes to its second bucket, its first
// bucket (full then, so slot 0 holds an entry) gets the overflow flag in slot 0, which is only
// ever written by that first claim and by these flags.  After kMaxKicks swaps it gives up and
// raises *fail: the host rebuilds with new hash seeds.  Every loop here is bounded.
constexpr int kMaxKicks = 128;

// A bucket is read in two 16-byte loads; a slot seen taken stays taken, and one seen empty is claimed
// with atomicCAS, so an old value costs a failed claim at most.
__device__ __forceinline__ bool cuckoo_try(unsigned long long* ent, uint32_t b, unsigned long long x) {
  unsigned long long* slot = &ent[4 * (uint64_t)b];
  const ulonglong2 lo = __ldcg((const ulonglong2*)slot), hi = __ldcg((const ulonglong2*)slot + 1);
  const unsigned long long seen[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (seen[j] == ZG_HASH_EMPTY && atomicCAS(&slot[j], ZG_HASH_EMPTY, x) == ZG_HASH_EMPTY) return true;
  return false;
}

__global__ void k_cuckoo_insert(const uint2* __restrict__ coo, uint64_t m, unsigned long long* ent, uint32_t bits,
                                uint64_t seed, unsigned long long* __restrict__ bloom, uint32_t bwords,
                                uint32_t* __restrict__ fail) {
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x) {
    const uint2 r = coo[e];
    unsigned long long k = zg_edge_key(r.x, r.y);
    unsigned long long x = ((unsigned long long)zg_fingerprint(k, seed) << 32) | e;
    const uint64_t h = zg_mix64(k ^ seed);
    atomicOr(&bloom[zg_bloom_word(h, bwords)], (unsigned long long)zg_bloom_bits(h));
    uint32_t from = 0xFFFFFFFFu;  // the bucket the carried entry was evicted from
    bool placed = false;
    for (int kick = 0; kick < kMaxKicks; ++kick) {
      const uint32_t b1 = zg_bucket1(k, seed, bits), b2 = zg_bucket2(k, seed, bits);
      if (cuckoo_try(ent, b1, x)) {
        placed = true;
        break;
      }
      if (b2 != b1 && cuckoo_try(ent, b2, x)) {
        atomicOr(&ent[4 * (uint64_t)b1], ZG_HASH_OVERFLOW);
        placed = true;
        break;
      }
      const uint32_t vb = from == b1 ? b2 : from == b2 ? b1 : (((e + kick) & 1) ? b2 : b1);
      if (vb != b1) atomicOr(&ent[4 * (uint64_t)b1], ZG_HASH_OVERFLOW);
      const unsigned long long old = atomicExch(&ent[4 * (uint64_t)vb + 1 + (e + (uint64_t)kick) % 3], x);
      if (old == ZG_HASH_EMPTY) {
        placed = true;
        break;
      }
      x = old;
      const uint2 ro = coo[(uint32_t)old];
      k = zg_edge_key(ro.x, ro.y);
      from = vb;
    }
    if (!placed) atomicOr(fail, 1u);
  }
}

// The first `checkers` blocks: every edge must be found in one of its two buckets (an insertion that gave up
// lost one), and one found only in its second bucket needs the overflow flag on its first.  The other blocks,
// half of them each: how many of kWedgeProbe first steps the filter leaves open, for triangles and for
// 4-cliques.
constexpr uint32_t kWedgeProbe = 4096;
__global__ void __launch_bounds__(256) k_cuckoo_check(ZgDevGraph g, const uint2* __restrict__ coo, uint32_t checkers,
                                                      BuildFlags::Table* __restrict__ t) {
  if (blockIdx.x >= checkers) {
    const uint32_t b = blockIdx.x - checkers;
    const bool clique = b & 1;
    Ctx c{0, (b >> 1) * 256u + threadIdx.x, 0, 0, nullptr, 0, 0, nullptr};
    Res r;
    res_init(r);
    const int n = __syncthreads_count(clique ? closing_pair_open<true>(g, c, r) : closing_pair_open<false>(g, c, r));
    if (threadIdx.x == 0) atomicAdd(clique ? &t->open_clique : &t->open_triangle, (uint32_t)n);
    return;
  }
  for (uint64_t e = blockIdx.x * 256ull + threadIdx.x; e < g.m; e += checkers * 256ull) {
    const uint2 r = coo[e];
    unsigned long long k = zg_edge_key(r.x, r.y);
    unsigned long long x = ((unsigned long long)zg_fingerprint(k, g.hseed) << 32) | e;
    const uint32_t b1 = zg_bucket1(k, g.hseed, g.hbits), b2 = zg_bucket2(k, g.hseed, g.hbits);
    bool in1 = false, in2 = false;
    for (int j = 0; j < 4; ++j) {
      in1 |= (g.hent[4 * (uint64_t)b1 + j] & ~ZG_HASH_OVERFLOW) == x;
      in2 |= (g.hent[4 * (uint64_t)b2 + j] & ~ZG_HASH_OVERFLOW) == x;
    }
    const unsigned long long s0 = g.hent[4 * (uint64_t)b1];
    const bool flagged = s0 != ZG_HASH_EMPTY && (s0 & ZG_HASH_OVERFLOW);
    if (!(in1 || (in2 && flagged))) atomicOr(&t->fail, 1u);
  }
}

// The L2's size (0 where it is not to be had) and a graph's sampling working set in the compact layout
// (records 16 B, edge-id adjacency 16 B, cuckoo table about 10 B per edge, offsets).
uint64_t l2_bytes() {
  int dev = 0, l2 = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev) == cudaSuccess)
    return (uint64_t)l2;
  cudaGetLastError();
  return 0;
}
uint64_t hot_bytes(uint64_t m, uint32_t nv) { return 42 * m + 4 * ((uint64_t)nv + 1); }

// The ways of a graph, from the open shares s3 (triangles) and s4 (4-cliques) of the probe.  The filter and
// the putting aside pay where most look-ups end at the filter; where most pairs are edges the one is a read
// more and the other runs the first step twice.  Ring lattices with a part of their edges rewired, ms per
// 2^23 samples (3-motif 2^22), packed records up to 9 M edges, wide at 36 M:
//   table alone / filter       s3 0.70        0.50         0.36         0.20         0.05
//   triangle    1.3 M       .166 / .188  .167 / .187  .168 / .184  .165 / .174  .156 / .155
//               3.0 M       .263 / .277  .259 / .258  .254 / .243  .248 / .222  .235 / .187
//               9.0 M       .542 / .563  .518 / .500  .501 / .441               .459 / .330
//                36 M       .711 / .730  .680 / .659  .648 / .594               .591 / .453
//   3-motif     1.3 M       .158 / .170  .160 / .170  .158 / .171  .158 / .157  .148 / .145
//               9.0 M       .318 / .343  .310 / .320  .306 / .304               .283 / .256
//   one by one / put aside (triangle without the filter at 1.3 M, with it beyond)
//   triangle    1.3 M       .166 / .218  .167 / .192  .168 / .169  .165 / .147  .156 / .127
//               3.0 M       .277 / .308  .258 / .269  .243 / .239  .222 / .203  .187 / .161
//               4.8 M       .390 / .428  .353 / .378  .318 / .344  .292 / .306  .233 / .231
//               9.0 M       .563 / .639  .500 / .570  .441 / .517               .330 / .352
//   4-clique                s4 0.75        0.59         0.47         0.33         0.22
//               1.3 M       .422 / .441  .407 / .383  .391 / .330  .359 / .268  .284 / .211
//               9.0 M       .973 / 1.03  .843 / .833  .722 / .683               .431 / .414
//   4-clique, uniform random      s4 - s3 0.52   0.46         0.38         0.32
//               0.2 to 0.6 M    .155 / .191  .162 / .185  .162 / .175  .154 / .179
// (R-MAT graphs lie at s3 0.02 to 0.16 and s4 0.05 to 0.22.)  So the filter is asked below 0.06 while the
// table takes 16 MB at most, both then being near the SMs, below 0.4 beyond, and below 0.6 on wide records;
// triangles are put aside below 0.3 while the working set is within 1.25 times the L2; 4-cliques below
// 0.65, unless 0.2 or more are open for a list's end alone (sparse graphs), which are soon decided.
uint32_t ways_for(const zg_graph* g, uint32_t bits, const BuildFlags::Table& t) {
  const double s3 = (double)t.open_triangle / kWedgeProbe, s4 = (double)t.open_clique / kWedgeProbe;
  const bool near_table = (sizeof(unsigned long long) * 4 << bits) <= (16u << 20);
  const bool near_graph = 4 * hot_bytes(g->d.m, g->d.nv) <= 5 * l2_bytes();
  return (s3 < (near_table ? 0.06 : g->wide ? 0.6 : 0.4) ? ZG_ASK_FILTER : 0u) |
         (s3 < 0.3 && near_graph ? ZG_DEFER_TRIANGLE : 0u) | (s4 < 0.65 && s4 - s3 < 0.2 ? ZG_DEFER_CLIQUE : 0u);
}

// log2 of the cuckoo table's buckets for a load of at most 0.8 (0.5, see below).
uint32_t hash_bits(uint64_t m, bool wide) {
  uint32_t bits = 1;
  // Load up to 0.8, or up to 0.5 for a graph far larger than L2 (wide records) whose table then
  // stays within 4 GiB: such a graph is read from HBM either way, and with more first buckets
  // holding an empty slot more absent edges are settled by one sector (edge_candidate).  Larger
  // tables keep the 0.8 load: doubling one of tens of GB cost more in address translation than
  // it saved (R-MAT scale 26: 709 -> 794 ms per batch; the 43 M-edge Chung-Lu batch: 74 -> 70 ms).
  while ((4ull << bits) * 4 < m * 5) ++bits;  // 4 * 2^bits slots >= m / 0.8
  uint32_t roomy = 1;
  while ((4ull << roomy) < m * 2) ++roomy;  // 4 * 2^roomy slots >= m / 0.5
  return wide && (8ull * (4ull << roomy)) <= (4ull << 30) ? roomy : bits;
}

// Words of the filter in front of the table (one at least): 16 bits per edge while that stays within
// a quarter of the L2, else 8.  A sample reads a word as often as a record or an entry, so a filter
// that fits L2 beside what is read once (draw_entry) costs no DRAM access; one that does not still
// meets L2 more often than the table, ten times its size.  Half the bits: 3 % of the absent edges go
// on to the table instead of 0.4 %.  Triangles / 4-cliques, ms per 2^24 (2^25 from 42 M edges on):
//   table alone                8 bits          16 bits
//   3.1 M edges  0.360 / 0.476  0.285 / 0.417  0.259 / 0.391   (R-MAT scale 20, ef 3)
//   8.8 M        0.909 / 0.967  0.593 / 0.660  0.584 / 0.652   (Chung-Lu, 1 M vertices)
//   42 M         2.05 / 2.15    1.38 / 1.51                    (Chung-Lu, 4.8 M vertices)
//   97 M         2.16 / 2.26    1.78 / 1.89                    (Chung-Lu, 11 M vertices)
//   779 M        2.37 / 2.45    2.19 / 2.27                    (R-MAT scale 25, ef 24)
// (12 bits at 42 M: 1.80 / 1.91 before the entries went first, where 8 took 1.73 / 1.85.)
constexpr uint64_t kBloomRoomy = 16ull << 20;
uint32_t bloom_words(uint64_t m) {
  return m == 0 ? 1 : (uint32_t)(m > kBloomRoomy ? (m + 7) / 8 : (m + 3) / 4);
}

// The cuckoo table in g->hent (2^bits buckets, allocated with the graph): up to 8 seeds, and the
// table doubled, in an allocation of its own, after 4 failed ones.  Releases `scratch`, the
// build's, before its first synchronisation.
int build_hash(zg_graph* g, const uint2* coo, uint32_t bits, BuildFlags* flags, ZgScratch& scratch, cudaStream_t s) {
  const uint64_t m = g->d.m;
  const int B = 256;
  for (int attempt = 0; attempt < 8; ++attempt) {
    if (attempt && attempt % 4 == 0) {
      ++bits;
      g->hent = nullptr;  // the graph's own allocation keeps the first table's place
      if (int rc = dev_alloc(&g->hent, 4ull << bits, s)) return rc;
    }
    const uint64_t slots = 4ull << bits;
    uint64_t seed = zg_mix64(0x5A4748415348ull + attempt);
    cudaError_t ce;
    if ((ce = cudaMemsetAsync(g->hent, 0xFF, sizeof(unsigned long long) * slots, s)) ||
        (ce = cudaMemsetAsync(&flags->table, 0, sizeof(flags->table), s)) ||
        (ce = cudaMemsetAsync(g->bloom, 0, sizeof(unsigned long long) * g->d.bwords, s)))
      return zg_check_cuda(ce, "hash memset");
    g->d.hent = g->hent;
    g->d.hbits = bits;
    g->d.hseed = seed;
    if (m) {
      k_cuckoo_insert<<<grid_for(m, B), B, 0, s>>>(coo, m, g->hent, bits, seed, g->bloom, g->d.bwords,
                                                   &flags->table.fail);
      k_cuckoo_check<<<grid_for(m, B) + 2 * kWedgeProbe / 256, B, 0, s>>>(g->d, coo, grid_for(m, B), &flags->table);
    }
    BuildFlags::Table t = {};
    ce = cudaMemcpyAsync(&t, &flags->table, sizeof(t), cudaMemcpyDeviceToHost, s);
    scratch.reset();
    if (ce || (ce = cudaStreamSynchronize(s))) return zg_check_cuda(ce, "hash build");
    if (!t.fail) {
      g->d.ways = ways_for(g, bits, t);
      g->bytes += slots * sizeof(unsigned long long);
      return ZG_OK;
    }
  }
  zg_set_error(ZG_ERR_CUDA, "cuckoo table of %llu edges did not build", (unsigned long long)m);
  return ZG_ERR_CUDA;
}

// Record layout of the graphs built from now on (zg_set_record_layout).
int g_record_layout = ZG_RECORDS_AUTO;

// Wide records when the compact layout's sampling working set is more than four times the L2: there nearly
// every first read misses L2 whatever its size, and the wide record saves a dependent read and two
// sectors per step.  Below, half the record bytes win.  Triangle / 4-clique / 3-chain / 4-chain, ms per
// 2^24 samples, wide and then compact or packed records (129 MB of L2):
//    6.1 M edges (2.0 x L2)  0.571 / 0.639 / 0.222 / 0.805   0.375 / 0.518 / 0.119 / 0.620
//    8.7 M       (2.9 x)     0.587 / 0.652 / 0.244 / 0.858   0.489 / 0.584 / 0.145 / 0.721
//   11.9 M       (3.9 x)     0.649 / 0.733 / 0.263 / 0.956   0.577 / 0.700 / 0.172 / 0.814
//   17.6 M       (5.8 x)     0.640 / 0.699 / 0.283 / 0.979   0.627 / 0.713 / 0.220 / 0.923
//   42.3 M       (13.9 x)    0.706 / 0.786 / 0.317 / 1.144   0.868 / 0.950 / 0.327 / 1.430
// The batch kernel, triangles and 3-motifs on the graph and four of its filters, ms wide / compact:
// 1.54 / 1.52 from 8.7 M edges, 1.73 / 1.86 from 17.6 M.  (The line lay at twice the L2 while each
// closure check read the table.)
bool wide_records(uint64_t m, uint32_t nv) {
  if (g_record_layout == ZG_RECORDS_WIDE) return true;
  if (g_record_layout == ZG_RECORDS_COMPACT || g_record_layout == ZG_RECORDS_PACKED) return false;
  const uint64_t l2 = l2_bytes();
  return l2 && hot_bytes(m, nv) > 4 * l2;
}

int check_size(uint64_t m, uint32_t nv) {
  // edge ids and adjacency positions (< 2m) are 32-bit
  if (m > 0x7FFFFFFFull)
    return zg_set_error(ZG_ERR_TOO_LARGE, "at most 2^31-1 edges (32-bit positions): m=%llu", (unsigned long long)m),
           ZG_ERR_TOO_LARGE;
  if (nv == 0 && m > 0) return zg_set_error(ZG_ERR_INVALID_GRAPH, "edges on a graph with 0 vertices"), ZG_ERR_INVALID_GRAPH;
  return ZG_OK;
}

// Builds a graph from a device COO (consumed: freed by the caller afterwards).
// sampling_only: skip the neighbour-ordered adjacency (exports only) and its duplicate check; for
// graphs derived from an already validated graph (filters, subsamples) that only sampling reads.
int build_graph(const uint2* d_coo, const uint32_t* d_w_in, uint64_t m, uint32_t nv,
                cudaStream_t s, zg_graph** out, bool sampling_only = false) {
  if (int rc = check_size(m, nv)) return rc;
  zg_graph* g = new zg_graph();
  memset(g, 0, sizeof(*g));
  int rc;
  auto fail = [&](int code) {
    zg_graph_free(g);
    return code;
  };
  const uint64_t n2 = 2 * m;
  const size_t nv1 = (size_t)nv + 1;
  g->wide = wide_records(m, nv);
  // packed records where the degrees allow it (else compact ones)
  const bool try_packed =
      !g->wide && m && (g_record_layout == ZG_RECORDS_AUTO || g_record_layout == ZG_RECORDS_PACKED);
  const size_t rec_bytes = (g->wide ? sizeof(ZgRec) : sizeof(uint4)) * m;
  const uint32_t hbits = hash_bits(m, g->wide);
  // one allocation: adj_e, 8 entries of slack (lb_eid_win's windows may read up to 7 entries past
  // the last one), off32, the records, the cuckoo table, and what only exports and filters read
  ZgCarve c;
  const size_t adj_bytes = sizeof(uint2) * (n2 + 8);
  const size_t o_adj = c.take(adj_bytes + sizeof(uint32_t) * nv1), o_rec = c.take(rec_bytes),
               o_hent = c.take(sizeof(unsigned long long) * (4ull << hbits)),
               o_bloom = c.take(sizeof(unsigned long long) * bloom_words(m)), o_off = c.take(sizeof(int64_t) * nv1),
               o_adjn = c.take(sampling_only ? 0 : sizeof(uint2) * n2), o_w = c.take(d_w_in ? sizeof(uint32_t) * m : 0);
  g->hot_bytes = c.at;
  if ((rc = dev_alloc((char**)&g->hot, g->hot_bytes, s))) return fail(rc);
  char* base = (char*)g->hot;
  g->adj_e = (uint2*)(base + o_adj);
  g->off32 = (uint32_t*)(base + o_adj + adj_bytes);
  g->rec = base + o_rec;
  g->hent = (unsigned long long*)(base + o_hent);
  g->d.bwords = bloom_words(m);
  g->bloom = (unsigned long long*)(base + o_bloom);
  g->d.bloom = g->bloom;
  g->off = (int64_t*)(base + o_off);
  if (!sampling_only) g->adj_n = (uint2*)(base + o_adjn);
  if (d_w_in) g->w = (uint32_t*)(base + o_w);
  g->bytes = rec_bytes + (sizeof(int64_t) + sizeof(uint32_t)) * nv1 + (sampling_only ? 1 : 2) * sizeof(uint2) * n2 +
             (d_w_in ? sizeof(uint32_t) * m : 0) + sizeof(unsigned long long) * g->d.bwords;
  // Scratch: half-edges before and after a sort, the places, the degrees.  The records, the table and
  // the filter are written last, so their part of the graph takes what fits of the sorts' arrays.  Least
  // free memory at which 34.6 M edges build, bytes an edge, full / as a batch's filter that keeps all: 154 /
  // 146 with allocations of their own, 162 / 164 with one for the graph and all scratch beside it, 106 /
  // 108 so.
  ZgCarve x, late;
  const size_t late_room = o_off - o_rec;
  struct Spot {
    bool in_graph;
    size_t at;
  };
  auto sort_array = [&](size_t bytes) {
    const bool fits = late.at + bytes <= late_room;
    return Spot{fits, (fits ? late : x).take(bytes)};
  };
  const int vb = bits_for(nv > 0 ? nv - 1 : 0);
  size_t tb = 0, tb_scan = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, tb, (uint32_t*)nullptr, (uint32_t*)nullptr, (unsigned long long*)nullptr,
                                  (unsigned long long*)nullptr, (int64_t)n2, 0, vb, s);
  cub::DeviceScan::ExclusiveSum(nullptr, tb_scan, (uint32_t*)nullptr, (uint32_t*)nullptr, (int64_t)nv1, s);
  const size_t o_deg = x.take(sizeof(uint32_t) * nv1), o_places = x.take(sizeof(uint32_t) * n2);
  const Spot o_tmp = sort_array(std::max(tb, tb_scan)), o_vals = sort_array(sizeof(unsigned long long) * n2),
             o_keys = sort_array(sizeof(uint32_t) * n2), o_keys2 = sort_array(sizeof(uint32_t) * n2);
  ZgScratch scratch(s), small(s);
  if ((rc = scratch.alloc(x.at)) || (rc = small.alloc(sizeof(BuildFlags)))) return fail(rc);
  auto at = [&](Spot o) { return o.in_graph ? base + o_rec + o.at : scratch.as<char>(o.at); };
  BuildFlags* flags = small.as<BuildFlags>();
  uint32_t *deg = scratch.as<uint32_t>(o_deg), *places = scratch.as<uint32_t>(o_places),
           *keys = (uint32_t*)at(o_keys), *keys2 = (uint32_t*)at(o_keys2);
  unsigned long long* vals = (unsigned long long*)at(o_vals);
  void* tmp = at(o_tmp);
  cudaError_t ce;
  if ((ce = cudaMemsetAsync(deg, 0, sizeof(uint32_t) * nv1, s)) ||
      (ce = cudaMemsetAsync(flags, 0, sizeof(BuildFlags), s)))
    return fail(zg_check_cuda(ce, "memset"));
  if (g->w && m && (ce = cudaMemcpyAsync(g->w, d_w_in, sizeof(uint32_t) * m, cudaMemcpyDeviceToDevice, s)))
    return fail(zg_check_cuda(ce, "copy weights"));
  const int B = 256;
  if (m) {
    k_half_edges<<<grid_for(m, B), B, 0, s>>>(d_coo, m, nv, (uint2*)keys, (ulonglong2*)vals, flags);
    cub::DeviceRadixSort::SortPairs(tmp, tb, keys, keys2, vals, (unsigned long long*)g->adj_e, (int64_t)n2, 0, vb, s);
    k_place<<<grid_for(n2, B), B, 0, s>>>(keys2, g->adj_e, n2, places, deg, sampling_only ? nullptr : keys,
                                          (uint2*)vals);
  }
  cub::DeviceScan::ExclusiveSum(tmp, tb_scan, deg, g->off32, (int64_t)nv1, s);
  k_offsets<<<std::min(grid_for(nv1, B), zg_num_sms() * 4), B, 0, s>>>(g->off32, nv, g->off, flags);
  if (m && !sampling_only) {
    cub::DeviceRadixSort::SortPairs(tmp, tb, keys, keys2, vals, (unsigned long long*)g->adj_n, (int64_t)n2, 0, vb, s);
    k_duplicates<<<grid_for(n2, B), B, 0, s>>>(keys2, g->adj_n, n2, flags);
  }
  BuildFlags h;
  if ((ce = cudaMemcpyAsync(&h, flags, sizeof(h), cudaMemcpyDeviceToHost, s)) || (ce = cudaStreamSynchronize(s)))
    return fail(zg_check_cuda(ce, "graph build"));
  if (h.bad) {
    zg_set_error(ZG_ERR_INVALID_GRAPH, "edge list holds a self-loop or a vertex id >= %u", nv);
    return fail(ZG_ERR_INVALID_GRAPH);
  }
  if (h.dup) {
    zg_set_error(ZG_ERR_INVALID_GRAPH, "edge list holds a duplicate edge");
    return fail(ZG_ERR_INVALID_GRAPH);
  }
  g->max_degree = h.max_degree;
  if (try_packed) {
    const uint32_t vbits = (uint32_t)vb, sb = (uint32_t)bits_for(g->max_degree), pb = (uint32_t)bits_for(n2 - 1);
    g->packed = 2 * vbits + sb <= 64 && sb + 2 * pb <= 64;
    g->d.pk_v = vbits;
    g->d.pk_s = sb;
    g->d.pk_p = pb;
  }
  if (m)
    k_records<<<grid_for(m, B), B, 0, s>>>(d_coo, m, (const uint2*)places, g->off32, g->rec, g->wide, g->packed,
                                           g->d.pk_v, g->d.pk_s, g->d.pk_p);
  g->d.nv = nv;
  g->d.m = m;
  g->d.wide = g->wide;
  g->d.packed = g->packed;
  g->d.off32 = g->off32;
  g->d.rec = g->rec;
  g->d.off = g->off;
  g->d.adj_e = g->adj_e;
  g->d.adj_n = g->adj_n;
  g->d.w = g->w;
  if ((rc = build_hash(g, d_coo, hbits, flags, scratch, s))) return fail(rc);
  ce = cudaGetLastError();
  if (ce != cudaSuccess) return fail(zg_check_cuda(ce, "graph build kernels"));
  g->num_edges = m;
  *out = g;
  return ZG_OK;
}

// An edge list with its data and parent indices, in scratch.
struct EdgeList {
  ZgScratch coo, w, parent;
  explicit EdgeList(cudaStream_t s) : coo(s), w(s), parent(s) {}
  int alloc(uint64_t m, bool weights, bool parents) {
    int rc = coo.alloc(sizeof(uint2) * m);
    if (rc == ZG_OK && weights) rc = w.alloc(sizeof(uint32_t) * m);
    if (rc == ZG_OK && parents) rc = parent.alloc(sizeof(unsigned long long) * m);
    return rc;
  }
  void reset() {
    coo.reset();
    w.reset();
    parent.reset();
  }
};

// `to` gets `from` in the seeded order.
int permute(const EdgeList& from, EdgeList& to, uint64_t m, uint64_t seed, cudaStream_t s) {
  if (int rc = to.alloc(m, from.w.p != nullptr, true)) return rc;
  if (m == 0) return ZG_OK;
  return zg_shuffle_edges(from.coo.as<uint2>(), from.w.as<uint32_t>(), from.parent.as<unsigned long long>(), m, seed, s,
                          to.coo.as<uint2>(), to.w.as<uint32_t>(), to.parent.as<unsigned long long>());
}

// What a call leaves in the pool beyond its bound goes back to the device here.
int settle(int rc, cudaStream_t s) {
  const cudaError_t e = cudaStreamSynchronize(s);
  return rc || e == cudaSuccess ? rc : zg_check_cuda(e, "graph build");
}

// Predicate flags for GraphFilter / keep draws for GraphSampler.
__global__ void k_select(uint64_t m, const uint32_t* __restrict__ w, int op, int64_t t0, int64_t t1,
                         double rate, uint64_t keep_seed, int mode, uint32_t* __restrict__ flag) {
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e <= m;
       e += (uint64_t)gridDim.x * blockDim.x) {
    bool keep;
    if (e == m) {  // the scan's last position is the total
      keep = false;
    } else if (mode == 0) {
      int64_t x = (int64_t)w[e];
      switch (op) {
        case ZG_PRED_GE: keep = x >= t0; break;
        case ZG_PRED_LT: keep = x < t0; break;
        case ZG_PRED_GT: keep = x > t0; break;
        case ZG_PRED_LE: keep = x <= t0; break;
        case ZG_PRED_EQ: keep = x == t0; break;
        case ZG_PRED_NE: keep = x != t0; break;
        default: keep = x >= t0 && x < t1; break;
      }
    } else {
      // src/Graph.cpp:652-664: rand_int(1, 2^30) <= (unsigned long long)(rate * 2^30)
      const unsigned long long max_rand_int = 1ull << 30;
      unsigned long long threshold = (unsigned long long)(rate * (double)max_rand_int);
      keep = zg_draw(keep_seed, ZG_STREAM_SUBSAMPLE, e, 0, 1, max_rand_int) <= threshold;
    }
    flag[e] = keep ? 1u : 0u;
  }
}

__global__ void k_compact(uint64_t m, const uint32_t* __restrict__ pos, const ZgDevGraph src,
                          const uint32_t* __restrict__ w, uint2* __restrict__ coo_out,
                          uint32_t* __restrict__ w_out, unsigned long long* __restrict__ parent) {
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < m;
       e += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t p = pos[e];
    if (pos[e + 1] == p) continue;  // dropped
    uint4 r = zg_rec_e(src, e);
    coo_out[p] = make_uint2(r.x, r.y);
    if (w) w_out[p] = w[e];
    parent[p] = e;
  }
}

// GraphFilter::generate_graph / GraphSampler::sample_graph on the device.
int derive(bool sampling_only, const zg_graph* g, int mode, int op, int64_t t0, int64_t t1, double rate,
           uint64_t keep_seed,
           uint64_t shuffle_seed, cudaStream_t s, uint64_t* parent_index, uint64_t* out_m, zg_graph** out) {
  if (!g || !out) return zg_set_error(ZG_ERR_INVALID_ARG, "null argument"), ZG_ERR_INVALID_ARG;
  if (mode == 0 && !g->w) return zg_set_error(ZG_ERR_INVALID_ARG, "graph has no edge weights"), ZG_ERR_INVALID_ARG;
  if (mode == 0 && (op < ZG_PRED_GE || op > ZG_PRED_RANGE))
    return zg_set_error(ZG_ERR_INVALID_ARG, "unknown predicate op %d", op), ZG_ERR_INVALID_ARG;
  const uint64_t m = g->d.m;
  const int B = 256;
  int rc;
  cudaError_t ce = cudaSuccess;
  uint32_t kept = 0;
  EdgeList list(s), shuffled(s);
  {
    ZgCarve c;
    size_t tb = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tb, (uint32_t*)nullptr, (uint32_t*)nullptr, (int64_t)m + 1, s);
    const size_t o_flag = c.take(4 * (m + 1)), o_pos = c.take(4 * (m + 1)), o_tmp = c.take(tb);
    ZgScratch x(s);
    if ((rc = x.alloc(c.at))) return rc;
    uint32_t *flag = x.as<uint32_t>(o_flag), *pos = x.as<uint32_t>(o_pos);
    k_select<<<grid_for(m + 1, B), B, 0, s>>>(m, g->w, op, t0, t1, rate, keep_seed, mode, flag);
    cub::DeviceScan::ExclusiveSum(x.as<char>(o_tmp), tb, flag, pos, (int64_t)m + 1, s);
    if ((ce = cudaMemcpyAsync(&kept, pos + m, 4, cudaMemcpyDeviceToHost, s)) || (ce = cudaStreamSynchronize(s)))
      return zg_check_cuda(ce, "filter count");
    if ((rc = list.alloc(kept, g->w != nullptr, true))) return rc;
    if (m)
      k_compact<<<grid_for(m, B), B, 0, s>>>(m, pos, g->d, g->w, list.coo.as<uint2>(), list.w.as<uint32_t>(),
                                             list.parent.as<unsigned long long>());
  }
  EdgeList* edges = &list;
  if (shuffle_seed != ZG_NO_SHUFFLE) {
    if ((rc = permute(list, shuffled, kept, shuffle_seed, s))) return settle(rc, s);
    edges = &shuffled;
    list.reset();
  }
  rc = build_graph(edges->coo.as<uint2>(), edges->w.as<uint32_t>(), kept, g->d.nv, s, out, sampling_only);
  if (rc == ZG_OK) {
    // src/GraphFilters.cpp:90-135 (identical in src/Graph.cpp:704-749)
    double sample_rate_after_partition =
        g->num_edges ? (double)g->d.m / (double)g->num_edges : 1.0;
    (*out)->num_edges = (uint64_t)(1. * (double)kept / sample_rate_after_partition);
    (*out)->max_degree = (uint64_t)((double)(*out)->max_degree / sample_rate_after_partition);
    if (parent_index && kept)
      ce = cudaMemcpyAsync(parent_index, edges->parent.p, 8ull * kept, cudaMemcpyDeviceToHost, s);
    if (ce != cudaSuccess) rc = zg_check_cuda(ce, "parent index");
  }
  if (out_m) *out_m = kept;
  edges->reset();
  return settle(rc, s);
}

int upload_coo(const uint32_t* edges, const uint32_t* weights, uint64_t m, EdgeList& list, cudaStream_t s) {
  if (int rc = list.alloc(m, weights != nullptr, false)) return rc;
  cudaError_t ce = cudaSuccess;
  if (m) ce = cudaMemcpyAsync(list.coo.p, edges, sizeof(uint2) * m, cudaMemcpyHostToDevice, s);
  if (ce == cudaSuccess && weights && m)
    ce = cudaMemcpyAsync(list.w.p, weights, sizeof(uint32_t) * m, cudaMemcpyHostToDevice, s);
  return zg_check_cuda(ce, "upload edges");
}

}  // namespace

// zg_graph_filter / zg_graph_subsample without the neighbour-ordered adjacency: derived graphs that
// only the sampling kernels read (the batch cache, the error profile's subsample).
int zg_graph_filter_sampling(const zg_graph* g, int pred_op, int64_t t0, int64_t t1, uint64_t shuffle_seed,
                             cudaStream_t s, uint64_t* out_m, zg_graph** out) {
  return derive(true, g, 0, pred_op, t0, t1, 0.0, 0, shuffle_seed, s, nullptr, out_m, out);
}
int zg_graph_subsample_sampling(const zg_graph* g, double rate, uint64_t keep_seed, uint64_t shuffle_seed,
                                cudaStream_t s, uint64_t* out_m, zg_graph** out) {
  return derive(true, g, 1, 0, 0, 0, rate, keep_seed, shuffle_seed, s, nullptr, out_m, out);
}

// A graph from a device COO in edge-id order (the device generators' entry into the build).
int zg_build_graph_device(const uint2* d_coo, const uint32_t* d_w, uint64_t m, uint32_t nv, cudaStream_t s,
                          zg_graph** out, bool sampling_only) {
  return build_graph(d_coo, d_w, m, nv, s, out, sampling_only);
}

extern "C" int zg_graph_create(const uint32_t* edges, uint64_t m, uint32_t num_vertices,
                               const uint32_t* weights, void* cuda_stream, zg_graph** out) {
  if (!out || (m && !edges)) return zg_set_error(ZG_ERR_INVALID_ARG, "null argument"), ZG_ERR_INVALID_ARG;
  cudaStream_t s = (cudaStream_t)cuda_stream;
  EdgeList list(s);
  int rc = check_size(m, num_vertices);
  if (rc == ZG_OK) rc = upload_coo(edges, weights, m, list, s);
  if (rc == ZG_OK) rc = build_graph(list.coo.as<uint2>(), list.w.as<uint32_t>(), m, num_vertices, s, out);
  list.reset();
  return settle(rc, s);
}

extern "C" int zg_graph_permuted(const uint32_t* edges, uint64_t m, uint32_t num_vertices,
                                 const uint32_t* weights, uint64_t shuffle_seed, void* cuda_stream,
                                 uint64_t* parent_index, zg_graph** out) {
  if (!out || (m && !edges)) return zg_set_error(ZG_ERR_INVALID_ARG, "null argument"), ZG_ERR_INVALID_ARG;
  cudaStream_t s = (cudaStream_t)cuda_stream;
  EdgeList list(s), shuffled(s);
  int rc = check_size(m, num_vertices);
  if (rc == ZG_OK) rc = upload_coo(edges, weights, m, list, s);
  if (rc == ZG_OK) rc = permute(list, shuffled, m, shuffle_seed, s);
  list.reset();
  if (rc == ZG_OK) rc = build_graph(shuffled.coo.as<uint2>(), shuffled.w.as<uint32_t>(), m, num_vertices, s, out);
  if (rc == ZG_OK && parent_index && m)
    rc = zg_check_cuda(cudaMemcpyAsync(parent_index, shuffled.parent.p, 8 * m, cudaMemcpyDeviceToHost, s), "parent index");
  shuffled.reset();
  return settle(rc, s);
}

extern "C" int zg_set_record_layout(int layout) {
  if (layout < ZG_RECORDS_AUTO || layout > ZG_RECORDS_PACKED)
    return zg_set_error(ZG_ERR_INVALID_ARG, "unknown record layout %d", layout), ZG_ERR_INVALID_ARG;
  g_record_layout = layout;
  return ZG_OK;
}

extern "C" int zg_graph_free(zg_graph* g) {
  if (!g) return ZG_OK;
  const char *h = (const char*)g->hent, *hot = (const char*)g->hot;
  if (h && (h < hot || h >= hot + g->hot_bytes)) cudaFree(g->hent);  // a table that was doubled
  if (g->hot) cudaFree(g->hot);
  delete g;
  return ZG_OK;
}

extern "C" int zg_graph_get_meta(const zg_graph* g, zg_graph_meta* out) {
  if (!g || !out) return zg_set_error(ZG_ERR_INVALID_ARG, "null argument"), ZG_ERR_INVALID_ARG;
  out->num_vertices = g->d.nv;
  out->weighted = g->w != nullptr;
  out->num_local_edges = g->d.m;
  out->num_edges = g->num_edges;
  out->max_degree = g->max_degree;
  out->device_bytes = g->bytes;
  out->record_bytes = g->wide ? (uint32_t)sizeof(ZgRec) : (uint32_t)sizeof(uint4);
  out->record_layout = g->wide ? ZG_RECORDS_WIDE : g->packed ? ZG_RECORDS_PACKED : ZG_RECORDS_COMPACT;
  return ZG_OK;
}

extern "C" int zg_graph_set_meta(zg_graph* g, uint64_t num_edges, uint64_t max_degree) {
  if (!g) return zg_set_error(ZG_ERR_INVALID_ARG, "null graph"), ZG_ERR_INVALID_ARG;
  g->num_edges = num_edges;
  g->max_degree = max_degree;
  return ZG_OK;
}

namespace {
// Edge e0 + i's (src, dst) and suffix sizes out of its record, in any layout.
__global__ void k_export_rec(ZgDevGraph g, uint64_t e0, uint64_t cnt, uint32_t* __restrict__ edges,
                             uint32_t* __restrict__ suffix) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < cnt; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint4 q = zg_rec_e(g, e0 + i);
    if (edges) reinterpret_cast<uint2*>(edges)[i] = make_uint2(q.x, q.y);
    if (suffix) reinterpret_cast<uint2*>(suffix)[i] = make_uint2(q.z, q.w);
  }
}
}  // namespace

extern "C" int zg_graph_download(const zg_graph* g, uint32_t* edges, uint32_t* weights, int64_t* offsets,
                                 uint32_t* adj_e, uint32_t* adj_n, uint32_t* suffix) {
  if (!g) return zg_set_error(ZG_ERR_INVALID_ARG, "null graph"), ZG_ERR_INVALID_ARG;
  uint64_t m = g->d.m;
  cudaError_t ce = cudaSuccess;
  if ((edges || suffix) && m) {
    // unpacked on the device in chunks of at most 2^27 edges (1 GiB per array), then copied out
    const uint64_t chunk = m < (1ull << 27) ? m : (1ull << 27);
    uint32_t *d_e = nullptr, *d_s = nullptr;
    if (edges) ce = cudaMalloc((void**)&d_e, 8 * chunk);
    if (ce == cudaSuccess && suffix) ce = cudaMalloc((void**)&d_s, 8 * chunk);
    for (uint64_t e0 = 0; ce == cudaSuccess && e0 < m; e0 += chunk) {
      const uint64_t cnt = m - e0 < chunk ? m - e0 : chunk;
      const int grid = (int)std::min<uint64_t>((cnt + 255) / 256, (uint64_t)zg_num_sms() * 16);
      k_export_rec<<<grid, 256>>>(g->d, e0, cnt, d_e, d_s);
      ce = cudaGetLastError();
      if (ce == cudaSuccess && edges) ce = cudaMemcpy(edges + 2 * e0, d_e, 8 * cnt, cudaMemcpyDeviceToHost);
      if (ce == cudaSuccess && suffix) ce = cudaMemcpy(suffix + 2 * e0, d_s, 8 * cnt, cudaMemcpyDeviceToHost);
    }
    if (d_e) cudaFree(d_e);
    if (d_s) cudaFree(d_s);
    if (ce != cudaSuccess) return zg_check_cuda(ce, "download records");
  }
  if (weights && g->w && m) ce = cudaMemcpy(weights, g->w, 4 * m, cudaMemcpyDeviceToHost);
  if (ce == cudaSuccess && offsets)
    ce = cudaMemcpy(offsets, g->off, 8 * ((size_t)g->d.nv + 1), cudaMemcpyDeviceToHost);
  if (ce == cudaSuccess && adj_e && m) ce = cudaMemcpy(adj_e, g->adj_e, 16 * m, cudaMemcpyDeviceToHost);
  if (adj_n && m && !g->adj_n)
    return zg_set_error(ZG_ERR_INVALID_ARG, "this derived graph has no neighbour-ordered adjacency"),
           ZG_ERR_INVALID_ARG;
  if (ce == cudaSuccess && adj_n && m) ce = cudaMemcpy(adj_n, g->adj_n, 16 * m, cudaMemcpyDeviceToHost);
  if (ce != cudaSuccess) return zg_check_cuda(ce, "download");
  return ZG_OK;
}

extern "C" int zg_graph_filter(const zg_graph* g, int pred_op, int64_t t0, int64_t t1, uint64_t shuffle_seed,
                               void* cuda_stream, uint64_t* parent_index, uint64_t* out_m, zg_graph** out) {
  return derive(false, g, 0, pred_op, t0, t1, 0.0, 0, shuffle_seed, (cudaStream_t)cuda_stream, parent_index, out_m,
                out);
}

extern "C" int zg_graph_subsample(const zg_graph* g, double rate, uint64_t keep_seed, uint64_t shuffle_seed,
                                  void* cuda_stream, uint64_t* parent_index, uint64_t* out_m, zg_graph** out) {
  if (!(rate >= 0.0 && rate <= 1.0))
    return zg_set_error(ZG_ERR_INVALID_ARG, "sample rate %g outside [0,1]", rate), ZG_ERR_INVALID_ARG;
  return derive(false, g, 1, 0, 0, 0, rate, keep_seed, shuffle_seed, (cudaStream_t)cuda_stream, parent_index, out_m,
                out);
}
