// zg_exact.cu — exact subgraph counts on the device, bit-exact with naive_implementation/:
//   triangles (TriangleCounting.cpp), wedges (ThreeChain.cpp), 3-edge paths (FourChain.cpp),
//   K1,4 stars (FiveStar.cpp), 4-cliques (FourClique.cpp), houses (FiveHouse.cpp), 4-edge paths
//   (FiveChain.cpp) and the predicate-weighted triangles (WeightedTriangleCounting.cpp,
//   AtLeastOneWeightedTriangleCounting.cpp).
//
// Degree orientation: every edge points from the endpoint with the smaller (degree, id) to the
// larger, which bounds every out-list by sqrt(2m) and counts each clique once from its lowest
// vertex.  The out-lists are filled by counting (no sort: their order does not matter).  Work is
// vertex-centred: out(u) goes into a hash table and the out-lists of its members are streamed
// through it, so one probe in shared memory answers what a binary search over a list in global
// memory would:
//   triangles  = sum over u, v in out(u), of |out(u) ∩ out(v)|
//   4-cliques  = the same pass keeps out(u) ∩ out(v) as one bit row per v; then, per set bit w of
//                row v, popc(row v & row w)
//   3-paths    = sum over edges of (d_u - 1)(d_v - 1) - 3 * triangles
//   wedges     = sum C(d,2),  stars = sum C(d,4)  (exact 128-bit; the naive FiveStar wraps in 64)
// A predicate on the edge data keeps only the passing edges in the orientation (weighted
// triangles: data >= T; at least one >= T: all triangles minus those whose edges are all < T).
// Houses and 4-edge paths come from per-edge triangle counts t(e) and 4-cycle counts c4(e), one
// warp per edge over the full sorted neighbour lists (identities checked against the naive walks
// in oracle/zg_oracle.c):
//   houses       = sum_e t(e) c4(e) - 2 sum_e t(e)^2 + 6 T
//   4-edge paths = (sum_v (S1(v)^2 - S2(v)) + 2 sum_e t(e)(3 - d_a - d_b) - 2 sum_e c4(e)) / 2
// with c4(a,b) = sum over x in N(a) \ {b} of (|N(x) ∩ N(b)| - 1), S1(v) = sum over w in N(v) of
// (d_w - 1), S2(v) the sum of the squares.  Sums are reduced per block in 128 bits (two's
// complement for the signed terms) and folded on the host.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <vector>

#include "zg_internal.cuh"

namespace {

constexpr int kB = 256;

constexpr uint32_t kNone = 0xFFFFFFFFu;  // no vertex has this id (there are at most 2^32 - 1 of them)

struct U128 {
  unsigned long long lo, hi;
};

__device__ __forceinline__ void add128(U128& a, unsigned long long v) {
  unsigned long long o = a.lo;
  a.lo += v;
  a.hi += a.lo < o;
}

__device__ __forceinline__ void add128w(U128& a, unsigned __int128 v) {
  add128(a, (unsigned long long)v);
  a.hi += (unsigned long long)(v >> 64);
}

__device__ void block_store(U128 a, U128* out) {
  __shared__ unsigned long long slo[kB], shi[kB];
  slo[threadIdx.x] = a.lo;
  shi[threadIdx.x] = a.hi;
  __syncthreads();
  if (threadIdx.x == 0) {
    U128 t = {0, 0};
    for (int i = 0; i < kB; ++i) {
      add128(t, slo[i]);
      t.hi += shi[i];
    }
    out[blockIdx.x] = t;
  }
}

__device__ __forceinline__ uint64_t deg(const ZgDevGraph& g, uint32_t v) { return (uint64_t)(g.off[v + 1] - g.off[v]); }

// Edge predicate of the weighted counts: 0 keeps every edge, 1 keeps data >= t, 2 keeps data < t.
__device__ __forceinline__ bool keep_edge(const ZgDevGraph& g, uint64_t e, int pred, uint32_t t) {
  if (pred == 0) return true;
  const uint32_t w = g.w[e];
  return pred == 1 ? w >= t : w < t;
}

// (degree, id) order: edge e as (lower, higher); its place in the lower one's out-list
__global__ void __launch_bounds__(kB) k_orient(ZgDevGraph g, int pred, uint32_t t, uint2* __restrict__ ab,
                                               uint32_t* __restrict__ slot, uint32_t* __restrict__ outdeg) {
  for (uint64_t e = blockIdx.x * (uint64_t)kB + threadIdx.x; e < g.m; e += (uint64_t)gridDim.x * kB) {
    if (!keep_edge(g, e, pred, t)) {
      ab[e] = make_uint2(kNone, kNone);
      continue;
    }
    const uint4 r = zg_rec_e(g, e);
    const uint32_t dx = g.off32[r.x + 1] - g.off32[r.x], dy = g.off32[r.y + 1] - g.off32[r.y];
    const bool up = dx < dy || (dx == dy && r.x < r.y);
    const uint32_t a = up ? r.x : r.y, b = up ? r.y : r.x;
    ab[e] = make_uint2(a, b);
    slot[e] = atomicAdd(&outdeg[a], 1u);
  }
}

__device__ __forceinline__ bool bsearch(const uint32_t* __restrict__ a, int64_t lo, int64_t hi, uint32_t key) {
  while (lo < hi) {
    int64_t mid = (lo + hi) >> 1;
    uint32_t x = __ldg(&a[mid]);
    if (x == key) return true;
    if (x < key)
      lo = mid + 1;
    else
      hi = mid;
  }
  return false;
}

// ---- triangles and 4-cliques over the out-lists ----------------------------------------------
// Vertices by out-degree k (one below 2 closes nothing): up to 32 one warp each, up to kMid and up
// to kBig one block each with the table and the bit rows in shared memory, beyond that one block
// each with both in a slab of global memory.  Bound by the probes (sum over edges of |out(v)|, each
// a few instructions and one shared-memory read); with one binary search per list entry in global
// memory instead, ms per count on one GB300, before -> now, triangles / 4-cliques:
//   R-MAT scale 13 ef 12 (96 k edges)  0.27 -> 0.11 / 2.6 -> 0.11
//   R-MAT scale 20 ef 3 (3.1 M)        2.4 -> 0.77 / 55 -> 0.86
//   R-MAT scale 20 ef 12 (12 M)        17.8 -> 6.3 / 3105 -> 8.9
//   R-MAT scale 22 ef 24 (95 M)        382 -> 201 / not run -> 509
// Where the lines lie: 32 members are one word a row and one lane each; 256 keep the block's table
// and rows at 15 KB, so a full SM of blocks is resident; 1 024 are the most whose rows fit beside
// the table (160 KB).
constexpr uint32_t kMid = 256, kBig = 1024;
constexpr int kClasses = 4;
struct DagHdr {
  unsigned long long lo, hi;  // the count, 128 bits
  uint32_t n[kClasses];       // vertices per class
  uint32_t next[kClasses];    // the blocks' work counters
  uint32_t kmax;              // the largest out-degree
};

// Fills the out-lists from the places k_orient handed out, and lists the vertices by class.
__global__ void __launch_bounds__(kB) k_fill(uint64_t m, uint32_t nv, const uint2* __restrict__ ab,
                                             const uint32_t* __restrict__ slot, const uint32_t* __restrict__ ooff,
                                             uint32_t* __restrict__ nbr, uint32_t* __restrict__ lists,
                                             DagHdr* __restrict__ hdr) {
  const uint64_t tid = blockIdx.x * (uint64_t)kB + threadIdx.x, stride = (uint64_t)gridDim.x * kB;
  for (uint64_t e = tid; e < m; e += stride) {
    const uint2 x = ab[e];
    if (x.x != kNone) nbr[ooff[x.x] + slot[e]] = x.y;
  }
  const uint32_t lane = threadIdx.x & 31;
  for (uint64_t v0 = tid - lane; v0 < nv; v0 += stride) {
    const uint64_t v = v0 + lane;
    const uint32_t k = v < nv ? ooff[v + 1] - ooff[v] : 0u;
    const int cls = k < 2 ? -1 : k <= 32 ? 0 : k <= kMid ? 1 : k <= kBig ? 2 : 3;
#pragma unroll
    for (int c = 0; c < kClasses; ++c) {
      const unsigned in = __ballot_sync(0xffffffffu, cls == c);
      if (!in) continue;
      uint32_t at = 0;
      if (lane == 0) at = atomicAdd(&hdr->n[c], (uint32_t)__popc(in));
      at = __shfl_sync(0xffffffffu, at, 0);
      if (cls == c) lists[(uint64_t)c * nv + at + __popc(in & ((1u << lane) - 1))] = (uint32_t)v;
    }
    if (cls == 3) atomicMax(&hdr->kmax, k);
  }
}

// Streams up to 32 lists, lane j's starting at nbr[start] with len entries, through body(j, x).
// Long lists go one after another with the whole warp on each; the short ones are laid end to end
// and every lane finds its list by a search over the running lengths, so that lists of a few
// entries (most of them) do not leave lanes idle.
template <class F>
__device__ __forceinline__ void stream_lists(const uint32_t* __restrict__ nbr, uint32_t start, uint32_t len, F&& body) {
  const uint32_t lane = threadIdx.x & 31;
  constexpr uint32_t kLong = 64;
  for (unsigned big = __ballot_sync(0xffffffffu, len >= kLong); big; big &= big - 1) {
    const int j = __ffs(big) - 1;
    const uint32_t s = __shfl_sync(0xffffffffu, start, j), n = __shfl_sync(0xffffffffu, len, j);
    uint32_t i = lane;
    for (; i + 96 < n; i += 128) {
      const uint32_t x0 = __ldg(&nbr[s + i]), x1 = __ldg(&nbr[s + i + 32]), x2 = __ldg(&nbr[s + i + 64]),
                     x3 = __ldg(&nbr[s + i + 96]);
      body(j, x0);
      body(j, x1);
      body(j, x2);
      body(j, x3);
    }
    for (; i < n; i += 32) body(j, __ldg(&nbr[s + i]));
  }
  const uint32_t mine = len >= kLong ? 0u : len;
  uint32_t incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= (uint32_t)o) incl += v;
  }
  const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
  const uint32_t shift = start - (incl - mine);  // flat position f of list j is nbr[shift + f]
  for (uint32_t f0 = 0; f0 < total; f0 += 32) {
    const uint32_t f = f0 + lane;
    int j = 0;  // the lists that end at or before f
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      if (__shfl_sync(0xffffffffu, incl, j + o - 1) <= f) j += o;
    const uint32_t at = __shfl_sync(0xffffffffu, shift, j) + f;
    if (f < total) body(j, __ldg(&nbr[at]));
  }
}

__device__ __forceinline__ uint32_t vhash(uint32_t x, uint32_t bits) { return (x * 0x9E3779B1u) >> (32 - bits); }

// The block's sum of c, added to the 128-bit count.
__device__ __forceinline__ void add_count(unsigned long long c, DagHdr* hdr) {
  U128 a = {c, 0};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long lo = __shfl_xor_sync(0xffffffffu, a.lo, o), hi = __shfl_xor_sync(0xffffffffu, a.hi, o);
    add128(a, lo);
    a.hi += hi;
  }
  if ((threadIdx.x & 31) == 0 && (a.lo | a.hi)) {
    const unsigned long long old = atomicAdd(&hdr->lo, a.lo);
    const unsigned long long up = a.hi + (old + a.lo < old);
    if (up) atomicAdd(&hdr->hi, up);
  }
}

// One warp per vertex of out-degree 2 .. 32: a 128-slot table and one 32-bit row per member.
template <bool CLIQUE>
__global__ void __launch_bounds__(kB) k_dag_warp(const uint32_t* __restrict__ list, const uint32_t* __restrict__ ooff,
                                                 const uint32_t* __restrict__ nbr, DagHdr* __restrict__ hdr) {
  __shared__ uint32_t s_key[kB / 32][128], s_row[kB / 32][32];
  __shared__ uint8_t s_idx[kB / 32][128];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t *key = s_key[warp], *row = s_row[warp];
  uint8_t* idx = s_idx[warp];
  for (int i = 0; i < 4; ++i) key[lane + 32 * i] = kNone;
  __syncwarp();
  const uint32_t count = hdr->n[0];
  unsigned long long c = 0;
  for (uint32_t w = blockIdx.x * (kB / 32) + warp; w < count; w += gridDim.x * (kB / 32)) {
    const uint32_t u = list[w], b = ooff[u], k = ooff[u + 1] - b;
    uint32_t start = 0, len = 0, slot = 0;
    row[lane] = 0;
    if (lane < k) {
      const uint32_t y = __ldg(&nbr[b + lane]);
      start = ooff[y];
      len = ooff[y + 1] - start;
      slot = vhash(y, 7);
      while (atomicCAS(&key[slot], kNone, y) != kNone) slot = (slot + 1) & 127;  // at most 32 of 128 slots are taken
      idx[slot] = (uint8_t)lane;
    }
    __syncwarp();
    stream_lists(nbr, start, len, [&](int j, uint32_t x) {
      for (uint32_t h = vhash(x, 7);; h = (h + 1) & 127) {
        const uint32_t y = key[h];
        if (y == x) {
          if (CLIQUE) atomicOr(&row[j], 1u << idx[h]);
          else ++c;
          break;
        }
        if (y == kNone) break;
      }
    });
    __syncwarp();
    if (CLIQUE) {
      const uint32_t r = row[lane];
      for (uint32_t bits = r; bits; bits &= bits - 1) c += __popc(r & row[__ffs(bits) - 1]);
      __syncwarp();
    }
    if (lane < k) key[slot] = kNone;
    __syncwarp();
  }
  add_count(c, hdr);
}

// One block per vertex u: key/idx a table of 2^hb >= 4k slots, mat k bit rows of R words at an odd
// stride.  GLOBAL: they lie in global memory (written through L2, so read there too).
template <bool CLIQUE, bool GLOBAL, int T>
__device__ __forceinline__ void dag_vertex(uint32_t u, const uint32_t* __restrict__ ooff,
                                           const uint32_t* __restrict__ nbr, uint32_t* key, uint16_t* idx,
                                           uint32_t* idx32, uint32_t* mat, uint32_t* s_next, unsigned long long& c) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t b = ooff[u], k = ooff[u + 1] - b;
  const uint32_t hb = 32 - __clz(4 * k - 1), mask = (1u << hb) - 1;
  const uint32_t R = (k + 31) / 32, RS = R | 1;
  auto ld = [](const uint32_t* p) { return GLOBAL ? __ldcg(p) : *p; };
  for (uint32_t i = threadIdx.x; i <= mask; i += T) key[i] = kNone;
  if (CLIQUE)
    for (uint64_t i = threadIdx.x; i < (uint64_t)k * RS; i += T) mat[i] = 0;
  if (threadIdx.x == 0) *s_next = 0;
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < k; i += T) {
    const uint32_t y = __ldg(&nbr[b + i]);
    uint32_t h = vhash(y, hb);
    while (atomicCAS(&key[h], kNone, y) != kNone) h = (h + 1) & mask;  // a quarter of the slots at most are taken
    if (GLOBAL) idx32[h] = i;
    else idx[h] = (uint16_t)i;
  }
  __syncthreads();
  // eight members at a time per warp: a vertex of 33 members already feeds five warps
  for (;;) {
    uint32_t j0 = 0;
    if (lane == 0) j0 = atomicAdd(s_next, 8u);
    j0 = __shfl_sync(0xffffffffu, j0, 0);
    if (j0 >= k) break;
    uint32_t start = 0, len = 0;
    if (lane < 8 && j0 + lane < k) {
      const uint32_t y = __ldg(&nbr[b + j0 + lane]);
      start = ooff[y];
      len = ooff[y + 1] - start;
    }
    stream_lists(nbr, start, len, [&](int j, uint32_t x) {
      for (uint32_t h = vhash(x, hb);; h = (h + 1) & mask) {
        const uint32_t y = ld(&key[h]);
        if (y == x) {
          if (CLIQUE) {
            const uint32_t i = GLOBAL ? __ldcg(&idx32[h]) : idx[h];
            atomicOr(&mat[(uint64_t)(j0 + j) * RS + i / 32], 1u << (i & 31));
          } else {
            ++c;
          }
          break;
        }
        if (y == kNone) break;
      }
    });
  }
  __syncthreads();
  if (CLIQUE) {
    for (uint64_t i = threadIdx.x; i < (uint64_t)k * R; i += T) {
      const uint32_t v = (uint32_t)(i / R), q = (uint32_t)(i % R);
      const uint32_t* rv = mat + (uint64_t)v * RS;
      for (uint32_t bits = ld(&rv[q]); bits; bits &= bits - 1) {
        const uint32_t* rw = mat + (uint64_t)(q * 32 + __ffs(bits) - 1) * RS;
        for (uint32_t l = 0; l < R; ++l) c += __popc(ld(&rv[l]) & ld(&rw[l]));
      }
    }
    __syncthreads();
  }
}

template <bool CLIQUE, uint32_t KMAX>
constexpr size_t dag_smem() {
  return 6u * 4 * KMAX + (CLIQUE ? 4u * KMAX * (KMAX / 32 + 1) : 0u);
}

template <bool CLIQUE, uint32_t KMAX, int T>
__global__ void __launch_bounds__(T) k_dag_block(int cls, const uint32_t* __restrict__ list,
                                                 const uint32_t* __restrict__ ooff, const uint32_t* __restrict__ nbr,
                                                 DagHdr* __restrict__ hdr) {
  extern __shared__ uint32_t smem[];
  __shared__ uint32_t s_item, s_next;
  uint32_t* key = smem;
  uint32_t* mat = smem + 4 * KMAX;
  uint16_t* idx = (uint16_t*)(mat + (CLIQUE ? KMAX * (KMAX / 32 + 1) : 0));
  const uint32_t count = hdr->n[cls];
  unsigned long long c = 0;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(&hdr->next[cls], 1u);
    __syncthreads();
    const uint32_t item = s_item;
    if (item >= count) break;
    dag_vertex<CLIQUE, false, T>(list[item], ooff, nbr, key, idx, nullptr, mat, &s_next, c);
    __syncthreads();
  }
  add_count(c, hdr);
}

// Vertices of more than kBig members, tables and rows in a slab of `slab` words per block.
template <bool CLIQUE, int T>
__global__ void __launch_bounds__(T) k_dag_global(const uint32_t* __restrict__ list, const uint32_t* __restrict__ ooff,
                                                  const uint32_t* __restrict__ nbr, uint32_t* __restrict__ slabs,
                                                  uint64_t slab, uint32_t table, DagHdr* __restrict__ hdr) {
  __shared__ uint32_t s_item, s_next;
  uint32_t* key = slabs + blockIdx.x * slab;
  const uint32_t count = hdr->n[3];
  unsigned long long c = 0;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(&hdr->next[3], 1u);
    __syncthreads();
    const uint32_t item = s_item;
    if (item >= count) break;
    dag_vertex<CLIQUE, true, T>(list[item], ooff, nbr, key, nullptr, key + table, key + 2ull * table, &s_next, c);
    __syncthreads();
  }
  add_count(c, hdr);
}

__global__ void k_low32(const unsigned long long* __restrict__ keys, uint64_t m, uint32_t* __restrict__ out) {
  for (uint64_t e = blockIdx.x * (uint64_t)kB + threadIdx.x; e < m; e += (uint64_t)gridDim.x * kB)
    out[e] = (uint32_t)keys[e];
}

// per-vertex degree terms and per-edge (d_u - 1)(d_v - 1)
__global__ void __launch_bounds__(kB) k_degree_terms(ZgDevGraph g, int kind, U128* __restrict__ parts) {
  U128 acc = {0, 0};
  uint64_t tid = blockIdx.x * (uint64_t)kB + threadIdx.x, stride = (uint64_t)gridDim.x * kB;
  if (kind == ZG_EXACT_THREE_PATH) {
    for (uint64_t e = tid; e < g.m; e += stride) {
      uint4 r = zg_rec_e(g, e);
      add128w(acc, (unsigned __int128)(deg(g, r.x) - 1) * (deg(g, r.y) - 1));
    }
  } else {
    for (uint64_t v = tid; v < g.nv; v += stride) {
      uint64_t d = deg(g, (uint32_t)v);
      if (kind == ZG_EXACT_WEDGE) add128(acc, d * (d - 1) / 2);
      else if (d >= 4) add128w(acc, (unsigned __int128)d * (d - 1) * (d - 2) * (d - 3) / 24);
    }
  }
  block_store(acc, parts);
}

struct Dev {
  void* p = nullptr;
  ~Dev() {
    if (p) cudaFree(p);
  }
};

int fold(U128* parts, int grid, cudaStream_t s, unsigned __int128* out) {
  std::vector<U128> h(grid);
  cudaError_t ce = cudaMemcpyAsync(h.data(), parts, sizeof(U128) * grid, cudaMemcpyDeviceToHost, s);
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(s);
  if (ce != cudaSuccess) return zg_check_cuda(ce, "exact count");
  unsigned __int128 t = 0;
  for (int i = 0; i < grid; ++i) t += ((unsigned __int128)h[i].hi << 64) | h[i].lo;
  *out = t;
  return ZG_OK;
}

int alloc(Dev& d, size_t bytes) {
  cudaError_t e = cudaMalloc(&d.p, bytes ? bytes : 1);
  if (e != cudaSuccess) {
    cudaGetLastError();
    d.p = nullptr;
    return zg_check_cuda(e, "exact count scratch");
  }
  return ZG_OK;
}

// Scratch from the library's pool, given back on the call's stream.
struct Pool {
  void* p = nullptr;
  cudaStream_t s;
  explicit Pool(cudaStream_t stream) : s(stream) {}
  ~Pool() {
    if (p) cudaFreeAsync(p, s);
  }
  int alloc(size_t bytes) {
    const cudaError_t e = zg_malloc_async(&p, bytes ? bytes : 1, s);
    if (e == cudaSuccess) return ZG_OK;
    cudaGetLastError();
    p = nullptr;
    return zg_check_cuda(e, "exact count scratch");
  }
};

template <bool CLIQUE>
int dag_launch(uint32_t nv, const uint32_t* lists, const uint32_t* ooff, const uint32_t* nbr, DagHdr* hdr,
               cudaStream_t s) {
  constexpr int TM = 256, TB = 512;
  constexpr size_t sm = dag_smem<CLIQUE, kMid>(), sb = dag_smem<CLIQUE, kBig>();
  cudaError_t e = cudaFuncSetAttribute(k_dag_block<CLIQUE, kBig, TB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sb);
  if (e != cudaSuccess) return zg_check_cuda(e, "exact count kernel");
  const int sms = zg_num_sms();
  // the largest vertices first: one of them is the longest single piece of work
  k_dag_block<CLIQUE, kBig, TB><<<sms, TB, sb, s>>>(2, lists + 2ull * nv, ooff, nbr, hdr);
  k_dag_block<CLIQUE, kMid, TM><<<sms * 8, TM, sm, s>>>(1, lists + nv, ooff, nbr, hdr);
  k_dag_warp<CLIQUE><<<sms * 8, kB, 0, s>>>(lists, ooff, nbr, hdr);
  return ZG_OK;
}

// The vertices past kBig: as many blocks as slabs fit a bounded share of the free memory.
int dag_launch_global(bool clique, const DagHdr& h, const uint32_t* list, const uint32_t* ooff, const uint32_t* nbr,
                      DagHdr* hdr, cudaStream_t s) {
  uint32_t table = 1;
  while (table < 4 * h.kmax) table <<= 1;
  const uint64_t R = (h.kmax + 31) / 32;
  const uint64_t slab = 2ull * table + (clique ? h.kmax * (R | 1) : 0);  // 32-bit words
  size_t free_b = 0, total_b = 0;
  cudaError_t e = cudaMemGetInfo(&free_b, &total_b);
  if (e != cudaSuccess) return zg_check_cuda(e, "exact count scratch");
  uint64_t blocks = std::min<uint64_t>({h.n[3], (uint64_t)zg_num_sms() * 2, (free_b / 4) / (4 * slab)});
  if (blocks < 1) blocks = 1;
  Pool slabs(s);
  int rc = slabs.alloc(4 * slab * blocks);
  if (rc) return rc;
  if (clique)
    k_dag_global<true, 512><<<(int)blocks, 512, 0, s>>>(list, ooff, nbr, (uint32_t*)slabs.p, slab, table, hdr);
  else
    k_dag_global<false, 512><<<(int)blocks, 512, 0, s>>>(list, ooff, nbr, (uint32_t*)slabs.p, slab, table, hdr);
  return ZG_OK;
}

// triangles (kind TRIANGLE) or 4-cliques over the degree-oriented DAG of the edges that pass the
// predicate (pred 0: every edge)
int dag_count(const zg_graph* g, int kind, int pred, uint32_t t, cudaStream_t s, unsigned __int128* out) {
  const uint64_t m = g->d.m;
  const uint32_t nv = g->d.nv;
  *out = 0;
  if (m == 0) return ZG_OK;
  // one block of scratch: (lower, higher) and place per edge, out-lists, offsets, class lists
  const size_t nv1 = (size_t)nv + 1;
  size_t tb = 0, at = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, tb, (uint32_t*)nullptr, (uint32_t*)nullptr, (int64_t)nv1, s);
  auto take = [&](size_t bytes) {
    const size_t p = at;
    at += (bytes + 255) & ~(size_t)255;
    return p;
  };
  const size_t o_hdr = take(sizeof(DagHdr)), o_deg = take(4 * nv1), o_off = take(4 * nv1), o_ab = take(8 * m),
               o_slot = take(4 * m), o_nbr = take(4 * m), o_list = take(4ull * kClasses * nv), o_tmp = take(tb);
  Pool pool(s);
  int rc = pool.alloc(at);
  if (rc) return rc;
  char* p = (char*)pool.p;
  DagHdr* hdr = (DagHdr*)(p + o_hdr);
  uint32_t *outdeg = (uint32_t*)(p + o_deg), *ooff = (uint32_t*)(p + o_off), *slot = (uint32_t*)(p + o_slot),
           *nbr = (uint32_t*)(p + o_nbr), *lists = (uint32_t*)(p + o_list);
  uint2* ab = (uint2*)(p + o_ab);
  cudaMemsetAsync(p + o_hdr, 0, o_off - o_hdr, s);  // the header and the out-degrees
  const int grid = (int)std::min<uint64_t>((m + kB - 1) / kB, (uint64_t)zg_num_sms() * 8);
  k_orient<<<grid, kB, 0, s>>>(g->d, pred, t, ab, slot, outdeg);
  cub::DeviceScan::ExclusiveSum(p + o_tmp, tb, outdeg, ooff, (int64_t)nv1, s);
  k_fill<<<grid, kB, 0, s>>>(m, nv, ab, slot, ooff, nbr, lists, hdr);
  const bool clique = kind == ZG_EXACT_FOUR_CLIQUE;
  if ((rc = clique ? dag_launch<true>(nv, lists, ooff, nbr, hdr, s) : dag_launch<false>(nv, lists, ooff, nbr, hdr, s)))
    return rc;
  DagHdr h;
  for (int pass = 0; pass < 2; ++pass) {
    cudaError_t ce = cudaMemcpyAsync(&h, hdr, sizeof(h), cudaMemcpyDeviceToHost, s);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(s);
    if (ce == cudaSuccess) ce = cudaGetLastError();
    if (ce != cudaSuccess) return zg_check_cuda(ce, "exact count kernel");
    if (pass || !h.n[3]) break;
    if ((rc = dag_launch_global(clique, h, lists + 3ull * nv, ooff, nbr, hdr, s))) return rc;
  }
  *out = ((unsigned __int128)h.hi << 64) | h.lo;
  return ZG_OK;
}

// ---- houses and 4-edge paths -------------------------------------------------------------------
// Sorted full neighbour lists aligned with g->off: from the neighbour-ordered adjacency when the
// graph has one, else by a radix sort of both directions' (src:dst) keys.
__global__ void k_both_keys(ZgDevGraph g, unsigned long long* __restrict__ keys) {
  for (uint64_t e = blockIdx.x * (uint64_t)kB + threadIdx.x; e < g.m; e += (uint64_t)gridDim.x * kB) {
    uint4 r = zg_rec_e(g, e);
    keys[2 * e] = ((unsigned long long)r.x << 32) | r.y;
    keys[2 * e + 1] = ((unsigned long long)r.y << 32) | r.x;
  }
}
__global__ void k_adj_nbr(const uint2* __restrict__ adj, uint64_t n, uint32_t* __restrict__ out) {
  for (uint64_t i = blockIdx.x * (uint64_t)kB + threadIdx.x; i < n; i += (uint64_t)gridDim.x * kB) out[i] = adj[i].x;
}

// |N(x) ∩ N(y)|: iterate the shorter list, binary-search the longer
__device__ __forceinline__ unsigned long long common(const uint32_t* __restrict__ nbr, const int64_t* __restrict__ off,
                                                     uint32_t x, uint32_t y) {
  int64_t bx = off[x], ex = off[x + 1], by = off[y], ey = off[y + 1];
  if (ex - bx > ey - by) {
    int64_t t0 = bx, t1 = ex;
    bx = by;
    ex = ey;
    by = t0;
    ey = t1;
  }
  unsigned long long c = 0;
  for (int64_t i = bx; i < ex; ++i) c += bsearch(nbr, by, ey, __ldg(&nbr[i]));
  return c;
}

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// one warp per edge (a, b), a the endpoint of smaller degree: t(e) and c4(e), then the edge's term
__global__ void __launch_bounds__(kB) k_house_chain(ZgDevGraph g, const uint32_t* __restrict__ nbr,
                                                    const int64_t* __restrict__ off, int kind, U128* __restrict__ parts) {
  U128 acc = {0, 0};
  const int lane = threadIdx.x & 31;
  const uint64_t warps = (uint64_t)gridDim.x * (kB / 32);
  for (uint64_t e = blockIdx.x * (uint64_t)(kB / 32) + (threadIdx.x >> 5); e < g.m; e += warps) {
    uint4 r = zg_rec_e(g, e);
    uint32_t a = r.x, b = r.y;
    int64_t da = off[a + 1] - off[a], db = off[b + 1] - off[b];
    if (da > db) {
      uint32_t t = a;
      a = b;
      b = t;
      int64_t x = da;
      da = db;
      db = x;
    }
    unsigned long long tl = 0;
    for (int64_t i = off[a] + lane; i < off[a + 1]; i += 32) tl += bsearch(nbr, off[b], off[b + 1], __ldg(&nbr[i]));
    const unsigned long long te = warp_sum(tl);
    if (kind == ZG_EXACT_FIVE_HOUSE && te == 0) continue;
    unsigned long long cl = 0;
    for (int64_t i = off[a] + lane; i < off[a + 1]; i += 32) {
      const uint32_t x = __ldg(&nbr[i]);
      if (x != b) cl += common(nbr, off, x, b) - 1;  // a is in both lists
    }
    const unsigned long long c4 = warp_sum(cl);
    if (lane == 0) {
      __int128 v;
      if (kind == ZG_EXACT_FIVE_HOUSE)
        v = (__int128)te * c4 - 2 * (__int128)te * te + 2 * (__int128)te;  // 6 T = 2 sum_e t(e)
      else
        v = 2 * (__int128)te * (3 - (__int128)da - (__int128)db) - 2 * (__int128)c4;
      add128w(acc, (unsigned __int128)v);
    }
  }
  block_store(acc, parts);
}

// one warp per vertex: S1(v)^2 - S2(v)
__global__ void __launch_bounds__(kB) k_chain_vertex(uint32_t nv, const uint32_t* __restrict__ nbr,
                                                     const int64_t* __restrict__ off, U128* __restrict__ parts) {
  U128 acc = {0, 0};
  const int lane = threadIdx.x & 31;
  const uint64_t warps = (uint64_t)gridDim.x * (kB / 32);
  for (uint64_t v = blockIdx.x * (uint64_t)(kB / 32) + (threadIdx.x >> 5); v < nv; v += warps) {
    unsigned long long s1 = 0;
    unsigned __int128 s2 = 0;
    for (int64_t i = off[v] + lane; i < off[v + 1]; i += 32) {
      const uint32_t w = __ldg(&nbr[i]);
      const unsigned long long dw = (unsigned long long)(off[w + 1] - off[w]) - 1;
      s1 += dw;
      s2 += (unsigned __int128)dw * dw;
    }
    s1 = warp_sum(s1);
    // exact 128-bit warp sum of s2: 64-bit halves, each low-half addition's carry into the high half
    unsigned long long slo = (unsigned long long)s2, shi = (unsigned long long)(s2 >> 64);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long olo = __shfl_xor_sync(0xffffffffu, slo, o), ohi = __shfl_xor_sync(0xffffffffu, shi, o);
      const unsigned long long n = slo + olo;
      shi += ohi + (n < slo);
      slo = n;
    }
    if (lane == 0) {
      const unsigned __int128 S2 = ((unsigned __int128)shi << 64) | slo;
      add128w(acc, (unsigned __int128)s1 * s1 - S2);
    }
  }
  block_store(acc, parts);
}

int house_chain(const zg_graph* g, int kind, cudaStream_t s, unsigned __int128* out) {
  const uint64_t m = g->d.m;
  const uint32_t nv = g->d.nv;
  if (m == 0) {
    *out = 0;
    return ZG_OK;
  }
  Dev nb, parts, k1, k2, tmp;
  int rc;
  const int grid = zg_num_sms() * 8;
  if ((rc = alloc(nb, 4 * 2 * m)) || (rc = alloc(parts, sizeof(U128) * 2 * grid))) return rc;
  if (g->adj_n) {
    k_adj_nbr<<<grid, kB, 0, s>>>(g->adj_n, 2 * m, (uint32_t*)nb.p);
  } else {
    if ((rc = alloc(k1, 8 * 2 * m)) || (rc = alloc(k2, 8 * 2 * m))) return rc;
    k_both_keys<<<grid, kB, 0, s>>>(g->d, (unsigned long long*)k1.p);
    size_t tb = 0;
    cub::DeviceRadixSort::SortKeys(nullptr, tb, (unsigned long long*)k1.p, (unsigned long long*)k2.p, (int64_t)(2 * m),
                                   0, 64, s);
    if ((rc = alloc(tmp, tb))) return rc;
    cub::DeviceRadixSort::SortKeys(tmp.p, tb, (unsigned long long*)k1.p, (unsigned long long*)k2.p, (int64_t)(2 * m),
                                   0, 64, s);
    k_low32<<<grid, kB, 0, s>>>((const unsigned long long*)k2.p, 2 * m, (uint32_t*)nb.p);
  }
  cudaMemsetAsync(parts.p, 0, sizeof(U128) * 2 * grid, s);
  k_house_chain<<<grid, kB, 0, s>>>(g->d, (const uint32_t*)nb.p, g->off, kind, (U128*)parts.p);
  if (kind == ZG_EXACT_FIVE_CHAIN)
    k_chain_vertex<<<grid, kB, 0, s>>>(nv, (const uint32_t*)nb.p, g->off, (U128*)parts.p + grid);
  cudaError_t ce = cudaGetLastError();
  if (ce != cudaSuccess) return zg_check_cuda(ce, "exact count kernel");
  unsigned __int128 r = 0;
  if ((rc = fold((U128*)parts.p, 2 * grid, s, &r))) return rc;
  *out = kind == ZG_EXACT_FIVE_CHAIN ? (unsigned __int128)((__int128)r / 2) : r;
  return ZG_OK;
}

int degree_terms(const zg_graph* g, int kind, cudaStream_t s, unsigned __int128* out) {
  int grid = zg_num_sms() * 8;
  Dev parts;
  int rc = alloc(parts, sizeof(U128) * grid);
  if (rc) return rc;
  k_degree_terms<<<grid, kB, 0, s>>>(g->d, kind, (U128*)parts.p);
  cudaError_t ce = cudaGetLastError();
  if (ce != cudaSuccess) return zg_check_cuda(ce, "exact count kernel");
  return fold((U128*)parts.p, grid, s, out);
}

}  // namespace

extern "C" int zg_exact_count(const zg_graph* g, int kind, void* cuda_stream, uint64_t out[2]) {
  if (!g || !out) return zg_set_error(ZG_ERR_INVALID_ARG, "null argument"), ZG_ERR_INVALID_ARG;
  if (kind < ZG_EXACT_TRIANGLE || kind > ZG_EXACT_FIVE_CHAIN)
    return zg_set_error(ZG_ERR_INVALID_ARG, "unknown exact-count kind %d (the weighted triangles take "
                        "zg_exact_count_weighted)", kind), ZG_ERR_INVALID_ARG;
  cudaStream_t s = (cudaStream_t)cuda_stream;
  unsigned __int128 r = 0, t = 0;
  int rc = ZG_OK;
  switch (kind) {
    case ZG_EXACT_TRIANGLE:
    case ZG_EXACT_FOUR_CLIQUE: rc = dag_count(g, kind, 0, 0, s, &r); break;
    case ZG_EXACT_WEDGE:
    case ZG_EXACT_FIVE_STAR: rc = degree_terms(g, kind, s, &r); break;
    case ZG_EXACT_THREE_PATH:
      rc = degree_terms(g, kind, s, &r);
      if (rc == ZG_OK) rc = dag_count(g, ZG_EXACT_TRIANGLE, 0, 0, s, &t);
      r -= 3 * t;
      break;
    case ZG_EXACT_FIVE_HOUSE:
    case ZG_EXACT_FIVE_CHAIN: rc = house_chain(g, kind, s, &r); break;
  }
  if (rc) return rc;
  out[0] = (uint64_t)r;
  out[1] = (uint64_t)(r >> 64);
  return ZG_OK;
}

extern "C" int zg_exact_count_weighted(const zg_graph* g, int kind, uint32_t threshold, void* cuda_stream,
                                       uint64_t out[2]) {
  if (!g || !out) return zg_set_error(ZG_ERR_INVALID_ARG, "null argument"), ZG_ERR_INVALID_ARG;
  if (kind != ZG_EXACT_WEIGHTED_TRIANGLE && kind != ZG_EXACT_AT_LEAST_ONE_TRIANGLE)
    return zg_set_error(ZG_ERR_INVALID_ARG, "unknown weighted exact-count kind %d", kind), ZG_ERR_INVALID_ARG;
  if (!g->w) return zg_set_error(ZG_ERR_INVALID_ARG, "the graph has no edge data"), ZG_ERR_INVALID_ARG;
  cudaStream_t s = (cudaStream_t)cuda_stream;
  unsigned __int128 r = 0, below = 0;
  int rc;
  if (kind == ZG_EXACT_WEIGHTED_TRIANGLE) {
    rc = dag_count(g, ZG_EXACT_TRIANGLE, 1, threshold, s, &r);
  } else {
    rc = dag_count(g, ZG_EXACT_TRIANGLE, 0, 0, s, &r);
    if (rc == ZG_OK) rc = dag_count(g, ZG_EXACT_TRIANGLE, 2, threshold, s, &below);
    r -= below;
  }
  if (rc) return rc;
  out[0] = (uint64_t)r;
  out[1] = (uint64_t)(r >> 64);
  return ZG_OK;
}
