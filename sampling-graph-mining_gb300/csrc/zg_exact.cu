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
// Houses and 4-edge paths come from per-edge triangle counts t(e) and 4-cycle counts c4(e)
// (identities checked against the naive walks in oracle/zg_oracle.c):
//   houses       = sum_e t(e) c4(e) - 2 sum_e t(e)^2 + 6 T,  T = sum_e t(e) / 3
//   4-edge paths = (sum_v (S1(v)^2 - S2(v)) + 2 sum_e t(e)(3 - d_a - d_b) - 2 sum_e c4(e)) / 2
// with S1(v) = sum over w in N(v) of (d_w - 1), S2(v) the sum of the squares.  t(e) is the triangle
// pass with one addition per edge of each triangle.  c4 is never stored: with the vertices in an
// order by degree, every 4-cycle is met at its last vertex a as two wedges a - x - y (x and y before
// a) that end in the same y.  cnt(y) such wedges make each of them part of cnt(y) - 1 cycles, all
// through the edges (a, x) and (x, y), so
//   sum_e t(e) c4(e) = sum over wedges of (cnt(y) - 1) (t(a, x) + t(x, y))
//   sum_e c4(e)      = 2 sum over wedges of (cnt(y) - 1)
// over sum_e min(d) wedges in all.  Sums are 128 bits.
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <type_traits>

#include "zg_scratch.cuh"

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

// Adds every thread's a to a 128-bit sum in global memory: a warp sum, then the low half's carry goes
// with the high half.
__device__ __forceinline__ void add_sum(U128 a, U128* sum) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long lo = __shfl_xor_sync(0xffffffffu, a.lo, o), hi = __shfl_xor_sync(0xffffffffu, a.hi, o);
    add128(a, lo);
    a.hi += hi;
  }
  if ((threadIdx.x & 31) == 0 && (a.lo | a.hi)) {
    const unsigned long long old = atomicAdd(&sum->lo, a.lo);
    const unsigned long long up = a.hi + (old + a.lo < old);
    if (up) atomicAdd(&sum->hi, up);
  }
}

__device__ __forceinline__ uint32_t deg(const ZgDevGraph& g, uint32_t v) { return g.off32[v + 1] - g.off32[v]; }

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
    const uint32_t dx = deg(g, r.x), dy = deg(g, r.y);
    const bool up = dx < dy || (dx == dy && r.x < r.y);
    const uint32_t a = up ? r.x : r.y, b = up ? r.y : r.x;
    ab[e] = make_uint2(a, b);
    slot[e] = atomicAdd(&outdeg[a], 1u);
  }
}

// ---- triangles and 4-cliques over the out-lists ----------------------------------------------
// Vertices by out-degree k (one below 2 closes nothing): up to 32 one warp each, up to kMid and up
// to kBig one block each with the table and the bit rows in shared memory, beyond that one block
// each with both in a slab of global memory.  Bound by the probes (sum over edges of |out(v)|, each
// a few instructions and one shared-memory read); with one binary search per list entry in global
// memory instead, ms per count on one GB300, before -> now, triangles / 4-cliques:
//   R-MAT scale 13 ef 12 (96 k edges)  0.27 -> 0.11 / 2.6 -> 0.11
//   R-MAT scale 20 ef 3 (3.1 M)        2.4 -> 0.62 / 55 -> 0.70
//   R-MAT scale 20 ef 12 (12 M)        17.8 -> 4.7 / 3105 -> 7.3
//   R-MAT scale 22 ef 24 (95 M)        382 -> 133 / not run -> 446
// Where the lines lie: 32 members are one word a row and one lane each; 256 keep the block's table
// and rows at 19 KB, so a full SM of blocks is resident; 1 024 are the most whose rows fit beside
// the table (176 KB).
constexpr uint32_t kMid = 256, kBig = 1024;
constexpr int kClasses = 4;
struct DagHdr {
  U128 sum;               // the count
  uint32_t n[kClasses];   // vertices per class
  uint32_t next[kClasses];  // the blocks' work counters
  uint32_t kmax;            // the largest out-degree
};

// What the pass over the out-lists computes: the triangles, the 4-cliques, or every edge's triangles
// (its out-list entries carry the edge ids), the sum then being not 0 when there are any.
enum { kTri, kClique, kPerEdge };
template <int MODE>
__device__ __forceinline__ void dag_result(unsigned long long c, DagHdr* hdr) {
  if (MODE != kPerEdge) add_sum(U128{c, 0}, &hdr->sum);
  else if (c && !__ldcg(&hdr->sum.lo)) hdr->sum.lo = 1;
}
template <int MODE>
using Entry = std::conditional_t<MODE == kPerEdge, uint2, uint32_t>;
__device__ __forceinline__ uint32_t vertex_of(uint32_t x) { return x; }
__device__ __forceinline__ uint32_t vertex_of(uint2 x) { return x.x; }
__device__ __forceinline__ void set_entry(uint32_t* p, uint32_t v, uint64_t) { *p = v; }
__device__ __forceinline__ void set_entry(uint2* p, uint32_t v, uint64_t e) { *p = make_uint2(v, (uint32_t)e); }
__device__ __forceinline__ uint32_t edge_of(uint32_t) { return 0; }
__device__ __forceinline__ uint32_t edge_of(uint2 x) { return x.y; }

// Fills the out-lists from the places k_orient handed out, and lists the vertices by class (`room`
// entries a class).
template <class E>
__global__ void __launch_bounds__(kB) k_fill(uint64_t m, uint32_t nv, const uint2* __restrict__ ab,
                                             const uint32_t* __restrict__ slot, const uint32_t* __restrict__ ooff,
                                             E* __restrict__ nbr, uint32_t* __restrict__ lists, uint64_t room,
                                             DagHdr* __restrict__ hdr) {
  const uint64_t tid = blockIdx.x * (uint64_t)kB + threadIdx.x, stride = (uint64_t)gridDim.x * kB;
  for (uint64_t e = tid; e < m; e += stride) {
    const uint2 x = ab[e];
    if (x.x != kNone) set_entry(&nbr[ooff[x.x] + slot[e]], x.y, e);
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
      if (cls == c) lists[c * room + at + __popc(in & ((1u << lane) - 1))] = (uint32_t)v;
    }
    if (cls == 3) atomicMax(&hdr->kmax, k);
  }
}

// Streams up to 32 lists, lane j's starting at nbr[start] with len entries, through body(j, x).
// Long lists go one after another with the whole warp on each; the short ones are laid end to end
// and every lane finds its list by a search over the running lengths, so that lists of a few
// entries (most of them) do not leave lanes idle.
template <class E, class F>
__device__ __forceinline__ void stream_lists(const E* __restrict__ nbr, uint32_t start, uint32_t len, F&& body) {
  const uint32_t lane = threadIdx.x & 31;
  constexpr uint32_t kLong = 64;
  for (unsigned big = __ballot_sync(0xffffffffu, len >= kLong); big; big &= big - 1) {
    const int j = __ffs(big) - 1;
    const uint32_t s = __shfl_sync(0xffffffffu, start, j), n = __shfl_sync(0xffffffffu, len, j);
    uint32_t i = lane;
    for (; i + 96 < n; i += 128) {
      const E x0 = __ldg(&nbr[s + i]), x1 = __ldg(&nbr[s + i + 32]), x2 = __ldg(&nbr[s + i + 64]),
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

// In front of a table, 32 signature bits per slot: a warp's probe would wait for the longest run of
// taken slots among its lanes (three or four at a quarter load), and with the bits it goes on at once
// unless a lane has a member or a false alarm (under 1 %).  Triangles and 4-cliques on R-MAT scale 20,
// ef 3: 1.44 -> 1.20 ms of kernels, on scale 22, ef 24: 201 + 509 -> 133 + 446 ms.

// One warp per vertex of out-degree 2 .. 32: a 128-slot table and one 32-bit row (per edge: one
// counter) per member.  (Bound by instructions: more vertices in flight, at fewer warps, were slower.)
template <int MODE>
__global__ void __launch_bounds__(kB) k_dag_warp(const uint32_t* __restrict__ list, const uint32_t* __restrict__ ooff,
                                                 const Entry<MODE>* __restrict__ nbr, uint32_t* __restrict__ tri,
                                                 DagHdr* __restrict__ hdr) {
  __shared__ uint32_t s_key[kB / 32][128], s_row[kB / 32][32], s_sig[kB / 32][128];
  __shared__ uint8_t s_idx[kB / 32][128];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t *key = s_key[warp], *row = s_row[warp], *sig = s_sig[warp];
  uint8_t* idx = s_idx[warp];
  for (int i = 0; i < 4; ++i) {
    key[lane + 32 * i] = kNone;
    sig[lane + 32 * i] = 0;
  }
  __syncwarp();
  const uint32_t count = hdr->n[0];
  unsigned long long c = 0;
  for (uint32_t w = blockIdx.x * (kB / 32) + warp; w < count; w += gridDim.x * (kB / 32)) {
    const uint32_t u = list[w], b = ooff[u], k = ooff[u + 1] - b;
    uint32_t start = 0, len = 0, slot = 0, own = 0;
    row[lane] = 0;
    if (lane < k) {
      const Entry<MODE> ent = __ldg(&nbr[b + lane]);
      const uint32_t y = vertex_of(ent);
      own = edge_of(ent);
      start = ooff[y];
      len = ooff[y + 1] - start;
      const uint32_t s = vhash(y, 12);
      atomicOr(&sig[s >> 5], 1u << (s & 31));
      slot = s >> 5;
      while (atomicCAS(&key[slot], kNone, y) != kNone) slot = (slot + 1) & 127;  // at most 32 of 128 slots are taken
      idx[slot] = (uint8_t)lane;
    }
    __syncwarp();
    stream_lists(nbr, start, len, [&](int j, Entry<MODE> ent) {
      const uint32_t x = vertex_of(ent), s = vhash(x, 12);
      if (!(sig[s >> 5] >> (s & 31) & 1)) return;
      for (uint32_t h = s >> 5;; h = (h + 1) & 127) {
        const uint32_t y = key[h];
        if (y == x) {
          if (MODE == kClique) {
            atomicOr(&row[j], 1u << idx[h]);
          } else {
            ++c;
            if (MODE == kPerEdge) {
              atomicAdd(&row[j], 1u);
              atomicAdd(&row[idx[h]], 1u);
              atomicAdd(&tri[edge_of(ent)], 1u);
            }
          }
          break;
        }
        if (y == kNone) break;
      }
    });
    __syncwarp();
    if (MODE == kClique) {
      const uint32_t r = row[lane];
      for (uint32_t bits = r; bits; bits &= bits - 1) c += __popc(r & row[__ffs(bits) - 1]);
      __syncwarp();
    }
    if (lane < k) {
      if (MODE == kPerEdge && row[lane]) atomicAdd(&tri[own], row[lane]);
      key[slot] = kNone;
    }
    for (int i = 0; i < 4; ++i) sig[lane + 32 * i] = 0;
    __syncwarp();
  }
  dag_result<MODE>(c, hdr);
}

// One block per vertex u: key/idx a table of 2^hb >= 4k slots with 32 signature bits each, mat k bit rows of R words at an odd
// stride (per edge: k counters).  GLOBAL: they lie in global memory (written through L2, so read
// there too).
template <int MODE, bool GLOBAL, int T>
__device__ __forceinline__ void dag_vertex(uint32_t u, const uint32_t* __restrict__ ooff,
                                           const Entry<MODE>* __restrict__ nbr, uint32_t* __restrict__ tri,
                                           uint32_t* key, uint32_t* sig, uint16_t* idx, uint32_t* idx32,
                                           uint32_t* mat, uint32_t* s_next, unsigned long long& c) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t b = ooff[u], k = ooff[u + 1] - b;
  const uint32_t hb = 32 - __clz(4 * k - 1), mask = (1u << hb) - 1;
  const uint32_t R = (k + 31) / 32, RS = MODE == kPerEdge ? 1 : R | 1;
  auto ld = [](const uint32_t* p) { return GLOBAL ? __ldcg(p) : *p; };
  for (uint32_t i = threadIdx.x; i <= mask; i += T) {  // one signature word per table slot
    key[i] = kNone;
    sig[i] = 0;
  }
  if (MODE != kTri)
    for (uint64_t i = threadIdx.x; i < (uint64_t)k * RS; i += T) mat[i] = 0;
  if (threadIdx.x == 0) *s_next = 0;
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < k; i += T) {
    const uint32_t y = vertex_of(__ldg(&nbr[b + i])), s = vhash(y, hb + 5);
    uint32_t h = s >> 5;
    atomicOr(&sig[h], 1u << (s & 31));
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
      const uint32_t y = vertex_of(__ldg(&nbr[b + j0 + lane]));
      start = ooff[y];
      len = ooff[y + 1] - start;
    }
    stream_lists(nbr, start, len, [&](int j, Entry<MODE> ent) {
      const uint32_t x = vertex_of(ent), s = vhash(x, hb + 5);
      if (!(ld(&sig[s >> 5]) >> (s & 31) & 1)) return;
      for (uint32_t h = s >> 5;; h = (h + 1) & mask) {
        const uint32_t y = ld(&key[h]);
        if (y == x) {
          if (MODE != kClique) ++c;
          if (MODE != kTri) {
            const uint32_t i = GLOBAL ? __ldcg(&idx32[h]) : idx[h];
            if (MODE == kClique) {
              atomicOr(&mat[(uint64_t)(j0 + j) * RS + i / 32], 1u << (i & 31));
            } else {
              atomicAdd(&mat[j0 + j], 1u);
              atomicAdd(&mat[i], 1u);
              atomicAdd(&tri[edge_of(ent)], 1u);
            }
          }
          break;
        }
        if (y == kNone) break;
      }
    });
  }
  __syncthreads();
  if (MODE == kClique) {
    for (uint64_t i = threadIdx.x; i < (uint64_t)k * R; i += T) {
      const uint32_t v = (uint32_t)(i / R), q = (uint32_t)(i % R);
      const uint32_t* rv = mat + (uint64_t)v * RS;
      for (uint32_t bits = ld(&rv[q]); bits; bits &= bits - 1) {
        const uint32_t* rw = mat + (uint64_t)(q * 32 + __ffs(bits) - 1) * RS;
        for (uint32_t l = 0; l < R; ++l) c += __popc(ld(&rv[l]) & ld(&rw[l]));
      }
    }
    __syncthreads();
  } else if (MODE == kPerEdge) {
    for (uint32_t i = threadIdx.x; i < k; i += T) {
      const uint32_t n = ld(&mat[i]);
      if (n) atomicAdd(&tri[edge_of(__ldg(&nbr[b + i]))], n);
    }
    __syncthreads();
  }
}

// 32-bit words of a vertex's rows or counters
template <int MODE>
__host__ __device__ constexpr uint64_t row_words(uint64_t k) {
  return MODE == kClique ? k * ((k + 31) / 32 | 1) : MODE == kPerEdge ? k : 0;
}
template <int MODE, uint32_t KMAX>
constexpr size_t dag_smem() {
  return 10u * 4 * KMAX + 4 * row_words<MODE>(KMAX);
}

template <int MODE, uint32_t KMAX, int T>
__global__ void __launch_bounds__(T) k_dag_block(int cls, const uint32_t* __restrict__ list,
                                                 const uint32_t* __restrict__ ooff,
                                                 const Entry<MODE>* __restrict__ nbr, uint32_t* __restrict__ tri,
                                                 DagHdr* __restrict__ hdr) {
  extern __shared__ uint32_t smem[];
  __shared__ uint32_t s_item, s_next;
  uint32_t* key = smem;
  uint32_t* sig = smem + 4 * KMAX;
  uint32_t* mat = smem + 8 * KMAX;
  uint16_t* idx = (uint16_t*)(mat + row_words<MODE>(KMAX));
  const uint32_t count = hdr->n[cls];
  unsigned long long c = 0;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(&hdr->next[cls], 1u);
    __syncthreads();
    const uint32_t item = s_item;
    if (item >= count) break;
    dag_vertex<MODE, false, T>(list[item], ooff, nbr, tri, key, sig, idx, nullptr, mat, &s_next, c);
    __syncthreads();
  }
  dag_result<MODE>(c, hdr);
}

// Vertices of more than kBig members, tables and rows in a slab of `slab` words per block.
template <int MODE, int T>
__global__ void __launch_bounds__(T) k_dag_global(const uint32_t* __restrict__ list, const uint32_t* __restrict__ ooff,
                                                  const Entry<MODE>* __restrict__ nbr, uint32_t* __restrict__ tri,
                                                  uint32_t* __restrict__ slabs, uint64_t slab, uint32_t table,
                                                  DagHdr* __restrict__ hdr) {
  __shared__ uint32_t s_item, s_next;
  uint32_t* key = slabs + blockIdx.x * slab;
  const uint32_t count = hdr->n[3];
  unsigned long long c = 0;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(&hdr->next[3], 1u);
    __syncthreads();
    const uint32_t item = s_item;
    if (item >= count) break;
    dag_vertex<MODE, true, T>(list[item], ooff, nbr, tri, key, key + table, nullptr, key + 2ull * table,
                              key + 3ull * table, &s_next, c);
    __syncthreads();
  }
  dag_result<MODE>(c, hdr);
}

// per-vertex degree terms and per-edge (d_u - 1)(d_v - 1)
__global__ void __launch_bounds__(kB) k_degree_terms(ZgDevGraph g, int kind, U128* __restrict__ sum) {
  U128 acc = {0, 0};
  uint64_t tid = blockIdx.x * (uint64_t)kB + threadIdx.x, stride = (uint64_t)gridDim.x * kB;
  if (kind == ZG_EXACT_THREE_PATH) {
    for (uint64_t e = tid; e < g.m; e += stride) {
      uint4 r = zg_rec_e(g, e);
      add128(acc, (uint64_t)(deg(g, r.x) - 1) * (deg(g, r.y) - 1));
    }
  } else {
    for (uint64_t v = tid; v < g.nv; v += stride) {
      uint64_t d = deg(g, (uint32_t)v);
      if (kind == ZG_EXACT_WEDGE) add128(acc, d * (d - 1) / 2);
      else if (d >= 4) add128w(acc, (unsigned __int128)d * (d - 1) * (d - 2) * (d - 3) / 24);
    }
  }
  add_sum(acc, sum);
}

int read_back(void* dst, const void* src, size_t bytes, cudaStream_t s) {
  cudaError_t ce = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s);
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(s);
  if (ce == cudaSuccess) ce = cudaGetLastError();
  return zg_check_cuda(ce, "exact count kernel");
}

unsigned __int128 wide(const U128& a) { return ((unsigned __int128)a.hi << 64) | a.lo; }

int grid_over(uint64_t n) {
  return (int)std::max<uint64_t>(1, std::min<uint64_t>((n + kB - 1) / kB, (uint64_t)zg_num_sms() * 8));
}

// The most vertices a class can have: each has an edge of its own (two in the out-lists' classes), so
// graphs of few edges among many ids take little.
uint64_t class_room(uint64_t m, uint32_t nv) { return std::min<uint64_t>(m, nv); }

template <int MODE>
int dag_launch(uint64_t room, const uint32_t* lists, const uint32_t* ooff, const Entry<MODE>* nbr, uint32_t* tri,
               DagHdr* hdr, cudaStream_t s) {
  constexpr int TM = 256, TB = 512;
  constexpr size_t sm = dag_smem<MODE, kMid>(), sb = dag_smem<MODE, kBig>();
  cudaError_t e = cudaFuncSetAttribute(k_dag_block<MODE, kBig, TB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sb);
  if (e != cudaSuccess) return zg_check_cuda(e, "exact count kernel");
  const int sms = zg_num_sms();
  // the largest vertices first: one of them is the longest single piece of work
  k_dag_block<MODE, kBig, TB><<<sms, TB, sb, s>>>(2, lists + 2 * room, ooff, nbr, tri, hdr);
  k_dag_block<MODE, kMid, TM><<<sms * 8, TM, sm, s>>>(1, lists + room, ooff, nbr, tri, hdr);
  k_dag_warp<MODE><<<sms * 8, kB, 0, s>>>(lists, ooff, nbr, tri, hdr);
  return ZG_OK;
}

// `words` 32-bit words for each of up to `want` blocks, within a quarter of the free memory.
int slab_blocks(uint64_t want, uint64_t words, ZgScratch& slabs, uint64_t* blocks) {
  size_t free_b = 0, total_b = 0;
  const cudaError_t e = cudaMemGetInfo(&free_b, &total_b);
  if (e != cudaSuccess) return zg_check_cuda(e, "exact count scratch");
  *blocks = std::max<uint64_t>(1, std::min<uint64_t>(want, (free_b / 4) / (4 * words)));
  return slabs.alloc(4 * words * *blocks);
}

// The vertices past kBig.
template <int MODE>
int dag_launch_global(const DagHdr& h, const uint32_t* list, const uint32_t* ooff, const Entry<MODE>* nbr,
                      uint32_t* tri, DagHdr* hdr, cudaStream_t s) {
  uint32_t table = 1;
  while (table < 4 * h.kmax) table <<= 1;
  const uint64_t slab = 3ull * table + row_words<MODE>(h.kmax);
  ZgScratch slabs(s);
  uint64_t blocks = 0;
  if (int rc = slab_blocks(std::min<uint64_t>(h.n[3], (uint64_t)zg_num_sms() * 2), slab, slabs, &blocks)) return rc;
  k_dag_global<MODE, 512><<<(int)blocks, 512, 0, s>>>(list, ooff, nbr, tri, (uint32_t*)slabs.p, slab, table, hdr);
  return ZG_OK;
}

// Where the pass over the out-lists keeps its arrays: the (lower, higher) ends and the place of every
// edge, the out-lists and their offsets, the class lists.  `bytes` is the last offset; what a caller
// takes before `edges` survives a reuse of the rest.
template <int MODE>
struct DagArrays {
  size_t hdr, outdeg, ooff, lists, tmp, tmp_bytes = 0, edges, ab, slot, nbr;
  DagArrays(ZgCarve& c, uint64_t m, uint32_t nv, cudaStream_t s) {
    const size_t nv1 = (size_t)nv + 1;
    cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, (uint32_t*)nullptr, (uint32_t*)nullptr, (int64_t)nv1, s);
    hdr = c.take(sizeof(DagHdr));
    outdeg = c.take(4 * nv1);
    ooff = c.take(4 * nv1);
    lists = c.take(4ull * kClasses * class_room(m, nv));
    tmp = c.take(tmp_bytes);
    edges = ab = c.take(8 * m);
    slot = c.take(4 * m);
    nbr = c.take(sizeof(Entry<MODE>) * m);
  }
};

// The pass over the degree-oriented out-lists of the edges that pass the predicate (pred 0: every
// edge); tri (kPerEdge): zeroed counters per edge.  *out (may be null) gets the count.
template <int MODE>
int dag_run(const zg_graph* g, int pred, uint32_t t, char* p, DagArrays<MODE> a, uint32_t* tri, cudaStream_t s,
            unsigned __int128* out) {
  const uint64_t m = g->d.m;
  const uint32_t nv = g->d.nv;
  DagHdr* hdr = (DagHdr*)(p + a.hdr);
  uint32_t *outdeg = (uint32_t*)(p + a.outdeg), *ooff = (uint32_t*)(p + a.ooff), *slot = (uint32_t*)(p + a.slot),
           *lists = (uint32_t*)(p + a.lists);
  Entry<MODE>* nbr = (Entry<MODE>*)(p + a.nbr);
  uint2* ab = (uint2*)(p + a.ab);
  const uint64_t room = class_room(m, nv);
  cudaMemsetAsync(p + a.hdr, 0, a.ooff - a.hdr, s);  // the header and the out-degrees
  k_orient<<<grid_over(m), kB, 0, s>>>(g->d, pred, t, ab, slot, outdeg);
  cub::DeviceScan::ExclusiveSum(p + a.tmp, a.tmp_bytes, outdeg, ooff, (int64_t)nv + 1, s);
  k_fill<<<grid_over(m), kB, 0, s>>>(m, nv, ab, slot, ooff, nbr, lists, room, hdr);
  int rc = dag_launch<MODE>(room, lists, ooff, nbr, tri, hdr, s);
  if (rc) return rc;
  DagHdr h;
  if ((rc = read_back(&h, hdr, sizeof(h), s))) return rc;
  if (h.n[3]) {
    if ((rc = dag_launch_global<MODE>(h, lists + 3 * room, ooff, nbr, tri, hdr, s)) ||
        (out && (rc = read_back(&h, hdr, sizeof(h), s))))
      return rc;
  }
  if (out) *out = wide(h.sum);
  return ZG_OK;
}

template <int MODE>
int dag_count(const zg_graph* g, int pred, uint32_t t, cudaStream_t s, unsigned __int128* out) {
  *out = 0;
  if (g->d.m == 0) return ZG_OK;
  ZgCarve c;
  const DagArrays<MODE> a(c, g->d.m, g->d.nv, s);
  ZgScratch pool(s);
  if (int rc = pool.alloc(c.at)) return rc;
  return dag_run<MODE>(g, pred, t, (char*)pool.p, a, nullptr, s, out);
}

int count_triangles(const zg_graph* g, int pred, uint32_t t, cudaStream_t s, unsigned __int128* out) {
  return dag_count<kTri>(g, pred, t, s, out);
}

// ---- houses and 4-edge paths -------------------------------------------------------------------
// The vertices in an order by degree: ranks go up through 256 buckets of degree (exact below 16,
// eight to an octave above), in any order within a bucket.
__device__ __forceinline__ uint32_t degree_bucket(uint32_t d) {
  if (d < 16) return d;
  const uint32_t l = 31 - __clz(d);
  return 16 + (l - 4) * 8 + ((d >> (l - 3)) & 7);  // at most 16 + 27 * 8 + 7 = 239
}

struct WedgeHdr {
  U128 sum;    // over the wedges
  U128 tt;     // sum of t(e)^2 (houses) or t(e) (d_a + d_b - 3) (paths)
  U128 t;      // sum of t(e)
  U128 s;      // sum over the vertices of S1^2 - S2 (paths)
  uint32_t hist[256], cursor[256];
  uint32_t n[kClasses], next[kClasses];
};

__global__ void __launch_bounds__(kB) k_degree_hist(ZgDevGraph g, WedgeHdr* __restrict__ hdr) {
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  for (uint64_t v = blockIdx.x * (uint64_t)kB + threadIdx.x; v < g.nv; v += (uint64_t)gridDim.x * kB)
    atomicAdd(&h[degree_bucket(deg(g, (uint32_t)v))], 1u);
  __syncthreads();
  if (h[threadIdx.x]) atomicAdd(&hdr->hist[threadIdx.x], h[threadIdx.x]);
}

__global__ void __launch_bounds__(kB) k_degree_rank(ZgDevGraph g, uint32_t* __restrict__ rank,
                                                    WedgeHdr* __restrict__ hdr) {
  __shared__ uint32_t base[256], h[256];
  // where each bucket starts, then this block's vertices counted, their places reserved, and given out
  base[threadIdx.x] = hdr->hist[threadIdx.x];
  h[threadIdx.x] = 0;
  __syncthreads();
  for (int o = 1; o < 256; o <<= 1) {
    const uint32_t v = threadIdx.x >= o ? base[threadIdx.x - o] : 0u;
    __syncthreads();
    base[threadIdx.x] += v;
    __syncthreads();
  }
  const uint64_t per = ((uint64_t)g.nv + gridDim.x - 1) / gridDim.x;
  const uint64_t lo = blockIdx.x * per, end = lo + per, hi = end < g.nv ? end : g.nv;
  for (uint64_t v = lo + threadIdx.x; v < hi; v += kB) atomicAdd(&h[degree_bucket(deg(g, (uint32_t)v))], 1u);
  __syncthreads();
  const uint32_t start = base[threadIdx.x] - hdr->hist[threadIdx.x];
  const uint32_t got = h[threadIdx.x] ? start + atomicAdd(&hdr->cursor[threadIdx.x], h[threadIdx.x]) : 0u;
  __syncthreads();
  h[threadIdx.x] = got;
  __syncthreads();
  for (uint64_t v = lo + threadIdx.x; v < hi; v += kB)
    rank[v] = atomicAdd(&h[degree_bucket(deg(g, (uint32_t)v))], 1u);
}

// The edge-id-ordered adjacency as (rank of the neighbour, edge id), and per vertex the wedges that
// start at it, at most: the degrees of its neighbours of lower rank, each less one for itself (at most 2m), with
// the number of those neighbours that start any from bit kWedgeBits on.  above: the degrees, less one, of the
// neighbours of higher rank (where given).
constexpr int kWedgeBits = 33;
constexpr unsigned long long kWedgeMask = (1ull << kWedgeBits) - 1;
__global__ void __launch_bounds__(kB) k_rank_adj(ZgDevGraph g, const uint32_t* __restrict__ rank,
                                                 uint2* __restrict__ radj, unsigned long long* __restrict__ wedges,
                                                 unsigned long long* __restrict__ above) {
  const uint64_t tid = blockIdx.x * (uint64_t)kB + threadIdx.x, stride = (uint64_t)gridDim.x * kB;
  for (uint64_t i = tid; i < 2 * g.m; i += stride) {
    const uint2 a = g.adj_e[i];
    radj[i] = make_uint2(rank[a.x], a.y);
  }
  for (uint64_t e = tid; e < g.m; e += stride) {
    const uint4 r = zg_rec_e(g, e);
    const bool up = rank[r.x] < rank[r.y];
    const uint32_t lo = up ? r.x : r.y, hi = up ? r.y : r.x, w = deg(g, lo) - 1;
    if (w) atomicAdd(&wedges[hi], (1ull << kWedgeBits) | w);
    if (above) atomicAdd(&above[lo], (unsigned long long)(deg(g, hi) - 1));
  }
}

// Classes by the larger of the wedges W at a vertex and its degree (the wedges of one neighbour close
// nothing, so a star's hub is in none): one warp with a
// 512-slot table up to 256; one block with the counters in shared memory, directly by rank where
// the whole graph's fit, else in a table, up to 2 048 and up to 8 192; beyond that one block with
// counters by rank, in global memory where they do not fit a block.  A warp's table is 4 KB, a block's
// 32 KB (six a SM) and 128 KB (one a SM); each is at most half full.  Bound by the wedges' additions and
// the gathers of t; ms, houses / 4-edge paths, per-edge list intersections by binary search -> this:
//   R-MAT scale 13 ef 12 (79 k edges)   37.3 -> 0.31 / 37.7 -> 0.27
//   R-MAT scale 14 ef 12 (165 k)         124 -> 0.48 / 123 -> 0.39
//   R-MAT scale 20 ef 3 (3.1 M)         not run -> 14.3 / 13.4
//   uniform random, 10^6 vertices, 2 M  0.68 -> 0.61 / 2.29 -> 0.64
//   grid of 1000 x 1000 (no triangle)   0.70 -> 0.31 / 1.97 -> 0.77
//   10^6 leaves on a hub, one triangle  0.85 -> 1.17 / 7.55 -> 1.2
// The last is the one that lost: all of a hub's neighbours go through one block, which looks at each twice.
constexpr uint32_t kWedge0 = 256, kWedge1 = 2048, kWedge2 = 8192;
constexpr uint32_t kDense = 24 << 10;  // vertices whose counters fit (96 KB: two blocks a SM)

__global__ void __launch_bounds__(kB) k_wedge_class(ZgDevGraph g, const unsigned long long* __restrict__ wedges,
                                                    uint32_t* __restrict__ lists, uint64_t room,
                                                    WedgeHdr* __restrict__ hdr) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t tid = blockIdx.x * (uint64_t)kB + threadIdx.x, stride = (uint64_t)gridDim.x * kB;
  for (uint64_t v0 = tid - lane; v0 < g.nv; v0 += stride) {
    const uint64_t v = v0 + lane;
    unsigned long long w = v < g.nv ? wedges[v] : 0ull;
    const bool closes = (w >> kWedgeBits) >= 2;
    if (closes) w = max(w & kWedgeMask, (unsigned long long)deg(g, (uint32_t)v));
    const int cls = !closes ? -1 : w <= kWedge0 ? 0 : w <= kWedge1 ? 1 : w <= kWedge2 ? 2 : 3;
#pragma unroll
    for (int c = 0; c < kClasses; ++c) {
      const unsigned in = __ballot_sync(0xffffffffu, cls == c);
      if (!in) continue;
      uint32_t at = 0;
      if (lane == 0) at = atomicAdd(&hdr->n[c], (uint32_t)__popc(in));
      at = __shfl_sync(0xffffffffu, at, 0);
      if (cls == c) lists[c * room + at + __popc(in & ((1u << lane) - 1))] = (uint32_t)v;
    }
  }
}

// The wedge counters of one vertex: a table of (rank, count) slots, or one count per rank in shared
// or global memory (the latter read where its additions are made, in L2).
enum { kTable, kShared, kGlobal };
template <int TAB>
struct Counters {
  uint32_t *key, *cnt;
  uint32_t bits;
  __device__ __forceinline__ void add(uint32_t r) const {
    if (TAB != kTable) {
      atomicAdd(&cnt[r], 1u);
      return;
    }
    const uint32_t mask = (1u << bits) - 1;
    uint32_t h = vhash(r, bits);
    for (;; h = (h + 1) & mask) {  // at most half of the slots are taken
      const uint32_t k = key[h];
      if (k == r) break;
      if (k != kNone) continue;
      const uint32_t was = atomicCAS(&key[h], kNone, r);
      if (was == kNone || was == r) break;
    }
    atomicAdd(&cnt[h], 1u);
  }
  __device__ __forceinline__ uint32_t get(uint32_t r) const {
    if (TAB == kGlobal) return __ldcg(&cnt[r]);
    if (TAB == kShared) return cnt[r];
    uint32_t h = vhash(r, bits);
    while (key[h] != r) h = (h + 1) & ((1u << bits) - 1);  // it was added
    return cnt[h];
  }
};

// The wedges through up to 32 neighbours of a: lane j's is entry `at` of the adjacency (its list is
// empty when it comes after a or among the `leaves` lowest ranks, those of degree 1 and below); te[j] gets
// t(a, x) where tri is given.  body(j, (rank of y, edge)).
template <class F>
__device__ __forceinline__ void wedges_of(const ZgDevGraph& g, const uint2* __restrict__ radj, bool in, uint32_t at,
                                          uint32_t ra, uint32_t leaves, const uint32_t* __restrict__ tri,
                                          uint32_t* te, F&& body) {
  uint32_t start = 0, len = 0;
  if (in) {
    const uint2 r = __ldg(&radj[at]);
    if (r.x < ra && r.x >= leaves) {
      const uint32_t x = __ldg(&g.adj_e[at]).x;
      start = g.off32[x];
      len = g.off32[x + 1] - start;
      if (tri) te[threadIdx.x & 31] = tri[r.y];
    }
  }
  if (!__any_sync(0xffffffffu, len)) return;
  __syncwarp();
  stream_lists(radj, start, len, [&](int j, uint2 y) {
    if (y.x < ra) body(j, y);
  });
  __syncwarp();
}

// A wedge's term once the counts are complete.
template <bool HOUSE, int TAB>
__device__ __forceinline__ void wedge_term(const Counters<TAB>& tab, uint2 y, uint32_t ta,
                                           const uint32_t* __restrict__ tri, U128& acc) {
  const uint32_t c = tab.get(y.x) - 1;
  if (!c) return;
  add128(acc, HOUSE ? (unsigned long long)c * ((unsigned long long)ta + __ldg(&tri[y.y])) : (unsigned long long)c);
}

template <bool HOUSE>
__global__ void __launch_bounds__(kB) k_wedge_warp(ZgDevGraph g, const uint32_t* __restrict__ list,
                                                   const uint32_t* __restrict__ rank, const uint2* __restrict__ radj,
                                                   const uint32_t* __restrict__ tri, WedgeHdr* __restrict__ hdr) {
  __shared__ uint32_t s_key[kB / 32][2 * kWedge0], s_cnt[kB / 32][2 * kWedge0], s_te[kB / 32][32];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Counters<kTable> tab{s_key[warp], s_cnt[warp], 9};
  uint32_t* te = s_te[warp];
  const uint32_t count = hdr->n[0], leaves = hdr->hist[0] + hdr->hist[1];
  U128 acc = {0, 0};
  for (uint32_t w = blockIdx.x * (kB / 32) + warp; w < count; w += gridDim.x * (kB / 32)) {
    const uint32_t a = list[w], ra = rank[a], b = g.off32[a], d = g.off32[a + 1] - b;
    for (uint32_t i = lane; i < 2 * kWedge0; i += 32) {
      tab.key[i] = kNone;
      tab.cnt[i] = 0;
    }
    __syncwarp();
    for (uint32_t j0 = 0; j0 < d; j0 += 32)
      wedges_of(g, radj, j0 + lane < d, b + j0 + lane, ra, leaves, nullptr, te, [&](int, uint2 y) { tab.add(y.x); });
    for (uint32_t j0 = 0; j0 < d; j0 += 32)
      wedges_of(g, radj, j0 + lane < d, b + j0 + lane, ra, leaves, HOUSE ? tri : nullptr, te,
                [&](int j, uint2 y) { wedge_term<HOUSE>(tab, y, HOUSE ? te[j] : 0u, tri, acc); });
  }
  add_sum(acc, &hdr->sum);
}

// The classes from cls down to last in one launch: with a launch for each, the blocks without one of the
// longest vertices waited for those before the next class began.  Counters in shared memory, us, houses /
// 4-edge paths: R-MAT scale 12 ef 12 266 / 244 -> 241 / 227, scale 13 ef 12 329 / 305 -> 306 / 288,
// scale 14 ef 12 508 / 438 -> 489 / 420.
template <bool HOUSE, int TAB, int T>
__global__ void __launch_bounds__(T) k_wedge_block(ZgDevGraph g, int cls, int last,
                                                   const uint32_t* __restrict__ lists, uint64_t room,
                                                   const uint32_t* __restrict__ rank, const uint2* __restrict__ radj,
                                                   const uint32_t* __restrict__ tri, uint32_t bits,
                                                   uint32_t* __restrict__ slabs, WedgeHdr* __restrict__ hdr) {
  extern __shared__ uint4 smem4[];
  __shared__ uint32_t s_item, s_next[2], s_te[T / 32][32];
  const uint32_t lane = threadIdx.x & 31;
  uint32_t* te = s_te[threadIdx.x >> 5];
  uint32_t* smem = (uint32_t*)smem4;
  const uint32_t leaves = hdr->hist[0] + hdr->hist[1];
  const Counters<TAB> tab{smem, TAB == kGlobal ? slabs + (uint64_t)blockIdx.x * g.nv
                                : TAB == kTable ? smem + (1u << bits) : smem, bits};
  U128 acc = {0, 0};
  for (;;) {
    if (threadIdx.x == 0) {
      s_item = atomicAdd(&hdr->next[cls], 1u);
      s_next[0] = s_next[1] = 0;
    }
    __syncthreads();
    const uint32_t item = s_item;
    if (item >= hdr->n[cls]) {  // the next class, once every thread has read this item
      if (cls-- == last) break;
      __syncthreads();
      continue;
    }
    const uint32_t a = lists[cls * room + item], ra = rank[a], b = g.off32[a], d = g.off32[a + 1] - b;
    if (TAB == kShared)
      for (uint32_t i = threadIdx.x; i < (ra + 3) / 4; i += T) smem4[i] = make_uint4(0, 0, 0, 0);
    if (TAB == kTable)
      for (uint32_t i = threadIdx.x; i < 1u << bits; i += T) {
        tab.key[i] = kNone;
        tab.cnt[i] = 0;
      }
    __syncthreads();
    const uint32_t step = d < 4 * T ? 8 : 32;  // neighbours at a time per warp
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      for (;;) {
        uint32_t j0 = 0;
        if (lane == 0) j0 = atomicAdd(&s_next[pass], step);
        j0 = __shfl_sync(0xffffffffu, j0, 0);
        if (j0 >= d) break;
        const bool in = lane < step && j0 + lane < d;
        if (pass == 0)
          wedges_of(g, radj, in, b + j0 + lane, ra, leaves, nullptr, te, [&](int, uint2 y) { tab.add(y.x); });
        else
          wedges_of(g, radj, in, b + j0 + lane, ra, leaves, HOUSE ? tri : nullptr, te,
                    [&](int j, uint2 y) { wedge_term<HOUSE>(tab, y, HOUSE ? te[j] : 0u, tri, acc); });
      }
      __syncthreads();
    }
    if (TAB == kGlobal) {  // back to zero, each warp the neighbours it comes to
      for (uint32_t j0 = threadIdx.x / 32 * step; j0 < d; j0 += T / 32 * step)
        wedges_of(g, radj, lane < step && j0 + lane < d, b + j0 + lane, ra, leaves, nullptr, te,
                  [&](int, uint2 y) { __stcg(&tab.cnt[y.x], 0u); });
      __syncthreads();
    }
  }
  add_sum(acc, &hdr->sum);
}

// The per-edge terms, and for the paths the per-vertex ones: S1(v) is what k_rank_adj found below and above
// v, and the sum of S2 over the vertices has d_w (d_w - 1)^2 from each w.
template <bool HOUSE>
__global__ void __launch_bounds__(kB) k_house_chain_terms(ZgDevGraph g, const uint32_t* __restrict__ tri,
                                                          const unsigned long long* __restrict__ wedges,
                                                          const unsigned long long* __restrict__ above,
                                                          WedgeHdr* __restrict__ hdr) {
  U128 tt = {0, 0}, t = {0, 0}, sv = {0, 0};
  const uint64_t tid = blockIdx.x * (uint64_t)kB + threadIdx.x, stride = (uint64_t)gridDim.x * kB;
  for (uint64_t e = tid; e < g.m; e += stride) {
    const uint64_t n = tri[e];
    if (!n) continue;
    if (HOUSE) {
      add128(t, n);
      add128(tt, n * n);
    } else {  // both ends of an edge of a triangle have degree 2 at least
      const uint4 r = zg_rec_e(g, e);
      add128w(tt, (unsigned __int128)n * ((uint64_t)deg(g, r.x) + deg(g, r.y) - 3));
    }
  }
  add_sum(tt, &hdr->tt);
  if (HOUSE) {
    add_sum(t, &hdr->t);
  } else {
    for (uint64_t v = tid; v < g.nv; v += stride) {
      const unsigned long long s1 = (wedges[v] & kWedgeMask) + above[v], d = deg(g, (uint32_t)v);  // s1 at most 2m
      add128w(sv, (unsigned __int128)s1 * s1);
      if (d) add128w(sv, ~((unsigned __int128)((d - 1) * (d - 1)) * d) + 1);
    }
    add_sum(sv, &hdr->s);
  }
}

constexpr uint32_t kSmallEdges = 20 << 10, kSmallVertices = 12 << 10;  // 48 KB of counters, and a little beside
constexpr uint64_t kSmallHub = 2048;  // the largest degree, as the graph's metadata has it (a hint here)
// A small graph in one launch: per vertex a (one block) the common-neighbour counts cnt(y) of a and
// every y by walking all two-step paths, so t(a, b) = cnt(b) and c4(a, b) = sum over y in N(b) of
// cnt(y), less d_a + d_b - 1 (y = a, and a itself in each of the others).  sum_v d^2 additions instead
// of sum_e min(d), but no order, no lists and no triangle pass: sixteen launches fewer.  Houses, us,
// this way / the other: R-MAT scale 8 ef 3 (620 edges) 28 / 140, scale 11 ef 12 (18 k) 96 / 201; with a warp
// for each neighbour, before, scale 12 ef 6 (20.7 k) took 169 / 190, scale 13 ef 3 (22.4 k) 218 / 194, and
// the line was drawn just below.
// A warp takes its share of a's neighbours, up to 32, at a time, their lists laid end to end: one warp for
// each neighbour took 1.72 ms on a star of 12 000 leaves, a chain of 1 500 reads.  Two-step paths through a
// hub and hubs in one block still cost most, so large degrees go the other way, this way / the other:
// houses and 4-edge paths, us, on that star 59 / 55 and 70 / 101, with 3 000 triangles on its leaves 268 /
// 147 and 385 / 160, on K(2, 10 000) 572 / 55 and 896 / 145; a star of 1 500 leaves takes 28 this way.  No
// graph was measured with its largest degree between.
template <bool HOUSE>
__global__ void __launch_bounds__(kB) k_house_chain_small(ZgDevGraph g, U128* __restrict__ sum) {
  extern __shared__ uint4 smem4[];
  __shared__ unsigned long long s_s1;
  __shared__ uint32_t s_te[kB / 32][32];
  uint32_t* cnt = (uint32_t*)smem4;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t* te = s_te[warp];
  U128 acc = {0, 0};  // signed terms, two's complement
  for (uint32_t a = blockIdx.x; a < g.nv; a += gridDim.x) {
    const uint32_t b0 = g.off32[a], d = g.off32[a + 1] - b0;
    if (d < 2) continue;  // no path or cycle turns at a
    for (uint32_t i = threadIdx.x; i < (g.nv + 3) / 4; i += kB) smem4[i] = make_uint4(0, 0, 0, 0);
    if (threadIdx.x == 0) s_s1 = 0;
    __syncthreads();
    const uint32_t step = min(32u, (d + kB / 32 - 1) / (kB / 32));
    auto lists = [&](uint32_t start, uint32_t len, auto&& body) {
      if (step > 1) return stream_lists(g.adj_e, start, len, body);
      const uint32_t s = __shfl_sync(0xffffffffu, start, 0), n = __shfl_sync(0xffffffffu, len, 0);
      for (uint32_t j = lane; j < n; j += 32) body(0, g.adj_e[s + j]);
    };
    unsigned long long s1 = 0;
    for (uint32_t i0 = warp * step; i0 < d; i0 += kB / 32 * step) {
      uint32_t start = 0, len = 0;
      if (lane < step && i0 + lane < d) {
        const uint32_t x = g.adj_e[b0 + i0 + lane].x;
        start = g.off32[x];
        len = g.off32[x + 1] - start;
        if (!HOUSE) {
          s1 += len - 1;
          add128w(acc, ~(unsigned __int128)((unsigned long long)(len - 1) * (len - 1)) + 1);
        }
      }
      lists(start, len, [&](int, uint2 y) { atomicAdd(&cnt[y.x], 1u); });
    }
    if (!HOUSE) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s1 += __shfl_xor_sync(0xffffffffu, s1, o);
      if (lane == 0 && s1) atomicAdd(&s_s1, s1);
    }
    __syncthreads();
    unsigned long long c = 0;  // the sum over b of t(a, b) times cnt over N(b), for paths of cnt alone
    for (uint32_t i0 = warp * step; i0 < d; i0 += kB / 32 * step) {
      uint32_t start = 0, len = 0;
      if (lane < step && i0 + lane < d) {
        const uint32_t b = g.adj_e[b0 + i0 + lane].x;
        const uint32_t t = b > a ? cnt[b] : 0u;
        te[lane] = t;
        if (b > a && (!HOUSE || t)) {
          start = g.off32[b];
          len = g.off32[b + 1] - start;
          const __int128 off_c4 = (__int128)d + len - 1;
          add128w(acc, (unsigned __int128)(HOUSE ? -(__int128)t * off_c4 - 2 * (__int128)t * t + 2 * (__int128)t
                                                 : 2 * (__int128)t * (3 - (__int128)d - len) + 2 * off_c4));
        }
      }
      __syncwarp();
      lists(start, len, [&](int j, uint2 y) { c += HOUSE ? (unsigned long long)te[j] * cnt[y.x] : cnt[y.x]; });
      __syncwarp();
    }
    add128w(acc, HOUSE ? (unsigned __int128)c : ~(2 * (unsigned __int128)c) + 1);
    if (!HOUSE && threadIdx.x == 0) add128w(acc, (unsigned __int128)s_s1 * s_s1);
    __syncthreads();
  }
  add_sum(acc, sum);
}

template <bool HOUSE>
int wedge_launch(const zg_graph* g, const uint32_t* lists, const uint32_t* rank, const uint2* radj,
                 const uint32_t* tri, WedgeHdr* hdr, cudaStream_t s) {
  const uint32_t nv = g->d.nv;
  const uint64_t room = class_room(g->d.m, nv);
  const int sms = zg_num_sms();
  cudaError_t e;
  const bool dense = nv <= kDense;
  if (dense) {
    // the limit belongs to the kernel, not to the call: always the largest, as another thread may be
    // about to launch on a larger graph
    constexpr int most = 4 * kDense;
    if ((e = cudaFuncSetAttribute(k_wedge_block<HOUSE, kShared, 1024>, cudaFuncAttributeMaxDynamicSharedMemorySize, most)) ||
        (e = cudaFuncSetAttribute(k_wedge_block<HOUSE, kShared, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize, most)))
      return zg_check_cuda(e, "exact count kernel");
    const size_t sm = ((size_t)nv + 3) / 4 * 16;
    const int fit = (int)std::max<size_t>(1, std::min<size_t>(8, (216 << 10) / (sm + 3072)));
    k_wedge_block<HOUSE, kShared, 1024><<<sms * std::min(2, fit), 1024, sm, s>>>(g->d, 3, 2, lists, room, rank, radj,
                                                                                 tri, 0, nullptr, hdr);
    k_wedge_block<HOUSE, kShared, 256><<<sms * fit, 256, sm, s>>>(g->d, 1, 1, lists, room, rank, radj, tri, 0, nullptr, hdr);
  } else {
    WedgeHdr h;
    if (int rc = read_back(&h, hdr, sizeof(h), s)) return rc;
    if (h.n[3]) {
      ZgScratch slabs(s);
      uint64_t blocks = 0;
      if (int rc = slab_blocks(std::min<uint64_t>(h.n[3], (uint64_t)sms * 2), nv, slabs, &blocks)) return rc;
      cudaMemsetAsync(slabs.p, 0, 4 * blocks * nv, s);
      k_wedge_block<HOUSE, kGlobal, 1024><<<(int)blocks, 1024, 0, s>>>(g->d, 3, 3, lists, room, rank, radj, tri, 0,
                                                                       (uint32_t*)slabs.p, hdr);
    }
    const size_t s2 = 16 * kWedge2, s1 = 16 * kWedge1;
    if ((e = cudaFuncSetAttribute(k_wedge_block<HOUSE, kTable, 512>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s2)))
      return zg_check_cuda(e, "exact count kernel");
    if (h.n[2])
      k_wedge_block<HOUSE, kTable, 512><<<sms, 512, s2, s>>>(g->d, 2, 2, lists, room, rank, radj, tri, 14, nullptr, hdr);
    if (h.n[1])
      k_wedge_block<HOUSE, kTable, 256><<<sms * 6, 256, s1, s>>>(g->d, 1, 1, lists, room, rank, radj, tri, 12, nullptr, hdr);
  }
  k_wedge_warp<HOUSE><<<sms * 6, kB, 0, s>>>(g->d, lists, rank, radj, tri, hdr);
  return ZG_OK;
}

template <bool HOUSE>
int house_chain(const zg_graph* g, cudaStream_t s, unsigned __int128* out) {
  const uint64_t m = g->d.m;
  const uint32_t nv = g->d.nv;
  *out = 0;
  if (m == 0) return ZG_OK;
  if (m <= kSmallEdges && nv <= kSmallVertices && g->max_degree < kSmallHub) {
    ZgScratch sum(s);
    int rc = sum.alloc(sizeof(U128));
    if (rc) return rc;
    cudaMemsetAsync(sum.p, 0, sizeof(U128), s);
    // always for the most vertices: the limit belongs to the kernel, not to the call
    const cudaError_t e = cudaFuncSetAttribute(k_house_chain_small<HOUSE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               4 * kSmallVertices);
    if (e != cudaSuccess) return zg_check_cuda(e, "exact count kernel");
    k_house_chain_small<HOUSE><<<(int)std::min<uint32_t>(nv, zg_num_sms() * 4), kB, ((size_t)nv + 3) / 4 * 16, s>>>(
        g->d, (U128*)sum.p);
    U128 h;
    if ((rc = read_back(&h, sum.p, sizeof(h), s))) return rc;
    *out = HOUSE ? wide(h) : (unsigned __int128)((__int128)wide(h) / 2);
    return ZG_OK;
  }
  ZgCarve c;
  const size_t o_hdr = c.take(sizeof(WedgeHdr)), o_wedges = c.take(8ull * nv), o_tri = c.take(4 * m), o_above = c.take(HOUSE ? 0 : 8ull * nv),
               o_rank = c.take(4ull * nv), o_lists = c.take(4ull * kClasses * class_room(m, nv));
  const DagArrays<kPerEdge> a(c, m, nv, s);
  const size_t o_radj = a.edges;  // 16 of the 20 bytes per edge the triangle pass is then done with
  ZgScratch pool(s);
  int rc = pool.alloc(c.at);
  if (rc) return rc;
  char* p = (char*)pool.p;
  WedgeHdr* hdr = (WedgeHdr*)(p + o_hdr);
  unsigned long long* wedges = (unsigned long long*)(p + o_wedges);
  uint32_t *tri = (uint32_t*)(p + o_tri), *rank = (uint32_t*)(p + o_rank), *lists = (uint32_t*)(p + o_lists);
  unsigned long long* above = HOUSE ? nullptr : (unsigned long long*)(p + o_above);
  uint2* radj = (uint2*)(p + o_radj);
  cudaMemsetAsync(p + o_hdr, 0, o_rank - o_hdr, s);  // the header and every count
  // without a triangle there is no house
  unsigned __int128 triangles = 0;
  if ((rc = dag_run<kPerEdge>(g, 0, 0, p, a, tri, s, HOUSE ? &triangles : nullptr)) || (HOUSE && !triangles)) return rc;
  k_degree_hist<<<grid_over(nv), kB, 0, s>>>(g->d, hdr);
  k_degree_rank<<<grid_over(nv), kB, 0, s>>>(g->d, rank, hdr);
  k_rank_adj<<<grid_over(2 * m), kB, 0, s>>>(g->d, rank, radj, wedges, above);
  k_wedge_class<<<grid_over(nv), kB, 0, s>>>(g->d, wedges, lists, class_room(m, nv), hdr);
  k_house_chain_terms<HOUSE><<<grid_over(std::max<uint64_t>(m, HOUSE ? 0 : nv)), kB, 0, s>>>(g->d, tri, wedges, above, hdr);
  if ((rc = wedge_launch<HOUSE>(g, lists, rank, radj, tri, hdr, s))) return rc;
  WedgeHdr h;
  if ((rc = read_back(&h, hdr, sizeof(h), s))) return rc;
  if (HOUSE)
    *out = wide(h.sum) - 2 * wide(h.tt) + 2 * wide(h.t);  // 6 T = 2 sum_e t(e)
  else
    *out = (unsigned __int128)((__int128)(wide(h.s) - 2 * wide(h.tt) - 4 * wide(h.sum)) / 2);
  return ZG_OK;
}

int degree_terms(const zg_graph* g, int kind, cudaStream_t s, unsigned __int128* out) {
  ZgScratch sum(s);
  int rc = sum.alloc(sizeof(U128));
  if (rc) return rc;
  cudaMemsetAsync(sum.p, 0, sizeof(U128), s);
  k_degree_terms<<<grid_over(std::max<uint64_t>(g->d.m, g->d.nv)), kB, 0, s>>>(g->d, kind, (U128*)sum.p);
  U128 h;
  if ((rc = read_back(&h, sum.p, sizeof(h), s))) return rc;
  *out = wide(h);
  return ZG_OK;
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
    case ZG_EXACT_TRIANGLE: rc = count_triangles(g, 0, 0, s, &r); break;
    case ZG_EXACT_FOUR_CLIQUE: rc = dag_count<kClique>(g, 0, 0, s, &r); break;
    case ZG_EXACT_WEDGE:
    case ZG_EXACT_FIVE_STAR: rc = degree_terms(g, kind, s, &r); break;
    case ZG_EXACT_THREE_PATH:
      rc = degree_terms(g, kind, s, &r);
      if (rc == ZG_OK) rc = count_triangles(g, 0, 0, s, &t);
      r -= 3 * t;
      break;
    case ZG_EXACT_FIVE_HOUSE: rc = house_chain<true>(g, s, &r); break;
    case ZG_EXACT_FIVE_CHAIN: rc = house_chain<false>(g, s, &r); break;
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
    rc = count_triangles(g, 1, threshold, s, &r);
  } else {
    rc = count_triangles(g, 0, 0, s, &r);
    if (rc == ZG_OK) rc = count_triangles(g, 2, threshold, s, &below);
    r -= below;
  }
  if (rc) return rc;
  out[0] = (uint64_t)r;
  out[1] = (uint64_t)(r >> 64);
  return ZG_OK;
}
