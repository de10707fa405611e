// The static count by decomposition: light pairs are counted, not visited.
//
// Call a pair of adjacent hyperedges heavy when it shares two or more members
// and light when it shares one. On the named workloads 85 to 99.9 % of the
// adjacent pairs are light, and a light pair is fully described by its one
// shared node, so triangles with at most one heavy pair have closed forms:
//
//   three light pairs   the three share one node u (a star: choose 3 of u's
//                       hyperedges), or the pairs use three distinct nodes
//                       x, y, z (choose one hyperedge per node pair: triangles
//                       of the node graph weighted by W(x, y), the number of
//                       hyperedges holding both x and y);
//   heavy pair (a, b)   with S = a & b: the third hyperedge meets a | b in one
//                       node of S (the hyperedges of that node), or in one
//                       node of a \ S and one of b \ S (the sum of W over
//                       those node pairs).
//
// Each form counts hyperedge triples with multiplicity, and every surplus
// comes from a triple with two or three heavy pairs (or from one hyperedge
// used twice), so those are the only triangles enumerated: a triangle with
// overlaps C and triple overlap g has
//   R = C_ab C_bc C_ca - g (C_ab + C_bc + C_ca) + 2 g
// ways to pick three distinct nodes, one per pair, and each heavy pair (x, y)
// of it with third hyperedge z is met (C_xz - g)(C_yz - g) times by the second
// heavy form and g times by the first. All sums are exact in uint64 modulo
// 2^64. The classes follow MoCHy's (MoCHy-master/motif_id.cpp:5-34) because
// every form fixes which of the seven regions are empty from the sizes alone.
//
// What is enumerated: for centre a (the lower-ranked end, by (degree, id), of
// the pair {a, c}), every heavy neighbour b of a and every heavy neighbour c
// of b ranked above a, tested against a's row. That is sum_b h(b)^2 / 2 tests,
// h the heavy degree, against sum_{(a, b)} d+(b) oriented entries in the
// enumeration of all triangles (hm_static.cu).
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "hm_classes.h"
#include "hm_device.h"
#include "hm_pairs.cuh"

namespace hm {
namespace {

constexpr unsigned kWarp = 32;
constexpr unsigned kBlock = 256;
constexpr unsigned kWarps = kBlock / kWarp;
constexpr uint32_t kEmpty = 0xffffffffu;

__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31u; }
__device__ __forceinline__ unsigned lanemask_lt() { return (1u << lane_id()) - 1u; }
__device__ __forceinline__ uint64_t gtid() { return (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; }
__device__ __forceinline__ uint64_t gstride() { return (uint64_t)gridDim.x * blockDim.x; }
__device__ __forceinline__ uint64_t global_warp() { return gtid() >> 5; }
__device__ __forceinline__ uint64_t n_warps() { return gstride() >> 5; }

__device__ __forceinline__ uint64_t warp_sum(uint64_t v) {
  for (int d = 16; d; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}

// Size category: 0 for |x| = 1, 1 for |x| = 2, 2 for |x| >= 3.
__device__ __forceinline__ uint32_t size_cat(uint32_t s) { return s >= 3 ? 2u : s - 1u; }

// ---- raw sums of one count (u64 each) ---------------------------------------------
// Stars by the sorted size categories of the three (10), triangles without a
// common node by how many of the three have a member of their own (4), the
// one-heavy-pair triangles through a shared node by (members of a beyond the
// pair, of b, category of c) (27), the enumerated triangles by class (30) and
// by the open-pair classes they remove (6), the open pairs (6), work queues.
constexpr unsigned kRawStar = 0, kRawDist = 10, kRawPair = 14, kRawClass = 41, kRawRem = 71, kRawOpen = 77,
                   kRawQueue = 83, kRawSize = 96;

__device__ __forceinline__ uint32_t star_index(uint32_t x, uint32_t y, uint32_t z) {  // any order
  const uint32_t lo = min(x, min(y, z)), hi = max(x, max(y, z)), mid = x + y + z - lo - hi;
  // 000 001 002 011 012 022 | 111 112 122 222
  return lo == 0 ? (mid == 0 ? hi : mid == 1 ? 2 + hi : 5u) : lo == 1 ? (mid == 1 ? 5 + hi : 8u) : 9u;
}
__device__ __forceinline__ uint32_t pair_index(uint32_t ua, uint32_t ub, uint32_t cat) {
  return (min(ua, 2u) * 3 + min(ub, 2u)) * 3 + cat;
}

// ---- preparation: ranks, heavy rows -------------------------------------------------

// Per slot: degree (sort key), heavy neighbours; sums: [0] h^2, [1] d^2,
// [2] node pairs of all hyperedges, [3] heavy entries, [4] node pairs of the
// marked hyperedges, [5] node triples of all hyperedges, [6] d^3 / n of those of
// more than 64 members, [7] how many those are; largest: [8] |a| |b| of a heavy
// pair, [9] members. A pair's larger hyperedge looks for [8], and only where it can
// be above large_pair: rows of nbr that are not needed are not read (50K wide-law
// hyperedges, batches of 4K: 2 % of the time). All blocks add to the same words, so a
// block adds its warps' sums up first.
constexpr unsigned kSums = 10;
__global__ void k_heavy_count(const uint64_t* off, const uint32_t* len, const uint32_t* nbr, const uint8_t* ovl,
                              const uint8_t* esize, const uint8_t* mark, uint32_t n, uint32_t large_pair,
                              uint32_t* heavy, uint32_t* ids, unsigned long long* sums) {
  __shared__ unsigned long long all[kSums];
  if (threadIdx.x < kSums) all[threadIdx.x] = 0;
  __syncthreads();
  unsigned long long h2 = 0, d2 = 0, np = 0, hs = 0, mp = 0, t3 = 0, d3 = 0, big = 0;
  uint32_t pair = 0, most = 0;
  for (uint64_t a = global_warp(); a < n; a += n_warps()) {
    const uint64_t s = off[a];
    const uint32_t l = len[a];
    const unsigned long long z = esize[a];
    uint32_t c = 0;
    if (z * z > max(large_pair, pair) && z * z > *(volatile unsigned long long*)&sums[8]) {
      for (uint32_t i = lane_id(); i < l; i += kWarp)
        if (ovl[s + i] >= 2) {
          ++c;
          pair = max(pair, (uint32_t)z * esize[nbr[s + i]]);
        }
    } else {
      for (uint32_t i = lane_id(); i < l; i += kWarp) c += ovl[s + i] >= 2;
    }
    for (int d = 16; d; d >>= 1) c += __shfl_xor_sync(0xffffffffu, c, d);
    if (lane_id() == 0) {
      heavy[a] = c;
      ids[a] = (uint32_t)a;
      most = max(most, (uint32_t)z);
      h2 += (unsigned long long)c * c;
      d2 += (unsigned long long)l * l;
      np += z * (z - (z > 0)) / 2;
      if (mark && mark[a]) mp += z * (z - (z > 0)) / 2;
      if (z >= 3) t3 += z * (z - 1) * (z - 2) / 6;
      if (z > 64) {
        d3 += (unsigned long long)l * l / n * l;
        ++big;
      }
      hs += c;
    }
  }
  for (int d = 16; d; d >>= 1) pair = max(pair, __shfl_xor_sync(0xffffffffu, pair, d));
  if (lane_id() == 0) {
    if (h2) atomicAdd(&all[0], h2);
    if (d2) atomicAdd(&all[1], d2);
    if (np) atomicAdd(&all[2], np);
    if (hs) atomicAdd(&all[3], hs);
    if (mp) atomicAdd(&all[4], mp);
    if (t3) atomicAdd(&all[5], t3);
    if (d3) atomicAdd(&all[6], d3);
    if (big) atomicAdd(&all[7], big);
    if (pair) atomicMax(&all[8], (unsigned long long)pair);
    if (most) atomicMax(&all[9], (unsigned long long)most);
  }
  __syncthreads();
  if (threadIdx.x < kSums && all[threadIdx.x]) {
    if (threadIdx.x < 8) atomicAdd(&sums[threadIdx.x], all[threadIdx.x]);
    else atomicMax(&sums[threadIdx.x], all[threadIdx.x]);
  }
}

__global__ void k_rank_scatter(const uint32_t* slot, uint32_t n, const uint32_t* heavy, uint32_t* rank,
                               uint32_t* hcnt) {
  for (uint64_t r = gtid(); r < n; r += gstride()) {
    const uint32_t s = slot[r];
    rank[s] = (uint32_t)r;
    hcnt[r] = heavy[s];
  }
}

// Heavy entries of every row, keyed (owner rank, neighbour rank), with their
// position in the owner's H2H row.
__global__ void k_heavy_emit(const uint32_t* slot, const uint32_t* rank, uint32_t n, const uint64_t* off,
                             const uint32_t* len, const uint32_t* nbr, const uint8_t* ovl, const uint64_t* hoff,
                             unsigned bits, uint64_t* key, uint32_t* pos) {
  for (uint64_t r = global_warp(); r < n; r += n_warps()) {
    uint64_t w = hoff[r];
    if (hoff[r + 1] == w) continue;
    const uint32_t a = slot[r];
    const uint64_t s = off[a];
    const uint32_t l = len[a];
    for (uint32_t i0 = 0; i0 < l; i0 += kWarp) {
      const uint32_t i = i0 + lane_id();
      const bool hv = i < l && ovl[s + i] >= 2;
      const unsigned m = __ballot_sync(0xffffffffu, hv);
      if (hv) {
        const uint64_t d = w + __popc(m & lanemask_lt());
        key[d] = (r << bits) | rank[nbr[s + i]];
        pos[d] = i;
      }
      w += __popc(m);
    }
  }
}

// An entry as the histogram kernel walks it: rank << 8 | (C - 2) * 8 +
// min(size, 8) - 1 for an overlap C of 2 to 4, low byte ~0 for a larger one.
__device__ __forceinline__ uint32_t walk_code(uint32_t rank, uint32_t os) {
  const uint32_t c = os & 0xffu;
  return (rank << 8) | (c <= 4 ? (c - 2) * 8 + min(os >> 8, 8u) - 1 : 0xffu);
}

// The sorted entries' fields; next = the first position of the neighbour's
// row that ranks above the owner (the owner is in that row: adjacency is
// symmetric).
__global__ void k_heavy_rows(const uint64_t* key, const uint32_t* pos, uint64_t nh, unsigned bits,
                             const uint32_t* slot, const uint64_t* off, const uint8_t* ovl, const uint8_t* esize,
                             const uint64_t* hoff, uint32_t* hnbr, uint32_t* hown, uint16_t* hos, uint32_t* hpos,
                             uint32_t* hnext, uint32_t* hcode) {
  const uint64_t low = (1ull << bits) - 1;
  for (uint64_t i = gtid(); i < nh; i += gstride()) {
    const uint64_t k = key[i];
    const uint32_t r = (uint32_t)(k >> bits), q = (uint32_t)(k & low);
    const uint32_t p = pos[i];
    hnbr[i] = q;
    hown[i] = r;
    const uint32_t os = ((uint32_t)esize[slot[q]] << 8) | ovl[off[slot[r]] + p];
    hos[i] = (uint16_t)os;
    hcode[i] = walk_code(q, os);
    hpos[i] = p;
    const uint64_t back = ((uint64_t)q << bits) | r;
    uint64_t lo = hoff[q], hi = hoff[q + 1];
    while (lo < hi) {
      const uint64_t mid = (lo + hi) >> 1;
      if (key[mid] <= back) lo = mid + 1;
      else hi = mid;
    }
    hnext[i] = (uint32_t)lo;
  }
}

// ---- preparation: node graph --------------------------------------------------------

// Hyperedges of each node by size category (3 per node); with marks, the
// marked ones alone into ncat_m too. classes: per kClass-th of an octave of the
// nodes' other members (hyperedge by hyperedge), the sums of about D and D^2, D
// the distinct ones among `even` nodes.
constexpr unsigned kClass = 4, kClasses = 33 * kClass;
__global__ void k_node_cats(const uint64_t* voff, const uint32_t* vlen, const uint32_t* vedge, const uint8_t* esize,
                            const uint8_t* mark, uint32_t n_nodes, float even, uint32_t* ncat, uint32_t* ncat_m, float* classes) {
  __shared__ float cls[2 * kClasses];
  for (unsigned k = threadIdx.x; k < 2 * kClasses; k += blockDim.x) cls[k] = 0;
  __syncthreads();
  for (uint64_t v = global_warp(); v < n_nodes; v += n_warps()) {
    const uint64_t s = voff[v];
    const uint32_t l = vlen[v];
    uint32_t c[6] = {0, 0, 0, 0, 0, 0};
    uint32_t others = 0;  // at most 254 of at most 2^24 hyperedges
    for (uint32_t i = lane_id(); i < l; i += kWarp) {
      const uint32_t e = vedge[s + i], z = esize[e];
      const bool m = mark && mark[e];
      others += z - 1;
      c[0] += z == 1;
      c[1] += z == 2;
      c[2] += z >= 3;
      c[3] += m && z == 1;
      c[4] += m && z == 2;
      c[5] += m && z >= 3;
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      for (int d = 16; d; d >>= 1) c[k] += __shfl_xor_sync(0xffffffffu, c[k], d);
      if (lane_id() == 0 && k < 3) ncat[3 * v + k] = c[k];
      if (lane_id() == 0 && k >= 3 && mark) ncat_m[3 * v + k - 3] = c[k];
    }
    for (int d = 16; d; d >>= 1) others += __shfl_xor_sync(0xffffffffu, others, d);
    if (lane_id() == 0 && others) {
      const float x = (float)others, distinct = even * (1.0f - expf(-x / even));
      const unsigned k = (unsigned)(log2f(x) * kClass);
      atomicAdd(&cls[2 * k], distinct);
      atomicAdd(&cls[2 * k + 1], distinct * distinct);
    }
  }
  __syncthreads();
  for (unsigned k = threadIdx.x; k < 2 * kClasses; k += blockDim.x)
    if (cls[k] != 0) atomicAdd(&classes[k], cls[k]);
}

// About the entries walked for the node triangles: a node of D neighbours, a share
// s of all neighbourhoods that of nodes of higher degree, is a neighbour in (1 - s)
// D rows and has s D entries in its own. Within 4 % of the walk on 19 graphs of
// even degrees, a fifth to a half of it on those with hubs.
double node_walk(const float* classes) {
  double total = 0, above = 0, walk = 0;
  for (unsigned k = 0; k < kClasses; ++k) total += classes[2 * k];
  for (unsigned k = kClasses; k-- > 0;) {
    const double own = classes[2 * k], s = total > 0 ? (above + own / 2) / total : 0;
    // within a class the shares run through own / total
    walk += (double)classes[2 * k + 1] * (s * (1 - s) - (total > 0 ? own * own / (total * total) / 12 : 0));
    above += own;
  }
  return walk;
}

// Node-pair table: open addressing over 16-byte entries {x, y, W2, W3},
// x < y, W2 / W3 the hyperedges of two / more members holding both; an entry
// of key 0 is empty (y > x >= 0). At most half full.
__device__ __forceinline__ uint32_t pair_hash(uint32_t x, uint32_t y) {
  uint32_t h = x * 2654435761u ^ (y * 2246822519u + 0x9E3779B9u);
  h ^= h >> 15;
  h *= 2246822519u;
  return h ^ (h >> 13);
}

// With wm (the marked hyperedges' weights, per table entry) those are returned.
__device__ __forceinline__ uint2 pair_weight(const uint4* tab, uint32_t mask, uint32_t x, uint32_t y,
                                             const uint2* wm = nullptr) {
  const uint32_t a = min(x, y), b = max(x, y);
  for (uint32_t h = pair_hash(a, b) & mask;; h = (h + 1) & mask) {
    const uint4 e = __ldg(tab + h);
    if (e.x == a && e.y == b) return wm ? __ldg(wm + h) : make_uint2(e.z, e.w);
    if (e.y == 0) return make_uint2(0, 0);
  }
}

// One warp per hyperedge, lanes over its node pairs (with only: those marked there).
__global__ void k_pair_insert(const uint64_t* off, const uint32_t* mem, const uint8_t* esize, const uint8_t* mark,
                              const uint8_t* only, uint32_t n, uint4* tab, uint2* wm, uint32_t mask) {
  for (uint64_t e = global_warp(); e < n; e += n_warps()) {
    const uint32_t s = esize[e];
    if (s < 2 || (only && !only[e])) continue;
    const uint32_t* m = mem + off[e];
    const uint32_t np = s * (s - 1) / 2;
    for (uint32_t t = lane_id(); t < np; t += kWarp) {
      // t-th pair (i < j): j the largest with j (j - 1) / 2 <= t
      uint32_t j = (uint32_t)((1.0f + sqrtf(8.0f * (float)t + 1.0f)) * 0.5f);
      while (j * (j - 1) / 2 > t) --j;
      while ((j + 1) * j / 2 <= t) ++j;
      const uint32_t x = m[t - j * (j - 1) / 2], y = m[j];
      const unsigned long long key = ((unsigned long long)y << 32) | x;  // memory order {x, y}
      uint32_t h = pair_hash(x, y) & mask;
      for (;; h = (h + 1) & mask) {
        const unsigned long long old = atomicCAS(reinterpret_cast<unsigned long long*>(tab + h), 0ull, key);
        if (old == 0ull || old == key) break;
      }
      atomicAdd(s == 2 ? &tab[h].z : &tab[h].w, 1u);
      if (mark && mark[e]) atomicAdd(s == 2 ? &wm[h].x : &wm[h].y, 1u);
    }
  }
}

__global__ void k_pair_degrees(const uint4* tab, uint64_t slots, uint32_t* deg) {
  for (uint64_t i = gtid(); i < slots; i += gstride()) {
    const uint4 e = tab[i];
    if (!e.y) continue;
    atomicAdd(&deg[e.x], 1u);
    atomicAdd(&deg[e.y], 1u);
  }
}

__device__ __forceinline__ bool owns(uint32_t x, uint32_t y, const uint32_t* deg) {  // x below y by (degree, id)
  const uint32_t dx = deg[x], dy = deg[y];
  return dx < dy || (dx == dy && x < y);
}

__global__ void k_pair_plus_count(const uint4* tab, uint64_t slots, const uint32_t* deg, uint32_t* plen) {
  for (uint64_t i = gtid(); i < slots; i += gstride()) {
    const uint4 e = tab[i];
    if (e.y) atomicAdd(&plen[owns(e.x, e.y, deg) ? e.x : e.y], 1u);
  }
}

__global__ void k_pair_plus_fill(const uint4* tab, const uint2* wm, uint64_t slots, const uint32_t* deg,
                                 const uint64_t* poff, uint32_t* cursor, uint32_t* nbr, uint2* w, uint2* w_m) {
  for (uint64_t i = gtid(); i < slots; i += gstride()) {
    const uint4 e = tab[i];
    if (!e.y) continue;
    const bool lo = owns(e.x, e.y, deg);
    const uint32_t u = lo ? e.x : e.y, v = lo ? e.y : e.x;
    const uint64_t d = poff[u] + atomicAdd(&cursor[u], 1u);
    nbr[d] = v;
    w[d] = make_uint2(e.z, e.w);
    if (wm) w_m[d] = wm[i];
  }
}

// ---- preparation: marked hyperedges ----------------------------------------------------
// Counting only the triples with a marked hyperedge (see count_touching_decomp):
// the marks by rank, each heavy row's marked neighbours as a row of their own,
// and per heavy entry where that row passes the entry's owner.

__global__ void k_rank_marks(const uint32_t* slot, uint32_t n, const uint8_t* mark, uint8_t* rmark) {
  for (uint64_t r = gtid(); r < n; r += gstride()) rmark[r] = mark[slot[r]];
}

__global__ void k_marked_count(const uint64_t* hoff, const uint32_t* hnbr, const uint8_t* rmark, uint32_t n,
                               uint32_t* cnt) {
  for (uint64_t r = global_warp(); r < n; r += n_warps()) {
    uint32_t c = 0;
    for (uint64_t e = hoff[r] + lane_id(); e < hoff[r + 1]; e += kWarp) c += rmark[hnbr[e]];
    for (int d = 16; d; d >>= 1) c += __shfl_xor_sync(0xffffffffu, c, d);
    if (lane_id() == 0) cnt[r] = c;
  }
}

__global__ void k_marked_fill(const uint64_t* hoff, const uint32_t* hnbr, const uint16_t* hos, const uint32_t* hpos,
                              const uint8_t* rmark, uint32_t n, const uint64_t* moff, uint32_t* mnbr, uint16_t* mos,
                              uint32_t* mpos, uint32_t* mcode) {
  for (uint64_t r = global_warp(); r < n; r += n_warps()) {
    uint64_t w = moff[r];
    if (moff[r + 1] == w) continue;
    for (uint64_t e0 = hoff[r]; e0 < hoff[r + 1]; e0 += kWarp) {
      const uint64_t e = e0 + lane_id();
      const bool keep = e < hoff[r + 1] && rmark[hnbr[e]];
      const unsigned m = __ballot_sync(0xffffffffu, keep);
      if (keep) {
        const uint64_t d = w + __popc(m & lanemask_lt());
        mnbr[d] = hnbr[e];
        mos[d] = hos[e];
        mcode[d] = walk_code(hnbr[e], hos[e]);
        mpos[d] = hpos[e];
      }
      w += __popc(m);
    }
  }
}

__global__ void k_marked_next(const uint32_t* hown, const uint32_t* hnbr, uint64_t nh, const uint64_t* moff,
                              const uint32_t* mnbr, uint32_t* mnext) {
  for (uint64_t e = gtid(); e < nh; e += gstride()) {
    const uint32_t r = hown[e];
    uint64_t lo = moff[hnbr[e]], hi = moff[hnbr[e] + 1];
    while (lo < hi) {
      const uint64_t mid = (lo + hi) >> 1;
      if (mnbr[mid] <= r) lo = mid + 1;
      else hi = mid;
    }
    mnext[e] = (uint32_t)lo;
  }
}

// ---- work lists -----------------------------------------------------------------------
// Items are put in (launch shape, log2 of their work) buckets, heaviest first
// within a shape; bucket codes are shape * 32 + 31 - log2(work), 255 for none.
constexpr unsigned kBuckets = 128;

__device__ __forceinline__ uint8_t bucket_code(unsigned shape, uint64_t work) {
  const unsigned lg = min(31u, (unsigned)(63 - __clzll((long long)work)));
  return (uint8_t)(shape * 32 + 31 - lg);
}

__global__ void k_bucket_starts(uint32_t* hist, uint32_t* starts, uint32_t* shape_end) {  // one block of kBuckets
  __shared__ uint32_t s[kBuckets];
  const unsigned t = threadIdx.x;
  s[t] = hist[t];
  __syncthreads();
  if (t == 0) {
    uint32_t run = 0;
    for (unsigned k = 0; k < kBuckets; ++k) {
      const uint32_t c = s[k];
      s[k] = run;
      run += c;
      if (k % 32 == 31) shape_end[k / 32] = run;
    }
  }
  __syncthreads();
  starts[t] = s[t];
}

__global__ void k_bucket_scatter(const uint8_t* code, uint32_t n, uint32_t* starts, uint32_t* list) {
  for (uint64_t i = gtid(); i < n; i += gstride()) {
    const uint8_t c = code[i];
    if (c < kBuckets) list[atomicAdd(&starts[c], 1u)] = (uint32_t)i;
  }
}

// Launch shapes of the enumeration: 0 a warp searching a's row (fewer tests
// than kTableMin or an eighth of the row, or a row no table holds), 1 and 2 the
// histogram kernel with 32-bit and 64-bit masks (up to 3072 entries ranked
// above a), 3 the large tables (up to 12288, and centres of more than 64
// members).
constexpr uint64_t kTableMin = 64;
// Up to this many heavy entries and tests (sum h^2) a graph is searched by entry,
// one or two entries for each warp of the launch. With 17,000 entries (100K
// hyperedges) the searches took 46 us of half the chip, the tables' launch 12 us.
constexpr uint64_t kEntriesFew = 1 << 13, kEntryTests = 1 << 18;
constexpr uint32_t kHHSmall = 3072, kHHLarge = 12288;
constexpr uint32_t kDenseSlots = 12288;  // up to this many hyperedges the tables are indexed by rank
__global__ void k_hh_codes(const uint32_t* slot, const uint32_t* rank, uint32_t n, const uint8_t* esize,
                           const uint64_t* off, const uint32_t* len, const uint32_t* nbr, const uint64_t* hoff,
                           const uint32_t* hnbr, const uint32_t* hnext, const uint8_t* rmark, const uint64_t* moff,
                           const uint32_t* mnext, uint8_t* code, uint32_t* hist) {
  for (uint64_t r = global_warp(); r < n; r += n_warps()) {
    uint64_t work = 0;
    for (uint64_t e = hoff[r] + lane_id(); e < hoff[r + 1]; e += kWarp) {
      const uint32_t q = hnbr[e];
      work += !rmark || rmark[r] || rmark[q] ? hoff[q + 1] - hnext[e] : moff[q + 1] - mnext[e];
    }
    work = warp_sum(work);
    uint8_t c = 255;
    if (work) {
      const uint32_t a = slot[r], l = len[a];
      unsigned shape = 0;
      if (work >= kTableMin && work * 8 >= l) {
        const bool narrow = esize[a] <= 32;
        uint32_t up = 0;
        if (!(narrow && n <= kDenseSlots)) {
          const uint64_t s = off[a];
          for (uint32_t i = lane_id(); i < l; i += kWarp) up += rank[nbr[s + i]] > r;
          for (int d = 16; d; d >>= 1) up += __shfl_xor_sync(0xffffffffu, up, d);
        }
        shape = up <= kHHSmall && esize[a] <= 64 ? (narrow ? 1u : 2u) : up <= kHHLarge ? 3u : 0u;
      }
      c = bucket_code(shape, work);
    }
    if (lane_id() == 0) {
      code[r] = c;
      if (c != 255) atomicAdd(&hist[c], 1u);
    }
  }
}

// Launch shapes of the node triangles: 0 one warp (short rows with little to
// probe: an item of 128 rows of 100 entries takes one warp 0.2 ms, longer than
// the rest of a 100K-hyperedge count), 1 and 2 blocks with 1024-slot and
// 4096-slot tables, 3 the largest table, or the global pair table past it.
constexpr uint32_t kNodeWarpRow = 128, kNodeWarpWork = 2048, kNodeSmall = 768, kNodeMid = 3072, kNodeLarge = 12288;
__global__ void k_node_codes(const uint64_t* poff, const uint32_t* plen, const uint32_t* nbr, uint32_t n,
                             uint8_t* code, uint32_t* hist, unsigned long long* total) {
  unsigned long long all = 0;  // entries the node triangles walk
  for (uint64_t u = global_warp(); u < n; u += n_warps()) {
    const uint32_t d = plen[u];
    uint8_t c = 255;
    if (d >= 2) {
      uint64_t work = 0;
      for (uint32_t i = lane_id(); i < d; i += kWarp) work += plen[nbr[poff[u] + i]];
      work = warp_sum(work);
      all += work;
      if (work)
        c = bucket_code(d <= kNodeWarpRow && work <= kNodeWarpWork ? 0u : d <= kNodeSmall ? 1u : d <= kNodeMid ? 2u : 3u,
                        work);
    }
    if (lane_id() == 0) {
      code[u] = c;
      if (c != 255) atomicAdd(&hist[c], 1u);
    }
  }
  if (lane_id() == 0 && all) atomicAdd(total, all);
}

// ---- counting: nodes, open pairs ------------------------------------------------------

__device__ __forceinline__ uint64_t choose2(uint64_t n) { return n * (n - (n > 0)) / 2; }
__device__ __forceinline__ uint64_t choose3(uint64_t n) {
  if (n < 3) return 0;
  const uint64_t p = choose2(n);
  return (n - 2) % 3 == 0 ? p * ((n - 2) / 3) : p / 3 * (n - 2);  // the division first: the product may pass 2^64
}

// All hyperedge triples through one node, by size categories.
__device__ void part_stars(unsigned vb, unsigned nb, const uint32_t* ncat, const uint32_t* ncat_m, uint32_t n_nodes,
                           unsigned long long* raw) {
  uint64_t s[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
  auto add = [&](uint64_t a, uint64_t b, uint64_t c, uint64_t f) {  // f: 1 or -1
    s[0] += f * choose3(a);
    s[1] += f * choose2(a) * b;
    s[2] += f * choose2(a) * c;
    s[3] += f * a * choose2(b);
    s[4] += f * a * b * c;
    s[5] += f * a * choose2(c);
    s[6] += f * choose3(b);
    s[7] += f * choose2(b) * c;
    s[8] += f * b * choose2(c);
    s[9] += f * choose3(c);
  };
  for (uint64_t v = (uint64_t)vb * kBlock + threadIdx.x; v < n_nodes; v += (uint64_t)nb * kBlock) {
    const uint64_t a = ncat[3 * v], b = ncat[3 * v + 1], c = ncat[3 * v + 2];
    add(a, b, c, 1);
    if (ncat_m) add(a - ncat_m[3 * v], b - ncat_m[3 * v + 1], c - ncat_m[3 * v + 2], ~0ull);  // those without a mark
  }
#pragma unroll
  for (int k = 0; k < 10; ++k) {
    const uint64_t t = warp_sum(s[k]);
    if (lane_id() == 0 && t) atomicAdd(&raw[kRawStar + k], (unsigned long long)t);
  }
}

// Open pairs of every centre (see k_open_pairs in hm_static.cu), from the
// heavy neighbours and the node counts: the light neighbours of a are the
// (node, other hyperedge) incidences of its members minus the overlaps of its
// heavy neighbours. Also takes back the node triangles a hyperedge forms
// alone, C(|a|, 3).
// With marks, the pairs with a marked hyperedge: of an unmarked centre, all
// pairs (pass 0) minus those of its unmarked neighbours (pass 1).
using OpenHist = uint32_t[kWarps][2][256];
struct OpenArgs {
  const uint32_t* slot;
  uint32_t n;
  const uint64_t* voff;
  const uint32_t* vmem;
  const uint8_t* esize;
  const uint32_t* h2h_len;
  const uint32_t* ncat;
  const uint32_t* ncat_m;
  const uint64_t* hoff;
  const uint32_t* hnbr;
  const uint16_t* hos;
  const uint8_t* rmark;
  unsigned long long* raw;
};
__device__ void part_open(unsigned vb, unsigned nb, OpenHist& hist, const OpenArgs& A) {
  const unsigned w = threadIdx.x / kWarp, lane = lane_id();
  uint64_t acc[6] = {0, 0, 0, 0, 0, 0};
  uint64_t alone = 0;
  for (uint64_t r = (uint64_t)vb * kWarps + w; r < A.n; r += (uint64_t)nb * kWarps) {
    const uint32_t a = A.slot[r];
    const uint32_t s = A.esize[a];
    const bool whole = !A.rmark || A.rmark[r];
    if (lane == 0 && whole) alone += choose3(s);
    if (A.h2h_len[a] < 2) continue;
    const bool heavy = A.hoff[r + 1] > A.hoff[r];
    const uint32_t* m = A.vmem + A.voff[a];
    for (int pass = 0; pass < (whole ? 1 : 2); ++pass) {
      if (heavy)
        for (uint32_t i = lane; i <= s; i += kWarp) {
          hist[w][0][i] = 0;
          hist[w][1][i] = 0;
        }
      uint32_t one[2] = {0, 0};
      for (uint32_t i = lane; i < s; i += kWarp) {
        const uint64_t v = 3 * (uint64_t)m[i];
        one[0] += A.ncat[v];
        one[1] += A.ncat[v + 1] + A.ncat[v + 2];
        if (pass) {
          one[0] -= A.ncat_m[v];
          one[1] -= A.ncat_m[v + 1] + A.ncat_m[v + 2];
        }
        one[s > 1] -= 1;  // a itself
      }
      __syncwarp();
      for (uint64_t e = A.hoff[r] + lane; e < A.hoff[r + 1]; e += kWarp) {
        if (pass && A.rmark[A.hnbr[e]]) continue;
        const uint32_t os = A.hos[e], c = os & 0xffu;
        one[1] -= c;  // a heavy neighbour has two members or more
        atomicAdd(&hist[w][c < (os >> 8)][c], 1u);
      }
      for (int d = 16; d; d >>= 1) {
        one[0] += __shfl_xor_sync(0xffffffffu, one[0], d);
        one[1] += __shfl_xor_sync(0xffffffffu, one[1], d);
      }
      __syncwarp();
      if (lane == 0 && !heavy) {
        // every overlap is 1: all pairs agree on [2 < |a|], the class is the ends' alone
        const uint32_t x = s > 2;
        const uint64_t f = pass ? ~0ull : 1ull;
        acc[x] += f * choose2(one[0]);
        acc[2 + x] += f * one[0] * one[1];
        acc[4 + x] += f * choose2(one[1]);
      } else if (lane == 0) {
        uint32_t* h0 = hist[w][0];
        uint32_t* h1 = hist[w][1];
        h0[1] += one[0];
        h1[1] += one[1];
        for (uint32_t k = 1; k <= s; ++k) {
          h0[k] += h0[k - 1];
          h1[k] += h1[k - 1];
        }
        open_pair_counts(h0, h1, s, acc, pass != 0);
      }
      __syncwarp();
    }
  }
  if (lane == 0) {
    for (int k = 0; k < 6; ++k)
      if (acc[k]) atomicAdd(&A.raw[kRawOpen + k], (unsigned long long)acc[k]);
    if (alone) atomicAdd(&A.raw[kRawDist + 3], 0ull - (unsigned long long)alone);
  }
}

// ---- counting: node triangles ----------------------------------------------------------

struct NodeArgs {
  const uint64_t* poff;
  const uint32_t* plen;
  const uint32_t* nbr;
  const uint2* w;
  const uint4* tab;  // the global pair table
  uint32_t tmask;
  const uint2* w_m;  // marked hyperedges' weights, per entry of nbr and per table entry (null: no marks)
  const uint2* tab_m;
  const uint32_t* work;
  uint32_t n_work;
  unsigned int* queue;
  unsigned long long* raw;
  uint32_t slices;  // part_nodes: item k is slice k % slices of node k / slices
};

__device__ __forceinline__ uint32_t node_hash(uint32_t key, uint32_t shift) { return (key * 2654435761u) >> shift; }

__device__ __forceinline__ void node_insert(uint32_t* keys, uint2* val, uint32_t shift, uint32_t mask, uint32_t key,
                                            uint2 v) {
  uint32_t h = node_hash(key, shift);
  while (atomicCAS(&keys[h], kEmpty, key) != kEmpty) h = (h + 1) & mask;
  val[h] = v;
}

// The node triangles a warp has found and not yet summed: per record the place
// of u's entry for v in u's row, the slot of the third node in u's table and
// the place of its entry in v's row. Most looked-up entries miss; a hit's three
// weights are loaded 32 hits at a time, instead of stalling the walk on each.
__device__ __forceinline__ uint64_t node_record(uint32_t i, uint32_t slot, uint64_t at) {
  return ((uint64_t)i << 48) | ((uint64_t)slot << 32) | at;  // i, slot < 2^14, at < 2^31
}
__device__ __forceinline__ void node_add(uint2 a, uint2 p, uint2 q, uint64_t f, uint64_t F[4]) {  // f: 1 or -1
  const uint64_t t0 = f * p.x * q.x, t1 = f * ((uint64_t)p.x * q.y + (uint64_t)p.y * q.x), t2 = f * p.y * q.y;
  F[0] += a.x * t0;
  F[1] += a.y * t0 + a.x * t1;
  F[2] += a.y * t1 + a.x * t2;
  F[3] += a.y * t2;
}
__device__ __forceinline__ uint2 less(uint2 a, uint2 b) { return make_uint2(a.x - b.x, a.y - b.y); }
// With marks (kTouch) the table's value is the place in u's row, and what the
// unmarked hyperedges give is taken off.
template <bool kTouch>
__device__ __forceinline__ void node_sum(uint64_t r, const uint2* val, const NodeArgs& A, uint64_t uo, uint64_t F[4]) {
  const uint32_t i = (uint32_t)(r >> 48), at = (uint32_t)r;
  const uint2 a = __ldg(A.w + uo + i), q = __ldg(A.w + at);
  uint2 p = val[(r >> 32) & 0xffffu];
  if (!kTouch) {
    node_add(a, p, q, 1, F);
    return;
  }
  const uint64_t ux = uo + p.x;
  p = __ldg(A.w + ux);
  const uint2 am = __ldg(A.w_m + uo + i), pm = __ldg(A.w_m + ux), qm = __ldg(A.w_m + at);
  if (!(am.x | am.y | pm.x | pm.y | qm.x | qm.y)) return;
  node_add(a, p, q, 1, F);
  node_add(less(a, am), less(p, pm), less(q, qm), ~0ull, F);
}

// Whole warp: the rows of u's neighbours i0, i0 + stride, ... (32 of them at
// most) against u's table. Their bounds are loaded at once, and each chunk of
// 32 entries while the one before is looked up. With filter (one bit per hash
// value in 1024, a word per lane) most misses are told by a shuffle.
template <bool kTouch, bool kFilter>
__device__ __forceinline__ void node_walk(const NodeArgs& A, const uint32_t* keys, const uint2* val, uint32_t shift,
                                          uint32_t mask, uint32_t filter, uint64_t uo, uint32_t d, uint32_t i0,
                                          uint32_t stride, uint64_t* q, uint32_t& qn, uint64_t F[4]) {
  const uint32_t* nbr = A.nbr;
  const unsigned lane = lane_id();
  const uint32_t mine = i0 + lane * stride;
  uint64_t vo = 0;
  uint32_t vl = 0;
  if (mine < d) {
    const uint32_t v = __ldg(nbr + uo + mine);
    vo = __ldg(A.poff + v);
    vl = __ldg(A.plen + v);
  }
  const uint32_t m = min(kWarp, (d - i0 + stride - 1) / stride);
  uint64_t o = __shfl_sync(0xffffffffu, vo, 0);
  uint32_t l = __shfl_sync(0xffffffffu, vl, 0), t = 0, j = lane;
  uint32_t x = j < l ? __ldg(nbr + o + j) : kEmpty;
  while (t < m) {
    const bool last = j - lane + kWarp >= l;  // the row's last chunk
    const uint32_t tn = t + last;
    const uint64_t on = __shfl_sync(0xffffffffu, vo, tn & 31u);
    const uint32_t ln = __shfl_sync(0xffffffffu, vl, tn & 31u), jn = last ? lane : j + kWarp;
    const uint32_t xn = tn < m && jn < ln ? __ldg(nbr + on + jn) : kEmpty;
    bool look = x != kEmpty;
    if (kFilter) {
      const uint32_t b = node_hash(x, 22);
      const uint32_t word = __shfl_sync(0xffffffffu, filter, b >> 5);
      look = look && ((word >> (b & 31u)) & 1u);
    }
    bool hit = false;
    uint32_t h = 0;
    if (look)
      for (h = node_hash(x, shift);; h = (h + 1) & mask) {
        const uint32_t k = keys[h];
        hit = k == x;
        if (hit || k == kEmpty) break;
      }
    const unsigned bal = __ballot_sync(0xffffffffu, hit);
    if (bal) {
      if (hit) q[qn + __popc(bal & lanemask_lt())] = node_record(i0 + t * stride, h, o + j);
      qn += (uint32_t)__popc(bal);
      __syncwarp();
      if (qn >= kWarp) {
        node_sum<kTouch>(q[lane], val, A, uo, F);
        __syncwarp();
        if (lane < qn - kWarp) q[lane] = q[kWarp + lane];
        __syncwarp();
        qn -= kWarp;
      }
    }
    t = tn;
    o = on;
    l = ln;
    j = jn;
    x = xn;
  }
}

__device__ __forceinline__ void node_flush(const uint64_t F[4], unsigned long long* raw) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint64_t t = warp_sum(F[k]);
    if (lane_id() == 0 && t) atomicAdd(&raw[kRawDist + k], (unsigned long long)t);
  }
}

// One warp per node with a short row: a table of up to 256 slots (load <= 1/2).
constexpr uint32_t kNodesAlone = 8192;  // items from which they get a launch of their own
constexpr uint32_t kNodeWarpSlots = 2 * kNodeWarpRow;
struct NodeWarp {
  uint2 val[kNodeWarpSlots];
  uint64_t q[2 * kWarp];
  uint32_t keys[kNodeWarpSlots];
  uint32_t filter[kWarp];
};
template <bool kTouch, bool kSliced>
__device__ void part_nodes(const NodeArgs& A, NodeWarp* S) {
  const uint32_t slices = kSliced ? A.slices : 1;
  const unsigned lane = lane_id();
  uint32_t* keys = S->keys;
  uint2* val = S->val;
  uint64_t F[4] = {0, 0, 0, 0};
  for (;;) {
    uint32_t it = 0;
    if (lane == 0) it = atomicAdd(A.queue, 1u);
    it = __shfl_sync(0xffffffffu, it, 0);
    if (it / slices >= A.n_work) break;
    const uint32_t u = A.work[it / slices], slice = it % slices;
    const uint64_t uo = A.poff[u];
    const uint32_t d = A.plen[u];
    if (slice >= d) continue;
    uint32_t slots = 64, qn = 0;
    while (slots < 2 * d && slots < kNodeWarpSlots) slots <<= 1;
    const uint32_t shift = 32u - (31u - (uint32_t)__clz(slots)), mask = slots - 1;
    for (uint32_t i = lane; i < slots; i += kWarp) keys[i] = kEmpty;
    S->filter[lane] = 0;
    __syncwarp();
    for (uint32_t i = lane; i < d; i += kWarp) {
      const uint32_t v = A.nbr[uo + i], b = node_hash(v, 22);
      node_insert(keys, val, shift, mask, v, kTouch ? make_uint2(i, 0) : A.w[uo + i]);
      atomicOr(&S->filter[b >> 5], 1u << (b & 31u));
    }
    __syncwarp();
    const uint32_t filter = S->filter[lane];
    for (uint32_t i0 = slice; i0 < d; i0 += kWarp * slices)
      node_walk<kTouch, true>(A, keys, val, shift, mask, filter, uo, d, i0, slices, S->q, qn, F);
    if (lane < qn) node_sum<kTouch>(S->q[lane], val, A, uo, F);  // the records name this node's table
    __syncwarp();
  }
  node_flush(F, A.raw);
}

// One block per node, kTab slots in shared memory (load <= 3/4); a longer row
// probes the global pair table instead.
template <bool kTouch, unsigned kTab, unsigned kThreads, unsigned kMinBlocks>
__global__ void __launch_bounds__(kThreads, kMinBlocks) k_node_tri(NodeArgs A) {
  constexpr unsigned kW = kThreads / kWarp;
  extern __shared__ uint64_t smem64[];
  uint2* val = reinterpret_cast<uint2*>(smem64);
  uint32_t* keys = reinterpret_cast<uint32_t*>(val + kTab);
  __shared__ uint64_t queues[kW][2 * kWarp];
  __shared__ uint32_t s_item;
  const unsigned w = threadIdx.x / kWarp, lane = lane_id();
  uint64_t F[4] = {0, 0, 0, 0};
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(A.queue, 1u);
    __syncthreads();
    const uint32_t it = s_item;
    if (it >= A.n_work) break;
    const uint32_t u = A.work[it];
    const uint64_t uo = A.poff[u];
    const uint32_t d = A.plen[u];
    if (d <= kTab / 4 * 3) {
      uint32_t slots = 64, qn = 0;
      while (slots < 2 * d && slots < kTab) slots <<= 1;
      const uint32_t shift = 32u - (31u - (uint32_t)__clz(slots)), mask = slots - 1;
      for (uint32_t i = threadIdx.x; i < slots; i += kThreads) keys[i] = kEmpty;
      __syncthreads();
      for (uint32_t i = threadIdx.x; i < d; i += kThreads)
        node_insert(keys, val, shift, mask, A.nbr[uo + i], kTouch ? make_uint2(i, 0) : A.w[uo + i]);
      __syncthreads();
      for (uint32_t i0 = w; i0 < d; i0 += kW * kWarp)
        node_walk<kTouch, false>(A, keys, val, shift, mask, 0, uo, d, i0, kW, queues[w], qn, F);
      __syncwarp();
      if (lane < qn) node_sum<kTouch>(queues[w][lane], val, A, uo, F);
    } else {
      for (uint32_t i = w; i < d; i += kW) {
        const uint32_t v = A.nbr[uo + i];
        const uint2 a = A.w[uo + i];
        const uint64_t o = A.poff[v];
        for (uint32_t j = lane; j < A.plen[v]; j += kWarp) {
          const uint32_t x = __ldg(A.nbr + o + j);
          const uint2 p = pair_weight(A.tab, A.tmask, u, x), q = __ldg(A.w + o + j);
          node_add(a, p, q, 1, F);
          if (kTouch)
            node_add(less(a, A.w_m[uo + i]), less(p, pair_weight(A.tab, A.tmask, u, x, A.tab_m)),
                     less(q, __ldg(A.w_m + o + j)), ~0ull, F);
        }
      }
    }
    __syncthreads();
  }
  node_flush(F, A.raw);
}

// ---- counting: heavy pairs --------------------------------------------------------------
// A heavy pair (a, b) is owned by its larger member (the lower rank at equal
// size). q(a, b), the sum of W over (a \ S) x (b \ S), is summed entry by entry
// for most pairs. A large owner with many partners first spreads
// y(w) = sum over v in a of W(v, w) over a node vector of its block, and then
//   q = sum_{w in b \ S} y(w) - sum_{v in S} self_b(v) + sum_{v != w in S} W(v, w),
// self_b(v) = sum_{w in b} W(v, w) kept per H2V entry: about |b| reads per pair.

struct PairArgs {
  const uint32_t* hown;
  const uint32_t* hnbr;
  const uint16_t* hos;
  const uint32_t* hpos;
  const uint32_t* hnext;
  const uint64_t* hoff;
  uint64_t nh;
  const uint32_t* slot;
  const uint64_t* off;   // H2H
  const uint64_t* mask;
  const uint64_t* voff;  // H2V
  const uint32_t* vmem;
  const uint8_t* esize;
  const uint32_t* ncat;
  const uint4* tab;
  uint32_t tmask;
  // with marks (else null): pairs of two unmarked hyperedges count their marked
  // third ones only, from the marked hyperedges' sums
  const uint8_t* rmark;
  const uint32_t* ncat_m;
  // the marked hyperedges' node pairs in a table of their own: with a twelfth of
  // 50K hyperedges marked it stays in L2 and most lookups end at an empty slot
  // (heavy pairs and spread of four counts 50.0 -> 44.6 ms, building it 1.1 ms)
  const uint4* tab_c;
  uint32_t cmask;
  const uint2* fw_m;
  uint2* self_m;
  const uint64_t* foff;  // the node graph's rows, both directions (for spreading)
  const uint32_t* fnbr;
  const uint2* fw;
  const uint8_t* spread;  // per rank: its owned pairs go through y
  const uint32_t* list;   // the ranks with spread set
  uint32_t n_list;
  uint2* self;            // per H2V entry {W2, W3}
  uint2* y;               // per block of k_spread_pairs: n_nodes entries (rounded up to even), zero between items
  uint32_t n_nodes;
  uint32_t per_warp, wide;  // entries a warp takes at once; combinations from which it takes a pair as a whole
  uint32_t slices;          // warps that share an entry (per_warp 1)
  unsigned int* queue;
  unsigned long long* raw;
};

__device__ __forceinline__ bool owns_pair(uint32_t ra, uint32_t sa, uint32_t rb, uint32_t sb) {
  return sa > sb || (sa == sb && ra < rb);
}

// The sums of one pair into the block's counters: q (third hyperedge of two /
// more members) and r (hyperedges of S's nodes by category, a and b included).
__device__ __forceinline__ void add_pair(unsigned long long* cnt, uint32_t sa, uint32_t sb, uint32_t C, uint64_t q2,
                                         uint64_t q3, uint64_t r0, uint64_t r1, uint64_t r2, bool unmarked) {
  const uint32_t ca = size_cat(sa), cb = size_cat(sb);
  const uint32_t n_ex = (sa > C + 1) + (sb > C + 1), n_big = (ca == 2) + (cb == 2);
  // a and b themselves are not third hyperedges (and not among the marked if unmarked)
  const uint64_t own = unmarked ? 0 : C;
  uint64_t r[3] = {r0, r1 - own * ((ca == 1) + (cb == 1)), r2 - own * ((ca == 2) + (cb == 2))};
  if (q2) {
    atomicAdd(&cnt[kRawDist + n_ex], (unsigned long long)q2);
    atomicAdd(&cnt[kRawDist + n_big], 0ull - (unsigned long long)q2 * C);
  }
  if (q3) {
    atomicAdd(&cnt[kRawDist + n_ex + 1], (unsigned long long)q3);
    atomicAdd(&cnt[kRawDist + n_big + 1], 0ull - (unsigned long long)q3 * C);
  }
#pragma unroll
  for (uint32_t k = 0; k < 3; ++k)
    if (r[k]) {
      atomicAdd(&cnt[kRawPair + pair_index(sa - C, sb - C, k)], (unsigned long long)r[k]);
      atomicAdd(&cnt[kRawStar + star_index(ca, cb, k)], 0ull - (unsigned long long)r[k]);
    }
  if (unmarked) return;
  // one hyperedge of the pair standing for two node pairs of a triangle
  const unsigned long long c2 = (unsigned long long)C * (C - 1) / 2;
  if (sa >= 3) atomicAdd(&cnt[kRawDist + 2 + (sb >= 3)], 0ull - c2 * (sa - 2));
  if (sb >= 3) atomicAdd(&cnt[kRawDist + 2 + (sa >= 3)], 0ull - c2 * (sb - 2));
}

__device__ __forceinline__ bool in_list(const uint32_t* list, uint32_t n, uint32_t key) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(list + mid) < key) lo = mid + 1;
    else hi = mid;
  }
  return lo < n && __ldg(list + lo) == key;
}

// Four entries per warp, eight lanes each over the |a| x |b| combinations, the
// positions in S read off the two entries' masks (members past 64: a search
// of the other list). Pairs of more than kPairWide combinations are taken by
// the whole warp, one after the other; with too few entries to fill the GPU
// that way (kPairFew) all are, one entry per warp.
constexpr uint32_t kPairWide = 384, kPairFew = 1u << 16;
using PairCounts = unsigned long long[kRawClass];
__device__ void part_pairs(unsigned vb, unsigned nb, PairCounts& cnt, const PairArgs& A) {
  const unsigned lane = lane_id(), grp = lane >> 3, sub = lane & 7u;
  for (unsigned k = threadIdx.x; k < kRawClass; k += kBlock) cnt[k] = 0;
  __syncthreads();
  const unsigned slice = threadIdx.x / kWarp % A.slices;
  for (uint64_t e0 = ((uint64_t)vb * kWarps + threadIdx.x / kWarp) / A.slices * A.per_warp; e0 < A.nh;
       e0 += (uint64_t)nb * kWarps / A.slices * A.per_warp) {
    const uint64_t e = e0 + grp;
    uint32_t sa = 0, sb = 0, C = 0;
    bool un = false;
    const uint32_t *pa = nullptr, *pb = nullptr;
    uint64_t ma = 0, mb = 0;
    if (grp < A.per_warp && e < A.nh) {
      const uint32_t ra = A.hown[e], rb = A.hnbr[e], os = A.hos[e];
      const uint32_t a = A.slot[ra];
      const uint32_t za = A.esize[a], zb = os >> 8;
      // (an unmarked owner spreads for its unmarked partners only)
      if (owns_pair(ra, za, rb, zb) && !(A.spread[ra] && (!A.rmark || A.rmark[ra] || !A.rmark[rb]))) {
        const uint32_t b = A.slot[rb];
        un = A.rmark && !A.rmark[ra] && !A.rmark[rb];
        sa = za;
        sb = zb;
        C = os & 0xffu;
        pa = A.vmem + A.voff[a];
        pb = A.vmem + A.voff[b];
        ma = A.mask[A.off[a] + A.hpos[e]];
        mb = A.mask[A.off[b] + A.hpos[A.hnext[e] - 1]];  // (b -> a) precedes b's entries above a
      }
    }
    uint64_t q2 = 0, q3 = 0, r0 = 0, r1 = 0, r2 = 0;
    // lanes first, first + step, ... of the |a| x |b| combinations; the
    // combinations of b's first member stand for a's member alone
    auto run = [&](uint32_t first, uint32_t step, uint32_t na, uint32_t nb, const uint32_t* xa, const uint32_t* xb,
                   uint64_t sma, uint64_t smb, bool unmarked) {
      const uint32_t* ncat = unmarked ? A.ncat_m : A.ncat;
      const uint4* tab = unmarked ? A.tab_c : A.tab;
      const uint32_t tmask = unmarked ? A.cmask : A.tmask;
      const uint32_t all = na * nb;
      for (uint32_t t = first; t < all; t += step) {
        const uint32_t i = t / nb, j = t - i * nb;
        const uint32_t v = __ldg(xa + i);
        if (i < 64 ? (sma >> i) & 1ull : in_list(xb, nb, v)) {
          if (j) continue;
          const uint32_t* c = ncat + 3 * (uint64_t)v;
          r0 += c[0];
          r1 += c[1];
          r2 += c[2];
          continue;
        }
        const uint32_t w = __ldg(xb + j);
        if (j < 64 ? (smb >> j) & 1ull : in_list(xa, na, w)) continue;
        const uint2 p = pair_weight(tab, tmask, v, w);
        q2 += p.x;
        q3 += p.y;
      }
    };
    const bool wide = sa * sb > A.wide;
    if (!wide) run(sub, 8, sa, sb, pa, pb, ma, mb, un);
    unsigned todo = __ballot_sync(0xffffffffu, wide && sub == 0);
    while (todo) {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1;
      const uint64_t k2 = q2, k3 = q3, s0 = r0, s1 = r1, s2 = r2;  // this lane's own pair, set aside
      q2 = q3 = r0 = r1 = r2 = 0;
      const uint32_t na = __shfl_sync(0xffffffffu, sa, src), nb = __shfl_sync(0xffffffffu, sb, src);
      const uint32_t* xa =
          reinterpret_cast<const uint32_t*>(__shfl_sync(0xffffffffu, (unsigned long long)pa, src));
      const uint32_t* xb =
          reinterpret_cast<const uint32_t*>(__shfl_sync(0xffffffffu, (unsigned long long)pb, src));
      const uint64_t sma = __shfl_sync(0xffffffffu, (unsigned long long)ma, src);
      const uint64_t smb = __shfl_sync(0xffffffffu, (unsigned long long)mb, src);
      const bool unmarked = __shfl_sync(0xffffffffu, (int)un, src) != 0;
      if (A.slices == 1) run(lane, 32, na, nb, xa, xb, sma, smb, unmarked);  // a fixed step: 2 % of a 100K count
      else run(slice * 32 + lane, A.slices * 32, na, nb, xa, xb, sma, smb, unmarked);
      __syncwarp();
      const uint64_t t2 = warp_sum(q2), t3 = warp_sum(q3), u0 = warp_sum(r0), u1 = warp_sum(r1), u2 = warp_sum(r2);
      // a further slice adds its sums alone, as an unmarked pair does
      if ((int)lane == src) add_pair(cnt, sa, sb, C, t2, t3, u0, u1, u2, un || slice);
      q2 = k2;
      q3 = k3;
      r0 = s0;
      r1 = s1;
      r2 = s2;
      __syncwarp();
    }
    uint64_t t[5] = {q2, q3, r0, r1, r2};
#pragma unroll
    for (int k = 0; k < 5; ++k)
      for (int d = 4; d; d >>= 1) t[k] += __shfl_xor_sync(0xffffffffu, t[k], d);
    if (sa && !wide && sub == 0) add_pair(cnt, sa, sb, C, t[0], t[1], t[2], t[3], t[4], un);
  }
  __syncthreads();
  for (unsigned k = threadIdx.x; k < kRawClass; k += kBlock)
    if (cnt[k]) atomicAdd(&A.raw[k], cnt[k]);
}

// Which owners spread: those whose entry-by-entry sums are longer than building
// and reading the vector (an increment and a clear per neighbour of a member),
// and long enough that one block's pass over it is not the slower one.
constexpr uint64_t kSpreadMin = 1u << 17;
__global__ void k_spread_flags(const uint32_t* slot, uint32_t n, const uint64_t* hoff, const uint32_t* hnbr,
                               const uint16_t* hos, const uint64_t* voff, const uint32_t* vmem, const uint8_t* esize,
                               const uint32_t* ndeg, uint8_t* spread, uint32_t* list, uint32_t* n_list) {
  for (uint64_t r = global_warp(); r < n; r += n_warps()) {
    const uint32_t a = slot[r], s = esize[a];
    uint64_t direct = 0, reads = 0;
    for (uint64_t e = hoff[r] + lane_id(); e < hoff[r + 1]; e += kWarp) {
      const uint32_t os = hos[e], z = os >> 8, C = os & 0xffu;
      if (!owns_pair((uint32_t)r, s, hnbr[e], z)) continue;
      direct += (uint64_t)(s - C) * (z - C);
      reads += z;
    }
    direct = warp_sum(direct);
    reads = warp_sum(reads);
    bool on = direct >= kSpreadMin && direct > reads;
    if (on) {
      uint64_t build = 0;
      for (uint32_t i = lane_id(); i < s; i += kWarp) build += ndeg[vmem[voff[a] + i]];
      on = direct > reads + 2 * warp_sum(build);
    }
    if (lane_id() == 0) {
      spread[r] = on;
      if (on) list[atomicAdd(n_list, 1u)] = (uint32_t)r;
    }
  }
}

__global__ void k_pair_rows_fill(const uint4* tab, const uint2* wm, uint64_t slots, const uint64_t* off,
                                 uint32_t* cursor, uint32_t* nbr, uint2* w, uint2* w_m) {
  for (uint64_t i = gtid(); i < slots; i += gstride()) {
    const uint4 e = tab[i];
    if (!e.y) continue;
    uint64_t d = off[e.x] + atomicAdd(&cursor[e.x], 1u);
    nbr[d] = e.y;
    w[d] = make_uint2(e.z, e.w);
    if (wm) w_m[d] = wm[i];
    d = off[e.y] + atomicAdd(&cursor[e.y], 1u);
    nbr[d] = e.x;
    w[d] = make_uint2(e.z, e.w);
    if (wm) w_m[d] = wm[i];
  }
}

// self_b(v) for every member v of every hyperedge with heavy neighbours.
__global__ void k_self_weights(PairArgs A, uint32_t n) {
  for (uint64_t r = global_warp(); r < n; r += n_warps()) {
    if (A.hoff[r + 1] == A.hoff[r]) continue;
    const uint32_t a = A.slot[r], s = A.esize[a];
    const uint64_t o = A.voff[a];
    for (uint32_t i = lane_id(); i < s; i += kWarp) {
      const uint32_t v = A.vmem[o + i];
      for (int k = 0; k < (A.rmark ? 2 : 1); ++k) {
        uint2 t = make_uint2(0, 0);
        for (uint32_t j = 0; j < s; ++j) {
          if (j == i) continue;
          const uint2 p = pair_weight(k ? A.tab_c : A.tab, k ? A.cmask : A.tmask, v, __ldg(A.vmem + o + j));
          t.x += p.x;
          t.y += p.y;
        }
        (k ? A.self_m : A.self)[o + i] = t;
      }
    }
  }
}

// One block per spreading owner a. In the vector a's own members hold
// {~0, ~0}, which tells S from b \ S.
constexpr unsigned kSpreadThreads = 1024;
__global__ void __launch_bounds__(kSpreadThreads) k_spread_pairs(PairArgs A) {
  __shared__ unsigned long long cnt[kRawClass];
  __shared__ uint32_t s_item;
  const unsigned w = threadIdx.x / kWarp, lane = lane_id();
  constexpr unsigned kW = kSpreadThreads / kWarp;
  const uint32_t vec = (A.n_nodes + 1) & ~1u;
  uint2* y = A.y + (uint64_t)blockIdx.x * vec;
  for (unsigned k = threadIdx.x; k < kRawClass; k += kSpreadThreads) cnt[k] = 0;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_item = atomicAdd(A.queue, 1u);
    __syncthreads();
    if (s_item >= A.n_list) break;
    const uint32_t ra = A.list[s_item], a = A.slot[ra], sa = A.esize[a];
    const uint32_t* pa = A.vmem + A.voff[a];
    // an unmarked owner's unmarked partners count marked third hyperedges only;
    // its few marked ones are left to part_pairs
    const bool un = A.rmark && !A.rmark[ra];
    const uint2* fw = un ? A.fw_m : A.fw;
    const uint32_t* ncat = un ? A.ncat_m : A.ncat;
    const uint2* self = un ? A.self_m : A.self;
    // the block takes the rows of the members one after another (a node's
    // row can be hundreds of times another's)
    uint64_t cells = 0;
#pragma unroll 4
    for (uint32_t i = 0; i < sa; ++i) {
      const uint32_t v = __ldg(pa + i);
      const uint64_t o = A.foff[v];
      const uint32_t l = (uint32_t)(A.foff[v + 1] - o);
      for (uint32_t k = threadIdx.x; k < l; k += kSpreadThreads) {
        const uint32_t x = __ldg(A.fnbr + o + k);
        const uint2 q = __ldg(fw + o + k);
        if (q.x) atomicAdd(&y[x].x, q.x);
        if (q.y) atomicAdd(&y[x].y, q.y);
      }
    }
    for (uint32_t i = 0; i < sa; ++i) cells += A.foff[pa[i] + 1] - A.foff[pa[i]];
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < sa; i += kSpreadThreads) y[pa[i]] = make_uint2(~0u, ~0u);
    __syncthreads();
    const uint64_t he = A.hoff[ra + 1];
    // eight lanes per pair: a pair is a chain of dependent loads, so the more
    // of them in flight the better
    for (uint64_t e0 = A.hoff[ra] + w * 4; e0 < he; e0 += kW * 4) {
      const uint64_t e = e0 + (lane >> 3);
      uint32_t sb = 0, C = 0;
      uint64_t bo = 0;
      if (e < he) {
        const uint32_t rb = A.hnbr[e], os = A.hos[e];
        if (owns_pair(ra, sa, rb, os >> 8) && !(un && A.rmark[rb])) {
          sb = os >> 8;
          C = os & 0xffu;
          bo = A.voff[A.slot[rb]];
        }
      }
      uint64_t t[5] = {0, 0, 0, 0, 0};  // q2, q3, r by category
      for (uint32_t j = lane & 7u; j < sb; j += 8) {
        const uint32_t v = __ldg(A.vmem + bo + j);
        const uint2 q = y[v];
        if (q.x != ~0u || q.y != ~0u) {
          t[0] += q.x;
          t[1] += q.y;
          continue;
        }
        const uint32_t* c = ncat + 3 * (uint64_t)v;
        t[2] += c[0];
        t[3] += c[1];
        t[4] += c[2];
        const uint2 z = self[bo + j];
        t[0] -= z.x;
        t[1] -= z.y;
        for (uint32_t k = 0; k < sb; ++k) {  // the other members of S
          if (k == j) continue;
          const uint32_t x = __ldg(A.vmem + bo + k);
          const uint2 u = y[x];
          if (u.x != ~0u || u.y != ~0u) continue;
          const uint2 p = pair_weight(un ? A.tab_c : A.tab, un ? A.cmask : A.tmask, v, x);
          t[0] += p.x;
          t[1] += p.y;
        }
      }
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 5; ++k)
        for (int d = 4; d; d >>= 1) t[k] += __shfl_xor_sync(0xffffffffu, t[k], d);
      if (sb && (lane & 7u) == 0) add_pair(cnt, sa, sb, C, t[0], t[1], t[2], t[3], t[4], un);
    }
    __syncthreads();
    if (A.n_nodes <= 4 * cells) {  // clear it all, two entries at a time (the vectors start at even entries)
      for (uint32_t i = threadIdx.x; i < vec / 2; i += kSpreadThreads)
        reinterpret_cast<uint4*>(y)[i] = make_uint4(0, 0, 0, 0);
    } else {
      for (uint32_t i = w; i < sa; i += kW) {
        const uint32_t v = __ldg(pa + i);
        if (lane == 0) y[v] = make_uint2(0, 0);
        for (uint64_t k = A.foff[v] + lane; k < A.foff[v + 1]; k += kWarp) {
          y[__ldg(A.fnbr + k)] = make_uint2(0, 0);
        }
      }
    }
  }
  for (unsigned k = threadIdx.x; k < kRawClass; k += kSpreadThreads)
    if (cnt[k]) atomicAdd(&A.raw[k], cnt[k]);
}

// ---- counting: triangles with two or three heavy pairs ------------------------------------

struct HHArgs {
  const uint32_t* slot;
  const uint32_t* rank;
  const uint64_t* hoff;   // heavy rows by rank
  const uint32_t* hnbr;
  const uint16_t* hos;
  const uint32_t* hpos;
  const uint32_t* hnext;
  const uint32_t* hcode;  // walk_code of every entry
  const uint64_t* off;    // H2H
  const uint32_t* len;
  const uint32_t* nbr;
  const uint8_t* ovl;
  const uint64_t* mask;
  const uint64_t* voff;   // H2V
  const uint32_t* vmem;
  const uint8_t* esize;
  // with marks (else null): b's marked neighbours alone, walked when neither a nor b is marked
  const uint8_t* rmark;
  const uint64_t* moff;
  const uint32_t* mnbr;
  const uint16_t* mos;
  const uint32_t* mpos;
  const uint32_t* mnext;
  const uint32_t* mcode;
  const uint32_t* work;   // ranks of the centres
  uint32_t n_work;
  uint32_t slices;        // k_hh_large: item k is slice k % slices of centre k / slices
  const uint32_t* hown;   // owner of every heavy entry
  uint64_t entries;       // by entry: that many heavy entries, no work list (0: by centre)
  unsigned int* queue;
  unsigned long long* raw;
};

// The part of b's heavy row past a that is walked for (a, b), entry e.
struct Walk {
  const uint32_t* nbr;
  const uint16_t* os;
  const uint32_t* pos;
  const uint32_t* code;
  uint64_t first, end;
};
__device__ __forceinline__ Walk walk_of(const HHArgs& A, uint32_t ra, uint32_t rb, uint64_t e) {
  if (!A.rmark || A.rmark[ra] || A.rmark[rb]) return Walk{A.hnbr, A.hos, A.hpos, A.hcode, A.hnext[e], A.hoff[rb + 1]};
  return Walk{A.mnbr, A.mos, A.mpos, A.mcode, A.mnext[e], A.moff[rb + 1]};
}

// |a & b & c| by a three-way merge (centres of more than 64 members).
__device__ uint32_t merge3(const HHArgs& A, uint32_t a, uint32_t b, uint32_t c) {
  const uint32_t* x = A.vmem + A.voff[a];
  const uint32_t* y = A.vmem + A.voff[b];
  const uint32_t* z = A.vmem + A.voff[c];
  const uint32_t nx = A.esize[a], ny = A.esize[b], nz = A.esize[c];
  uint32_t i = 0, j = 0, k = 0, g = 0;
  while (i < nx && j < ny && k < nz) {
    const uint32_t u = x[i], v = y[j], t = z[k];
    const uint32_t m = max(u, max(v, t));
    if (u == m && v == m && t == m) {
      ++g; ++i; ++j; ++k;
    } else {
      i += (u < m);
      j += (v < m);
      k += (t < m);
    }
  }
  return g;
}

// Counters a triangle adds to, 32-bit, one of kCol columns per lane (lanes of
// a warp often meet the same counter): 30 classes, 6 removals, 4 stars by the
// number of hyperedges with three members or more, 18 pair entries (ua, ub,
// c of three or more).
constexpr unsigned kSmClass = 0, kSmRem = 30, kSmStar = 36, kSmPair = 40, kSmRows = 58;
// A test adds at most 3 x 255 to one 32-bit counter: flushed every 2^22 tests,
// none can wrap.
constexpr uint32_t kFlushTests = 1u << 22;

template <unsigned kCol>
struct WarpCounts {
  unsigned long long dist[4][kWarp];  // per lane: no conflicts, no atomics
  uint32_t c[kSmRows][kCol];
};

template <unsigned kCol>
__device__ __forceinline__ void clear_counts(WarpCounts<kCol>* W) {
  for (unsigned k = 0; k < 4; ++k) W->dist[k][lane_id()] = 0;
  for (unsigned k = lane_id(); k < kSmRows * kCol; k += kWarp) (&W->c[0][0])[k] = 0;
  __syncwarp();
}

template <unsigned kCol>
__device__ __forceinline__ void flush_counts(WarpCounts<kCol>* W, unsigned long long* raw) {
  __syncwarp();
  for (unsigned k = 0; k < 4; ++k) {
    const uint64_t t = warp_sum(W->dist[k][lane_id()]);
    if (lane_id() == 0 && t) atomicAdd(&raw[kRawDist + k], (unsigned long long)t);
  }
  for (unsigned k = lane_id(); k < kSmRows; k += kWarp) {
    unsigned long long t = 0;
    for (unsigned j = 0; j < kCol; ++j) t += W->c[k][j];
    if (!t) continue;
    if (k < kSmRem) atomicAdd(&raw[kRawClass + k], t);
    else if (k < kSmStar) atomicAdd(&raw[kRawRem + (k - kSmRem)], t);
    else if (k < kSmPair) atomicAdd(&raw[kRawStar + 6 + (k - kSmStar)], t);  // sorted categories 111 112 122 222
    else {
      const uint32_t q = k - kSmPair;  // (ua, ub) * 2 + big, taken back
      atomicAdd(&raw[kRawPair + (q >> 1) * 3 + 1 + (q & 1u)], 0ull - t);
    }
  }
  __syncwarp();
  clear_counts(W);
}

// The same for n triangles without a common node: each pair has nodes of its
// own, so the class (26 to 29) and the removals follow from how many of the
// three have a member outside the others, as for the closed forms, and R and
// the products reduce to P = C_ab C_bc C_ac.
template <unsigned kCol>
__device__ __forceinline__ void add_triangle0(WarpCounts<kCol>* W, uint32_t sa, uint32_t sb, uint32_t sc, uint32_t cab,
                                              uint32_t cbc, uint32_t cac, uint32_t n) {
  const unsigned lane = lane_id();
  const uint32_t ba = sa >= 3, bb = sb >= 3, bc = sc >= 3;
  const uint32_t eab = cab >= 2 ? cac * cbc : 0u, ebc = cbc >= 2 ? cab * cac : 0u, eac = cac >= 2 ? cab * cbc : 0u;
  const uint32_t dk = cab * cbc * cac * ((cab >= 2) + (cbc >= 2) + (cac >= 2) - 1);
  W->dist[(sa > cab + cac) + (sb > cab + cbc) + (sc > cac + cbc)][lane] += n;
  W->dist[ba + bb + bc][lane] += (unsigned long long)dk * n;
  if (eab) W->dist[(sa > cab + 1) + (sb > cab + 1) + bc][lane] -= (unsigned long long)eab * n;
  if (ebc) W->dist[(sb > cbc + 1) + (sc > cbc + 1) + ba][lane] -= (unsigned long long)ebc * n;
  if (eac) W->dist[(sa > cac + 1) + (sc > cac + 1) + bb][lane] -= (unsigned long long)eac * n;
}

// One triangle with overlaps cab, cbc, cac (two of them heavy or all) and
// triple overlap g: its class and removals, and what the closed forms counted
// it for (see the head of this file).
template <unsigned kCol>
__device__ __forceinline__ void add_triangle(WarpCounts<kCol>* W, const int8_t* cls, uint32_t sa, uint32_t sb,
                                             uint32_t sc, uint32_t cab, uint32_t cbc, uint32_t cac, uint32_t g,
                                             uint32_t n = 1) {
  if (!g) {
    add_triangle0(W, sa, sb, sc, cab, cbc, cac, n);
    return;
  }
  const unsigned lane = lane_id(), col = lane & (kCol - 1);
  const int k = cls[region_pattern((int)sa, (int)sb, (int)sc, (int)cab, (int)cbc, (int)cac, (int)g)];
  atomicAdd(&W->c[kSmClass + k][col], n);
  const uint32_t oa = (cab + cac < sa) + 2 * ((cab < sb) + (cac < sc));
  const uint32_t ob = (cab + cbc < sb) + 2 * ((cab < sa) + (cbc < sc));
  const uint32_t oc = (cac + cbc < sc) + 2 * ((cac < sa) + (cbc < sb));
  atomicAdd(&W->c[kSmRem + oa][col], n);
  atomicAdd(&W->c[kSmRem + ob][col], n);
  atomicAdd(&W->c[kSmRem + oc][col], n);
  const uint32_t ba = sa >= 3, bb = sb >= 3, bc = sc >= 3;
  const uint32_t xab = cab - g, xbc = cbc - g, xac = cac - g;
  // below 2^26 in absolute value: sizes are at most 255
  int dk = (int)(g * (cab + cbc + cac)) - 2 * (int)g - (int)(cab * cbc * cac);  // -R
  const uint32_t eab = cab >= 2 ? xac * xbc : 0u, ebc = cbc >= 2 ? xab * xac : 0u, eac = cac >= 2 ? xab * xbc : 0u;
  dk += (int)(cab * eab + cbc * ebc + cac * eac);
  W->dist[ba + bb + bc][lane] += (unsigned long long)((long long)dk * n);
  if (eab) W->dist[(sa > cab + 1) + (sb > cab + 1) + bc][lane] -= (unsigned long long)eab * n;
  if (ebc) W->dist[(sb > cbc + 1) + (sc > cbc + 1) + ba][lane] -= (unsigned long long)ebc * n;
  if (eac) W->dist[(sa > cac + 1) + (sc > cac + 1) + bb][lane] -= (unsigned long long)eac * n;
  const uint32_t gn = g * n;
  atomicAdd(&W->c[kSmStar + ba + bb + bc][col], gn * ((cab >= 2) + (cbc >= 2) + (cac >= 2) - 1));
  auto pair = [&](uint32_t ux, uint32_t uy, uint32_t big) {
    atomicAdd(&W->c[kSmPair + (min(ux, 2u) * 3 + min(uy, 2u)) * 2 + big][col], gn);
  };
  if (cab >= 2) pair(sa - cab, sb - cab, bc);
  if (cbc >= 2) pair(sb - cbc, sc - cbc, ba);
  if (cac >= 2) pair(sa - cac, sc - cac, bb);
}

// A record packs |b|, |c|, C_ab, C_bc, C_ac and g, 8 bits each, and how many
// triangles it stands for, 16 bits.
__device__ __forceinline__ uint64_t pack6(uint32_t sb, uint32_t sc, uint32_t cab, uint32_t cbc, uint32_t cac,
                                          uint32_t g, uint32_t n = 1) {
  return (uint64_t)(sb | (sc << 8) | (cab << 16) | (cbc << 24)) | ((uint64_t)(cac | (g << 8) | (n << 16)) << 32);
}
template <unsigned kCol>
__device__ __forceinline__ void add_record(WarpCounts<kCol>* W, const int8_t* cls, uint32_t sa, uint64_t r) {
  const uint32_t lo = (uint32_t)r, hi = (uint32_t)(r >> 32);
  add_triangle(W, cls, sa, lo & 0xffu, (lo >> 8) & 0xffu, (lo >> 16) & 0xffu, lo >> 24, hi & 0xffu, (hi >> 8) & 0xffu,
               hi >> 16);
}

// Whole warp: appends the lanes' records to the warp's queue (64 places) and
// hands 32 at a time to add.
template <class Add>
__device__ __forceinline__ void queue_records(bool push, uint64_t rec, uint64_t* q, uint32_t& qn, Add&& add) {
  const unsigned bal = __ballot_sync(0xffffffffu, push);
  if (!bal) return;
  if (push) q[qn + __popc(bal & lanemask_lt())] = rec;
  qn += (uint32_t)__popc(bal);
  __syncwarp();
  if (qn >= kWarp) {
    add(q[lane_id()]);
    __syncwarp();
    if (lane_id() < qn - kWarp) q[lane_id()] = q[kWarp + lane_id()];
    __syncwarp();
    qn -= kWarp;
  }
}

__device__ __forceinline__ void fill_classes(int8_t* cls) {
  for (unsigned p = threadIdx.x; p < 128; p += blockDim.x) {
    const int k = static_class_of_pattern((int)p);
    cls[p] = (int8_t)(k < 0 ? 0 : k);  // a closed triangle always has a class
  }
}

// Searches: each c of b's heavy row past a is looked up in a's id-sorted row.
// By centre (a warp takes all of a's heavy neighbours) for those with few
// tests; by entry (a warp takes one heavy pair (a, b)) where the whole graph has
// few, as then every search is in flight at once and no launch is needed for the
// tables: with the counters in the last block, 1K hyperedges of 558 heavy
// entries went from 75 to 72 us per count.
constexpr unsigned kSearchCol = 4;
struct SearchShared {
  WarpCounts<kSearchCol> wc[kWarps];
  int8_t cls[128];
};
__device__ void part_search(unsigned vb, unsigned nb, const HHArgs& A, SearchShared& S) {
  const unsigned lane = lane_id();
  WarpCounts<kSearchCol>* W = &S.wc[threadIdx.x / kWarp];
  int8_t* cls = S.cls;
  fill_classes(cls);
  clear_counts(W);
  __syncthreads();
  uint32_t tests = 0;
  uint64_t it = (uint64_t)vb * kWarps + threadIdx.x / kWarp;  // by entry: every nb * kWarps-th
  for (;;) {
    uint64_t e, he;
    uint32_t ra;
    if (A.entries) {
      if (it >= A.entries) break;
      e = it;
      he = it + 1;
      ra = A.hown[e];
      it += (uint64_t)nb * kWarps;
    } else {
      uint32_t k = 0;
      if (lane == 0) k = atomicAdd(A.queue, 1u);
      k = __shfl_sync(0xffffffffu, k, 0);
      if (k >= A.n_work) break;
      ra = A.work[k];
      e = A.hoff[ra];
      he = A.hoff[ra + 1];
    }
    const uint32_t a = A.slot[ra];
    const uint64_t ao = A.off[a];
    const uint32_t al = A.len[a];
    const uint32_t sa = A.esize[a];
    for (; e < he; ++e) {
      const uint32_t rb = A.hnbr[e], osb = A.hos[e];
      const uint64_t mab = A.mask[ao + A.hpos[e]];
      const Walk B = walk_of(A, ra, rb, e);
      for (uint64_t j0 = B.first; j0 < B.end; j0 += kWarp) {
        const uint64_t j = j0 + lane;
        if (j < B.end) {
          const uint32_t rc = B.nbr[j], osc = B.os[j], c = A.slot[rc];
          uint32_t lo = 0, hi = al;
          while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (__ldg(A.nbr + ao + mid) < c) lo = mid + 1;
            else hi = mid;
          }
          if (lo < al && A.nbr[ao + lo] == c) {
            const uint32_t cac = A.ovl[ao + lo];
            if (cac < 2 || rb > rc) {  // three heavy pairs: once, b ranked highest
              const uint32_t g = sa <= 64 ? (uint32_t)__popcll(mab & A.mask[ao + lo]) : merge3(A, a, A.slot[rb], c);
              add_triangle(W, cls, sa, osb >> 8, osc >> 8, osb & 0xffu, osc & 0xffu, cac, g);
            }
          }
        }
        __syncwarp();
        if ((tests += kWarp) >= kFlushTests) {
          flush_counts(W, A.raw);
          tests = 0;
        }
      }
    }
  }
  flush_counts(W, A.raw);
}

// One block per centre a: the entries of a's row ranked above a in a shared
// table keyed by rank (4 keys per 16-byte bucket, load <= 3/4), each with its
// place in a's row. Warps take b among a's heavy neighbours, lanes walk b's
// heavy row past a. For the longest rows and centres of more than 64 members,
// few and long (23,000 neighbours at 60K hyperedges): a centre's b are dealt to
// several blocks where there are fewer centres than places.
constexpr unsigned kHHSlots = 16384, kHHThreads = 1024, kHHCol = 4;
constexpr size_t kHHSmem = kHHSlots * 2 * sizeof(uint32_t) +
                           kHHThreads / kWarp * (sizeof(WarpCounts<kHHCol>) + 2 * kWarp * sizeof(uint64_t));
static_assert(kHHSmem <= 226 * 1024 && kHHLarge <= kHHSlots * 3 / 4, "one block per SM, table load");
__global__ void __launch_bounds__(kHHThreads, 1) k_hh_large(HHArgs A) {
  constexpr unsigned kSlots = kHHSlots, kThreads = kHHThreads, kCol = kHHCol, kW = kThreads / kWarp;
  extern __shared__ uint64_t smem64[];
  uint32_t* val = reinterpret_cast<uint32_t*>(smem64);
  uint32_t* keys = val + kSlots;
  WarpCounts<kCol>* W = reinterpret_cast<WarpCounts<kCol>*>(keys + kSlots) + threadIdx.x / kWarp;
  uint64_t* q = reinterpret_cast<uint64_t*>(reinterpret_cast<WarpCounts<kCol>*>(keys + kSlots) + kW) +
                (threadIdx.x / kWarp) * 2 * kWarp;
  __shared__ int8_t cls[128];
  __shared__ uint32_t s_item;
  const unsigned w = threadIdx.x / kWarp, lane = lane_id();
  fill_classes(cls);
  clear_counts(W);
  uint32_t qn = 0, tests = 0;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(A.queue, 1u);
    __syncthreads();
    const uint32_t it = s_item;
    if (it >= A.n_work * A.slices) break;
    const uint32_t ra = A.work[it / A.slices], a = A.slot[ra], slice = it % A.slices;
    const uint64_t ao = A.off[a];
    const uint32_t al = A.len[a];
    const uint32_t sa = A.esize[a];
    const bool exact = sa <= 64;
    uint32_t slots = 64;
    while (slots < 2 * al && slots < kSlots) slots <<= 1;
    const uint32_t shift = 32u - (31u - (uint32_t)__clz(slots / 4)), bmask = slots / 4 - 1;
    for (uint32_t i = threadIdx.x; i < slots; i += kThreads) keys[i] = kEmpty;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < al; i += kThreads) {
      const uint32_t key = __ldg(A.rank + __ldg(A.nbr + ao + i));
      if (key <= ra) continue;
      uint32_t bk = (key * 2654435761u) >> shift, h = 0;
      for (bool done = false; !done; bk = (bk + 1) & bmask)
        for (uint32_t t = 0; t < 4; ++t)
          if (atomicCAS(&keys[4 * bk + t], kEmpty, key) == kEmpty) {
            h = 4 * bk + t;
            done = true;
            break;
          }
      val[h] = i;
    }
    __syncthreads();
    const uint64_t he = A.hoff[ra + 1];
    for (uint64_t e = A.hoff[ra] + slice * kW + w; e < he; e += kW * A.slices) {
      const uint32_t rb = A.hnbr[e], osb = A.hos[e];
      // the masks of the triple overlap: over a's members, or over b's when a
      // has more than 64 (b's entry of a precedes its entries above a)
      const bool by_b = !exact && (osb >> 8) <= 64;
      const uint64_t bo = A.off[A.slot[rb]];
      const uint64_t mab = exact ? A.mask[ao + A.hpos[e]] : by_b ? A.mask[bo + A.hpos[A.hnext[e] - 1]] : 0;
      const Walk B = walk_of(A, ra, rb, e);
      uint64_t j = B.first + lane;
      uint32_t rc = kEmpty, osc = 0;
      if (j < B.end) {
        rc = __ldg(B.nbr + j);
        osc = __ldg(B.os + j);
      }
      for (uint64_t j0 = B.first; j0 < B.end; j0 += kWarp) {
        j += kWarp;  // the next round's entries are loaded before this round's tests
        uint32_t rn = kEmpty, on = 0;
        if (j < B.end) {
          rn = __ldg(B.nbr + j);
          on = __ldg(B.os + j);
        }
        bool push = false;
        uint64_t rec = 0;
        if (rc != kEmpty) {
          uint32_t bk = (rc * 2654435761u) >> shift;
          int t;
          for (;;) {
            const uint4 k4 = reinterpret_cast<const uint4*>(keys)[bk];
            t = k4.x == rc ? 0 : k4.y == rc ? 1 : k4.z == rc ? 2 : k4.w == rc ? 3 : -1;
            if (t >= 0 || k4.w == kEmpty) break;
            bk = (bk + 1) & bmask;
          }
          if (t >= 0) {
            const uint64_t at = ao + val[4 * bk + (uint32_t)t];
            const uint64_t v = exact ? __ldg(A.mask + at) : (uint64_t)__ldg(A.ovl + at);
            const uint32_t cac = exact ? (uint32_t)__popcll(v) : (uint32_t)v;
            if (cac < 2 || rb > rc) {  // three heavy pairs: once, b ranked highest
              const uint32_t g = exact  ? (uint32_t)__popcll(mab & v)
                                 : by_b ? (uint32_t)__popcll(mab & __ldg(A.mask + bo + B.pos[j - kWarp]))
                                        : merge3(A, a, A.slot[rb], A.slot[rc]);
              push = true;
              rec = pack6(osb >> 8, osc >> 8, osb & 0xffu, osc & 0xffu, cac, g);
            }
          }
        }
        queue_records(push, rec, q, qn, [&](uint64_t r) { add_record(W, cls, sa, r); });
        if ((tests += kWarp) >= kFlushTests) {
          flush_counts(W, A.raw);
          tests = 0;
        }
        rc = rn;
        osc = on;
      }
    }
    __syncwarp();
    if (lane < qn) add_record(W, cls, sa, q[lane]);  // the centre's last triangles (they depend on |a|)
    qn = 0;
    __syncthreads();
  }
  flush_counts(W, A.raw);
}

// The same for centres of at most 32 members (32-bit masks, the bulk) or 64,
// with most triangles counted in a histogram instead of queued. For given
// |a|, |b| and C_ab a triangle's contributions depend on C_bc, C_ac, g and |c|
// (only up to C_bc + C_ac + 1), and most overlaps are small: those go to 288
// bins per warp, which become weighted records when the warp has walked the
// rows of all its b alike in |b| and C_ab (of 32 taken together). Fewer than
// kHistMin tests queue every triangle. The enumeration is issue-bound (86 % of
// the issue slots with a record per triangle, 31 ms on a 60K-hyperedge wide
// graph), so instructions per test are what counts. Graphs of up to kDenseSlots
// hyperedges index their table by rank and need no hash.
constexpr uint32_t kHistMin = 96, kHistMax = 1u << 16, kHistBins = 288;
constexpr unsigned kFastThreads = 512, kFastWarps = kFastThreads / kWarp, kFastCol = 4, kFastSlots = 4096;
struct FastWarp {
  WarpCounts<kFastCol> counts;
  uint64_t q[2 * kWarp];     // weighted records
  uint64_t late[2 * kWarp];  // triangles outside the bins
  uint32_t hist[kHistBins];
};
template <class Mask>
constexpr size_t fast_smem() { return kFastWarps * sizeof(FastWarp) + kFastSlots * (sizeof(uint32_t) + sizeof(Mask)); }
constexpr size_t kDenseSmem = kFastWarps * sizeof(FastWarp) + (kDenseSlots + 4) * sizeof(uint32_t);
static_assert(fast_smem<uint64_t>() <= 113 * 1024 && kDenseSmem <= 113 * 1024, "two blocks per SM");

template <bool kDense, class Mask>
__global__ void __launch_bounds__(kFastThreads, 2) k_hh_fast(HHArgs A, uint32_t n_ranks) {
  extern __shared__ uint64_t smem64[];
  FastWarp* F = reinterpret_cast<FastWarp*>(smem64) + threadIdx.x / kWarp;
  WarpCounts<kFastCol>* W = &F->counts;
  Mask* val = reinterpret_cast<Mask*>(reinterpret_cast<FastWarp*>(smem64) + kFastWarps);
  uint32_t* keys = reinterpret_cast<uint32_t*>(val + kFastSlots);  // hash only
  auto bits = [](Mask m) { return (uint32_t)(sizeof(Mask) == 8 ? __popcll(m) : __popc((uint32_t)m)); };
  __shared__ int8_t cls[128];
  __shared__ uint32_t s_item;
  const unsigned w = threadIdx.x / kWarp, lane = lane_id();
  fill_classes(cls);
  clear_counts(W);
  for (unsigned k = lane; k < kHistBins; k += kWarp) F->hist[k] = 0;
  uint32_t qn = 0, ln = 0, tests = 0;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(A.queue, 1u);
    __syncthreads();
    const uint32_t it = s_item;
    if (it >= A.n_work) break;
    const uint32_t ra = A.work[it], a = A.slot[ra];
    const uint64_t ao = A.off[a];
    const uint32_t al = A.len[a];
    const uint32_t sa = A.esize[a];
    uint32_t shift = 0, bmask = 0;
    if (kDense) {
      const uint32_t quads = (n_ranks - ra) / 4 + 1;  // places ra + 1 .. n_ranks, at rank - ra; the last stays 0
      for (uint32_t i = threadIdx.x; i < quads; i += kFastThreads)
        reinterpret_cast<uint4*>(val)[i] = make_uint4(0, 0, 0, 0);
    } else {
      uint32_t slots = 64;
      while (slots < 2 * al && slots < kFastSlots) slots <<= 1;
      shift = 32u - (31u - (uint32_t)__clz(slots / 4));
      bmask = slots / 4 - 1;
      for (uint32_t i = threadIdx.x; i < slots; i += kFastThreads) keys[i] = kEmpty;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < al; i += kFastThreads) {
      const uint32_t key = __ldg(A.rank + __ldg(A.nbr + ao + i));
      if (key <= ra) continue;
      const Mask m = (Mask)__ldg(A.mask + ao + i);
      if (kDense) {
        val[key - ra] = m;
      } else {
        uint32_t bk = (key * 2654435761u) >> shift, h = 0;
        for (bool done = false; !done; bk = (bk + 1) & bmask)
          for (uint32_t t = 0; t < 4; ++t)
            if (atomicCAS(&keys[4 * bk + t], kEmpty, key) == kEmpty) {
              h = 4 * bk + t;
              done = true;
              break;
            }
        val[h] = m;
      }
    }
    __syncthreads();
    const uint64_t he = A.hoff[ra + 1];
    // a waiting triangle: the place of c's entry (bit 31: among the marked
    // rows), C_ac, g, C_ab and |b|
    auto late = [&](uint64_t r) {
      const uint32_t at = (uint32_t)r, hi = (uint32_t)(r >> 32);
      const uint32_t osc = __ldg((at >> 31 ? A.mos : A.hos) + (at & 0x7fffffffu));
      add_triangle(W, cls, sa, hi >> 24, osc >> 8, (hi >> 16) & 0xffu, osc & 0xffu, hi & 0xffu, (hi >> 8) & 0xffu);
    };
    // the warp takes every kFastWarps-th b, 32 at a time, a lane reading each
    for (uint64_t e0 = A.hoff[ra] + w; e0 < he; e0 += kFastWarps * kWarp) {
      const uint64_t e = e0 + (uint64_t)lane * kFastWarps;
      uint32_t my_rb = 0, my_os = 0, my_first = 0, my_n = 0;
      Mask my_mab = 0;
      bool marked_row = false;
      if (e < he) {
        my_rb = A.hnbr[e];
        my_os = A.hos[e];
        my_mab = (Mask)A.mask[ao + A.hpos[e]];
        const Walk B = walk_of(A, ra, my_rb, e);
        my_first = (uint32_t)B.first;
        my_n = (uint32_t)(B.end - B.first);
        marked_row = B.code != A.hcode;
      }
      const unsigned in_marked = __ballot_sync(0xffffffffu, marked_row);
      unsigned todo = __ballot_sync(0xffffffffu, my_n != 0);
      while (todo) {
        const int lead = __ffs(todo) - 1;
        const uint32_t osb = __shfl_sync(0xffffffffu, my_os, lead);
        unsigned peers = todo & __ballot_sync(0xffffffffu, my_os == osb);
        uint32_t total = (peers >> lane) & 1u ? min(my_n, kHistMax) : 0u;
        for (int d = 16; d; d >>= 1) total += __shfl_xor_sync(0xffffffffu, total, d);
        if (total >= kHistMax) {  // a bin's count has to fit a record's 16 bits
          peers = 1u << lead;
          total = __shfl_sync(0xffffffffu, my_n, lead);
        }
        todo &= ~peers;
        const bool bins = total >= kHistMin && total < kHistMax;
        const uint32_t bias = bins ? 0u : 4u;
        for (unsigned left = peers; left; left &= left - 1) {
          const int src = __ffs(left) - 1;
          const uint32_t rb = __shfl_sync(0xffffffffu, my_rb, src), first = __shfl_sync(0xffffffffu, my_first, src),
                         n = __shfl_sync(0xffffffffu, my_n, src);
          const Mask mab = __shfl_sync(0xffffffffu, my_mab, src);
          const bool sub = (in_marked >> src) & 1u;
          const uint32_t* hc = (sub ? A.mcode : A.hcode) + first;
          const uint64_t part = ((uint64_t)osb << 48) | (sub ? 0x80000000u : 0u);
          // One round: the entries cur of the lanes, at hc + at. An entry past
          // the row's end has a rank no table holds.
          auto round = [&](uint32_t cur, uint32_t at) {
            const uint32_t rc = cur >> 8, code = cur & 0xffu;
            Mask v = 0;
            if (kDense) {
              v = val[min(rc - ra, n_ranks - ra)];
            } else {
              uint32_t bk = (rc * 2654435761u) >> shift;
              int t;
              for (;;) {
                const uint4 k4 = reinterpret_cast<const uint4*>(keys)[bk];
                t = k4.x == rc ? 0 : k4.y == rc ? 1 : k4.z == rc ? 2 : k4.w == rc ? 3 : -1;
                if (t >= 0 || k4.w == kEmpty) break;
                bk = (bk + 1) & bmask;
              }
              if (t >= 0) v = val[4 * bk + (uint32_t)t];
            }
            const uint32_t cac = bits(v), g = bits(v & mab);
            const bool take = cac == 1 || (cac > 1 && rb > rc);  // three heavy pairs: once, b ranked highest
            const bool slow = cac + ((code & 0x80u) >> 5) + bias > 3;
            if (take && !slow) atomicAdd(&F->hist[g * 72 + cac * 24 + code - 24], 1u);
            // the others wait as their entry's place and what is known of the
            // triangle; |c| and C_bc are read when 32 have come together
            queue_records(take && slow, part | ((uint64_t)(cac | (g << 8)) << 32) | (first + at), F->late, ln, late);
          };
          for (uint32_t c0 = 0; c0 < n; c0 += kHistMax) {
            const uint32_t c1 = min(n, c0 + kHistMax);
            // two rounds at a time, their successors' entries loaded before them
            uint32_t at = c0 + lane;
            uint32_t x = at < c1 ? __ldg(hc + at) : kEmpty, y = at + kWarp < c1 ? __ldg(hc + at + kWarp) : kEmpty;
            for (uint32_t j0 = c0; j0 < c1; j0 += 2 * kWarp) {
              const uint32_t to = at + 2 * kWarp;
              const uint32_t xn = to < c1 ? __ldg(hc + to) : kEmpty,
                             yn = to + kWarp < c1 ? __ldg(hc + to + kWarp) : kEmpty;
              round(x, at);
              if (j0 + kWarp < c1) round(y, at + kWarp);
              at = to;
              x = xn;
              y = yn;
            }
            if (c1 < n) flush_counts(W, A.raw);
          }
        }
        if ((tests += min(total, kHistMax)) >= kFlushTests - 2 * kHistMax) {
          flush_counts(W, A.raw);
          tests = 0;
        }
        if (!bins) continue;
        __syncwarp();
#pragma unroll 1
        for (uint32_t k0 = 0; k0 < kHistBins; k0 += kWarp) {
          const uint32_t k = k0 + lane;  // |c| - 1 (7 for 8 or more) + 8 (C_bc - 2) + 24 (C_ac - 1) + 72 g
          const uint32_t c = F->hist[k], g = k / 72, m = k - 72 * g, r = m % 24;
          if (c) F->hist[k] = 0;
          queue_records(c != 0, pack6(osb >> 8, (r & 7u) + 1, osb & 0xffu, 2 + (r >> 3), m / 24 + 1, g, c), F->q, qn,
                        [&](uint64_t x) { add_record(W, cls, sa, x); });
        }
      }
    }
    __syncwarp();
    if (lane < qn) add_record(W, cls, sa, F->q[lane]);  // the centre's last triangles (they depend on |a|)
    if (lane < ln) late(F->late[lane]);
    qn = ln = 0;
    __syncthreads();
  }
  flush_counts(W, A.raw);
}

static_assert(kHHSmall <= kFastSlots * 3 / 4, "table load");
constexpr size_t node_smem(unsigned slots) { return slots * (sizeof(uint2) + sizeof(uint32_t)); }
static_assert(kNodeSmall == 1024 / 4 * 3 && kNodeMid == 4096 / 4 * 3 && kNodeLarge == 16384 / 4 * 3, "table load");

// The short node rows alone (k_parts takes them too when they are few): at the
// registers of its own it keeps 6 blocks per SM, k_parts 4.
template <bool kTouch>
__global__ void __launch_bounds__(kBlock, 6) k_node_tri_warp(NodeArgs A) {
  __shared__ NodeWarp S[kWarps];
  part_nodes<kTouch, false>(A, &S[threadIdx.x / kWarp]);
}

// The counter block of the static count (hm_static.cu: 30 closed classes, 6
// removals, 6 open-pair counts) from the raw sums, by one block: a thread per
// sum adds it to the few counters it belongs to.
struct FinishShared {
  unsigned long long o[42];
};
__device__ void finish(FinishShared& S, const unsigned long long* raw, unsigned long long* out) {
  unsigned long long* o = S.o;
  const unsigned t = threadIdx.x;
  auto sum = [&](unsigned k) { return __ldcg(raw + k); };  // written by other blocks' atomics, in L2
  if (t < 42) o[t] = sum(t < 30 ? kRawClass + t : t < 36 ? kRawRem + t - 30 : kRawOpen + t - 36);
  __syncthreads();
  auto add = [&](unsigned k, unsigned long long n) { atomicAdd(&o[k], n); };
  if (t < 4) {
    const unsigned long long n = sum(kRawDist + t);
    add(26 + t, n);
    add(35, t * n);
    add(34, (3 - t) * n);
  } else if (t >= 32 && t < 42) {
    const unsigned i = t - 32;  // the order of star_index
    const unsigned x = i < 6 ? 0 : i < 9 ? 1 : 2, y = i < 6 ? (i < 3 ? 0 : i < 5 ? 1 : 2) : i < 8 ? 1 : 2;
    const unsigned z = i < 6 ? (i < 3 ? i : i < 5 ? i - 2 : 2) : i < 8 ? i - 5 : 2;
    const unsigned long long n = sum(kRawStar + i);
    const unsigned ex = x > 0, ey = y > 0, ez = z > 0;
    add(ex + ey + ez, n);
    add(30 + (x == 2) + 2 * (ey + ez), n);
    add(30 + (y == 2) + 2 * (ex + ez), n);
    add(30 + (z == 2) + 2 * (ex + ey), n);
  } else if (t >= 64 && t < 91) {
    const unsigned i = t - 64, ua = i / 9, ub = i / 3 % 3, c = i % 3;
    const unsigned long long n = sum(kRawPair + i);
    const unsigned ea = ua > 0, eb = ub > 0, l = c > 0;
    // regions: a's and b's own, the pair's, the common node, c's own if it has a second member
    const int pat = (int)(ea | (eb << 1) | (l << 2) | (1u << 3) | (1u << 6));
    add(static_class_of_pattern(pat), n);
    add(30 + (ua > 1) + 2 * (eb + l), n);
    add(30 + (ub > 1) + 2 * (ea + l), n);
    add(30 + (c == 2) + 4, n);
  }
  __syncthreads();
  if (t < 42) out[t] = o[t];
}

// The parts of a count that run in small blocks, side by side in one launch:
// blocks [0, end[0]) search, [end[0], end[1]) sum the heavy pairs, then node
// triangles of the short rows, open pairs, stars. At small sizes each part is
// one wave of latency, so one launch takes as long as its slowest part. It is
// the count's last launch but for the counters, which its last block to end makes
// from the sums where the grid is one wave (a launch of one block took 4 us of a
// 1K-hyperedge count's 75); over several waves each block's wait for its own
// sums to land cost more than that launch (7 us of 484 at 100K hyperedges).
struct PartArgs {
  HHArgs search;
  PairArgs pairs;
  NodeArgs nodes;
  OpenArgs open;
  unsigned end[5];
  unsigned int* ended;      // blocks that have added their sums (null: k_decomp_finish follows)
  unsigned long long* out;  // 42 counters
};
union PartShared {
  SearchShared search;
  PairCounts pairs;
  NodeWarp nodes[kWarps];
  OpenHist open;
  FinishShared finish;
};
template <bool kTouch>
__global__ void __launch_bounds__(kBlock, 4) k_parts(const __grid_constant__ PartArgs A) {
  __shared__ __align__(16) unsigned char mem[sizeof(PartShared)];
  PartShared& S = *reinterpret_cast<PartShared*>(mem);
  const unsigned b = blockIdx.x;
  if (b < A.end[0]) {
    part_search(b, A.end[0], A.search, S.search);
  } else if (b < A.end[1]) {
    part_pairs(b - A.end[0], A.end[1] - A.end[0], S.pairs, A.pairs);
  } else if (b < A.end[2]) {
    part_nodes<kTouch, true>(A.nodes, &S.nodes[threadIdx.x / kWarp]);
  } else if (b < A.end[3]) {
    part_open(b - A.end[2], A.end[3] - A.end[2], S.open, A.open);
  } else {
    part_stars(b - A.end[3], A.end[4] - A.end[3], A.pairs.ncat, A.pairs.ncat_m, A.pairs.n_nodes, A.search.raw);
  }
  if (!A.ended) return;
  __shared__ bool last;
  __threadfence();  // this thread's sums before the block's count
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(A.ended, 1u) == gridDim.x - 1;
  __syncthreads();
  if (last) {
    __threadfence();
    finish(S.finish, A.search.raw, A.out);
  }
}

__global__ void k_decomp_finish(const unsigned long long* raw, unsigned long long* out) {
  __shared__ FinishShared S;
  finish(S, raw, out);
}

unsigned bits_for(uint64_t n) {  // bits of the values 0 .. n - 1
  unsigned b = 1;
  while ((1ull << b) < n) ++b;
  return b;
}

}  // namespace

static int decomp_attrs() {
  HM_CUDA(cudaFuncSetAttribute(k_hh_large, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kHHSmem));
  HM_CUDA(cudaFuncSetAttribute(k_hh_fast<true, uint32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kDenseSmem));
  HM_CUDA(cudaFuncSetAttribute(k_hh_fast<false, uint32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)fast_smem<uint32_t>()));
  HM_CUDA(cudaFuncSetAttribute(k_hh_fast<false, uint64_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)fast_smem<uint64_t>()));
  auto node = [](auto* big, auto* mid) -> int {
    HM_CUDA(cudaFuncSetAttribute(big, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)node_smem(16384)));
    HM_CUDA(cudaFuncSetAttribute(mid, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)node_smem(4096)));
    return HM_OK;
  };
  HM_TRY(node(k_node_tri<false, 16384, 1024, 1>, k_node_tri<false, 4096, 512, 2>));
  HM_TRY(node(k_node_tri<true, 16384, 1024, 1>, k_node_tri<true, 4096, 512, 2>));
  return HM_OK;
}

// Whether the decomposition is the cheaper count, and its structures if so.
// It enumerates sum h^2 / 2 tests; the oriented rows hold about a quarter of
// sum d^2 / 2 entries to probe (measured 0.24 to 0.30 on the named laws), and
// a test costs about as much as a probe, so it needs sum h^2 <= sum d^2 / 4. Then
// the node graph has to be worth it: W entries walked for its triangles, P node
// pairs, and the latency of the largest items, which a few warps sum while the rest
// of the GPU is done: Z members at most, X = |a| |b| of a heavy pair at most, a share
// L of the GPU's warps with a heavy pair. With nnz = sum d and B = sum d^3 / n over
// the hyperedges of more than 64 members times their share of all (their triangles
// are merged, not masked), in ns beside 60 us each:
//   decomposed  0.0014 h^2 + 0.008 W + 0.06 P + 3.7 Z^2 + 16 X L
//   enumerated  0.0011 d^2 + 12.6 sqrt(d^2) + 0.048 nnz + 0.3 B
// and for the touched triples of m of n hyperedges, whose walk goes through c entries
// (and whose tables are built for one count)
//   decomposed  0.0014 h^2 min(1, 3 m / n) + 0.01 W + 0.3 P + 3.7 Z^2 + 16 X L
//   walked      0.003 c.
// Fitted on 300 graphs timed both ways, of 100 to 50K hyperedges of all laws and
// sizes: the way the sums name takes 1.4 % more than the better one on average, at
// most 1.8 times as long. Decomposed / enumerated, ms: 8K hub hyperedges 13.7 /
// 146, 100K of 4 to 8 members over 200K nodes 0.31 / 0.56, 3,458 hyperedges, a few of
// them of up to 120 members, 0.66 / 0.10, 20K of 20 to 40 over 20K nodes 25.4 / 18.6,
// 20K of 60 to 100 over 2M nodes 23.5 / 1.2 (and 54 / 0.7 to prepare). Before the
// table is built W is taken from node_walk, or 3/2 of the hyperedges' own node
// triples (the least measured).
// With mark (per slot) the structures of a touched-triple count of `marked`
// hyperedges and walk cost `cost`.
static int build_decomp(hm_graph* g, Decomp& P, const uint8_t* mark, uint32_t marked = 0, uint64_t cost = 0) {
  hm_ctx* ctx = g->ctx;
  cudaStream_t st = ctx->stream;
  const uint32_t E = g->n_slots, V = g->n_nodes;
  P.release();
  P.decided = true;
  if (!E || !V) return HM_OK;
  DArr<uint32_t> heavy, ids, deg, hcnt;
  DArr<unsigned long long> sums;
  HM_TRY(heavy.alloc(ctx, E));
  HM_TRY(ids.alloc(ctx, E));
  HM_TRY(deg.alloc(ctx, E));
  HM_TRY(hcnt.alloc(ctx, E));
  HM_TRY(sums.alloc(ctx, kSums + kClasses));  // and the nodes' classes
  HM_TRY(P.rank.alloc(ctx, E));
  HM_TRY(P.slot.alloc(ctx, E));
  HM_TRY(P.hoff.alloc(ctx, (size_t)E + 1));
  HM_TRY(P.ncat.alloc(ctx, 3 * (size_t)V));
  if (mark) HM_TRY(P.ncat_m.alloc(ctx, 3 * (size_t)V));
  HM_CUDA(cudaMemsetAsync(sums.p, 0, (kSums + kClasses) * sizeof(unsigned long long), st));
  // as many nodes of one degree would give the adjacency there is
  const double mem = (double)g->h2v_nnz;
  const float even = (float)std::max(1.0, std::min((double)V, mem * mem / ((double)g->h2h_nnz + mem + 1.0)));
  k_node_cats<<<grid_for((uint64_t)V * 32, kBlock), kBlock, 0, st>>>(g->v2h_off.p, g->v2h_len.p, g->v2h_edge.p,
                                                                    g->esize.p, mark, V, even, P.ncat.p, P.ncat_m.p,
                                                                    reinterpret_cast<float*>(sums.p + kSums));
  HM_LAUNCH_CHECK();
  // a heavy pair's 16 ns |a| |b| below 9 us, or a hundredth of the other way's least
  // time (sum d^2 >= nnz^2 / n), cannot decide
  const double least = mark ? 0.003 * (double)cost : 0.0011 * (double)g->h2h_nnz * (double)g->h2h_nnz / E;
  const uint32_t large_pair = (uint32_t)std::min(65025.0, std::max(576.0, 0.01 * least / 16));
  k_heavy_count<<<grid_for((uint64_t)E * 32, kBlock), kBlock, 0, st>>>(
      g->h2h_off.p, g->h2h_len.p, g->h2h_nbr.p, g->h2h_ovl.p, g->esize.p, mark, E, large_pair, heavy.p, ids.p, sums.p);
  HM_LAUNCH_CHECK();
  const unsigned bits = bits_for(E);
  {
    size_t tb = 0;
    HM_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, g->h2h_len.p, deg.p, ids.p, P.slot.p, (int64_t)E, 0, (int)bits,
                                            st));
    DArr<uint8_t> tmp;
    HM_TRY(tmp.alloc(ctx, tb));
    HM_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, tb, g->h2h_len.p, deg.p, ids.p, P.slot.p, (int64_t)E, 0, (int)bits,
                                            st));
  }
  k_rank_scatter<<<grid_for(E, kBlock), kBlock, 0, st>>>(P.slot.p, E, heavy.p, P.rank.p, hcnt.p);
  HM_LAUNCH_CHECK();
  HM_TRY(exclusive_scan(ctx, hcnt.p, P.hoff.p, E));
  unsigned long long hs[kSums + kClasses];
  HM_CUDA(cudaMemcpyAsync(hs, sums.p, sizeof(hs), cudaMemcpyDeviceToHost, st));
  HM_CUDA(cudaStreamSynchronize(st));
  float hc[2 * kClasses];
  std::memcpy(hc, hs + kSums, sizeof(hc));
  const uint64_t h2 = hs[0], d2 = hs[1], pairs = hs[2], nh = hs[3];
  uint64_t tslots = 1024;
  while (tslots < 2 * pairs) tslots <<= 1;
  uint64_t cslots = 1024;  // the marked hyperedges' own table
  while (cslots < 2 * hs[4]) cslots <<= 1;
  const size_t need = tslots * (sizeof(uint4) + (mark ? sizeof(uint2) : 0)) + (mark ? cslots * sizeof(uint4) : 0) + pairs * (mark ? 60 : 36) +
                      nh * (22 + 24 + (mark ? 18 : 0));
  const size_t room = ctx->budget ? ctx->budget - std::min<size_t>(ctx->budget, ctx->used.load()) : SIZE_MAX;
  auto worth = [&](double walk) {
    if (g->force_decomp) return true;
    if (h2 > d2 / 4) return false;
    const double lone = std::min(1.0, (double)nh / (ctx->n_sms * 8.0 * kWarps));
    const double largest = 3.7 * (double)hs[9] * (double)hs[9] + 16.0 * (double)hs[8] * lone;
    if (mark)
      return 0.0014 * (double)h2 * std::min(1.0, 3.0 * marked / E) + 0.01 * walk + 0.3 * (double)pairs + largest <=
             0.003 * (double)cost;
    return 0.0014 * (double)h2 + 0.008 * walk + 0.06 * (double)pairs + largest <=
           0.0011 * (double)d2 + 12.6 * std::sqrt((double)d2) + 0.048 * (double)g->h2h_nnz +
               0.3 * (double)hs[6] * (double)hs[7] / E;
  };
  P.need = need;
  if (!worth(std::max(1.5 * (double)hs[5], node_walk(hc))) || nh >= (1ull << 31) || tslots > (1ull << 31)) {
    P.release();
    P.decided = true;
    return HM_OK;
  }
  if (need > room / 2) return set_error(HM_ERR_NOMEM, "decomposition: %zu bytes of %zu", need, room);
  P.nh = nh;
  P.by_entry = nh <= kEntriesFew && h2 <= kEntryTests;
  HM_TRY(P.hnbr.alloc(ctx, nh));
  HM_TRY(P.hown.alloc(ctx, nh));
  HM_TRY(P.hos.alloc(ctx, nh));
  HM_TRY(P.hpos.alloc(ctx, nh));
  HM_TRY(P.hnext.alloc(ctx, nh));
  HM_TRY(P.hcode.alloc(ctx, nh));
  if (nh) {
    DArr<uint64_t> key, key_s;
    DArr<uint32_t> pos, pos_s;
    HM_TRY(key.alloc(ctx, nh));
    HM_TRY(key_s.alloc(ctx, nh));
    HM_TRY(pos.alloc(ctx, nh));
    HM_TRY(pos_s.alloc(ctx, nh));
    k_heavy_emit<<<grid_for((uint64_t)E * 32, kBlock), kBlock, 0, st>>>(P.slot.p, P.rank.p, E, g->h2h_off.p,
                                                                       g->h2h_len.p, g->h2h_nbr.p, g->h2h_ovl.p,
                                                                       P.hoff.p, bits, key.p, pos.p);
    HM_LAUNCH_CHECK();
    size_t tb = 0;
    HM_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, key.p, key_s.p, pos.p, pos_s.p, (int64_t)nh, 0,
                                            (int)(2 * bits), st));
    DArr<uint8_t> tmp;
    HM_TRY(tmp.alloc(ctx, tb));
    HM_CUDA(cub::DeviceRadixSort::SortPairs(tmp.p, tb, key.p, key_s.p, pos.p, pos_s.p, (int64_t)nh, 0,
                                            (int)(2 * bits), st));
    k_heavy_rows<<<grid_for(nh, kBlock), kBlock, 0, st>>>(key_s.p, pos_s.p, nh, bits, P.slot.p, g->h2h_off.p,
                                                          g->h2h_ovl.p, g->esize.p, P.hoff.p, P.hnbr.p, P.hown.p,
                                                          P.hos.p, P.hpos.p, P.hnext.p, P.hcode.p);
    HM_LAUNCH_CHECK();
  }
  if (mark) {
    HM_TRY(P.rmark.alloc(ctx, E));
    HM_TRY(P.moff.alloc(ctx, (size_t)E + 1));
    HM_TRY(P.mnbr.alloc(ctx, nh));
    HM_TRY(P.mos.alloc(ctx, nh));
    HM_TRY(P.mpos.alloc(ctx, nh));
    HM_TRY(P.mnext.alloc(ctx, nh));
    HM_TRY(P.mcode.alloc(ctx, nh));
    k_rank_marks<<<grid_for(E, kBlock), kBlock, 0, st>>>(P.slot.p, E, mark, P.rmark.p);
    HM_LAUNCH_CHECK();
    k_marked_count<<<grid_for((uint64_t)E * 32, kBlock), kBlock, 0, st>>>(P.hoff.p, P.hnbr.p, P.rmark.p, E, hcnt.p);
    HM_LAUNCH_CHECK();
    HM_TRY(exclusive_scan(ctx, hcnt.p, P.moff.p, E));
    k_marked_fill<<<grid_for((uint64_t)E * 32, kBlock), kBlock, 0, st>>>(P.hoff.p, P.hnbr.p, P.hos.p, P.hpos.p,
                                                                        P.rmark.p, E, P.moff.p, P.mnbr.p, P.mos.p,
                                                                        P.mpos.p, P.mcode.p);
    HM_LAUNCH_CHECK();
    if (nh) {
      k_marked_next<<<grid_for(nh, kBlock), kBlock, 0, st>>>(P.hown.p, P.hnbr.p, nh, P.moff.p, P.mnbr.p, P.mnext.p);
      HM_LAUNCH_CHECK();
    }
    HM_TRY(P.tab_m.alloc(ctx, tslots));
    HM_TRY(P.nw_m.alloc(ctx, pairs));
    HM_CUDA(cudaMemsetAsync(P.tab_m.p, 0, sizeof(uint2) * tslots, st));
    P.cslots = cslots;
    HM_TRY(P.tab_c.alloc(ctx, cslots));
    HM_CUDA(cudaMemsetAsync(P.tab_c.p, 0, sizeof(uint4) * cslots, st));
  }
  // node graph
  P.tslots = tslots;
  HM_TRY(P.tab.alloc(ctx, tslots));
  HM_TRY(P.noff.alloc(ctx, (size_t)V + 1));
  HM_TRY(P.nlen.alloc(ctx, V));
  HM_TRY(P.nnbr.alloc(ctx, pairs));
  HM_TRY(P.nw.alloc(ctx, pairs));
  HM_TRY(P.hwork.alloc(ctx, E));
  HM_TRY(P.nwork.alloc(ctx, V));
  HM_TRY(P.spread.alloc(ctx, E));
  HM_TRY(P.slist.alloc(ctx, E));
  DArr<uint32_t> ndeg;     // V degrees, then V write cursors
  DArr<uint32_t> bk;       // per list: kBuckets counts, kBuckets starts, 4 shape ends
  DArr<uint8_t> hcode, ncode;
  constexpr uint32_t kBk = 2 * kBuckets + 4;
  HM_TRY(ndeg.alloc(ctx, 2 * (size_t)V));
  // and the number of spreading owners, nothing, the node triangles' walk (8 bytes)
  constexpr uint32_t kBkAll = 2 * kBk + 4;
  HM_TRY(bk.alloc(ctx, kBkAll));
  HM_TRY(hcode.alloc(ctx, E));
  HM_TRY(ncode.alloc(ctx, V));
  HM_CUDA(cudaMemsetAsync(P.tab.p, 0, sizeof(uint4) * tslots, st));
  HM_CUDA(cudaMemsetAsync(P.nlen.p, 0, sizeof(uint32_t) * V, st));
  HM_CUDA(cudaMemsetAsync(ndeg.p, 0, sizeof(uint32_t) * 2 * V, st));
  HM_CUDA(cudaMemsetAsync(bk.p, 0, sizeof(uint32_t) * kBkAll, st));
  const uint32_t tmask = (uint32_t)(tslots - 1);
  k_pair_insert<<<grid_for((uint64_t)E * 32, kBlock), kBlock, 0, st>>>(g->h2v_off.p, g->h2v_mem.p, g->esize.p, mark,
                                                                      nullptr, E, P.tab.p, P.tab_m.p, tmask);
  HM_LAUNCH_CHECK();
  if (mark) {
    k_pair_insert<<<grid_for((uint64_t)E * 32, kBlock), kBlock, 0, st>>>(
        g->h2v_off.p, g->h2v_mem.p, g->esize.p, nullptr, mark, E, P.tab_c.p, nullptr, (uint32_t)(cslots - 1));
    HM_LAUNCH_CHECK();
  }
  k_pair_degrees<<<grid_for(tslots, kBlock), kBlock, 0, st>>>(P.tab.p, tslots, ndeg.p);
  HM_LAUNCH_CHECK();
  k_pair_plus_count<<<grid_for(tslots, kBlock), kBlock, 0, st>>>(P.tab.p, tslots, ndeg.p, P.nlen.p);
  HM_LAUNCH_CHECK();
  HM_TRY(exclusive_scan(ctx, P.nlen.p, P.noff.p, V));
  k_pair_plus_fill<<<grid_for(tslots, kBlock), kBlock, 0, st>>>(P.tab.p, P.tab_m.p, tslots, ndeg.p, P.noff.p,
                                                               ndeg.p + V, P.nnbr.p, P.nw.p, P.nw_m.p);
  HM_LAUNCH_CHECK();
  if (!P.by_entry) {
    k_hh_codes<<<grid_for((uint64_t)E * 32, kBlock), kBlock, 0, st>>>(P.slot.p, P.rank.p, E, g->esize.p, g->h2h_off.p,
                                                                   g->h2h_len.p, g->h2h_nbr.p, P.hoff.p, P.hnbr.p,
                                                                   P.hnext.p, P.rmark.p, P.moff.p, P.mnext.p, hcode.p, bk.p);
    HM_LAUNCH_CHECK();
  }
  k_spread_flags<<<grid_for((uint64_t)E * 32, kBlock), kBlock, 0, st>>>(
      P.slot.p, E, P.hoff.p, P.hnbr.p, P.hos.p, g->h2v_off.p, g->h2v_mem.p, g->esize.p, ndeg.p, P.spread.p, P.slist.p,
      bk.p + 2 * kBk);
  HM_LAUNCH_CHECK();
  k_node_codes<<<grid_for((uint64_t)V * 32, kBlock), kBlock, 0, st>>>(P.noff.p, P.nlen.p, P.nnbr.p, V, ncode.p,
                                                                     bk.p + kBk,
                                                                     reinterpret_cast<unsigned long long*>(bk.p + 2 * kBk + 2));
  HM_LAUNCH_CHECK();
  for (int l = P.by_entry ? 1 : 0; l < 2; ++l) {
    uint32_t* b = bk.p + l * kBk;
    k_bucket_starts<<<1, kBuckets, 0, st>>>(b, b + kBuckets, b + 2 * kBuckets);
    HM_LAUNCH_CHECK();
    const uint32_t n = l ? V : E;
    k_bucket_scatter<<<grid_for(n, kBlock), kBlock, 0, st>>>(l ? ncode.p : hcode.p, n, b + kBuckets,
                                                            l ? P.nwork.p : P.hwork.p);
    HM_LAUNCH_CHECK();
  }
  uint32_t ends[kBkAll];
  HM_CUDA(cudaMemcpyAsync(ends, bk.p, sizeof(ends), cudaMemcpyDeviceToHost, st));
  HM_CUDA(cudaStreamSynchronize(st));
  unsigned long long walk = 0;
  std::memcpy(&walk, ends + 2 * kBk + 2, sizeof(walk));
  if (!worth((double)walk)) {
    P.release();
    P.decided = true;
    return HM_OK;
  }
  std::memcpy(P.hend, ends + 2 * kBuckets, sizeof(P.hend));
  std::memcpy(P.nend, ends + kBk + 2 * kBuckets, sizeof(P.nend));
  P.n_spread = ends[2 * kBk];
  if (P.n_spread) {
    // one node vector per block of k_spread_pairs, a sixteenth of the room at most
    const size_t vec = ((size_t)V + 1) & ~(size_t)1;
    P.y_blocks = (uint32_t)std::max<size_t>(
        1, std::min<size_t>({(size_t)ctx->n_sms, (size_t)P.n_spread, room / 16 / (sizeof(uint2) * vec)}));
    const size_t y_all = (size_t)P.y_blocks * vec;
    HM_TRY(P.self.alloc(ctx, g->h2v_tail));
    if (mark) HM_TRY(P.self_m.alloc(ctx, g->h2v_tail));
    if (mark) HM_TRY(P.fw_m.alloc(ctx, 2 * pairs));
    HM_TRY(P.y.alloc(ctx, y_all));
    HM_CUDA(cudaMemsetAsync(P.y.p, 0, sizeof(uint2) * y_all, st));
    HM_TRY(P.foff.alloc(ctx, (size_t)V + 1));
    HM_TRY(P.fnbr.alloc(ctx, 2 * pairs));
    HM_TRY(P.fw.alloc(ctx, 2 * pairs));
    HM_TRY(exclusive_scan(ctx, ndeg.p, P.foff.p, V));
    HM_CUDA(cudaMemsetAsync(ndeg.p + V, 0, sizeof(uint32_t) * V, st));
    k_pair_rows_fill<<<grid_for(tslots, kBlock), kBlock, 0, st>>>(P.tab.p, P.tab_m.p, tslots, P.foff.p, ndeg.p + V,
                                                                 P.fnbr.p, P.fw.p, P.fw_m.p);
    HM_LAUNCH_CHECK();
  }
  HM_TRY(P.raw.alloc(ctx, kRawSize));
  HM_TRY(decomp_attrs());
  P.usable = true;
  return HM_OK;
}

int prepare_decomp(hm_graph* g) {
  hm_ctx* ctx = g->ctx;
  Decomp& P = g->decomp;
  auto others = [&] { return ctx->used.load() - std::min(ctx->used.load(), plus_bytes(g)); };
  auto room = [&] { return ctx->budget - std::min(ctx->budget, ctx->used.load()); };
  if (P.decided && !(P.need && others() < P.others && P.need <= room() / 2)) return HM_OK;
  const int s = build_decomp(g, P, nullptr);
  const size_t need = P.need;
  if (s < 0) P.release();
  if (s == HM_ERR_NOMEM) {  // no room for it: the enumeration of all triangles needs less
    P.decided = true;
    P.need = std::max<size_t>(need, 1);
    P.others = others();
    return HM_OK;
  }
  P.need = 0;
  if (P.usable) release_groups(g);  // a full count walks them no more
  return s;
}

// Warps that share an item of k_parts where there are few: a power of two, as
// many as the chip holds and a block has at most. A warp alone took 19 us for the largest
// heavy pair and 15 us for the longest node row of a 1K-hyperedge count.
static uint32_t slices_of(uint64_t items, unsigned sms) {
  uint32_t s = 1;
  while (s < kWarps && items * s * 2 <= (uint64_t)sms * 8 * kWarps) s *= 2;
  return s;
}

// One count: the raw sums cleared, the block-per-item launches, the small
// parts side by side, and the counter block from the sums.
template <bool kTouch>
static int launch_parts(hm_graph* g, Decomp& P, unsigned long long* counters, Launches& L) {
  hm_ctx* ctx = g->ctx;
  const unsigned sms = (unsigned)ctx->n_sms;
  const uint32_t E = g->n_slots, V = g->n_nodes;
  unsigned int* queue = reinterpret_cast<unsigned int*>(P.raw.p + kRawQueue);
  HM_TRY(L.zero(P.raw.p, kRawSize));
  PartArgs A;
  A.search = HHArgs{P.slot.p, P.rank.p, P.hoff.p, P.hnbr.p, P.hos.p, P.hpos.p, P.hnext.p, P.hcode.p, g->h2h_off.p, g->h2h_len.p,
                    g->h2h_nbr.p, g->h2h_ovl.p, g->h2h_mask.p, g->h2v_off.p, g->h2v_mem.p, g->esize.p, P.rmark.p,
                    P.moff.p, P.mnbr.p, P.mos.p, P.mpos.p, P.mnext.p, P.mcode.p, nullptr, 0, 1, P.hown.p,
                    P.by_entry ? P.nh : 0, nullptr, P.raw.p};
  A.pairs = PairArgs{P.hown.p, P.hnbr.p, P.hos.p, P.hpos.p, P.hnext.p, P.hoff.p, P.nh, P.slot.p, g->h2h_off.p,
                     g->h2h_mask.p, g->h2v_off.p, g->h2v_mem.p, g->esize.p, P.ncat.p, P.tab.p,
                     (uint32_t)(P.tslots - 1), P.rmark.p, P.ncat_m.p, P.tab_c.p,
                     (uint32_t)(P.cslots ? P.cslots - 1 : 0), P.fw_m.p, P.self_m.p, P.foff.p,
                     P.fnbr.p, P.fw.p, P.spread.p, P.slist.p, P.n_spread, P.self.p, P.y.p,
                     V, P.nh < kPairFew ? 1u : 4u, P.nh < kPairFew ? 0u : kPairWide,
                     slices_of(P.nh, sms), queue + 8, P.raw.p};
  A.nodes = NodeArgs{P.noff.p, P.nlen.p, P.nnbr.p, P.nw.p, P.tab.p, (uint32_t)(P.tslots - 1), P.nw_m.p, P.tab_m.p,
                     nullptr, 0, nullptr, P.raw.p, 1};
  A.open = OpenArgs{P.slot.p, E, g->h2v_off.p, g->h2v_mem.p, g->esize.p, g->h2h_len.p, P.ncat.p, P.ncat_m.p, P.hoff.p,
                    P.hnbr.p, P.hos.p, P.rmark.p, P.raw.p};
  auto hh_part = [&](int k) {
    const uint32_t b = k ? P.hend[k - 1] : 0;
    A.search.work = P.hwork.p + b;
    A.search.n_work = P.hend[k] - b;
    A.search.queue = queue + k;
    return A.search.n_work;
  };
  auto node_part = [&](int k) {
    const uint32_t b = k ? P.nend[k - 1] : 0;
    A.nodes.work = P.nwork.p + b;
    A.nodes.n_work = P.nend[k] - b;
    A.nodes.queue = queue + 4 + k;
    return A.nodes.n_work;
  };
  if (const uint32_t n = hh_part(3)) {
    A.search.slices = std::min(16u, std::max(1u, 8 * sms / n));
    HM_TRY(L.run(k_hh_large, std::min(sms, n * A.search.slices), kHHThreads, kHHSmem, A.search));
  }
  if (const uint32_t n = hh_part(2))
    HM_TRY(L.run(k_hh_fast<false, uint64_t>, std::min(sms * 2, n), kFastThreads, fast_smem<uint64_t>(), A.search, E));
  if (const uint32_t n = hh_part(1)) {
    if (E <= kDenseSlots)
      HM_TRY(L.run(k_hh_fast<true, uint32_t>, std::min(sms * 2, n), kFastThreads, kDenseSmem, A.search, E));
    else
      HM_TRY(L.run(k_hh_fast<false, uint32_t>, std::min(sms * 2, n), kFastThreads, fast_smem<uint32_t>(), A.search, E));
  }
  if (P.n_spread) {
    HM_TRY(L.run(k_self_weights, grid_for((uint64_t)E * 32, kBlock), kBlock, 0, A.pairs, E));
    HM_TRY(L.run(k_spread_pairs, P.y_blocks, kSpreadThreads, 0, A.pairs));
  }
  if (const uint32_t n = node_part(3))
    HM_TRY(L.run(k_node_tri<kTouch, 16384, 1024, 1>, std::min(sms, n), 1024, node_smem(16384), A.nodes));
  if (const uint32_t n = node_part(2))
    HM_TRY(L.run(k_node_tri<kTouch, 4096, 512, 2>, std::min(sms * 4, n), 512, node_smem(4096), A.nodes));
  if (const uint32_t n = node_part(1))
    HM_TRY(L.run(k_node_tri<kTouch, 1024, 256, 6>, std::min(sms * 6, n), 256, node_smem(1024), A.nodes));
  const uint32_t n_search = hh_part(0);
  uint32_t n_nodes = node_part(0);
  if (n_nodes > kNodesAlone) {
    HM_TRY(L.run(k_node_tri_warp<kTouch>, std::min(sms * 12, (n_nodes + kWarps - 1) / kWarps), kBlock, 0, A.nodes));
    n_nodes = 0;
  }
  auto blocks = [&](uint64_t warps, unsigned most) {
    return (unsigned)std::min<uint64_t>(sms * most, (warps + kWarps - 1) / kWarps);
  };
  unsigned end = 0;
  A.end[0] = end += blocks(P.by_entry ? P.nh : n_search, 4);
  A.end[1] = end += blocks((P.nh * A.pairs.slices + A.pairs.per_warp - 1) / A.pairs.per_warp, 8);
  A.nodes.slices = n_nodes ? slices_of(n_nodes, sms) : 1;
  A.end[2] = end += blocks((uint64_t)n_nodes * A.nodes.slices, 8);
  A.end[3] = end += blocks(E, 8);
  A.end[4] = end += std::min<unsigned>(sms * 2, (V + kBlock - 1) / kBlock);
  A.ended = end <= sms * 4 ? queue + 12 : nullptr;
  A.out = counters;
  HM_TRY(L.run(k_parts<kTouch>, end, kBlock, 0, A));
  if (!A.ended)
    HM_TRY(L.run(k_decomp_finish, 1, 128, 0, P.raw.p, counters));
  return HM_OK;
}

void routes_of(const Decomp& P, uint32_t* by_entry, uint32_t centres[4], uint32_t* spread) {
  *by_entry = P.by_entry;
  for (int k = 0; k < 4; ++k) centres[k] = P.hend[k] - (k ? P.hend[k - 1] : 0);
  *spread = P.n_spread;
}

int launch_decomp(hm_graph* g, Launches& L) { return launch_parts<false>(g, g->decomp, g->counters.p, L); }

// The triples with a marked hyperedge, count(G) - count(G without them), by the
// same forms: every sum over nodes, node pairs and heavy pairs minus the same
// sum over the unmarked hyperedges (linear in the marked ones' weights where a
// pair is unmarked), and only the triangles with two or three heavy pairs that
// hold a mark enumerated. *done = false (and nothing counted) where the graph
// does not suit the decomposition or the device has no room for it.
int count_touching_decomp(hm_graph* g, const uint8_t* mark, uint32_t marked, uint64_t cost, uint64_t out30[30],
                          bool* done) {
  *done = false;
  Decomp P;
  DArr<unsigned long long> cnt;
  int s = build_decomp(g, P, mark, marked, cost);
  if (s >= 0) s = cnt.alloc(g->ctx, 42);
  if (s == HM_ERR_NOMEM || (s >= 0 && !P.usable)) return HM_OK;
  HM_TRY(s);
  Launches L{g->ctx->stream};
  HM_TRY(launch_parts<true>(g, P, cnt.p, L));
  unsigned long long h[42];
  HM_CUDA(cudaMemcpyAsync(h, cnt.p, sizeof(h), cudaMemcpyDeviceToHost, g->ctx->stream));
  HM_CUDA(cudaStreamSynchronize(g->ctx->stream));
  for (int k = 0; k < 30; ++k) out30[k] = h[k];
  for (int k = 0; k < 6; ++k) out30[20 + k] += h[36 + k] - h[30 + k];
  routes_of(P, &g->routes.touch_by_entry, g->routes.touch_centres, &g->routes.touch_spread);
  *done = true;
  return HM_OK;
}

}  // namespace hm
