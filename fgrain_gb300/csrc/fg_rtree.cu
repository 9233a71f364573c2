// Device builder of the reference tree (BVH::build / subdivide, bvh.rs:157-295); see fg_rtree.cuh.
//
// The tree's topology is built top-down, one level at a time over all tiles of a batch, by one
// cooperative kernel (k_rt_levels) whose blocks pass the phases of a level together:
//   decide  leaf or split (largest centroid extent, midpoint 0.5 (lo + hi)), children ids;
//   flag    every element of a splitting node: centroid >= mid ("big"), with the running number of
//           bigs (a prefix sum along each tile, chunk by chunk); P and Q list the positions of the
//           bigs and of the smalls by that number;
//   place   every element moves to where the reference's swap partition puts it (below), and its
//           centroid joins its child's centroid box (min / max on order-preserving keys: exact
//           whatever the order, and on the integer pipes).
// The splits read only the centroids (bvh.rs:196-258), so each element's three order-preserving
// centroid keys travel with it, and every pass reads them in order.  A centroid is the midpoint of
// the FP64 max_dim box, which for FP32 crystals without expansion is the FP32 position itself: such
// trees carry 32-bit keys, the others 64-bit ones.  Nodes of at most RT_CTA_MAX elements leave the
// global levels: one thread block each builds their subtree with the elements in shared memory, the
// same passes per level, all levels down to the leaves.  The leaf boxes (the union of the elements'
// boxes) are formed by a pass over the leaves; the boxes above them, which only the walks need,
// bottom up (min and max are exact, so the order does not matter).
//
// The swap partition (bvh.rs:244-258: i from the left, j from the right; a small at i stays and i
// advances, a big at i is swapped with j and j retreats) examines the range as two streams: the
// left stream runs while it sees smalls, the right stream while it sees bigs.  With S the number
// of smalls, K = the number of bigs among the first S positions (the pairs the swaps exchange) and
// Q_0 = n, the left stream covers [0, li) where li = S + 1 if position S holds a big, else S; and
// the element at relative position r goes to
//   r < li, small:            r                      (stays)
//   r < li, the m-th big:     Q_{m-1} - 1            (bigs fill the right end in examination order)
//   r >= li, the m-th small from the right:  P_m     (takes the place of the m-th big)
//   r >= li, big:             r - 1                  (shifts one place towards the middle)
// where P_m is the m-th big from the left and Q_m the m-th small from the right; S is the left
// child's size.  A simulation of the reference loop confirms the rule and the closed forms of K and
// li on random ranges.
#include <algorithm>
#include <climits>
#include <cmath>
#include <type_traits>

#include "fg_internal.h"
#include "fg_rtree.cuh"

namespace fg {

namespace {

constexpr unsigned RT_BLOCK = 256;

// Most global split levels for trees of up to emax elements: halving down to the per-block size,
// plus a wide margin for uneven splits (the kernel ends with the last level that has work).
constexpr int RT_LEVELS = 44;
int levels_for(uint32_t emax) {
  if (emax <= static_cast<uint32_t>(RT_CTA_MAX)) return 0;
  int lv = 0;
  while ((static_cast<unsigned long long>(RT_CTA_MAX) << lv) < emax) ++lv;
  return std::min(lv + 8, RT_LEVELS);
}

// Work goes by chunks of consecutive positions (a tile's chunks start at its first): wpw words of 32
// positions for each of a block's eight warps.  A warp's words follow one another, so small builds
// take short chunks: enough blocks, and less latency in a row.  The line is drawn by capacity (about 1.33 times a
// synthesized tile's crystals).  Trees and cells of one t-max tile with two words and with eight, in ms: 260 k
// crystals .346 and .364, 301 k .362 and .364, 342 k (455 k of capacity) .391 and .377, 382 k .418 and .384,
// 502 k .521 and .445, 1.0 M .847 and .630; scan stages with all of them developed (64-bit keys): .681 and
// .726, .730 and .755, .809 and .801, .844 and .810, .996 and .961, 1.715 and 1.465.  Tri-x is within 2 % of these.
// Several tiles have fewer levels of the same elements, and the two are even a little later: 4 to 36 tiles of
// 360 k crystals in all .23 - .30 and .25 - .33, 415 k (550 k of capacity) .36 and .34, 500 k .38 and .35.
constexpr int RT_WARPS = RT_BLOCK / 32;
constexpr int RT_WPW_LARGE = 8, RT_WPW_SMALL = 2;
constexpr unsigned long long RT_LARGE = 520ull * 1000ull;  // elements from which chunks are long
// Blocks per SM that a build's registers leave (32-bit keys: trees of a 1400 x 1400 px t-max image in
// 6.77 ms with four, 6.33 with five, 6.51 with six; 64-bit keys: a gradient step in 4.07, 4.30, 4.36).
constexpr int rt_blocks(bool wide) { return wide ? 4 : 5; }
constexpr unsigned rt_chunk(int wpw) { return 32u * RT_WARPS * static_cast<unsigned>(wpw); }
constexpr unsigned RT_CNT_BAR = 4;               // RtArgs::cnt: the grid barrier's arrivals
constexpr unsigned RT_CNT_TILES = 16;            // first of ntiles + 1 words: chunks before each tile

__device__ __forceinline__ unsigned long long ord64(double v) {
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(v));
  return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double unord64(unsigned long long u) {
  const unsigned long long b = (u & 0x8000000000000000ull) ? (u & 0x7fffffffffffffffull) : ~u;
  return __longlong_as_double(static_cast<long long>(b));
}
__device__ __forceinline__ uint32_t ord32(float v) {
  const uint32_t b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float unord32(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}
__device__ __forceinline__ unsigned long long umin64(unsigned long long a, unsigned long long b) { return a < b ? a : b; }
__device__ __forceinline__ unsigned long long umax64(unsigned long long a, unsigned long long b) { return a > b ? a : b; }

// The split of a node whose centroids span lo .. hi (subdivide, bvh.rs:200-243): the axis of the largest
// extent, -1 for a leaf (degenerate centroids), and the midpoint.
__device__ __forceinline__ int split64(const double lo[3], const double hi[3], double& mid) {
  const double ex = __dsub_rn(hi[0], lo[0]), ey = __dsub_rn(hi[1], lo[1]), ez = __dsub_rn(hi[2], lo[2]);
  const int axis = (ex >= ey && ex >= ez) ? 0 : (ey >= ez ? 1 : 2);
  const double ext = axis == 0 ? ex : (axis == 1 ? ey : ez);
  const double a = axis == 0 ? lo[0] : (axis == 1 ? lo[1] : lo[2]), b = axis == 0 ? hi[0] : (axis == 1 ? hi[1] : hi[2]);
  mid = __dmul_rn(0.5, __dadd_rn(a, b));
  return ext <= 1e-7 ? -1 : axis;
}

// Centroid keys of either width: made so that -0 orders as +0, as the FP64 comparisons see them.
// split: as split64, with the midpoint as a key: key >= thr iff the centroid >= the midpoint.
struct Key32 {
  using T = uint32_t;
  static constexpr bool WIDE = false;
  // As split64, in float arithmetic (FP64 instructions are slow on sm_103a, and a level waits for this
  // chain).  32-bit keys are those of synthesized crystals, whose coordinates are 0 or at least 1/1024 of
  // one of at most 16,000 cells: 48 bits hold any difference or sum of two, so the FP64 ones are exact.
  // Here they are exact float pairs, compared word by word.
  __device__ static int split(const T lo[3], const T hi[3], T& thr) {
    float e[3], el[3];
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      const float a = unord32(hi[f]), b = unord32(lo[f]);
      e[f] = __fsub_rn(a, b);
      const float t = __fsub_rn(e[f], a);
      el[f] = __fsub_rn(__fsub_rn(a, __fsub_rn(e[f], t)), __fadd_rn(b, t));
    }
    auto ge = [&](int f, int g) { return e[f] > e[g] || (e[f] == e[g] && el[f] >= el[g]); };
    const int axis = ge(0, 1) && ge(0, 2) ? 0 : (ge(1, 2) ? 1 : 2);
    const float ext = axis == 0 ? e[0] : (axis == 1 ? e[1] : e[2]);
    const float exl = axis == 0 ? el[0] : (axis == 1 ? el[1] : el[2]);
    const float a = unord32(axis == 0 ? lo[0] : (axis == 1 ? lo[1] : lo[2]));
    const float b = unord32(axis == 0 ? hi[0] : (axis == 1 ? hi[1] : hi[2]));
    thr = ord32(__fmul_rn(0.5f, __fadd_ru(a, b)) + 0.0f);
    if (ext > 1.1e-7f) return axis;
    return __dadd_rn(static_cast<double>(ext), static_cast<double>(exl)) <= 1e-7 ? -1 : axis;
  }
  __device__ static T warp_min(T k) { return __reduce_min_sync(0xffffffffu, k); }
  __device__ static T warp_max(T k) { return __reduce_max_sync(0xffffffffu, k); }
  __device__ static void make(const RTile& t, uint32_t s, T k[3]) {
    const float4 a = t.a[s];
    k[0] = ord32(a.x + 0.0f);
    k[1] = ord32(a.y + 0.0f);
    k[2] = ord32(a.z + 0.0f);
  }
};
struct Key64 {
  using T = unsigned long long;
  static constexpr bool WIDE = true;
  __device__ static int split(const T lo[3], const T hi[3], T& thr) {
    double clo[3], chi[3];
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      clo[f] = unord64(lo[f]);
      chi[f] = unord64(hi[f]);
    }
    double mid;
    const int axis = split64(clo, chi, mid);
    thr = ord64(mid);
    return axis;
  }
  // As two 32-bit reductions: the high words, then the low words of the lanes holding that high word.
  __device__ static T warp_min(T k) {
    const uint32_t hi = static_cast<uint32_t>(k >> 32), h = __reduce_min_sync(0xffffffffu, hi);
    const uint32_t l = __reduce_min_sync(0xffffffffu, hi == h ? static_cast<uint32_t>(k) : 0xffffffffu);
    return (static_cast<T>(h) << 32) | l;
  }
  __device__ static T warp_max(T k) {
    const uint32_t hi = static_cast<uint32_t>(k >> 32), h = __reduce_max_sync(0xffffffffu, hi);
    const uint32_t l = __reduce_max_sync(0xffffffffu, hi == h ? static_cast<uint32_t>(k) : 0u);
    return (static_cast<T>(h) << 32) | l;
  }
  __device__ static void make(const RTile& t, uint32_t s, T k[3]) {
    double lo[3], hi[3], cc[3];
    rt_box_pm(rt_pm(t, s), lo, hi, cc);
#pragma unroll
    for (int i = 0; i < 3; ++i) k[i] = ord64(__dadd_rn(cc[i], 0.0));
  }
};

struct RtArgs {
  RTile* tiles;
  int ntiles;
  unsigned long long E, N;
  uint32_t* idx[2];
  // Keys of the element at position x, field f at key[c][f * E + x]: centroid xyz (Key32 or Key64).
  void* key[2];
  uint32_t* nof[2];
  uint32_t* bits;   // big flags, 32 positions a word (chunk by chunk)
  uint32_t* wp;     // bigs of the tile before each word
  unsigned long long* blk;  // per chunk: level tag, state and count of the running sum
  uint32_t* P;      // positions of the tile's bigs and smalls by number (tile-relative, at ebase)
  uint32_t* Q;
  uint32_t* ridx;
  unsigned long long* acc;
  double* box64;
  uint32_t* parent;  // parent id of each node (RT_NONE for a root)
  uint32_t *nstart, *ncount, *ntile, *ndepth;
  int* nsplit;
  unsigned long long* nthr;  // split threshold (a key)
  int2* nchild;
  uint32_t* wl[2];  // nodes pending for the levels of either parity
  uint32_t* bq;     // block queue: nodes of at most RT_CTA_MAX elements
  uint32_t* bqpar;  // and the buffer parity holding their elements
  uint32_t* cnt;    // [0], [1] worklist counts, [2] block queue count, RT_CNT_BAR, RT_CNT_TILES
  uint32_t* err;
};

// Node allocation: two tile-local ids, or none when the tile's node capacity is spent.
__device__ __forceinline__ bool alloc_pair(const RtArgs& A, int t, uint32_t& l) {
  l = atomicAdd(&A.tiles[t].nodes, 2u);
  if (l + 2 > A.tiles[t].ncap) {
    atomicOr(A.err, ERR_LIST_OVERFLOW);
    return false;
  }
  return true;
}

constexpr uint32_t RT_NONE = 0xffffffffu;

// Hands a new node of n elements (held in buffer `par`) to the phase that builds it: the global
// levels (more than RT_CTA_MAX elements) or one block.
__device__ __forceinline__ void rt_enqueue(const RtArgs& A, uint32_t id, uint32_t n, int par) {
  A.nsplit[id] = -1;
  if (n > static_cast<uint32_t>(RT_CTA_MAX)) {
    A.wl[par][atomicAdd(&A.cnt[par], 1u)] = id;
  } else if (n > 0) {
    const uint32_t q = atomicAdd(&A.cnt[2], 1u);
    A.bq[q] = id;
    A.bqpar[q] = static_cast<uint32_t>(par);
  }
}

// Empties a node's centroid accumulators (minima, then maxima).
__device__ __forceinline__ void rt_acc_clear(const RtArgs& A, uint32_t id) {
  unsigned long long* a = A.acc + 6ull * id;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    a[k] = ~0ull;
    a[3 + k] = 0ull;
  }
}

// One warp's running centroid box of one node, per lane; flush adds it to the node's accumulators.
template <class K>
struct RtRun {
  typename K::T lo[3], hi[3];
  __device__ void clear() {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      lo[i] = ~static_cast<typename K::T>(0);
      hi[i] = 0;
    }
  }
  __device__ void add(const typename K::T k[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      lo[i] = min(lo[i], k[i]);
      hi[i] = max(hi[i], k[i]);
    }
  }
  // All 32 lanes; lanes 0-5 do one atomic each.
  __device__ void flush(const RtArgs& A, uint32_t id) {
    unsigned long long v = 0;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const typename K::T l = K::warp_min(lo[i]), h = K::warp_max(hi[i]);
      if (lane == i) v = l;
      if (lane == 3 + i) v = h;
    }
    unsigned long long* a = A.acc + 6ull * id;
    if (lane < 3) atomicMin(a + lane, v);
    else if (lane < 6) atomicMax(a + lane, v);
    clear();
  }
};

// All blocks of the (cooperative) grid arrive before any leaves; what they wrote is visible then.
// The wait is bounded: false (error set) when it gives up, and the kernel then ends.
__device__ bool rt_grid_sync(const RtArgs& A) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    if (gridDim.x > 1) {
      __threadfence();
      volatile uint32_t* bar = A.cnt + RT_CNT_BAR;
      const uint32_t ticket = atomicAdd(A.cnt + RT_CNT_BAR, 1u);
      const uint32_t target = (ticket / gridDim.x + 1u) * gridDim.x;
      uint32_t spins = 0;
      while (static_cast<int32_t>(*bar - target) < 0) {
        if (++spins > (1u << 24)) {
          atomicOr(A.err, ERR_SPIN_LIMIT);
          ok = 0;
          break;
        }
        __nanosleep(32);
      }
      __threadfence();
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// Running sum of the chunk counts along a tile: chunk ch (first: the tile's first) adds `total` and
// gets the sum of the tile's earlier chunks.  One warp calls it.  A chunk publishes its own count,
// then looks back over the counts or sums of the chunks before it until it meets a sum; chunks are
// taken in increasing order by blocks that all run, so every count arrives.  The wait is bounded.
// Words are tagged with the level, so they need no clearing between levels.
__device__ __forceinline__ uint32_t rt_chunk_sum(const RtArgs& A, uint32_t ch, uint32_t first, uint32_t level,
                                                 uint32_t total) {
  const unsigned long long tag = static_cast<unsigned long long>(level + 1u) << 40;
  const unsigned long long COUNT = 1ull << 32, SUM = 2ull << 32;
  const uint32_t lane = threadIdx.x & 31;
  if (ch == first) {
    if (lane == 0) atomicExch(A.blk + ch, tag | SUM | total);
    return 0;
  }
  if (lane == 0) atomicExch(A.blk + ch, tag | COUNT | total);
  uint32_t sum = 0, spins = 0;
  for (uint32_t back = ch;;) {  // chunks back - 1 - lane
    const bool in = lane < back - first;
    const unsigned long long w = in ? *(volatile unsigned long long*)(A.blk + (back - 1 - lane)) : tag | SUM;
    const bool ready = (w >> 40) == (tag >> 40);
    if (!__all_sync(0xffffffffu, ready)) {
      if (++spins > (1u << 22)) {
        if (lane == 0) atomicOr(A.err, ERR_SPIN_LIMIT);
        break;
      }
      continue;
    }
    const unsigned sums = __ballot_sync(0xffffffffu, (w & SUM) != 0);
    const int last = sums ? __ffs(sums) - 1 : 31;
    sum += __reduce_add_sync(0xffffffffu, static_cast<int>(lane) <= last ? static_cast<uint32_t>(w) : 0u);
    if (sums) break;
    back -= 32;
  }
  if (lane == 0) atomicExch(A.blk + ch, tag | SUM | (sum + total));
  return sum;
}

// Bigs of the tile before tile-relative position r (word base wb of the tile).
__device__ __forceinline__ uint32_t rt_rank(const RtArgs& A, uint32_t wb, uint32_t r) {
  const uint32_t w = wb + (r >> 5);
  return A.wp[w] + __popc(A.bits[w] & ((1u << (r & 31u)) - 1u));
}
__device__ __forceinline__ uint32_t rt_big(const RtArgs& A, uint32_t wb, uint32_t r) {
  return (A.bits[wb + (r >> 5)] >> (r & 31u)) & 1u;
}

// The chunk's tile (the last whose first chunk is <= ch), by one thread.
__device__ __forceinline__ int rt_chunk_tile(const uint32_t* start, int ntiles, uint32_t ch) {
  int lo = 0, hi = ntiles - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (start[mid] <= ch) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Element order, keys and the global levels, all of them.  Work goes by chunks of the tiles' elements
// (tiles with few elements in a large range cost only what they hold); a warp takes WPW words of 32
// consecutive positions.  One launch instead of eight per level, levels without work
// included: a level of few elements costs three grid barriers.
//
// Bound by latency more than by the streams (Key32: about 56 B per element and level, a third of the
// copy bandwidth): each word's node, element and keys are read while the word before is placed.
// Against eight launches per level with 64-bit keys, 18.9 M elements in 25 tiles: 11.5 -> 4.3 ms; the
// whole build of one tile's 3,556: 0.19 -> 0.10 ms, of 309 k: 0.60 -> 0.35 ms.
template <class K, int WPW>
__global__ void __launch_bounds__(RT_BLOCK, rt_blocks(K::WIDE)) k_rt_levels(RtArgs A, int levels) {
  using T = typename K::T;
  constexpr unsigned RT_CHUNK = rt_chunk(WPW), RT_WORDS = RT_CHUNK / 32;
  __shared__ int s_tile;
  __shared__ uint32_t s_wsum[RT_BLOCK / 32], s_base;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt = (1u << lane) - 1u;
  uint32_t* cst = A.cnt + RT_CNT_TILES;
  const unsigned g0 = blockIdx.x * RT_BLOCK + tid, gs = gridDim.x * RT_BLOCK;
  // Roots, and the first chunk of every tile (block 0).
  for (int t = static_cast<int>(g0); t < A.ntiles; t += static_cast<int>(gs)) {
    RTile& R = A.tiles[t];
    R.nodes = 2;
    R.depth = R.n ? 1 : 0;
    const uint32_t root = static_cast<uint32_t>(R.nbase + 1);
    A.nstart[root] = static_cast<uint32_t>(R.ebase);
    A.ncount[root] = R.n;
    A.ntile[root] = static_cast<uint32_t>(t);
    A.ndepth[root] = 1;
    A.parent[root] = RT_NONE;
    rt_acc_clear(A, root);
    rt_enqueue(A, root, R.n, 0);
  }
  if (blockIdx.x == 0) {
    uint32_t carry = 0;
    for (int base = 0; base < A.ntiles; base += RT_BLOCK) {
      const int t = base + tid;
      const uint32_t v = t < A.ntiles ? (A.tiles[t].n + RT_CHUNK - 1) / RT_CHUNK : 0u;
      uint32_t incl = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) s_wsum[warp] = incl;
      __syncthreads();
      uint32_t off = carry, tot = 0;
      for (int w = 0; w < static_cast<int>(RT_BLOCK / 32); ++w) {
        if (w < warp) off += s_wsum[w];
        tot += s_wsum[w];
      }
      if (t < A.ntiles) cst[t] = off + incl - v;
      carry += tot;
      __syncthreads();
    }
    if (tid == 0) cst[A.ntiles] = carry;
  }
  if (!rt_grid_sync(A)) return;
  const uint32_t nch = *(volatile uint32_t*)(cst + A.ntiles);
  // Order, keys and the roots' centroid boxes.
  {
    T* key = static_cast<T*>(A.key[0]);
    for (uint32_t ch = blockIdx.x; ch < nch; ch += gridDim.x) {
      if (tid == 0) s_tile = rt_chunk_tile(cst, A.ntiles, ch);
      __syncthreads();
      const RTile& R = A.tiles[s_tile];
      const uint32_t r0 = (ch - cst[s_tile]) * RT_CHUNK + warp * (32 * WPW);
      const bool big = R.n > static_cast<uint32_t>(RT_CTA_MAX);
      RtRun<K> run;
      run.clear();
#pragma unroll
      for (int j = 0; j < WPW; ++j) {
        const uint32_t r = r0 + j * 32 + lane;
        if (r >= R.n) continue;
        const unsigned long long x = R.ebase + r;
        const uint32_t slot = R.order ? static_cast<uint32_t>(R.order[r] - R.obase) : r;
        T k[3];
        K::make(R, slot, k);
        A.idx[0][x] = slot;
#pragma unroll
        for (int f = 0; f < 3; ++f) key[f * A.E + x] = k[f];
        if (big) run.add(k);
        A.nof[0][x] = big ? static_cast<uint32_t>(R.nbase + 1) : RT_DONE;
      }
      __syncwarp();
      if (big) run.flush(A, static_cast<uint32_t>(R.nbase + 1));
      __syncthreads();
    }
  }
  if (!rt_grid_sync(A)) return;
  int L = 0;
  for (; L < levels; ++L) {
    const int c = L & 1, o = c ^ 1;
    const T* key = static_cast<const T*>(A.key[c]);
    T* keyo = static_cast<T*>(A.key[o]);
    const uint32_t nw = *(volatile uint32_t*)(A.cnt + c);
    if (nw == 0) break;
    // Leaf or split for every pending node of this level (subdivide, bvh.rs:200-270).  (Each warp
    // deciding for the nodes it meets saves a barrier but repeats the FP64 chain: 5.4 ms against 4.9
    // on 18.9 M elements, 261 us against 242 on 309 k.)
    if (g0 == 0) A.cnt[o] = 0;  // read by all before the last barrier; filled by the place phase
    for (uint32_t i = g0; i < nw; i += gs) {
      const uint32_t node = A.wl[c][i];
      const int t = static_cast<int>(A.ntile[node]);
      const unsigned long long* a = A.acc + 6ull * node;
      T clo[3], chi[3], thr;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        clo[k] = static_cast<T>(__ldcg(a + k));
        chi[k] = static_cast<T>(__ldcg(a + 3 + k));
      }
      const int axis = K::split(clo, chi, thr);
      uint32_t l = 0;
      if (axis < 0 || !alloc_pair(A, t, l)) {
        A.nsplit[node] = -1;  // leaf (degenerate centroids, or no node capacity left)
        continue;
      }
      A.nsplit[node] = axis;
      A.nthr[node] = thr;
      const uint32_t id = static_cast<uint32_t>(A.tiles[t].nbase + l);
      A.nchild[node] = make_int2(static_cast<int>(id), static_cast<int>(id + 1));
      A.parent[id] = node;
      A.parent[id + 1] = node;
      rt_acc_clear(A, id);
      rt_acc_clear(A, id + 1);
    }
    if (!rt_grid_sync(A)) return;
    // Flags, their running number, and the positions of bigs and smalls by number.
    for (uint32_t ch = blockIdx.x; ch < nch; ch += gridDim.x) {
      if (tid == 0) s_tile = rt_chunk_tile(cst, A.ntiles, ch);
      __syncthreads();
      const RTile& R = A.tiles[s_tile];
      const uint32_t first = cst[s_tile];
      const uint32_t r0 = (ch - first) * RT_CHUNK + warp * (32 * WPW);
      uint32_t mybits = 0, myact = 0;  // lane j: word j's flags and its positions of splitting nodes
      uint32_t cur = RT_NONE;
      int axis = -1;
      T thr = 0;
      uint32_t nodes[WPW];
#pragma unroll
      for (int j = 0; j < WPW; ++j) {
        const uint32_t r = r0 + j * 32 + lane;
        nodes[j] = r < R.n ? A.nof[c][R.ebase + r] : RT_DONE;
      }
#pragma unroll
      for (int j = 0; j < WPW; ++j) {
        const uint32_t r = r0 + j * 32 + lane;
        const uint32_t node = nodes[j];
        bool act = false, flag = false;
        for (unsigned todo = __ballot_sync(0xffffffffu, !(node & RT_DONE)); todo;) {
          const uint32_t nd = __shfl_sync(0xffffffffu, node, __ffs(todo) - 1);
          if (nd != cur) {
            cur = nd;
            axis = A.nsplit[nd];
            thr = static_cast<T>(A.nthr[nd]);
          }
          if (node == nd && axis >= 0) {
            act = true;
            flag = key[axis * A.E + R.ebase + r] >= thr;
          }
          todo &= ~__ballot_sync(0xffffffffu, node == nd);
        }
        const unsigned b = __ballot_sync(0xffffffffu, flag), a = __ballot_sync(0xffffffffu, act);
        if (lane == j) {
          mybits = b;
          myact = a;
        }
      }
      uint32_t incl = __popc(mybits);
#pragma unroll
      for (int d = 1; d < WPW; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += y;
      }
      if (lane == WPW - 1) s_wsum[warp] = incl;
      __syncthreads();
      uint32_t off = 0, tot = 0;
      for (int w = 0; w < static_cast<int>(RT_BLOCK / 32); ++w) {
        if (w < warp) off += s_wsum[w];
        tot += s_wsum[w];
      }
      if (warp == 0) {
        const uint32_t b = rt_chunk_sum(A, ch, first, static_cast<uint32_t>(L), tot);
        if (lane == 0) s_base = b;
      }
      __syncthreads();
      const uint32_t mywp = s_base + off + incl - __popc(mybits);
      if (lane < WPW) {
        const uint32_t w = ch * RT_WORDS + warp * WPW + lane;
        A.bits[w] = mybits;
        A.wp[w] = mywp;
      }
      for (int j = 0; j < WPW; ++j) {
        const uint32_t b = __shfl_sync(0xffffffffu, mybits, j), a = __shfl_sync(0xffffffffu, myact, j);
        const uint32_t p = __shfl_sync(0xffffffffu, mywp, j) + __popc(b & lt);
        const uint32_t r = r0 + j * 32 + lane;
        if (!((a >> lane) & 1u) || p > r) continue;
        if ((b >> lane) & 1u) A.P[R.ebase + p] = r; else A.Q[R.ebase + (r - p)] = r;
      }
      __syncthreads();
    }
    if (!rt_grid_sync(A)) return;
    // Every element of a splitting node moves to its place after the reference's swap partition and
    // joins its child's centroid box; elements of new leaves are done; the children are set up.
    for (uint32_t ch = blockIdx.x; ch < nch; ch += gridDim.x) {
      if (tid == 0) s_tile = rt_chunk_tile(cst, A.ntiles, ch);
      __syncthreads();
      const RTile& R = A.tiles[s_tile];
      const uint32_t first = cst[s_tile], wb = first * RT_WORDS;
      const uint32_t r0 = (ch - first) * RT_CHUNK + warp * (32 * WPW);
      // The node at hand: split axis, start and size, bigs before it, smalls, end of the left stream,
      // left child's size, children.
      uint32_t cur = RT_NONE, s = 0, n = 0, bs = 0, St = 0, li = 0, Sp = 0;
      int axis = -1;
      int2 kid = make_int2(0, 0);
      RtRun<K> run[2];
      run[0].clear();
      run[1].clear();
      auto flush = [&]() {
        if (axis < 0) return;
        if (Sp > static_cast<uint32_t>(RT_CTA_MAX)) run[0].flush(A, static_cast<uint32_t>(kid.x));
        if (n - Sp > static_cast<uint32_t>(RT_CTA_MAX)) run[1].flush(A, static_cast<uint32_t>(kid.y));
      };
      // A word's node, element and keys are read while the word before is placed.
      uint32_t pnode = RT_DONE, pel = 0;
      T pk[3] = {0, 0, 0};
      auto fetch = [&](uint32_t q) {
        pnode = RT_DONE;
        if (q >= R.n) return;
        pnode = A.nof[c][R.ebase + q];
        if (pnode & RT_DONE) return;
        pel = A.idx[c][R.ebase + q];
#pragma unroll
        for (int f = 0; f < 3; ++f) pk[f] = key[f * A.E + R.ebase + q];
      };
      fetch(r0 + lane);
#pragma unroll 1
      for (int j = 0; j < WPW; ++j) {
        const uint32_t q = r0 + j * 32 + lane;  // tile-relative position
        const unsigned long long x = R.ebase + q;
        const bool in = q < R.n;
        const uint32_t node = pnode, el = pel;
        const T k[3] = {pk[0], pk[1], pk[2]};
        if (j + 1 < WPW) fetch(q + 32);
        if (in && (node & RT_DONE)) A.nof[o][x] = RT_DONE;
        for (unsigned todo = __ballot_sync(0xffffffffu, !(node & RT_DONE)); todo;) {
          const uint32_t nd = __shfl_sync(0xffffffffu, node, __ffs(todo) - 1);
          if (nd != cur) {
            flush();
            run[0].clear();
            run[1].clear();
            cur = nd;
            axis = A.nsplit[nd];
            s = A.nstart[nd] - static_cast<uint32_t>(R.ebase);
            n = A.ncount[nd];
            if (axis >= 0) {
              bs = rt_rank(A, wb, s);
              uint32_t Bt = rt_rank(A, wb, s + n - 1) + rt_big(A, wb, s + n - 1) - bs;
              if (Bt > n) {  // only after a wait that gave up
                atomicOr(A.err, ERR_BAD_INDEX);
                Bt = n;
              }
              St = n - Bt;
              li = St + (St < n ? rt_big(A, wb, s + St) : 0u);
              // The reference splits at count / 2 when every centroid fell on one side (bvh.rs:260-265).
              Sp = (St == 0 || St == n) ? n / 2 : St;
              kid = A.nchild[nd];
            }
          }
          if (node == nd) {
            if (axis < 0) {  // a leaf of this level: its order is final
              A.ridx[x] = el;
              A.nof[o][x] = RT_DONE;
            } else {
              const uint32_t r = q - s;
              const uint32_t w = A.bits[wb + (q >> 5)];
              const uint32_t Bb = A.wp[wb + (q >> 5)] + __popc(w & lt) - bs;
              const bool big = (w >> lane) & 1u;
              // Where P or Q gives the place: the big's partner Q_{m-1} (m - 1 = Bb), the small's P_m.
              uint32_t dest = r;
              const bool look = (r < li) == big && !(big && Bb == 0);
              if (look) {
                const uint32_t at = big ? s - bs + (St - Bb) : bs + (St - (r - Bb)) - 1;
                dest = at < R.n ? (big ? A.Q[R.ebase + at] : A.P[R.ebase + at]) - s : n;
                if (big) --dest;
              } else if (big) {
                dest = r < li ? n - 1 : r - 1;
              }
              if (index_ok(dest < n, A.err, SITE_TREE, dest, n)) {
                const bool left = dest < Sp;
                const uint32_t csize = left ? Sp : n - Sp;
                const unsigned long long y = R.ebase + s + dest;
                const bool deep = csize > static_cast<uint32_t>(RT_CTA_MAX);
#pragma unroll
                for (int f = 0; f < 3; ++f) keyo[f * A.E + y] = k[f];
                A.idx[o][y] = el;
                A.nof[o][y] = deep ? static_cast<uint32_t>(left ? kid.x : kid.y) : RT_DONE;
                if (deep) {
                  if (left) run[0].add(k); else run[1].add(k);
                }
              }
              if (r == 0) {
                const uint32_t dep = A.ndepth[nd] + 1;
#pragma unroll
                for (int side = 0; side < 2; ++side) {
                  const uint32_t id = static_cast<uint32_t>(side ? kid.y : kid.x), cs = side ? n - Sp : Sp;
                  A.nstart[id] = static_cast<uint32_t>(R.ebase) + s + (side ? Sp : 0u);
                  A.ncount[id] = cs;
                  A.ntile[id] = static_cast<uint32_t>(s_tile);
                  A.ndepth[id] = dep;
                  rt_enqueue(A, id, cs, o);
                }
                atomicMax(&A.tiles[s_tile].depth, dep);
              }
            }
          }
          todo &= ~__ballot_sync(0xffffffffu, node == nd);
        }
      }
      flush();
      __syncthreads();
    }
    if (!rt_grid_sync(A)) return;
  }
  if (g0 == 0 && *(volatile uint32_t*)(A.cnt + (L & 1)) != 0) atomicOr(A.err, ERR_LIST_OVERFLOW);  // levels spent
}

// Segment-wise reduction over a warp's 32 consecutive positions: lanes with equal `seg` form
// contiguous runs (a node is a contiguous range of positions, so equal values at two lanes mean
// the same node in between).  On return the first lane of each run holds the run's minima
// (k[0..2]) and maxima (k[3..5]); the return value says whether this lane is a run's first.
// Lanes without a node pass a seg value no other lane has.  All 32 lanes call it.
__device__ __forceinline__ bool rt_seg_reduce(uint32_t seg, uint32_t k[6]) {
  const int lane = threadIdx.x & 31;
  if (__all_sync(0xffffffffu, __shfl_sync(0xffffffffu, seg, 0) == seg)) {  // one node across the warp
#pragma unroll
    for (int i = 0; i < 6; ++i) k[i] = i < 3 ? __reduce_min_sync(0xffffffffu, k[i]) : __reduce_max_sync(0xffffffffu, k[i]);
    return lane == 0;
  }
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t ns = __shfl_down_sync(0xffffffffu, seg, o);
    const bool take = lane + o < 32 && ns == seg;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const uint32_t y = __shfl_down_sync(0xffffffffu, k[i], o);
      if (take) k[i] = i < 3 ? min(k[i], y) : max(k[i], y);
    }
  }
  const uint32_t up = __shfl_up_sync(0xffffffffu, seg, 1);
  return lane == 0 || up != seg;
}

// The block queue: one block builds the whole subtree of a node of at most RT_CTA_MAX elements
// with its elements in shared memory.  Each level runs the passes of the global levels over all
// of the level's nodes of more than RT_LEAF_MAX elements at once (segment-wise reduce, decide, flags
// with their prefix sum and P / Q, children, place); a child of at most RT_LEAF_MAX elements is a leaf
// (bvh.rs:200-204), whose fields one thread writes at the start of the next level.
constexpr int RT_CTA_T = 256;                                // threads per block
constexpr int RT_CTA_PER = RT_CTA_MAX / RT_CTA_T;            // positions per thread
constexpr int RT_LEAF_MAX = 4;                               // subdivide's leaf size
constexpr int RT_CTA_LV = RT_CTA_MAX / (RT_LEAF_MAX + 1);    // nodes of more than 4 per level (204)
constexpr int RT_CTA_SL = 2 * RT_CTA_LV;                     // leaves of at most 4 made by one level
constexpr uint8_t RT_CTA_FREE = 0xff;                        // position of a finished range
static_assert(RT_CTA_LV < RT_CTA_FREE, "level slots must fit a byte");
static_assert(RT_CTA_MAX <= 2048, "positions are packed in 11 bits");

// A node of the level as split: x: offset | count << 16; y: bigs before it | smalls in it << 16; z: left
// child's size | end of the left stream << 16; w: next-level slots of the children (RT_CTA_FREE for a
// small leaf) | << 8, | 1 << 16 when it splits.
template <class K>
struct RtCtaSmem {
  typename K::T key[3][RT_CTA_MAX];  // the job's centroid keys, at their load position (home)
  // Per level: the nodes' centroid boxes (reduce to decide), by words of 32 positions; then the flags' prefix sum, P, Q
  // and the nodes as split (flags to place); the two uses do not overlap.
  union {
    struct {
      typename K::T acc[RT_CTA_LV][6];      // minima, maxima of a node (64-bit keys: from its start to the end of that word)
      typename K::T head[RT_CTA_MAX / 32][6];  // 64-bit keys: of the node's elements at the start of a word
    } c;
    struct {
      uint4 node[RT_CTA_LV];                // what placing reads of a node (as above)
      alignas(8) uint16_t bb[RT_CTA_MAX + 4];  // flag << 15 | exclusive prefix sum of the flags
      uint16_t P[RT_CTA_MAX], Q[RT_CTA_MAX];  // positions of the bigs and of the others, by number
    } r;
  } u;
  typename K::T thr[RT_CTA_LV];           // split threshold
  uint32_t idx[RT_CTA_MAX];               // element slot
  alignas(8) uint16_t home[RT_CTA_MAX];   // element's load position (its keys)
  uint32_t id[2][RT_CTA_LV];              // this level's nodes and the next's
  uint32_t sl[RT_CTA_SL];                 // small leaves: position | count << 11 | depth << 14
  uint32_t slid[RT_CTA_SL];
  uint32_t scan[RT_CTA_T / 32];
  uint16_t off[2][RT_CTA_LV], cnt[2][RT_CTA_LV];
  alignas(4) uint8_t nd[RT_CTA_MAX];      // level slot of the position's node, RT_CTA_FREE when done
  uint8_t dep[2][RT_CTA_LV];
  int8_t axis[RT_CTA_LV];
  int nl, nsl, nnext, nslnew;
  uint32_t maxdep;
};

// What bounds it: latency.  A level is seven barriers with short chains of shared-memory reads between
// them, 7,200 cycles (32-bit keys; 10,100 with 64-bit ones) for 1,024 elements.  With the ranks in a
// pass of their own, a global atomic and FP64 decisions in the chain, and 64-bit minima accumulated in
// shared memory, the blocks of a 64 x 64 px tri-x tile took 50 us (64-bit keys 58), now 38 (45); the
// 18.9 M elements of a 1600 x 1600 px t-max image 2.40 ms, now 2.05.
//
// Four blocks per SM (64 registers; the block's shared memory is about 53 KB with 64-bit keys): 9 %
// faster than two.
template <class K>
__global__ void __launch_bounds__(RT_CTA_T, 4) k_rt_cta(RtArgs A) {
  using T = typename K::T;
  extern __shared__ __align__(32) unsigned char rt_cta_raw[];
  RtCtaSmem<K>& S = *reinterpret_cast<RtCtaSmem<K>*>(rt_cta_raw);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const uint32_t nq = A.cnt[2];
  for (uint32_t q = blockIdx.x; q < nq; q += gridDim.x) {
    const uint32_t root = A.bq[q], par = A.bqpar[q];
    const uint32_t s = A.nstart[root];
    const int n = static_cast<int>(min(A.ncount[root], static_cast<uint32_t>(RT_CTA_MAX)));
    const uint32_t t = A.ntile[root];
    const unsigned long long nb = A.tiles[t].nbase;
    const uint32_t ncap = A.tiles[t].ncap;
    const uint32_t dep0 = min(A.ndepth[root], 255u);
    for (int x = tid; x < RT_CTA_MAX; x += RT_CTA_T) {
      if (x < n) {
#pragma unroll
        for (int f = 0; f < 3; ++f) S.key[f][x] = static_cast<const T*>(A.key[par])[f * A.E + s + x];
        S.home[x] = static_cast<uint16_t>(x);
        S.idx[x] = A.idx[par][s + x];
        S.nd[x] = n > RT_LEAF_MAX ? 0 : RT_CTA_FREE;
      } else {
        S.nd[x] = RT_CTA_FREE;
      }
    }
    if (tid == 0) {
      S.maxdep = 0;
      if (n > RT_LEAF_MAX) {
        S.nl = 1;
        S.nsl = 0;
        S.id[0][0] = root;
        S.off[0][0] = 0;
        S.cnt[0][0] = static_cast<uint16_t>(n);
        S.dep[0][0] = static_cast<uint8_t>(dep0);
      } else {
        S.nl = 0;
        S.nsl = 1;
        S.sl[0] = static_cast<uint32_t>(n) << 11 | dep0 << 14;
        S.slid[0] = root;
      }
    }
    __syncthreads();
    int cur = 0;
    for (;;) {
      const int nl = S.nl, nsl = S.nsl;
      // Leaves of at most four elements made by the previous level (or a small root).
      for (int i = tid; i < nsl; i += RT_CTA_T) {
        const uint32_t e = S.sl[i], id = S.slid[i];
        const int o0 = static_cast<int>(e & 2047u), cn = static_cast<int>((e >> 11) & 7u);
        const uint32_t dp = e >> 14;
        A.nstart[id] = s + static_cast<uint32_t>(o0);
        A.ncount[id] = static_cast<uint32_t>(cn);
        A.ntile[id] = t;
        A.ndepth[id] = dp;
        A.nsplit[id] = -1;
        atomicMax(&S.maxdep, dp);
      }
      if (nl == 0) break;
      if (!K::WIDE) {
        for (int i = tid; i < nl * 6; i += RT_CTA_T) S.u.c.acc[i / 6][i % 6] = (i % 6) < 3 ? ~static_cast<T>(0) : static_cast<T>(0);
        __syncthreads();
      }
      if (tid == 0) {
        S.nnext = 0;
        S.nslnew = 0;
      }
      // Reduce: position x = k * RT_CTA_T + tid, so a warp holds 32 consecutive positions, those of at
      // most eight nodes (of more than four elements each).  32-bit keys: the nodes' runs reduced side by
      // side, their heads joined in shared memory.  64-bit keys, whose minimum in shared memory is a
      // loop: a reduction over the warp for each node; its box in the word goes to the word when the
      // node may start before it, else to the node, so nothing is accumulated in place.  (The other way
      // round: 25 k cycles a block against 20 with 32-bit keys, 37 against 22 with 64-bit ones.)
#pragma unroll 2
      for (int k = 0; k < RT_CTA_PER; ++k) {
        const int x = k * RT_CTA_T + tid;
        const uint32_t node = S.nd[x];
        const bool act = node != RT_CTA_FREE;
        unsigned todo = __ballot_sync(0xffffffffu, act);
        if (!todo) continue;
        T kk[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) kk[i] = S.key[i][act ? S.home[x] : 0];
        if constexpr (!K::WIDE) {
          T box[6];
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            box[i] = act ? kk[i] : ~static_cast<T>(0);
            box[3 + i] = act ? kk[i] : static_cast<T>(0);
          }
          if (rt_seg_reduce(act ? node : (0x100u | static_cast<uint32_t>(lane)), box) && act) {
#pragma unroll
            for (int i = 0; i < 3; ++i) {
              atomicMin(&S.u.c.acc[node][i], box[i]);
              atomicMax(&S.u.c.acc[node][3 + i], box[3 + i]);
            }
          }
        } else {
          while (todo) {
            const int src = __ffs(todo) - 1;
            const uint32_t nd = __shfl_sync(0xffffffffu, node, src);
            const bool in = node == nd;
            todo &= ~__ballot_sync(0xffffffffu, in);
            T lo[3], hi[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
              lo[i] = K::warp_min(in ? kk[i] : ~static_cast<T>(0));
              hi[i] = K::warp_max(in ? kk[i] : static_cast<T>(0));
            }
            if (lane == src) {
              T* out = src == 0 ? S.u.c.head[k * (RT_CTA_T / 32) + w] : S.u.c.acc[nd];
#pragma unroll
              for (int i = 0; i < 3; ++i) {
                out[i] = lo[i];
                out[3 + i] = hi[i];
              }
            }
          }
        }
      }
      __syncthreads();
      // Decide (subdivide, bvh.rs:200-270), one thread per node of the level.  The ids of its children
      // are asked for here and used after the flags: the counter is a microsecond away.
      static_assert(RT_CTA_LV <= RT_CTA_T, "a thread to a node");
      int axis = -1;
      uint32_t l = 0;
      if (tid < nl) {
        T clo[3], chi[3], thr;
        const int o0 = S.off[cur][tid], cn = S.cnt[cur][tid];
        const bool own = !K::WIDE || (o0 & 31) != 0;
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          clo[m] = own ? S.u.c.acc[tid][m] : ~static_cast<T>(0);
          chi[m] = own ? S.u.c.acc[tid][3 + m] : static_cast<T>(0);
        }
        for (int word = (o0 + 31) >> 5; K::WIDE && word <= (o0 + cn - 1) >> 5; ++word)
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            clo[m] = min(clo[m], S.u.c.head[word][m]);
            chi[m] = max(chi[m], S.u.c.head[word][3 + m]);
          }
        axis = cn > RT_LEAF_MAX ? K::split(clo, chi, thr) : -1;
        if (axis >= 0) {
          l = atomicAdd(&A.tiles[t].nodes, 2u);
          S.thr[tid] = thr;
        }
        S.axis[tid] = static_cast<int8_t>(axis);
      }
      __syncthreads();
      // Flags, their exclusive prefix sum, and the positions of the bigs and of the others by number:
      // thread tid owns positions RT_CTA_PER * tid + k.
      {
        static_assert(RT_CTA_PER == 4, "four positions to a thread");
        const uint32_t nd4 = *reinterpret_cast<const uint32_t*>(S.nd + RT_CTA_PER * tid);
        const uint2 home4 = *reinterpret_cast<const uint2*>(S.home + RT_CTA_PER * tid);
        uint32_t f[RT_CTA_PER], sum = 0;
#pragma unroll
        for (int k = 0; k < RT_CTA_PER; ++k) {
          const uint32_t node = (nd4 >> (8 * k)) & 0xffu;
          const uint32_t home = ((k < 2 ? home4.x : home4.y) >> (16 * (k & 1))) & 0xffffu;
          f[k] = 0;
          if (node != RT_CTA_FREE) {
            const int ax = S.axis[node];
            if (ax >= 0) f[k] = S.key[ax][home] < S.thr[node] ? 0u : 1u;
          }
          sum += f[k];
        }
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += y;
        }
        if (lane == 31) S.scan[w] = incl;
        __syncthreads();
        uint32_t acc = incl - sum;
        for (int i = 0; i < w; ++i) acc += S.scan[i];
        uint32_t b[RT_CTA_PER];
#pragma unroll
        for (int k = 0; k < RT_CTA_PER; ++k) {
          const uint32_t x = RT_CTA_PER * tid + k;
          b[k] = f[k] << 15 | acc;
          if (f[k]) S.u.r.P[acc] = static_cast<uint16_t>(x); else S.u.r.Q[x - acc] = static_cast<uint16_t>(x);
          acc += f[k];
        }
        *reinterpret_cast<uint2*>(S.u.r.bb + RT_CTA_PER * tid) = make_uint2(b[0] | b[1] << 16, b[2] | b[3] << 16);
        if (tid == RT_CTA_T - 1) S.u.r.bb[RT_CTA_MAX] = static_cast<uint16_t>(acc);
      }
      __syncthreads();
      // The nodes, and the children of those that split: to the next level (more than four elements) or
      // small leaves.
      if (tid < nl) {
        const uint32_t id = S.id[cur][tid], dep = S.dep[cur][tid];
        const int o0 = S.off[cur][tid], cn = S.cnt[cur][tid];
        A.nstart[id] = s + static_cast<uint32_t>(o0);
        A.ncount[id] = static_cast<uint32_t>(cn);
        A.ntile[id] = t;
        A.ndepth[id] = dep;
        atomicMax(&S.maxdep, dep);
        if (axis >= 0 && l + 2 > ncap) {  // no node capacity left
          atomicOr(A.err, ERR_LIST_OVERFLOW);
          axis = -1;
        }
        A.nsplit[id] = axis;
        uint4 N = make_uint4(static_cast<uint32_t>(o0) | static_cast<uint32_t>(cn) << 16, 0u, 0u, 0u);
        if (axis >= 0) {
          const int bs = S.u.r.bb[o0] & 0x7fff, Bt = (S.u.r.bb[o0 + cn] & 0x7fff) - bs, St = cn - Bt;
          const int li = St + (St < cn ? S.u.r.bb[o0 + St] >> 15 : 0);
          const int Sp = (St == 0 || St == cn) ? cn / 2 : St;  // bvh.rs:260-265
          const uint32_t kid = static_cast<uint32_t>(nb + l);
          A.nchild[id] = make_int2(static_cast<int>(kid), static_cast<int>(kid + 1));
          A.parent[kid] = id;
          A.parent[kid + 1] = id;
          const uint32_t cd = min(dep + 1u, 255u);  // saturates past the depth check
          uint32_t slots = 0;
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const uint32_t cid = kid + static_cast<uint32_t>(c);
            const int coff = o0 + (c ? Sp : 0), csz = c ? cn - Sp : Sp;
            if (csz > RT_LEAF_MAX) {
              const int slot = atomicAdd(&S.nnext, 1);
              S.id[cur ^ 1][slot] = cid;
              S.off[cur ^ 1][slot] = static_cast<uint16_t>(coff);
              S.cnt[cur ^ 1][slot] = static_cast<uint16_t>(csz);
              S.dep[cur ^ 1][slot] = static_cast<uint8_t>(cd);
              slots |= static_cast<uint32_t>(slot) << (8 * c);
            } else {
              const int qi = atomicAdd(&S.nslnew, 1);
              S.sl[qi] = static_cast<uint32_t>(coff) | static_cast<uint32_t>(csz) << 11 | cd << 14;
              S.slid[qi] = cid;
              slots |= static_cast<uint32_t>(RT_CTA_FREE) << (8 * c);
            }
          }
          N.y = static_cast<uint32_t>(bs) | static_cast<uint32_t>(St) << 16;
          N.z = static_cast<uint32_t>(Sp) | static_cast<uint32_t>(li) << 16;
          N.w = slots | 1u << 16;
        }
        S.u.r.node[tid] = N;
      }
      __syncthreads();
      // Place: every element of a splitting node moves to its place after the swap partition.
      uint16_t vp[RT_CTA_PER];
      uint32_t vi[RT_CTA_PER];
      int dst[RT_CTA_PER];
      uint8_t vn[RT_CTA_PER];
#pragma unroll
      for (int k = 0; k < RT_CTA_PER; ++k) {
        // Without branches: the four positions' chains of reads run side by side.
        const int x = k * RT_CTA_T + tid;
        const uint32_t node = S.nd[x];
        const bool act = node != RT_CTA_FREE;
        vp[k] = S.home[x];
        vi[k] = S.idx[x];
        const uint4 N = S.u.r.node[act ? node : 0u];
        const uint32_t b = S.u.r.bb[x];
        const bool move = act && (N.w >> 16) != 0;  // else a leaf of this level (its order is final), or done
        const int o0 = static_cast<int>(N.x & 0xffffu), cn = static_cast<int>(N.x >> 16);
        const int bs = static_cast<int>(N.y & 0xffffu), St = static_cast<int>(N.y >> 16);
        const int Sp = static_cast<int>(N.z & 0xffffu), li = static_cast<int>(N.z >> 16);
        const int r = x - o0, Bb = static_cast<int>(b & 0x7fffu) - bs;
        const bool big = (b >> 15) != 0, look = move && (r < li) == big && !(big && Bb == 0);
        const int at = big ? o0 - bs + (St - Bb) : bs + (St - (r - Bb)) - 1;
        const int got = (big ? S.u.r.Q : S.u.r.P)[look ? at : 0];
        // Block position: P's; one before Q's, or before the node's end for the first big; one less; the same.
        const int d = look ? (big ? got - 1 : got) : (big && move ? (r < li ? o0 + cn : x) - 1 : x);
        dst[k] = act ? d : -1;
        vn[k] = static_cast<uint8_t>(!move ? RT_CTA_FREE : (d - o0 < Sp ? N.w : N.w >> 8));
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < RT_CTA_PER; ++k) {
        if (dst[k] < 0) continue;
        S.home[dst[k]] = vp[k];
        S.idx[dst[k]] = vi[k];
        S.nd[dst[k]] = vn[k];
      }
      if (tid == 0) {
        S.nl = S.nnext;
        S.nsl = S.nslnew;
      }
      cur ^= 1;
      __syncthreads();
    }
    for (int x = tid; x < n; x += RT_CTA_T) A.ridx[s + x] = S.idx[x];
    __syncthreads();  // the last level's leaves have joined S.maxdep; the next job may write the rest
    if (tid == 0) atomicMax(&A.tiles[t].depth, S.maxdep);
  }
}

// Leaves, by tile (blockIdx.y): the leaf box (the union of its elements' max_dim boxes, bvh.rs:196-204),
// the leaf-of map and the elements' ranks (the walk takes the right subtree first, so leaves in
// descending element position, and a leaf's elements in index order); rleaf (may be null) gets the
// element range.  Boxes fold as order-preserving integers, or, for FP32 crystals without expansion
// (FP32), as the exact float pairs p -+ m, rounded to FP64 once per leaf: GB300's FP64 pipe is narrow.
template <bool FP32>
__global__ void k_rt_leaves(RtArgs A, uint2* rleaf, uint32_t* leafof, unsigned long long leafof_n, uint32_t* rank) {
  const RTile& T = A.tiles[blockIdx.y];
  if (blockIdx.x == 0 && threadIdx.x == 0 && T.depth > static_cast<uint32_t>(RT_MAX_DEPTH))
    atomicOr(A.err, ERR_STACK_OVERFLOW);
  if (T.n == 0) return;
  const uint32_t nodes = min(T.nodes, T.ncap);
  // (After a failed node allocation, ids below the capacity may never have been set up; the build
  // has flagged the error, and the checks below keep this pass inside its buffers.)
  for (uint32_t id = 1 + blockIdx.x * blockDim.x + threadIdx.x; id < nodes; id += gridDim.x * blockDim.x) {
    const unsigned long long g = T.nbase + id;
    if (A.nsplit[g] >= 0) continue;
    const uint32_t st = A.nstart[g], cn = A.ncount[g];
    if (st < T.ebase || st - T.ebase + static_cast<unsigned long long>(cn) > T.n) {
      atomicOr(A.err, ERR_BAD_INDEX);
      continue;
    }
    const uint32_t r0 = static_cast<uint32_t>(st - T.ebase);
    if (rleaf) rleaf[g] = make_uint2(r0, cn);
    unsigned long long k[6];
    float h[6], l[6];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      k[m] = ~0ull;
      k[3 + m] = 0ull;
      h[m] = INFINITY;
      h[3 + m] = -INFINITY;
      l[m] = l[3 + m] = 0.0f;
    }
    for (uint32_t j = 0; j < cn; ++j) {
      const uint32_t slot = A.ridx[st + j];
      if (T.ebase + slot >= leafof_n) {
        atomicOr(A.err, ERR_BAD_INDEX);
        continue;
      }
      leafof[T.ebase + slot] = id;
      if (rank) rank[T.ebase + slot] = T.n - r0 - cn + j;
      if (FP32) {
        const float4 a = T.a[slot], d = T.d[slot];
        const float p[3] = {a.x, a.y, a.z}, dm = fmaxf(fmaxf(d.x, d.y), d.z);
#pragma unroll
        for (int m = 0; m < 6; ++m) {
          // p -+ dm as an exact pair (Knuth's two-sum).
          const float q = p[m % 3], w = m < 3 ? -dm : dm;
          const float s = q + w, z = s - q, e = (q - (s - z)) + (w - z);
          const bool take = m < 3 ? (s < h[m] || (s == h[m] && e < l[m])) : (s > h[m] || (s == h[m] && e > l[m]));
          if (take) {
            h[m] = s;
            l[m] = e;
          }
        }
        continue;
      }
      const double4_32a v = rt_pm(T, slot);
      const double p[3] = {v.x, v.y, v.z};
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        k[m] = umin64(k[m], ord64(__dsub_rn(p[m], v.w)));
        k[3 + m] = umax64(k[3 + m], ord64(__dadd_rn(p[m], v.w)));
      }
    }
#pragma unroll
    for (int m = 0; m < 6; ++m)
      A.box64[6ull * g + m] = FP32 ? __dadd_rn(static_cast<double>(h[m]), static_cast<double>(l[m])) : unord64(k[m]);
  }
}

// Node boxes above the leaves (the BVHNode aabb: the union of the node's elements' max_dim boxes,
// bvh.rs:196-204), for the walks.  One thread per leaf climbs: at each parent the first child to
// arrive stops and the second forms the parent's box as the union of both children's.  Boxes are
// published with a fence before the arrival count and read through L2.  `arrive` holds one zeroed
// counter per node.
__global__ void k_rt_refit(RtArgs A, uint32_t* arrive) {
  const RTile& T = A.tiles[blockIdx.y];
  const unsigned long long nlo = T.nbase, nhi = T.nbase + T.ncap;
  const uint32_t nodes = T.n ? min(T.nodes, T.ncap) : 0;
  for (uint32_t id = 1 + blockIdx.x * blockDim.x + threadIdx.x; id < nodes; id += gridDim.x * blockDim.x) {
    unsigned long long node = T.nbase + id;
    if (A.nsplit[node] >= 0) continue;
    for (int up = 0; up <= RT_MAX_DEPTH; ++up) {
      const uint32_t p = A.parent[node];
      if (p == RT_NONE) break;
      if (p < nlo || p >= nhi) {
        atomicOr(A.err, ERR_BAD_INDEX);
        break;
      }
      __threadfence();
      if (atomicAdd(&arrive[p], 1u) == 0u) break;  // the other child forms the parent's box
      __threadfence();
      const int2 ch = A.nchild[p];
      if (static_cast<unsigned long long>(ch.x) < nlo || static_cast<unsigned long long>(ch.y) >= nhi) {
        atomicOr(A.err, ERR_BAD_INDEX);
        break;
      }
      const double* a = A.box64 + 6ull * static_cast<unsigned long long>(ch.x);
      const double* b = A.box64 + 6ull * static_cast<unsigned long long>(ch.y);
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        const unsigned long long l = umin64(ord64(__ldcg(a + m)), ord64(__ldcg(b + m)));
        const unsigned long long h = umax64(ord64(__ldcg(a + 3 + m)), ord64(__ldcg(b + 3 + m)));
        A.box64[6ull * p + m] = unord64(l);
        A.box64[6ull * p + 3 + m] = unord64(h);
      }
      node = p;
    }
  }
}

// Walk records, one thread per node: the root and every internal node at odd depth write their
// four-wide record (fg_rtree.cuh), the
// grandchildren in the reference's visiting order (right before left, a leaf child in one slot).
// An internal slot's box is rounded outward, padded and extended by the reach; a leaf slot's box
// is rounded to nearest.
__global__ void k_rt_records(RtArgs A, Node4* rec) {
  const unsigned long long stride = static_cast<unsigned long long>(gridDim.x) * blockDim.x;
  for (unsigned long long g = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; g < A.N;
       g += stride) {
    int lo_ = 0, hi_ = A.ntiles - 1;
    while (lo_ < hi_) {
      const int mid = (lo_ + hi_ + 1) >> 1;
      if (A.tiles[mid].nbase <= g) lo_ = mid; else hi_ = mid - 1;
    }
    const RTile& T = A.tiles[lo_];
    const uint32_t id = static_cast<uint32_t>(g - T.nbase);
    // (After a failed node allocation, ids below the capacity may never have been set up; the
    // build has flagged the error, and the checks below keep this pass inside its buffers.)
    if (id >= min(T.nodes, T.ncap)) continue;
    Node4* R = rec + T.rbase;
    float bx[6][4];
    int ref[4] = {INT32_MIN, INT32_MIN, INT32_MIN, INT32_MIN};
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int c = 0; c < 6; ++c) bx[c][k] = 0.0f;
    auto put = [&](int k, Node4* out) {
      Node4 nd;
      nd.lox = make_float4(bx[0][0], bx[0][1], bx[0][2], bx[0][3]);
      nd.loy = make_float4(bx[1][0], bx[1][1], bx[1][2], bx[1][3]);
      nd.loz = make_float4(bx[2][0], bx[2][1], bx[2][2], bx[2][3]);
      nd.hix = make_float4(bx[3][0], bx[3][1], bx[3][2], bx[3][3]);
      nd.hiy = make_float4(bx[4][0], bx[4][1], bx[4][2], bx[4][3]);
      nd.hiz = make_float4(bx[5][0], bx[5][1], bx[5][2], bx[5][3]);
      nd.ref = make_int4(ref[0], ref[1], ref[2], ref[3]);
      nd._pad = make_int4(k, 0, 0, 0);
      *out = nd;
    };
    if (id == 0) {  // the super-root slot: an empty tree's record 0
      if (T.n == 0 && T.rcap > 0) put(0, R);
      continue;
    }
    if (id == 1 && T.n == 0) continue;
    const bool leaf = A.nsplit[g] < 0;
    if (id != 1 && (leaf || !(A.ndepth[g] & 1u))) continue;
    // Slot k takes node c (a global id inside the tile): its box and reference.
    int k = 0;
    bool bad = false;
    auto add = [&](unsigned long long c) {
      if (c < T.nbase || c >= T.nbase + T.ncap || k >= 4) {
        bad = true;
        return;
      }
      const double* b = A.box64 + 6ull * c;
      const int local = static_cast<int>(c - T.nbase);
      float f[6];
      if (A.nsplit[c] < 0) {
#pragma unroll
        for (int m = 0; m < 6; ++m) f[m] = __double2float_rn(b[m]);
        ref[k] = ~local;
      } else {
        const int2 ch = A.nchild[c];
        const long long r = (static_cast<long long>(ch.x) - static_cast<long long>(T.nbase)) >> 1;
        if (r < 1 || r >= static_cast<long long>(T.rcap)) {
          bad = true;
          return;
        }
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          f[m] = __double2float_rd(b[m]) - T.pad - T.reach;
          f[3 + m] = __double2float_ru(b[3 + m]) + T.pad + T.reach;
        }
        ref[k] = static_cast<int>(r);
      }
#pragma unroll
      for (int m = 0; m < 6; ++m) bx[m][k] = f[m];
      ++k;
    };
    unsigned long long at = 0;  // record index
    if (leaf) {  // a root leaf
      add(g);
    } else {
      const int2 ch = A.nchild[g];
      if (id != 1) at = (static_cast<unsigned long long>(ch.x) - T.nbase) >> 1;
      const unsigned long long cs[2] = {static_cast<unsigned long long>(ch.y), static_cast<unsigned long long>(ch.x)};
#pragma unroll
      for (int q = 0; q < 2; ++q) {  // right child first
        const unsigned long long c = cs[q];
        if (c < T.nbase || c >= T.nbase + T.ncap) {
          bad = true;
          break;
        }
        if (A.nsplit[c] < 0) {
          add(c);
        } else {
          const int2 gc = A.nchild[c];
          add(static_cast<unsigned long long>(gc.y));
          add(static_cast<unsigned long long>(gc.x));
        }
      }
    }
    if (bad || at >= T.rcap) {
      atomicOr(A.err, ERR_BAD_INDEX);
      continue;
    }
    put(k, R + at);
  }
}

}  // namespace

RtArgs rt_args(RTreeBufs& B, uint32_t* err) {
  RtArgs A;
  A.tiles = B.tiles.p;
  A.ntiles = B.ntiles;
  A.E = B.E;
  A.N = B.N;
  A.idx[0] = B.idx0.p;
  A.idx[1] = B.idx1.p;
  A.key[0] = B.key0.p;
  A.key[1] = B.key1.p;
  A.nof[0] = B.nof0.p;
  A.nof[1] = B.nof1.p;
  A.bits = B.bits.p;
  A.wp = B.wp.p;
  A.blk = B.blk.p;
  A.P = B.P.p;
  A.Q = B.Q.p;
  A.ridx = B.ridx.p;
  A.acc = B.acc.p;
  A.box64 = B.box64.p;
  A.parent = B.parent.p;
  A.nstart = B.nstart.p;
  A.ncount = B.ncount.p;
  A.ntile = B.ntile.p;
  A.ndepth = B.ndepth.p;
  A.nsplit = B.nsplit.p;
  A.nthr = B.nthr.p;
  A.nchild = B.nchild.p;
  A.wl[0] = B.wl0.p;
  A.wl[1] = B.wl1.p;
  A.bq = B.bq.p;
  A.bqpar = B.bqpar.p;
  A.cnt = B.cnt.p;
  A.err = err;
  return A;
}

void rtree_alloc(RTreeBufs& B, std::vector<RTile>& tiles, bool want_leafof, cudaStream_t st, double node_frac,
                 size_t leafof_slots, bool want_rank, bool walks) {
  B.ntiles = static_cast<int>(tiles.size());
  unsigned long long e = 0, nn = 0;
  uint32_t emax = 0;
  unsigned long long nch = 0;  // chunks
  unsigned long long rr = 0;
  for (auto& t : tiles) {
    t.ebase = e;
    t.ncap = static_cast<uint32_t>(std::min<double>(t.ecap + 2.0, std::ceil(t.ecap * node_frac) + 64.0));
    t.nbase = nn;
    t.rcap = t.ncap / 2 + 1;
    t.rbase = static_cast<uint32_t>(rr);
    e += t.ecap;
    nn += t.ncap;
    rr += t.rcap;
    emax = std::max(emax, t.ecap);
  }
  B.wpw = e < RT_LARGE ? RT_WPW_SMALL : RT_WPW_LARGE;
  const unsigned chunk = rt_chunk(B.wpw);
  for (auto& t : tiles) nch += (std::max(t.ecap, 1u) + chunk - 1) / chunk;
  FG_REQUIRE(e < 0x7fffffffull && nn < 0x7fffffffull, "too many elements for one reference-tree build");
  B.E = e;
  B.N = nn;
  B.R = rr;
  B.levels = levels_for(emax);
  const size_t E1 = static_cast<size_t>(std::max<unsigned long long>(e, 1));
  const size_t N1 = static_cast<size_t>(std::max<unsigned long long>(nn, 1));
  // Pending nodes have more than RT_CTA_MAX elements; the walks' refit counts every node's arrivals.
  const size_t wl = walks ? N1 : static_cast<size_t>(e / RT_CTA_MAX + tiles.size() + 1);
  B.tiles.alloc(tiles.size(), st);
  FG_CUDA(cudaMemcpyAsync(B.tiles.p, tiles.data(), tiles.size() * sizeof(RTile), cudaMemcpyHostToDevice, st));
  B.idx0.alloc(E1, st);
  B.idx1.alloc(E1, st);
  B.key0.alloc(3 * E1, st);
  B.key1.alloc(3 * E1, st);
  B.nof0.alloc(E1, st);
  B.nof1.alloc(E1, st);
  B.nblk = nch;
  B.bits.alloc(nch * (chunk / 32), st);
  B.wp.alloc(nch * (chunk / 32), st);
  B.blk.alloc(nch, st);
  B.P.alloc(E1, st);
  B.Q.alloc(E1, st);
  B.ridx.alloc(E1, st);
  B.acc.alloc(6 * N1, st);
  B.box64.alloc(6 * N1, st);
  B.parent.alloc(N1, st);
  B.nstart.alloc(N1, st);
  B.ncount.alloc(N1, st);
  B.ntile.alloc(N1, st);
  B.ndepth.alloc(N1, st);
  B.nsplit.alloc(N1, st);
  B.nthr.alloc(N1, st);
  B.nchild.alloc(N1, st);
  B.wl0.alloc(wl, st);
  B.wl1.alloc(wl, st);
  B.bq.alloc(N1, st);
  B.bqpar.alloc(N1, st);
  B.cnt.alloc(RT_CNT_TILES + tiles.size() + 1, st);
  if (walks) {
    B.rnode.alloc(std::max<unsigned long long>(rr, 1), st);
    B.rleaf.alloc(N1, st);
  }
  if (want_leafof) B.leafof.alloc(std::max(E1, leafof_slots), st);
  if (want_rank) B.rank.alloc(std::max(E1, leafof_slots), st);
  FG_CUDA(cudaMemsetAsync(B.ridx.p, 0, E1 * sizeof(uint32_t), st));
}

namespace {

// Carves the buffers of a one-tile tree from `base` (or only counts the bytes when base is null).
size_t carve(RTreeBufs* B, uint32_t ecap, bool want_leafof, uint32_t leafof_slots, unsigned char* base) {
  const size_t E1 = std::max<uint32_t>(ecap, 1);
  const size_t N1 = rt_attach_nodes(E1);
  const size_t nblk = rt_attach_blocks(E1);
  static_assert(rt_chunk(RT_WPW_LARGE) == 2048, "rt_attach_blocks assumes chunks of 2048 positions");
  size_t off = 0;
  auto take = [&](auto& buf, size_t count) {
    using T = typename std::remove_reference<decltype(*buf.p)>::type;
    off = (off + 255) / 256 * 256;
    if (base) buf.view(reinterpret_cast<T*>(base + off), count);
    off += count * sizeof(T);
  };
  RTreeBufs dummy;
  RTreeBufs& b = B ? *B : dummy;
  take(b.tiles, 1);
  take(b.idx0, E1);
  take(b.idx1, E1);
  take(b.key0, 3 * E1);
  take(b.key1, 3 * E1);
  take(b.nof0, E1);
  take(b.nof1, E1);
  take(b.bits, E1 + 1);
  take(b.wp, E1 + 1);
  take(b.blk, nblk);
  take(b.P, E1);
  take(b.Q, E1);
  take(b.ridx, E1);
  take(b.acc, 6 * N1);
  take(b.box64, 6 * N1);
  take(b.parent, N1);
  take(b.nstart, N1);
  take(b.ncount, N1);
  take(b.ntile, N1);
  take(b.ndepth, N1);
  take(b.nsplit, N1);
  take(b.nthr, N1);
  take(b.nchild, N1);
  take(b.wl0, N1);
  take(b.wl1, N1);
  take(b.bq, N1);
  take(b.bqpar, N1);
  take(b.cnt, RT_CNT_TILES + 2);
  take(b.rnode, N1 / 2 + 1);
  take(b.rleaf, N1);
  if (want_leafof) take(b.leafof, std::max<uint32_t>(leafof_slots, 1));
  if (B) {
    B->ntiles = 1;
    B->E = E1;
    B->N = N1;
    B->R = N1 / 2 + 1;
    B->nblk = nblk;
    B->wpw = RT_WPW_LARGE;
    B->levels = levels_for(ecap);
  }
  return (off + 255) / 256 * 256;
}

}  // namespace

size_t rtree_scratch_bytes(uint32_t ecap, bool want_leafof, uint32_t leafof_slots) {
  return carve(nullptr, ecap, want_leafof, leafof_slots, nullptr);
}

void rtree_attach(RTreeBufs& B, RTile tile, bool want_leafof, uint32_t leafof_slots, unsigned char* base,
                  size_t bytes, cudaStream_t st) {
  const size_t need = carve(nullptr, tile.ecap, want_leafof, leafof_slots, nullptr);
  FG_REQUIRE(need == rtree_attach_bytes(tile.ecap, want_leafof, leafof_slots), "tree scratch layout mismatch");
  FG_REQUIRE(need <= bytes, "tree scratch too small");
  FG_REQUIRE(tile.ecap >= rt_chunk(RT_WPW_LARGE), "tree scratch: the flag words need a chunk's worth of elements");
  carve(&B, tile.ecap, want_leafof, leafof_slots, base);
  tile.ebase = 0;
  tile.nbase = 0;
  tile.ncap = static_cast<uint32_t>(B.N);
  tile.rbase = 0;
  tile.rcap = static_cast<uint32_t>(B.R);
  FG_CUDA(cudaMemcpyAsync(B.tiles.p, &tile, sizeof(RTile), cudaMemcpyHostToDevice, st));
}

namespace {

template <class K>
void build_topology(const RTreeBufs& B, const RtArgs& A, cudaStream_t st) {
  int dev = 0, sms = 0;
  FG_CUDA(cudaGetDevice(&dev));
  FG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  // The launch bounds let that many blocks share an SM, so the whole grid runs at once.
  const unsigned long long room = 1ull * rt_blocks(K::WIDE) * sms;
  const unsigned GL = static_cast<unsigned>(std::max<unsigned long long>(std::min<unsigned long long>(B.nblk, room), 1));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(GL);
  cfg.blockDim = dim3(RT_BLOCK);
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeCooperative;
  at.val.cooperative = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  FG_CUDA(B.wpw == RT_WPW_SMALL ? cudaLaunchKernelEx(&cfg, k_rt_levels<K, RT_WPW_SMALL>, A, B.levels)
                                : cudaLaunchKernelEx(&cfg, k_rt_levels<K, RT_WPW_LARGE>, A, B.levels));
  const unsigned GC = static_cast<unsigned>(
      std::min<unsigned long long>(B.E / (RT_LEAF_MAX + 1) + static_cast<unsigned long long>(B.ntiles), 152ull * 8));
  static_assert(sizeof(RtCtaSmem<K>) <= 56 * 1024, "four blocks of the block phase must fit an SM");
  FG_CUDA(cudaFuncSetAttribute(k_rt_cta<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(sizeof(RtCtaSmem<K>))));
  k_rt_cta<K><<<GC, RT_CTA_T, sizeof(RtCtaSmem<K>), st>>>(A);
  FG_CUDA(cudaGetLastError());
}

}  // namespace

void rtree_build(RTreeBufs& B, uint32_t* err, cudaStream_t st, bool walks, bool key32, RTile* tiles_dev) {
  if (B.ntiles == 0) return;
  FG_REQUIRE(B.ntiles <= 65535, "too many trees for one build");
  RtArgs A = rt_args(B, err);
  if (tiles_dev) A.tiles = tiles_dev;
  FG_CUDA(cudaMemsetAsync(B.cnt.p, 0, RT_CNT_TILES * sizeof(uint32_t), st));
  FG_CUDA(cudaMemsetAsync(B.blk.p, 0, static_cast<size_t>(B.nblk) * sizeof(unsigned long long), st));
  if (key32) build_topology<Key32>(B, A, st); else build_topology<Key64>(B, A, st);
  // Per-tile grids over the nodes (about 0.67 per element).
  const unsigned long long per = (B.N / static_cast<unsigned long long>(B.ntiles) + RT_BLOCK) / RT_BLOCK;
  const unsigned GX = static_cast<unsigned>(std::max<unsigned long long>(std::min<unsigned long long>(per, 152ull * 16), 1));
  const dim3 GN(GX, static_cast<unsigned>(B.ntiles));
  if (key32) k_rt_leaves<true><<<GN, RT_BLOCK, 0, st>>>(A, B.rleaf.p, B.leafof.p, B.leafof.n, B.rank.p);
  else k_rt_leaves<false><<<GN, RT_BLOCK, 0, st>>>(A, B.rleaf.p, B.leafof.p, B.leafof.n, B.rank.p);
  if (walks) {
    // The worklist is spent: its words count the children that reached each node.
    FG_CUDA(cudaMemsetAsync(B.wl0.p, 0, static_cast<size_t>(B.N) * sizeof(uint32_t), st));
    k_rt_refit<<<GN, RT_BLOCK, 0, st>>>(A, B.wl0.p);
    k_rt_records<<<static_cast<unsigned>(std::min<unsigned long long>((B.N + RT_BLOCK - 1) / RT_BLOCK, 152ull * 16)),
                   RT_BLOCK, 0, st>>>(A, B.rnode.p);
  }
  FG_CUDA(cudaGetLastError());
}

// Element lists of an emulsion in crystal-id order: all crystals (their slots), or the developed
// ones (flag, exclusive sum, scatter).
__global__ void k_rt_id_slots(const uint32_t* id2s, uint32_t n, const uint8_t* developed, uint32_t* flag) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const uint32_t s = id2s ? id2s[k] : k;
  flag[k] = developed[s] ? 1u : 0u;
}
__global__ void k_rt_id_scatter(const uint32_t* id2s, uint32_t n, const uint32_t* flag, const uint32_t* pos,
                                uint32_t* list) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n || !flag[k]) return;
  list[pos[k]] = id2s ? id2s[k] : k;
}

void build_emulsion_tree(fg_engine* e, const fg_emulsion* em, bool developed_only, RTreeBufs& B,
                         DBuf<uint32_t>& list, bool walks) {
  cudaStream_t st = e->stream;
  const uint32_t n = em->n;
  RTile t{};
  t.a = em->a.p;
  t.d = em->d.p;
  t.pos64 = em->has64 ? em->pos64.p : nullptr;
  t.dims64 = em->has64 ? em->dims64.p : nullptr;
  t.exp64 = developed_only ? em->exp64.p : nullptr;
  t.pad = static_cast<float>(std::max(em->extent, std::max(em->cfg.width, em->cfg.height)) * 2e-6 + 1e-5);
  t.reach = developed_only ? 0.0f : rt_reach(em->any_cubic ? em->max_half_dim : 0.0);
  const uint32_t* id2s = em->h_s2id.empty() ? nullptr : em->id_to_sorted.p;
  uint32_t m = n;
  if (developed_only && n) {
    DBuf<uint32_t> flag(n + 1, st), pos(n + 1, st);
    FG_CUDA(cudaMemsetAsync(flag.p + n, 0, sizeof(uint32_t), st));
    k_rt_id_slots<<<grid_for(n, 256), 256, 0, st>>>(id2s, n, em->developed.p, flag.p);
    exclusive_scan_u32(flag.p, pos.p, n + 1, st);
    FG_CUDA(cudaMemcpyAsync(&m, pos.p + n, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    FG_CUDA(cudaStreamSynchronize(st));
    list.alloc(std::max<uint32_t>(m, 1), st);
    k_rt_id_scatter<<<grid_for(n, 256), 256, 0, st>>>(id2s, n, flag.p, pos.p, list.p);
    FG_CUDA(cudaGetLastError());
    t.order = list.p;
  } else {
    t.order = id2s;
  }
  t.ecap = developed_only ? std::max<uint32_t>(m, 1) : std::max<uint32_t>(n, 1);
  t.n = developed_only ? m : n;
  std::vector<RTile> v{t};
  rtree_alloc(B, v, true, st, 1.0, n, !developed_only, walks);
  // The developed crystals of a set that was accepted can be more uneven than the set.
  if (developed_only) B.levels = std::max(B.levels, m > static_cast<uint32_t>(RT_CTA_MAX) ? RT_LEVELS : 0);
  // FP32 crystals without expansion: the centroids are the positions themselves.
  rtree_build(B, e->d_err, st, walks, !em->has64 && !developed_only && std::isfinite(em->max_half_dim));
  B.count = t.n;
}

unsigned rtree_kernel_launches(const RTreeBufs& B, bool walks) {
  return B.ntiles ? (walks ? 5u : 3u) : 0u;
}

}  // namespace fg

extern "C" fg_status fg_emulsion_reference_tree(fg_engine* e, const fg_emulsion* em, int developed_only,
                                                uint32_t* order, uint32_t* leaves, double* leaf_boxes, size_t cap,
                                                size_t* nelem, size_t* nleaves) {
  using namespace fg;
  return guard(e, [&] {
    FG_REQUIRE(em, "null emulsion");
    cudaStream_t st = e->stream;
    begin_call(e);
    RTreeBufs local;
    DBuf<uint32_t> list;
    const RTreeBufs* T = &em->rt;
    if (developed_only) {
      build_emulsion_tree(e, em, true, local, list);
      T = &local;
    }
    RTile tile{};
    if (T->ntiles) FG_CUDA(cudaMemcpyAsync(&tile, T->tiles.p, sizeof(RTile), cudaMemcpyDeviceToHost, st));
    FG_CUDA(cudaStreamSynchronize(st));
    end_call(e);  // raises a build error first
    const uint32_t n = T->ntiles ? tile.n : 0, nn = T->ntiles ? std::min(tile.nodes, tile.ncap) : 0;
    std::vector<uint32_t> ridx(n), nstart(nn), ncount(nn);
    std::vector<int> nsplit(nn);
    std::vector<double> box(6ull * nn);
    if (n) FG_CUDA(cudaMemcpyAsync(ridx.data(), T->ridx.p, n * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    if (nn) {
      FG_CUDA(cudaMemcpyAsync(nstart.data(), T->nstart.p, nn * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
      FG_CUDA(cudaMemcpyAsync(ncount.data(), T->ncount.p, nn * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
      FG_CUDA(cudaMemcpyAsync(nsplit.data(), T->nsplit.p, nn * sizeof(int), cudaMemcpyDeviceToHost, st));
      FG_CUDA(cudaMemcpyAsync(box.data(), T->box64.p, 6ull * nn * sizeof(double), cudaMemcpyDeviceToHost, st));
    }
    FG_CUDA(cudaStreamSynchronize(st));
    if (nelem) *nelem = n;
    if (order)
      for (uint32_t k = 0; k < n && k < cap; ++k) order[k] = em->h_s2id.empty() ? ridx[k] : em->h_s2id[ridx[k]];
    std::vector<uint32_t> lf;
    for (uint32_t id = 1; id < nn && n; ++id)
      if (nsplit[id] < 0) lf.push_back(id);
    std::sort(lf.begin(), lf.end(), [&](uint32_t a, uint32_t b) { return nstart[a] < nstart[b]; });
    if (nleaves) *nleaves = lf.size();
    for (size_t k = 0; k < lf.size() && k < cap; ++k) {
      if (leaves) {
        leaves[2 * k] = nstart[lf[k]];
        leaves[2 * k + 1] = ncount[lf[k]];
      }
      if (leaf_boxes)
        for (int j = 0; j < 6; ++j) leaf_boxes[6 * k + j] = box[6ull * lf[k] + j];
    }
  });
}
