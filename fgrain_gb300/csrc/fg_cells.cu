// Builds the cells of fg_cells.cuh: count the crystals of every cell, prefix sum, then write each
// crystal's record at its position with its leaf box and walk rank from the reference tree; place
// then holds the position of each slot.
//
// Both passes stream the crystals in slot order (compact blocks of the film), so the counters and
// the scattered records of a warp fall into few cache lines.
#include "fg_internal.h"
#include "fg_transport.cuh"

namespace fg {

__device__ __forceinline__ int cells_tile_of(const TileDesc* tiles, int ntiles, unsigned long long g) {
  int lo = 0, hi = ntiles - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tiles[mid].cbase <= g) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ unsigned long long cell_index(const CellGrid& c, const float4& a) {
  const uint32_t x = static_cast<uint32_t>(cell_coord(a.x, c.x.inv, c.x.last));
  const uint32_t y = static_cast<uint32_t>(cell_coord(a.y, c.y.inv, c.y.last));
  const uint32_t z = static_cast<uint32_t>(cell_coord(a.z, c.z.inv, c.z.last));
  return c.cell_base + (static_cast<unsigned long long>(y) * c.z.n + z) * c.x.n + x;
}

// Counts; place[g] is the crystal's number inside its cell (any order: hits are put in rank order).
// *unfit (may be null) is set when a cell holds more than `limit` crystals or a centre lies outside
// the box.
__global__ void k_cells_count(const TileDesc* __restrict__ tiles, int ntiles, unsigned long long ncap,
                              const float4* __restrict__ A, uint32_t* __restrict__ cnt, uint32_t* __restrict__ place,
                              uint32_t limit, uint32_t* unfit) {
  const unsigned long long g = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x;
  if (g >= ncap) return;
  const TileDesc& t = tiles[cells_tile_of(tiles, ntiles, g)];
  if (g - t.cbase >= t.n) return;
  const float4 a = A[g];
  const uint32_t k = atomicAdd(&cnt[cell_index(t.cells, a)], 1u);
  place[g] = k;
  const bool in = a.x >= 0.0f && a.y >= 0.0f && a.z >= 0.0f && a.x <= t.cells.hx && a.y <= t.cells.hy && a.z <= t.cells.hz;
  if (unfit && (k == limit || !in)) *unfit = 1u;
}

// The density about a crystal over the mean one, times crystals: the sum of n_b^2 / v_b over blocks of about 80
// crystals (4 mean spacings in x and y, 5 in z), n_b the block's crystals and v_b its cells.
constexpr uint32_t UNEVEN_X = 20, UNEVEN_Y = 4, UNEVEN_Z = 2;
__global__ void k_cells_uneven(CellAxis x, CellAxis y, CellAxis z, const uint32_t* __restrict__ off, double* out) {
  const uint32_t bx = (x.n + UNEVEN_X - 1) / UNEVEN_X, by = (y.n + UNEVEN_Y - 1) / UNEVEN_Y;
  const unsigned long long blocks = 1ull * bx * by * ((z.n + UNEVEN_Z - 1) / UNEVEN_Z);
  double sum = 0.0;
  for (unsigned long long b = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; b < blocks;
       b += 1ull * gridDim.x * blockDim.x) {
    const uint32_t x0 = static_cast<uint32_t>(b % bx) * UNEVEN_X, y0 = static_cast<uint32_t>(b / bx % by) * UNEVEN_Y;
    const uint32_t z0 = static_cast<uint32_t>(b / bx / by) * UNEVEN_Z;
    const uint32_t x1 = min(x0 + UNEVEN_X, x.n), y1 = min(y0 + UNEVEN_Y, y.n), z1 = min(z0 + UNEVEN_Z, z.n);
    uint32_t n = 0;
    for (uint32_t j = y0; j < y1; ++j)
      for (uint32_t k = z0; k < z1; ++k) {
        const uint32_t* row = off + (j * z.n + k) * x.n;
        n += row[x1] - row[x0];
      }
    sum += static_cast<double>(n) * n / ((x1 - x0) * (y1 - y0) * (z1 - z0));
  }
  if (sum != 0.0) atomicAdd(out, sum);
}

void launch_cells_uneven(const CellGrid& g, double* out, cudaStream_t st) {
  k_cells_uneven<<<256, 128, 0, st>>>(g.x, g.y, g.z, g.off, out);
  FG_CUDA(cudaGetLastError());
}

__global__ void k_cells_fill(const TileDesc* __restrict__ tiles, int ntiles, unsigned long long ncap,
                             const float4* __restrict__ A, const float4* __restrict__ Q, const float4* __restrict__ D,
                             const uint32_t* __restrict__ off, uint32_t* __restrict__ place,
                             const uint32_t* __restrict__ rank, const uint32_t* __restrict__ leafof,
                             const double* __restrict__ box64, float4* __restrict__ pos, float4* __restrict__ q,
                             float4* __restrict__ d, float4* __restrict__ leaf, uint2* __restrict__ by_rank,
                             uint32_t* err) {
  const unsigned long long g = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x;
  if (g >= ncap) return;
  const TileDesc& t = tiles[cells_tile_of(tiles, ntiles, g)];
  const unsigned long long s = g - t.cbase;
  if (s >= t.n) return;
  const float4 a = A[g], dd = D[g];
  const uint32_t p = off[cell_index(t.cells, a)] + place[g];
  const uint32_t r = rank[g], lf = leafof[g];
  if (!index_ok(p < t.cells.npos && r < t.n && lf < t.nnodes, err, SITE_CELL, p, r)) return;
  place[g] = p;
  pos[p] = make_float4(a.x, a.y, a.z, cell_ball2(dd));
  q[p] = Q[g];
  d[p] = dd;
  // The leaf box as the reference's test sees it in the FP32 walk: rounded to nearest.
  const double* b = box64 + 6ull * (t.nbase + lf);
  leaf[2ull * p] = make_float4(__double2float_rn(b[0]), __double2float_rn(b[1]), __double2float_rn(b[2]),
                               __double2float_rn(b[3]));
  leaf[2ull * p + 1] = make_float4(__double2float_rn(b[4]), __double2float_rn(b[5]), __uint_as_float(r),
                                   __uint_as_float(static_cast<uint32_t>(s)));
  by_rank[t.cbase + r] = make_uint2(static_cast<uint32_t>(s), __float_as_uint(a.w));
}

void launch_cells_count(const TileDesc* tiles, int ntiles, unsigned long long ncap, const float4* A, uint32_t* cnt,
                        uint32_t* place, cudaStream_t st, uint32_t limit, uint32_t* unfit) {
  if (ncap == 0) return;
  k_cells_count<<<grid_for(ncap, 256), 256, 0, st>>>(tiles, ntiles, ncap, A, cnt, place, limit, unfit);
  FG_CUDA(cudaGetLastError());
}

void launch_cells_fill(const TileDesc* tiles, int ntiles, unsigned long long ncap, const float4* A, const float4* Q,
                       const float4* D, const RTreeBufs& tree, const CellBufs& c, uint32_t* err, cudaStream_t st) {
  if (ncap == 0) return;
  k_cells_fill<<<grid_for(ncap, 256), 256, 0, st>>>(tiles, ntiles, ncap, A, Q, D, c.off.p, c.place.p, tree.rank.p,
                                                    tree.leafof.p, tree.box64.p, c.pos.p, c.q.p, c.d.p, c.leaf.p,
                                                    c.by_rank.p, err);
  FG_CUDA(cudaGetLastError());
}

void CellBufs::alloc(unsigned long long ncap, unsigned long long cells, cudaStream_t st) {
  const size_t n = static_cast<size_t>(ncap > 0 ? ncap : 1);
  ncells = cells;
  cnt.alloc(cells + 1, st);
  off.alloc(cells + 1, st);
  place.alloc(n, st);
  pos.alloc(n, st);
  q.alloc(n, st);
  d.alloc(n, st);
  leaf.alloc(2 * n, st);
  by_rank.alloc(n, st);
}

void CellBufs::attach(CellGrid& g, unsigned long long cbase) const {
  g.pos = pos.p;
  g.q = q.p;
  g.d = d.p;
  g.leaf = leaf.p;
  g.off = off.p + g.cell_base;
  g.by_rank = by_rank.p + cbase;
  g.npos = static_cast<uint32_t>(pos.n);
}

}  // namespace fg
