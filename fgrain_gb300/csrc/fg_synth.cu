// Device crystal synthesis: column-parallel Bridson, thinning to the reference density, Morton
// compaction and crystal attributes.  See fg_synth.cuh for the scheme.
#include <algorithm>

#include "fg_internal.h"
#include "fg_synth.cuh"

namespace fg {

enum : uint32_t {
  TAG_CAND = 0x43410000u,
  TAG_SEED = 0x53450000u,
  TAG_THIN = 0x54480000u,
};

// True when the point of an occupied cell (word w) is closer than r to the candidate, (ox, oy, oz)
// being the cell's corner relative to the candidate (fixed point), oz less SYN_OCC_Z: the word's
// occupancy bit comes down with its z.
constexpr int SYN_OCC_Z = static_cast<int>(OCC >> 20);
__device__ __forceinline__ bool syn_conflict(uint32_t w, int ox, int oy, int oz) {
  const int ex = ox + static_cast<int>(w & 1023u);
  const int ey = oy + static_cast<int>((w >> 10) & 1023u);
  const int ez = oz + static_cast<int>(w >> 20);
  return ex * ex + ey * ey + ez * ez < SYN_R2X;
}

// Occupancy rows of the staged region: word (rz, ry) holds the cells of row (rz, ry) in bits 0-15
// (bit rx) and those of row (rz, ry + 1) in bits 16-31, so the 3 x 3 x 3 cells around a cell are
// six words.  About one cell in nine holds a point: a candidate visits the occupied cells only.
__device__ __forceinline__ void syn_mark(uint32_t* rows, int row, int rx) {
  atomicOr(rows + row, 1u << rx);
  atomicOr(rows + row - 1, 0x10000u << rx);
}

// The 27 cells of the inner block in the order of syn_near_free's mask bits: the rows above and
// below in y of the three layers (6 bits a layer), then the rows of the candidate's own y, its own
// row last.  The last bits are visited first: they are the likeliest to hold a conflict.
// An entry: the cell's corner offset (fixed point, z less SYN_OCC_Z) and its region index offset.
__device__ __forceinline__ int4 syn_near_entry(int k) {
  const int dx = k % 3 - 1;
  const int dy = k < 18 ? ((k / 3) % 2 ? 1 : -1) : 0;
  const int dz = k < 18 ? k / 6 - 1 : (k < 21 ? -1 : (k < 24 ? 1 : 0));
  return make_int4(dx * SYN_Q, dy * SYN_Q, dz * SYN_Q - SYN_OCC_Z, (dz * SYN_R + dy) * SYN_R + dx);
}

// First half of the candidate test, one lane per candidate: the points in the 27 cells of the inner
// 3x3x3 block.  They reject about 87 % of Bridson candidates, so the lanes that survive are few and
// the rest of the test runs warp-cooperatively (syn_outer_free).  A point in the candidate's own
// cell always conflicts (two points of a cell are less than r apart).
__device__ __forceinline__ bool syn_near_free(const uint32_t* grid, const uint32_t* rows, const int4* cells27, int rx,
                                              int row, int rb, int lx, int ly, int lz) {
  const uint32_t* w = rows + row;
  const int sh = rx - 1;
  const uint32_t a0 = w[-SYN_R - 1] >> sh, c0 = w[-SYN_R + 1] >> sh;
  const uint32_t a1 = w[-1] >> sh, c1 = w[1] >> sh;
  const uint32_t a2 = w[SYN_R - 1] >> sh, c2 = w[SYN_R + 1] >> sh;
  if (a1 & 0x20000u) return false;
  uint32_t m = (a0 & 7u) | ((c0 & 7u) << 3) | ((a1 & 7u) << 6) | ((c1 & 7u) << 9) | ((a2 & 7u) << 12) |
               ((c2 & 7u) << 15) | ((a0 & 0x70000u) << 2) | ((a2 & 0x70000u) << 5) | ((a1 & 0x70000u) << 8);
  while (m) {
    const int k = 31 - __clz(static_cast<int>(m));
    m ^= 1u << k;
    const int4 c = cells27[k];
    if (syn_conflict(grid[rb + c.w], c.x - lx, c.y - ly, c.z - lz)) return false;
  }
  return true;
}

// Whether the candidate at region cell cb = row * SYN_R + rx, fixed-point offsets (cx, cy, cz) inside
// it, has a point within r in the 90 cells of the 5x5x5 neighbourhood outside the inner block
// (without its eight corners, which cannot hold a point within r = sqrt(3) cells): lane 5 (dz + 2) +
// dy + 2 takes the row at (dy, dz), its occupied cells only.  All 32 lanes call it with the same
// candidate; the answer is the same in every lane.
__device__ __forceinline__ bool syn_outer_hit(const uint32_t* grid, const uint32_t* rows, int cb, int cx, int cy,
                                              int cz, int lane) {
  bool hit = false;
  if (lane < 25) {
    const int dz = lane / 5 - 2, dy = lane % 5 - 2;
    const bool ez = dz == -2 || dz == 2, ey = dy == -2 || dy == 2;
    const int row = cb / SYN_R, rx = cb - row * SYN_R;
    const int r2 = row + dz * SYN_R + dy;
    // Bits 0-4: the cells at dx = -2 .. 2.
    uint32_t m = (rows[r2] >> (rx - 2)) & (ez && ey ? 0x0eu : (ez || ey ? 0x1fu : 0x11u));
    const uint32_t* g = grid + r2 * SYN_R + rx - 2;
    while (m) {
      const int k = 31 - __clz(static_cast<int>(m));
      m ^= 1u << k;
      if (syn_conflict(g[k], (k - 2) * SYN_Q - cx, dy * SYN_Q - cy, dz * SYN_Q - SYN_OCC_Z - cz)) {
        hit = true;
        break;
      }
    }
  }
  return __any_sync(0xffffffffu, hit);
}

// Second half of the test for the lanes whose candidates passed syn_near_free: the warp takes the
// survivors one at a time, in lane order, until one also passes the outer cells: the step's first
// valid candidate, the only lane left valid.  The survivors after it stay untested (`rest`, the
// same in every lane): the round's resolution needs another candidate only when that one
// conflicts with a point accepted for an earlier warp, and tests them then.  All 32 lanes call it.
__device__ __forceinline__ bool syn_outer_free(const uint32_t* grid, const uint32_t* rows, bool valid, int rb, int lx,
                                               int ly, int lz, int lane, unsigned& rest) {
  unsigned sm = __ballot_sync(0xffffffffu, valid);
  int win = -1;
  while (sm) {
    const int c = __ffs(sm) - 1;
    sm &= sm - 1;
    const int cb = __shfl_sync(0xffffffffu, rb, c);
    const int cx = __shfl_sync(0xffffffffu, lx, c);
    const int cy = __shfl_sync(0xffffffffu, ly, c);
    const int cz = __shfl_sync(0xffffffffu, lz, c);
    if (!syn_outer_hit(grid, rows, cb, cx, cy, cz, lane)) {
      win = c;
      break;
    }
  }
  rest = sm;
  return lane == win;
}

// Exact test of a fixed-point candidate against the staged grid: every point within r.  The eight
// corner cells of the 5x5x5 neighbourhood cannot hold a point within r = sqrt(3) cells.  The
// outer loop stays rolled (small code), the first point within r ends the test.
__device__ __forceinline__ bool syn_free(const uint32_t* grid, int nz, int rx, int ry, int rz, int X, int Y, int Z,
                                         int cx, int cy, int cz, uint32_t* err) {
  // The neighbourhood must lie inside the staged region (it does for candidates within 2r of a
  // point of the column); a candidate that fails the check is rejected.
  if (!index_ok(rx >= 2 && rx <= SYN_R - 3 && ry >= 2 && ry <= SYN_R - 3 && rz >= 2 && rz <= nz - 3, err,
                SITE_SYN_REGION, static_cast<uint32_t>(rx | (ry << 8) | (rz << 16)), blockIdx.x))
    return false;
#pragma unroll 1
  for (int dz = -2; dz <= 2; ++dz) {
    const bool zedge = dz == -2 || dz == 2;
#pragma unroll
    for (int dy = -2; dy <= 2; ++dy) {
      const int row = ((rz + dz) * SYN_R + (ry + dy)) * SYN_R + rx;
#pragma unroll
      for (int dx = -2; dx <= 2; ++dx) {
        if (zedge && (dx == -2 || dx == 2) && (dy == -2 || dy == 2)) continue;
        const uint32_t w = grid[row + dx];
        if (w & OCC) {
          const int ex = (cx + dx) * SYN_Q + static_cast<int>(w & 1023u) - X;
          const int ey = (cy + dy) * SYN_Q + static_cast<int>((w >> 10) & 1023u) - Y;
          const int ez = (cz + dz) * SYN_Q + static_cast<int>((w >> 20) & 1023u) - Z;
          if (ex * ex + ey * ey + ez * ez < SYN_R2X) return false;
        }
      }
    }
  }
  return true;
}

__device__ __forceinline__ uint32_t syn_word(int X, int Y, int Z) {
  return OCC | (static_cast<uint32_t>(Z & 1023) << 20) | (static_cast<uint32_t>(Y & 1023) << 10) |
         static_cast<uint32_t>(X & 1023);
}

// philox with its ten round keys from a table (the same in every step of a column): eighteen
// additions a draw less.
__device__ __forceinline__ P4 philox_keys(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, const uint4* keys) {
#pragma unroll
  for (int r = 0; r < 5; ++r) {
    const uint4 k = keys[r];  // the keys of two rounds
    const uint32_t a0 = __umulhi(PHILOX_M1, c2) ^ c1 ^ k.x, a2 = __umulhi(PHILOX_M0, c0) ^ c3 ^ k.y;
    const uint32_t a1 = PHILOX_M1 * c2, a3 = PHILOX_M0 * c0;
    c0 = __umulhi(PHILOX_M1, a2) ^ a1 ^ k.z;
    c1 = PHILOX_M1 * a2;
    c2 = __umulhi(PHILOX_M0, a0) ^ a3 ^ k.w;
    c3 = PHILOX_M0 * a0;
  }
  return P4{c0, c1, c2, c3};
}

// The draws of a step's lane (thread `slot` of the column): a lane that places a candidate gets its
// offset from the active point in the shell [r, 2 r] (fixed point), the last lane the bits (.x) that
// pick the active point.
__device__ __forceinline__ float3 syn_draw(int iter, int slot, int lane, uint32_t colkey, const uint4* keys) {
  const P4 r = philox_keys(static_cast<uint32_t>(iter), static_cast<uint32_t>(slot), colkey, TAG_CAND, keys);
  const float u = uf(r.x);
  const float ct = uf(r.y) * 2.0f - 1.0f;
  const float st = sqrtf(fmaxf(1.0f - ct * ct, 0.0f));
  float sp, cp;
  sincospif(uf(r.z) * 2.0f, &sp, &cp);
  const float rad = cbrtf(7.0f * u + 1.0f) * 1.7320508075688772f * SYN_Q;  // r = sqrt(3) cells
  const float x = __fmul_rn(rad * st, cp);
  return make_float3(lane < SYN_K ? x : __uint_as_float(r.x), __fmul_rn(rad * st, sp), __fmul_rn(rad, ct));
}

// An entry of the active list: the cell's region coordinates (SYN_R < 16; a region that fits in
// shared memory has at most 256 layers).
static_assert(SYN_R <= 16 && bridson_smem(253) > BRIDSON_SMEM_MAX, "4 + 4 + 8 bits hold a position");
__device__ __forceinline__ uint16_t syn_pos(int rx, int ry, int rz) {
  return static_cast<uint16_t>(rx | ry << 4 | rz << 8);
}

// What bounds it: issue slots (76 % issue activity at 24 of 32 lanes; DRAM 1 %): about 620 warp
// instructions a step, 31 rounds of 8 steps for the 115 points of a t-max column, which is within
// 10 % of one step per point kept and one per point retired.  Visiting only the occupied cells (one
// in nine, from the occupancy rows) instead of testing all 27 + 90 took the kernel from 38.8 to
// 28.5 ms on a 1600 x 1600 px t-max image; the instructions taken out since (one bounds check by
// subtraction in each axis, round keys and neighbour cells from shared memory, positions packed by
// coordinate) and the shorter resolution took it to 24.6 ms, and from 7.7 to 6.6 ms on a
// 2048 x 2048 px tri-x one.
//
// Launch bounds of 8 CTAs per SM (32 registers): more columns in flight hide the round's barriers.
// A column with its one-cell spill and the halo stages 14 x 14 cells per layer, and its list of active
// points has an entry for each that can fit (26 a layer), so eight CTAs fit in the SM's 228 KB of shared
// memory for depths up to 24 cells.  With an entry for each of the 64 cells of a layer seven ran at 23
// cells, tri-x-1600's depth (1600 x 1600 px of tri-x pushed two stops: 3.87 ms, now 3.69; 22 cells are
// the same), two instead of three at 77 (36.8, now 30.0).
//
// FEW: with few columns in flight the latency of a round counts instead (5,600 cycles, of which 1,950
// are the resolution by one warp).  4 CTAs per SM leave 64 registers, and the seven warps that wait
// draw the next round's candidates meanwhile.  The classes run nearly one after another, so 20
// columns an SM are about five in flight: on t-max films of 25 .. 1,936 columns it takes .34 - .45
// against .40 - .51 ms, at 2,601 .521 against .581, at 3,249 (21 an SM) .617 against .621, at 4,356
// .814 against .726.
constexpr unsigned SYN_FEW = 20;  // columns an SM
// All columns of all four colour classes in one launch, class after class in block order.  A column
// starts once the columns of lower classes next to it have written their cells back (their done
// flags), which gives every column the cell state it would see if the classes ran one launch
// after another: only the eight neighbouring columns share cells with it, and a neighbour of a
// higher class waits for it in turn.  The flags are waited on by lower block indices only, so
// the wait ends as the earlier blocks finish; it is bounded all the same (ERR_SPIN_LIMIT).
template <bool FEW>
__global__ void __launch_bounds__(SYN_WARPS * 32, FEW ? 4 : 8) k_bridson(const SynthTile* __restrict__ tiles,
                                                            int ntiles, uint4 class_base, int nz,
                                                            uint32_t* __restrict__ cells,
                                                            uint32_t* __restrict__ npts, uint32_t* done,
                                                            uint32_t* err, uint32_t wait_limit,
                                                            const uint32_t* probe) {
  extern __shared__ uint32_t syn_sm[];
  uint32_t* grid = syn_sm;                                   // SYN_R^2 * nz cell words
  uint32_t* rows = grid + SYN_R * SYN_R * nz;                // SYN_R * nz occupancy rows (syn_mark)
  uint16_t* active = reinterpret_cast<uint16_t*>(rows + SYN_R * nz);  // syn_active_cap(nz - 4)
  __shared__ int s_nact, s_wsum[SYN_WARPS];
  __shared__ int s_ncom;  // points this column commits (each fills one empty cell of its tile)
  __shared__ int4 s_pick[SYN_WARPS / 4];   // the steps' picks
  __shared__ int4 s_win[SYN_WARPS];        // the step's winner from the region's corner; w: whether it has one
  __shared__ unsigned s_rmask[SYN_WARPS];  // later candidates that passed the near cells, untested
  __shared__ uint32_t s_cxy[SYN_WARPS][32];  // those: x | y << 16 from the region's corner
  __shared__ int s_cz[SYN_WARPS][32];
  __shared__ int4 s_near[27];
  __shared__ uint4 s_key[5];              // Philox round keys
  __shared__ float3 s_off[FEW ? 32 : 1];  // the next round's draws of the resolving warp
  static_assert(FEW || 8 * (bridson_smem(24) + sizeof(s_nact) + sizeof(s_wsum) + sizeof(s_ncom) + sizeof(s_pick) +
                            sizeof(s_win) + sizeof(s_rmask) + sizeof(s_cxy) + sizeof(s_cz) + sizeof(s_near) +
                            sizeof(s_key) + sizeof(s_off) + 1024) <= 228 * 1024,
                "eight CTAs of 24 cells (and 1 KB each) in an SM's shared memory");

  // Column of this CTA: colour class, tile, then the j-th column of this class in that tile.
  const uint32_t cb[4] = {class_base.x, class_base.y, class_base.z, class_base.w};
  const int color = blockIdx.x >= cb[3] ? 3 : (blockIdx.x >= cb[2] ? 2 : (blockIdx.x >= cb[1] ? 1 : 0));
  const uint32_t bidx = blockIdx.x - cb[color];
  int lo = 0, hi = ntiles - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tiles[mid].col_base[color] <= bidx) lo = mid; else hi = mid - 1;
  }
  const SynthTile& t = tiles[lo];
  const uint32_t j = bidx - t.col_base[color];
  const uint32_t cxn = (t.nbx - (color & 1) + 1) / 2;
  const uint32_t bx = 2 * (j % cxn) + (color & 1), by = 2 * (j / cxn) + (color >> 1);
  const int x0 = static_cast<int>(bx) * SYN_B, y0 = static_cast<int>(by) * SYN_B;
  const int x1 = min(x0 + SYN_B, static_cast<int>(t.gw)), y1 = min(y0 + SYN_B, static_cast<int>(t.gh));
  const int gd = static_cast<int>(t.gd);
  const int ox = x0 - SYN_HALO, oy = y0 - SYN_HALO;
  const uint32_t colkey = by * t.nbx + bx;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ncell = SYN_R * SYN_R * nz;
  const int acap = syn_active_cap(nz - 4);  // active list capacity
  uint32_t* tc = cells + t.cell_base;

  // Wait for the neighbouring columns of lower classes.
  if (tid == 0 && color > 0) {
    for (int dy = -1; dy <= 1; ++dy)
      for (int dx = -1; dx <= 1; ++dx) {
        const int nx = static_cast<int>(bx) + dx, ny = static_cast<int>(by) + dy;
        if ((dx == 0 && dy == 0) || nx < 0 || ny < 0 || nx >= static_cast<int>(t.nbx) || ny >= static_cast<int>(t.nby))
          continue;
        const int nc = (nx & 1) | ((ny & 1) << 1);
        if (nc >= color) continue;
        const uint32_t ncxn = (t.nbx - (nc & 1) + 1) / 2;
        const uint32_t id = cb[nc] + t.col_base[nc] + static_cast<uint32_t>(ny >> 1) * ncxn + static_cast<uint32_t>(nx >> 1);
        const volatile uint32_t* f = done + id;
        uint32_t spins = 0;
        while (*f == 0u) {
          if (++spins > wait_limit) {
            atomicOr(err, ERR_SPIN_LIMIT);
            break;
          }
          __nanosleep(64);
        }
      }
    __threadfence();
  }
  // Failure drill: a flag that nothing sets, waited on with the same bound.
  if (tid == 0 && probe) {
    const volatile uint32_t* f = probe;
    uint32_t spins = 0;
    while (*f == 0u) {
      if (++spins > wait_limit) {
        atomicOr(err, ERR_SPIN_LIMIT);
        break;
      }
      __nanosleep(64);
    }
  }
  __syncthreads();

  // Stage the region (column + halo) of the cell grid (through L2: neighbours wrote it).
  for (int i = tid; i < ncell; i += blockDim.x) {
    const int rx = i % SYN_R, ry = (i / SYN_R) % SYN_R, rz = i / (SYN_R * SYN_R);
    const int gx = ox + rx, gy = oy + ry, gz = rz - 2;
    uint32_t w = 0;
    if (gx >= 0 && gy >= 0 && gz >= 0 && gx < static_cast<int>(t.gw) && gy < static_cast<int>(t.gh) && gz < gd)
      w = __ldcg(tc + (static_cast<size_t>(gz) * t.gh + gy) * t.gw + gx);
    grid[i] = w;
  }
  if (tid < 5) {
    const uint32_t a = t.k0 + 2 * tid * PHILOX_W0, b = t.k1 + 2 * tid * PHILOX_W1;
    s_key[tid] = make_uint4(a, b, a + PHILOX_W0, b + PHILOX_W1);
  }
  if (tid < 27) s_near[tid] = syn_near_entry(tid);
  if (tid == 0) {
    s_nact = 0;
    s_ncom = 0;
  }
  __syncthreads();
  for (int j = tid; j < SYN_R * nz; j += blockDim.x) {
    uint32_t m = 0;
#pragma unroll
    for (int x = 0; x < SYN_R; ++x) m |= (grid[j * SYN_R + x] >> 31) << x;
    uint16_t* h = reinterpret_cast<uint16_t*>(rows);
    h[2 * j] = static_cast<uint16_t>(m);
    if (j > 0) h[2 * j - 1] = static_cast<uint16_t>(m);
  }
  __syncthreads();
  // Active list: the column's points in cell order (deterministic block-wide compaction).
  const int bw = x1 - x0, bh = y1 - y0;
  const int bcells = bw * bh * gd;
  for (int base = 0; base < bcells; base += blockDim.x) {
    const int i = base + tid;
    const int lx = i % bw, ly = (i / bw) % bh, lz = i / (bw * bh);
    const bool o =
        i < bcells && (grid[((lz + 2) * SYN_R + (ly + SYN_HALO)) * SYN_R + (lx + SYN_HALO)] & OCC) != 0;
    const unsigned m = __ballot_sync(0xffffffffu, o);
    if (lane == 0) s_wsum[warp] = __popc(m);
    __syncthreads();
    int off = s_nact;
    for (int w = 0; w < warp; ++w) off += s_wsum[w];
    const int at = off + __popc(m & ((1u << lane) - 1u));
    if (o) active[min(at, acap - 1)] = syn_pos(lx + SYN_HALO, ly + SYN_HALO, lz + 2);
    __syncthreads();
    if (tid == 0)
      for (int w = 0; w < SYN_WARPS; ++w) s_nact += s_wsum[w];
    __syncthreads();
  }
  // (Past the capacity only after a wait that gave up, which has set the error: the neighbours' points may
  // then be too close.)
  if (tid == 0) s_nact = min(s_nact, acap);
  // An empty column starts from one random point (poisson.rs:46-57), up to 30 tries.
  if (tid == 0 && s_nact == 0 && bw > 0 && bh > 0) {
    for (int k = 0; k < SYN_K; ++k) {
      const P4 r = philox(static_cast<uint32_t>(k), 0, colkey, TAG_SEED, t.k0, t.k1);
      const int X = x0 * SYN_Q + static_cast<int>(uf(r.x) * static_cast<float>(bw * SYN_Q));
      const int Y = y0 * SYN_Q + static_cast<int>(uf(r.y) * static_cast<float>(bh * SYN_Q));
      const int Z = static_cast<int>(uf(r.z) * static_cast<float>(t.ZW));
      if (X >= static_cast<int>(t.XW) || Y >= static_cast<int>(t.YW) || Z >= static_cast<int>(t.ZW)) continue;
      const int cx = X >> 10, cy = Y >> 10, cz = Z >> 10;
      const int rx = cx - ox, ry = cy - oy, rz = cz + 2;
      if (!syn_free(grid, nz, rx, ry, rz, X, Y, Z, cx, cy, cz, err)) continue;
      const int ridx = (rz * SYN_R + ry) * SYN_R + rx;
      grid[ridx] = syn_word(X, Y, Z);
      syn_mark(rows, rz * SYN_R + ry, rx);
      ++s_ncom;
      if (index_ok(s_nact < acap, err, SITE_SYN_ACTIVE, s_nact, blockIdx.x)) active[s_nact++] = syn_pos(rx, ry, rz);
      break;
    }
  }
  float3 off = FEW ? syn_draw(0, tid, lane, colkey, s_key) : float3{};
  const int max_iter = 16 * SYN_B * SYN_B * gd + 64;
  for (int iter = 0;; ++iter) {
    __syncthreads();
    const int nact = s_nact;
    if (nact == 0) break;
    if (iter >= max_iter) {
      if (tid == 0) atomicOr(err, ERR_SPIN_LIMIT);
      break;
    }
    // One Bridson step per warp on a random active point (poisson.rs:59-129): 30 candidates in
    // the shell [r, 2r], one per lane; the lowest valid lane is the step's winner.  Every lane
    // draws one Philox block of the warp's stream: lanes 0-29 place the candidates and lane 31's
    // draw picks the active point (shuffled to the warp); lane 0 records the pick for the
    // retirement.
    static_assert(SYN_HALO - SYN_SPILL == 2, "a candidate's neighbourhood reaches two cells");
    static_assert(SYN_K < 32, "lane 31 draws the pick");
    if (!FEW) {
      off = syn_draw(iter, tid, lane, colkey, s_key);
    } else if (warp == 0 && iter > 0) {
      off = s_off[lane];
    }
    const uint32_t rpick = __shfl_sync(0xffffffffu, __float_as_uint(off.x), 31);
    const int pick = static_cast<int>((static_cast<unsigned long long>(rpick) * static_cast<unsigned>(nact)) >> 32);
    if (lane == 0) reinterpret_cast<int*>(s_pick)[warp] = pick;
    const int pr = active[pick];
    const int prx = pr & 15, pry = (pr >> 4) & 15, prz = pr >> 8;
    const uint32_t pw = grid[(prz * SYN_R + pry) * SYN_R + prx];
    const int BX = (prx + ox) * SYN_Q + static_cast<int>(pw & 1023u);
    const int BY = (pry + oy) * SYN_Q + static_cast<int>((pw >> 10) & 1023u);
    const int BZ = (prz - 2) * SYN_Q + static_cast<int>((pw >> 20) & 1023u);
    bool valid = false;
    int X = 0, Y = 0, Z = 0, rb = 0;
    if (lane < SYN_K) {
      // Rounded down, so a negative coordinate fails the unsigned bound.
      X = __float2int_rd(__fadd_rn(static_cast<float>(BX), off.x));
      Y = __float2int_rd(__fadd_rn(static_cast<float>(BY), off.y));
      Z = __float2int_rd(__fadd_rn(static_cast<float>(BZ), off.z));
      // Candidates lie in the column and its spill; those of the staged region's cells 2 .. SYN_R - 3
      // in x and y (x1 <= x0 + SYN_B) and 2 .. nz - 3 in z (ZW <= gd * SYN_Q), so their
      // neighbourhoods lie inside the region.
      const int rx = (X >> 10) - ox, ry = (Y >> 10) - oy, rz = (Z >> 10) + 2;
      if (static_cast<uint32_t>(X) < t.XW && static_cast<uint32_t>(Y) < t.YW && static_cast<uint32_t>(Z) < t.ZW &&
          static_cast<uint32_t>(rx - (SYN_HALO - SYN_SPILL)) < static_cast<uint32_t>(x1 - x0 + 2 * SYN_SPILL) &&
          static_cast<uint32_t>(ry - (SYN_HALO - SYN_SPILL)) < static_cast<uint32_t>(y1 - y0 + 2 * SYN_SPILL)) {
        const int row = rz * SYN_R + ry;
        rb = row * SYN_R + rx;
        valid = syn_near_free(grid, rows, s_near, rx, row, rb, X & 1023, Y & 1023, Z & 1023);
      }
    }
    unsigned rest;
    const bool first = syn_outer_free(grid, rows, valid, rb, X & 1023, Y & 1023, Z & 1023, lane, rest);
    const bool none = __ballot_sync(0xffffffffu, first) == 0u;
    if (first || (none && lane == 0)) s_win[warp] = make_int4(X - ox * SYN_Q, Y - oy * SYN_Q, Z, first);
    if ((rest >> lane) & 1u) {
      s_cxy[warp][lane] = static_cast<uint32_t>(X - ox * SYN_Q) | static_cast<uint32_t>(Y - oy * SYN_Q) << 16;
      s_cz[warp][lane] = Z;
    }
    if (lane == 0) s_rmask[warp] = rest;
    __syncthreads();
    if (warp != 0) {
      // With registers to spare, the other warps draw for the next round meanwhile, one of them for
      // the resolving warp too.
      if (FEW) {
        if (warp == 1) s_off[lane] = syn_draw(iter + 1, lane, lane, colkey, s_key);
        off = syn_draw(iter + 1, tid, lane, colkey, s_key);
      }
    } else {
      // The round's steps in warp order, exactly as if they ran one after another: warp w keeps its
      // first candidate (lane order) that is free in the grid and at least r from the points
      // accepted for warps < w; with none left, its point retires.  The other warps wait meanwhile:
      // this is the round's serial part, kept short.
      //
      // Lane w speaks for warp w and holds its winner (first grid-free candidate).  That order keeps
      // a winner unless it lies within r of a point accepted for an earlier warp, so the warps keep
      // their winners in runs up to the next warp whose winner conflicts; only that warp searches
      // its other candidates against the points accepted so far.  The 64 pairs of winners are tested
      // two to a lane: lane 4 w + q holds warp w's against those of warps q and q + 4.
      static_assert(SYN_WARPS == 8, "two pairs of winners to a lane");
      auto close = [](const int4& p, const int4& q) {
        const int ex = p.x - q.x, ey = p.y - q.y, ez = p.z - q.z;
        return ex * ex + ey * ey + ez * ez < SYN_R2X;
      };
      int4 P = s_win[lane & 7];
      const int4 pw4 = s_win[lane >> 2];
      const unsigned b0 = __ballot_sync(0xffffffffu, close(pw4, s_win[lane & 3]));
      const unsigned b1 = __ballot_sync(0xffffffffu, close(pw4, s_win[(lane & 3) + 4]));
      const unsigned has = __ballot_sync(0xffffffffu, lane < SYN_WARPS && P.w != 0);  // warps with a winner
      const int sh = 4 * (lane & 7);
      // Bit u: this lane's winner conflicts with warp u's (u < lane).
      const unsigned cm = (((b0 >> sh) & 15u) | ((b1 >> sh) & 15u) << 4) & has & ((1u << (lane & 7)) - 1u);
      unsigned accw = 0, acc = 0;  // warps that keep their winner; warps that keep a point
      bool near = false;           // this lane's winner lies within r of a point kept instead of a winner
      for (int cur = 0; cur < SYN_WARPS;) {
        // A warp from cur on keeps its winner unless it conflicts with a kept point; up to the first
        // such warp, every warp with a winner keeps it.
        const unsigned from = ~((1u << cur) - 1u);
        const bool bad = lane >= cur && ((has >> lane) & 1u) != 0u && (near || (cm & (accw | from)) != 0u);
        const unsigned bm = __ballot_sync(0xffffffffu, bad);
        const int wb = bm ? __ffs(bm) - 1 : SYN_WARPS;
        const unsigned run = has & from & ((1u << wb) - 1u);
        accw |= run;
        acc |= run;
        if (wb == SYN_WARPS) break;
        // Warp wb: its first candidate after the winner that is at least r from every point kept
        // for warps < wb and passes the outer test, in lane order (the grid is as the candidate
        // phase saw it: the round commits after it is resolved).
        bool ok = (s_rmask[wb] >> lane) & 1u;
        int4 C = make_int4(0, 0, 0, 1);
        if (ok) {
          const uint32_t xy = s_cxy[wb][lane];
          C.x = static_cast<int>(xy & 0xffffu);
          C.y = static_cast<int>(xy >> 16);
          C.z = s_cz[wb][lane];
        }
        for (unsigned a = __any_sync(0xffffffffu, ok) ? acc : 0u; a; a &= a - 1u)
          if (close(C, s_win[__ffs(a) - 1])) ok = false;
        unsigned okm = __ballot_sync(0xffffffffu, ok);
        while (okm) {
          const int l = __ffs(okm) - 1;
          okm &= okm - 1;
          const int lx_ = __shfl_sync(0xffffffffu, C.x, l), ly_ = __shfl_sync(0xffffffffu, C.y, l);
          const int lz_ = __shfl_sync(0xffffffffu, C.z, l);
          const int cb = (((lz_ >> 10) + 2) * SYN_R + (ly_ >> 10)) * SYN_R + (lx_ >> 10);
          if (!syn_outer_hit(grid, rows, cb, lx_ & 1023, ly_ & 1023, lz_ & 1023, lane)) {
            if (lane == l) s_win[wb] = C;
            __syncwarp();
            const int4 N = s_win[wb];
            acc |= 1u << wb;
            if (lane == wb) P = N;
            near = near || close(P, N);  // looked at for the warps after wb only
            break;
          }
        }
        cur = wb + 1;
      }
      // Commit the kept points, appending to the active list in warp order.
      bool inside = false, committed = false;
      uint16_t cpos = 0;
      if (lane < SYN_WARPS && ((acc >> lane) & 1u)) {
        const int rx = P.x >> 10, ry = P.y >> 10, rz = (P.z >> 10) + 2;
        if (index_ok(rx >= 1 && rx < SYN_R && ry >= 1 && ry < SYN_R && rz >= 0 && rz < nz, err, SITE_SYN_COMMIT,
                     static_cast<uint32_t>(rx | (ry << 8) | (rz << 16)), blockIdx.x)) {
          cpos = syn_pos(rx, ry, rz);
          grid[(rz * SYN_R + ry) * SYN_R + rx] = syn_word(P.x, P.y, P.z);
          syn_mark(rows, rz * SYN_R + ry, rx);
          committed = true;
          inside = rx >= SYN_HALO && rx < SYN_HALO + bw && ry >= SYN_HALO && ry < SYN_HALO + bh;
        }
      }
      const unsigned im = __ballot_sync(0xffffffffu, inside);
      if (inside) {
        const int pos = nact + __popc(im & ((1u << lane) - 1u));
        if (index_ok(pos < acap, err, SITE_SYN_ACTIVE, pos, blockIdx.x)) active[pos] = cpos;
      }
      const unsigned cmm = __ballot_sync(0xffffffffu, committed);
      const int n0 = min(nact + __popc(im), acap);
      __syncwarp();  // the appended entries are visible to the retirement below
      // Retire the points of failed steps, each once, as if removed one after another in descending
      // list order, each by moving the list's current last entry into its place (a swap-remove).
      // The removal of rank k takes the entry then at n0 - 1 - k; when that position was itself
      // refilled by the removal of a lower rank, its entry is the one that removal took, and so on
      // down.  Nibble k of `tail` holds 1 + the rank of the pick at n0 - 1 - k, 0 for none.
      const int mypick = reinterpret_cast<const int*>(s_pick)[lane & 7];
      unsigned eq = 0, gt = 0;  // warps with this lane's pick; with a later one
#pragma unroll
      for (int h = 0; h < SYN_WARPS / 4; ++h) {
        const int4 q = s_pick[h];
        eq |= (q.x == mypick ? 1u : 0u) << (4 * h) | (q.y == mypick ? 2u : 0u) << (4 * h) |
              (q.z == mypick ? 4u : 0u) << (4 * h) | (q.w == mypick ? 8u : 0u) << (4 * h);
        gt |= (q.x > mypick ? 1u : 0u) << (4 * h) | (q.y > mypick ? 2u : 0u) << (4 * h) |
              (q.z > mypick ? 4u : 0u) << (4 * h) | (q.w > mypick ? 8u : 0u) << (4 * h);
      }
      const bool first = lane < SYN_WARPS && ((acc >> lane) & 1u) == 0u && (eq & ~acc & ((1u << lane) - 1u)) == 0u;
      const unsigned dm = __ballot_sync(0xffffffffu, first);
      int k = __popc(gt & dm);  // rank
      const unsigned at = static_cast<unsigned>(n0 - 1 - mypick);
      const unsigned tail = __reduce_or_sync(0xffffffffu, first && at < 8u ? static_cast<unsigned>(k + 1) << (4 * at) : 0u);
      if (tail && first) {
        for (int e; (e = static_cast<int>(tail >> (4 * k) & 15u)) != 0 && e - 1 < k;) k = e - 1;
      }
      const int src = n0 - 1 - k;
      uint16_t moved = 0;
      if (first && index_ok(src >= 0 && src < n0, err, SITE_SYN_ACTIVE, src, blockIdx.x)) moved = active[src];
      __syncwarp();
      if (first && src >= 0 && src < n0) active[mypick] = moved;
      if (lane == 0) {
        s_nact = n0 - __popc(dm);
        s_ncom += __popc(cmm);
      }
    }
  }
  __syncthreads();
  // Write back the column and its spill zone.
  for (int i = tid; i < ncell; i += blockDim.x) {
    const int rx = i % SYN_R, ry = (i / SYN_R) % SYN_R, rz = i / (SYN_R * SYN_R);
    if (rx < 2 || ry < 2 || rx >= SYN_R - 2 || ry >= SYN_R - 2) continue;
    const int gx = ox + rx, gy = oy + ry, gz = rz - 2;
    if (gx >= 0 && gy >= 0 && gz >= 0 && gx < static_cast<int>(t.gw) && gy < static_cast<int>(t.gh) && gz < gd)
      tc[(static_cast<size_t>(gz) * t.gh + gy) * t.gw + gx] = grid[i];
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    if (s_ncom) atomicAdd(npts + lo, static_cast<uint32_t>(s_ncom));
    atomicExch(done + blockIdx.x, 1u);
  }
}

// Cell of compaction slot sl: the brick (2D Morton over the high x, y bits) in the bits above
// 3 * brick_bits, the cell inside it (3D Morton, x lowest) below.
__device__ __forceinline__ void slot_cell(const SynthTile& t, uint32_t sl, uint32_t& x, uint32_t& y, uint32_t& z) {
  const uint32_t L = t.brick_bits;
  const uint32_t lo = sl & ((1u << (3 * L)) - 1u), hi = sl >> (3 * L);
  x = (morton2_compact(hi) << L) | morton3_compact(lo);
  y = (morton2_compact(hi >> 1) << L) | morton3_compact(lo >> 1);
  z = morton3_compact(lo >> 2);
}

// A part's cells as a warp reads them, word j of 16, one cell a lane.  A part of a brick of 8 cells or
// more is a cube of 8 x 8 x 8, read in rows of 8 (a sector) and not in slot order; of a smaller brick,
// 512 consecutive slots.
struct PartCells {
  bool cube, in;               // in: some cells lie inside the grid (its first slot, the lowest corner, does)
  uint32_t lin, row4, layer;   // cube: the lane's cell of word 0 (linear index), steps of 4 rows, of a layer
  uint32_t words;              // cube: bit j: the lane's cell of word j is inside the grid
};
__device__ __forceinline__ PartCells part_cells(const SynthTile& t, uint32_t p, uint32_t lane) {
  PartCells c;
  uint32_t x, y, z;
  slot_cell(t, p * SYN_PART, x, y, z);
  c.in = x < t.gw && y < t.gh && z < t.gd;
  c.cube = t.brick_bits >= 3;
  x += lane & 7u;
  y += lane >> 3;
  c.row4 = 4u * t.gw;
  c.layer = t.gh * t.gw;
  c.lin = z * c.layer + y * t.gw + x;
  const uint32_t nz = min(t.gd - z, 8u);  // layers inside
  c.words = x >= t.gw ? 0u
                      : (y < t.gh ? 0x5555u : 0u) & ((1u << (2 * nz)) - 1u) |
                            (y + 4u < t.gh ? 0xaaaau : 0u) & ((1u << (2 * nz)) - 1u);
  return c;
}
// The linear index of the lane's cell of word j, NO_CELL outside the grid; its slot in the part.
constexpr uint32_t NO_CELL = 0xffffffffu;
__device__ __forceinline__ uint32_t part_cell(const SynthTile& t, const PartCells& c, uint32_t p, uint32_t j, uint32_t lane) {
  if (c.cube) return (c.words >> j) & 1u ? c.lin + (j & 1u) * c.row4 + (j >> 1) * c.layer : NO_CELL;
  uint32_t x, y, z;
  const uint32_t sl = p * SYN_PART + j * 32 + lane;
  slot_cell(t, sl, x, y, z);
  return sl < t.slots && x < t.gw && y < t.gh && z < t.gd ? (z * t.gh + y) * t.gw + x : NO_CELL;
}
__device__ __forceinline__ uint32_t part_slot(const PartCells& c, uint32_t j, uint32_t lane) {
  if (!c.cube) return j * 32 + lane;
  const uint32_t x = lane & 7u, y = lane >> 3, z = j >> 1;
  return (x & 1u) | (x & 2u) << 2 | (x & 4u) << 4 | (y & 1u) << 1 | (y & 2u) << 3 | (j & 1u) << 7 | (z & 1u) << 2 |
         (z & 2u) << 4 | (z & 4u) << 6;
}
// Bit j: the lane's cell of word j holds a point (the loads are in flight together).
__device__ __forceinline__ uint32_t part_points(const SynthTile& t, const PartCells& c, const uint32_t* tc, uint32_t p,
                                                uint32_t lane) {
  uint32_t occ = 0;
  if (c.cube) {
#pragma unroll
    for (uint32_t j = 0; j < SYN_PART / 32; ++j)
      occ |= ((c.words >> j) & 1u ? tc[c.lin + (j & 1u) * c.row4 + (j >> 1) * c.layer] >> 31 : 0u) << j;
  } else {
    for (uint32_t j = 0; j < SYN_PART / 32; ++j) {
      const uint32_t lin = part_cell(t, c, p, j, lane);
      occ |= (lin != NO_CELL ? tc[lin] >> 31 : 0u) << j;
    }
  }
  return occ;
}

// Thinning to the Bridson-expected count (a point goes with the probability of the excess, n points as
// counted by k_bridson), and the points left per part, a warp to a part.  The draws run over the
// part's points, with the lanes busy.  blockIdx.y is the tile.
//
// Bound by the latency of its loads (DRAM 15 %).  A pass for thinning and one for the counts, a block to
// a brick of up to 32^3 cells, took 320 + 420 us on a 1600 x 1600 px t-max image, this one 438; for the
// four bricks of a 64 x 64 px tri-x tile 3.5 + 24 us, now 7.4.
constexpr int PART_T = 256;
__global__ void __launch_bounds__(PART_T) k_thin_count(const SynthTile* __restrict__ tiles, uint32_t* __restrict__ cells,
                                                       const uint32_t* __restrict__ npts, uint32_t* __restrict__ counts) {
  const SynthTile& t = tiles[blockIdx.y];
  const uint32_t nparts = syn_parts(t), lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
  const uint32_t n = npts[blockIdx.y];
  const bool thin = n > t.target;
  const float excess = 1.0f - static_cast<float>(t.target) / static_cast<float>(n);
  uint32_t* tc = cells + t.cell_base;
  __shared__ uint32_t s_q[PART_T / 32][SYN_PART];  // the part's points
  uint32_t* q = s_q[threadIdx.x >> 5];
  for (uint32_t p = blockIdx.x * (PART_T / 32) + (threadIdx.x >> 5); p < nparts; p += gridDim.x * (PART_T / 32)) {
    const PartCells c = part_cells(t, p, lane);
    uint32_t left = 0;
    if (c.in) {
      const uint32_t occ = part_points(t, c, tc, p, lane);
      left = __popc(occ);
      if (thin) {
        uint32_t fill = 0;
        for (uint32_t j = 0; j < SYN_PART / 32; ++j) {
          const unsigned m = __ballot_sync(0xffffffffu, (occ >> j) & 1u);
          if ((occ >> j) & 1u) q[fill + __popc(m & lt)] = part_cell(t, c, p, j, lane);
          fill += __popc(m);
        }
        __syncwarp();
        for (uint32_t i = lane; i < fill; i += 32) {
          const uint32_t lin = q[i];
          if (uf(philox(lin, 0, 0, TAG_THIN, t.k0, t.k1).x) < excess) {
            tc[lin] = 0;
            --left;
          }
        }
        __syncwarp();
      }
      left = __reduce_add_sync(0xffffffffu, left);
    }
    if (lane == 0) counts[t.slot_base + p] = left;
  }
}

// Crystal k of a tile, the one of cell (x, y, z): position from the fixed-point cell
// word, attributes from the tile's Philox stream keyed by the cell (emulsion.rs:162-200).
__device__ __forceinline__ void emit_crystal(const SynthTile& t, const uint32_t* __restrict__ cells, uint32_t x,
                                             uint32_t y, uint32_t z, uint32_t k, float4* A, float4* Q, float4* D) {
  const uint32_t lin = (z * t.gh + y) * t.gw + x;
  const uint32_t w = cells[t.cell_base + lin];
  const float px = static_cast<float>(static_cast<int>(x) * SYN_Q + static_cast<int>(w & 1023u)) * (t.cell / SYN_Q);
  const float py = static_cast<float>(static_cast<int>(y) * SYN_Q + static_cast<int>((w >> 10) & 1023u)) * (t.cell / SYN_Q);
  const float pz = static_cast<float>(static_cast<int>(z) * SYN_Q + static_cast<int>((w >> 20) & 1023u)) * (t.cell / SYN_Q);
  const P4 r0 = philox(lin, 0, 0, TAG_ATTR, t.k0, t.k1);
  const P4 r1 = philox(lin, 1, 0, TAG_ATTR, t.k0, t.k1);
  // Two normals from one Box-Muller pair: radius (log-normal) and sensitivity.
  const float bm = sqrtf(-2.0f * logf(1.0f - uf(r0.x)));
  float s2, c2;
  sincospif(2.0f * uf(r0.y), &s2, &c2);
  const float radius = fminf(fmaxf(expf(t.mu + t.sg * bm * c2), 0.15f), t.rmax);
  const float sens = fmaxf(t.base_sens + 0.15f * bm * s2, 0.1f);
  float4 q, d;
  if (t.morph == 1) {
    // Tabular: thickness r / AR (>= 0.05), tilt +-0.17 rad about a random in-plane axis.
    const float ht = fmaxf(radius / t.aspect, 0.05f);
    const float tilt = uf(r0.z) * 0.34f - 0.17f;
    float ax = uf(r0.w) * 2.0f - 1.0f, ay = uf(r1.x) * 2.0f - 1.0f;
    const float n = rsqrtf(fmaxf(ax * ax + ay * ay, 1e-30f));
    ax *= n;
    ay *= n;
    float sh, ch;
    sincosf(0.5f * tilt, &sh, &ch);
    q = make_float4(ax * sh, ay * sh, 0.0f, ch);
    d = make_float4(radius, radius, ht, __int_as_float(1));
  } else {
    // Cubic / octahedral: UnitQuaternion::from_euler_angles(2 pi u1, pi u2, 2 pi u3).
    float sr, cr, sp, cp, sy, cy;
    sincospif(uf(r0.z), &sr, &cr);        // roll / 2 = pi u1
    sincospif(0.5f * uf(r0.w), &sp, &cp); // pitch / 2 = pi u2 / 2
    sincospif(uf(r1.x), &sy, &cy);        // yaw / 2 = pi u3
    q = make_float4(sr * cp * cy - cr * sp * sy, cr * sp * cy + sr * cp * sy, cr * cp * sy - sr * sp * cy,
                    cr * cp * cy + sr * sp * sy);
    d = make_float4(radius, radius, radius, __int_as_float(t.morph));
  }
  const unsigned long long o = t.cbase + k;
  A[o] = make_float4(px, py, pz, sens);
  Q[o] = q;
  D[o] = d;
}

// The crystals of each part in slot order (slot_cell), numbered after the points of the earlier parts
// (scan: exclusive sum of k_thin_count).  A warp to a part, without the block's barriers: a part's words
// are loaded together, and as about one cell in nine holds a point, the warp queues the occupied ones
// and makes 32 crystals at a time, with every lane busy; the queue outlives the part.
// blockIdx.y is the tile.
//
// Bound by the latency of its loads.  A block to a brick, with its barriers, took 85 us for the four
// bricks of a 64 x 64 px tri-x tile (now 9.8), 475 us for a 2048 x 2048 px image (now 213) and 1,100 us for
// 1600 x 1600 px of t-max (now 683).
__global__ void __launch_bounds__(PART_T) k_emit(const SynthTile* __restrict__ tiles,
                                                 const uint32_t* __restrict__ cells,
                                                 const uint32_t* __restrict__ scan, float4* A, float4* Q,
                                                 float4* D, uint32_t* err) {
  const SynthTile& t = tiles[blockIdx.y];
  const uint32_t nparts = syn_parts(t);
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
  const uint32_t* tc = cells + t.cell_base;
  const uint32_t kbase = scan[t.slot_base];
  __shared__ uint2 s_q[PART_T / 32][64];             // queued crystals: number and slot
  __shared__ uint32_t s_m[PART_T / 32][SYN_PART / 32];  // the part's points in slot order
  uint32_t* pts = s_m[warp];
  uint2* q = s_q[warp];
  uint32_t fill = 0;  // the same in every lane
  auto emit = [&](uint2 c) {
    if (c.x >= t.ccap) {  // past the tile's capacity
      atomicOr(err, ERR_LIST_OVERFLOW);
      return;
    }
    uint32_t x, y, z;
    slot_cell(t, c.y, x, y, z);
    emit_crystal(t, cells, x, y, z, c.x, A, Q, D);
  };
  for (uint32_t p = blockIdx.x * (PART_T / 32) + warp; p < nparts; p += gridDim.x * (PART_T / 32)) {
    const uint32_t k0 = scan[t.slot_base + p];
    if (scan[t.slot_base + p + 1] == k0) continue;
    uint32_t k = k0 - kbase;
    const PartCells c = part_cells(t, p, lane);
    const uint32_t occ = part_points(t, c, tc, p, lane);
    if (lane < SYN_PART / 32) pts[lane] = 0;
    __syncwarp();
#pragma unroll
    for (uint32_t j = 0; j < SYN_PART / 32; ++j)
      if ((occ >> j) & 1u) {
        const uint32_t sl = part_slot(c, j, lane);
        atomicOr(pts + (sl >> 5), 1u << (sl & 31u));
      }
    __syncwarp();
    for (uint32_t j = 0; j < SYN_PART / 32; ++j) {
      const unsigned m = pts[j];
      const bool o = (m >> lane) & 1u;
      const uint32_t r = __popc(m & lt);
      if (o) q[fill + r] = make_uint2(k + r, p * SYN_PART + j * 32 + lane);
      k += __popc(m);
      fill += __popc(m);
      __syncwarp();
      if (fill >= 32) {
        const uint2 mine = q[lane];
        const uint32_t rest = fill - 32;
        const uint2 moved = lane < rest ? q[32 + lane] : make_uint2(0u, 0u);
        __syncwarp();
        if (lane < rest) q[lane] = moved;
        fill = rest;
        __syncwarp();
        emit(mine);
      }
    }
  }
  if (lane < fill) emit(q[lane]);
}

// Host wrappers (launch on `st`; all buffers preallocated so the sequence can be graph-captured).
// cols[c] columns of class c; done holds one flag per column (zeroed here).
void launch_bridson(const SynthTile* tiles, int ntiles, const unsigned cols[4], int gdmax, uint32_t* cells,
                    uint32_t* npts, uint32_t* done, uint32_t* err, cudaStream_t st, int sms, uint32_t wait_limit,
                    const uint32_t* probe) {
  const unsigned total = cols[0] + cols[1] + cols[2] + cols[3];
  if (total == 0) return;
  const int nz = gdmax + 4;
  const size_t smem = bridson_smem(gdmax);
  FG_CUDA(cudaMemsetAsync(done, 0, total * sizeof(uint32_t), st));
  const auto kernel = total <= SYN_FEW * static_cast<unsigned>(sms) ? k_bridson<true> : k_bridson<false>;
  // The most that any launch asks for, whatever this one does: the attribute is the process's, and another
  // thread's launch may come between.
  FG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(BRIDSON_SMEM_MAX)));
  const uint4 cb = make_uint4(0u, cols[0], cols[0] + cols[1], cols[0] + cols[1] + cols[2]);
  kernel<<<total, SYN_WARPS * 32, smem, st>>>(tiles, ntiles, cb, nz, cells, npts, done, err,
                                                  wait_limit ? wait_limit : (1u << 22), probe);
  FG_CUDA(cudaGetLastError());
}

static unsigned part_blocks(unsigned long long max_parts) {
  return static_cast<unsigned>(std::min<unsigned long long>((max_parts + PART_T / 32 - 1) / (PART_T / 32), 4096));
}
// Per-tile grids (blockIdx.y is the tile): max_parts: the largest tile's.
void launch_synth_post(const SynthTile* tiles, int ntiles, unsigned long long max_parts, uint32_t* cells,
                       const uint32_t* npts, uint32_t* counts, cudaStream_t st) {
  if (ntiles == 0) return;
  FG_REQUIRE(ntiles <= 65535, "too many tiles for one launch");
  k_thin_count<<<dim3(part_blocks(max_parts), ntiles), PART_T, 0, st>>>(tiles, cells, npts, counts);
  FG_CUDA(cudaGetLastError());
}

void launch_emit(const SynthTile* tiles, int ntiles, unsigned long long max_parts, const uint32_t* cells,
                 const uint32_t* scan, float4* A, float4* Q, float4* D, uint32_t* err, cudaStream_t st) {
  if (ntiles == 0) return;
  FG_REQUIRE(ntiles <= 65535, "too many tiles for one launch");
  k_emit<<<dim3(part_blocks(max_parts), ntiles), PART_T, 0, st>>>(tiles, cells, scan, A, Q, D, err);
  FG_CUDA(cudaGetLastError());
}

}  // namespace fg
