// Crystals in uniform cells, for the transport's segments and the development's touch queries.
//
// A walk of the reference's tree is needed only for what it decides: which leaves a segment
// reaches, and the order of its hits.  Both are static per crystal: a crystal is hit iff its
// geometry is hit and its leaf's box passes the reference's slab test (an ancestor's box contains
// the leaf's, so it passes too), and the walk visits leaves in one fixed order (right subtree
// first), so every crystal has a rank in it.  The candidates themselves come from cells: each
// crystal is listed once, in the cell of its centre, and a segment visits the rows of cells within
// the crystals' reach of it.  Cells are x-fastest, so the crystals of a row's x span are one
// contiguous range.
#pragma once
#include <math.h>

#include "fg_device.cuh"

namespace fg {

// One axis of a grid of cells: n cells of edge `edge` um from 0 (inv = 1 / edge, last = n - 1).
struct __align__(16) CellAxis {
  float inv, edge, last;
  uint32_t n;
};

// One tile's (or emulsion's) cells over the box from the origin; every crystal's centre lies in the
// box.  Positions (crystals in cell order) count over the whole allocation; off holds the first
// position of each of the tile's cells and of the one after.
struct __align__(16) CellGrid {
  CellAxis x, y, z;
  const float4* pos;      // centre xyz, squared radius of the ball the crystal lies in (with margin)
  const uint32_t* off;
  uint32_t npos;          // positions of the allocation (bounds the ranges read from off)
  float reach;            // how far from a segment the centre of a crystal it hits can lie
  float slack;            // um, far above FP32 rounding of the coordinates
  float _pad;
  const float4* q;
  const float4* d;
  const float4* leaf;     // two per position: leaf box lo xyz, hi x; hi y, hi z, rank, slot (bits)
  const uint2* by_rank;   // per rank: crystal slot, sensitivity (bits)
  unsigned long long cell_base;  // first cell of this tile in the allocation
  float hx, hy, hz;       // the box
};

// Sets the reach of a set whose largest half-dimension is m (a cube reaches sqrt(3) m).
inline void cells_reach(CellGrid& g, double m, bool cubes) {
  g.reach = static_cast<float>(m * (cubes ? 1.7320508075688773 : 1.0) * 1.002) + g.slack;
}

// Cells suit a crystal set whose crystals reach no further than the mean spacing and that fills the
// box evenly: then a segment tests a handful of crystals per layer of cells.  One giant crystal
// drags every segment's rows out to its reach, a set bunched in a corner puts many crystals into one
// cell, and a centre outside the box has no cell; such sets keep the tree walk, whose cost follows
// the boxes.  Measured with one giant among the crystals of a 140 um film (ms, cells / walk): none
// (reach 0.4 spacings for t-max's, 0.7 for tri-x's) 0.49 / 0.92 and 0.47 / 0.72; reach 1 spacing
// 0.92 / 0.93 and 0.63 / 0.82; 1.5 spacings 1.45 / 0.90 and 0.97 / 0.91.
constexpr double CELLS_MAX_REACH = 1.0;      // mean spacings, of an emulsion's largest crystal
constexpr uint32_t CELLS_MAX_COUNT = 16;     // crystals in one cell (half a crystal on average)
constexpr uint32_t CELLS_UNEVEN_MIN = 512;   // crystals from which the set's unevenness is looked at
// A synthesized tile's reach is that of nearly all its crystals; 200-256 px of t-max crystals thicker than wide
// (ms, cells / walk): 2.0 spacings 2.79 / 3.40, 2.7 spacings 5.90 / 5.43, 4.0 spacings 13.3 / 10.0.
constexpr double CELLS_MAX_REACH_ALL = 2.5;
// A segment of many hits is visited again for every twelve, so its cost grows with the square of its hits
// (cells_hits: H), the walk's with the hits.  Transport of 200 x 200 px films, 10 to 60 um deep, mean free path
// 20 um to none (cells / walk): tri-x H 9 .57, 13 .71 - .86, 18 .82 - .98, 20 .99, 23 1.03 - 1.15, 27 1.14 - 1.32,
// 40 1.76; hp5 H 19 .69, 23 .88; t-max H 8 .58.
constexpr double CELLS_MAX_HITS = 20.0;
// In uploaded sets it also grows with the crystals' reach.  Lattices, reach in spacings and where cells
// and walk are even: .42 H 18 - 20, .6 H 16, .72 H 14, .9 H 11 - 14, .99 H 9 (H 16: 1.2 - 1.6; H 78: 4 - 6).  Uneven
// sets, by the density about a crystal (H, reach in its spacings, cells / walk): 6.5 .45 .57 - .63; 9.9 .52 .67 - .87;
// 12 .56 .74 - .96; 11 .72 1.04 - 1.27; 14 .77 1.02 - 1.35; 16 .61 1.2 - 1.5; 18 .85 1.8 - 2.3.
constexpr double CELLS_MAX_HITS_REACH = 7.5;  // hits times spacings of reach, uploaded sets

// Hits that a segment expects to absorb, weighted by hits (E[h^2] / E[h]): per_um of them per um of a free
// path of mean 1 / mu_t that ends after `length` um at the latest: the film's smallest extent (photons leave
// a narrow film by its sides: exposing 14 x 14 um of tri-x 50 um deep takes .26 ms by the cells, .54 by the walk;
// 30 x 30 um .45 and .82; 90 x 90 um, where the depth is the smallest, 1.23 and 1.27).
inline double cells_hits(double per_um, double mu_t, double length) {
  const double x = mu_t * length;
  if (!(x > 1e-3)) return per_um * length;
  const double e = std::exp(-x);
  return per_um * 2.0 * (1.0 - e * (1.0 + x)) / (mu_t * (1.0 - e));
}

// Mean projected area (um^2) of a crystal of half-sizes a, b, c: a quarter of a box's surface (Cauchy); for the
// ellipsoid shapes pi times the mean product of two.
inline double cells_area(double a, double b, double c, bool cube) {
  return (a * b + b * c + c * a) * (cube ? 2.0 : 1.0471975511965976);
}

// Cell edges in units of the mean crystal spacing a = (volume / crystals)^(1/3).  Rows run along x,
// so x cells are short (a row's span is cut close to the segment at no cost); rows are wide and
// layers high enough that a row holds a few crystals near the segment.  Transport of 800 x 800 px
// t-max / 1600 x 1600 tri-x / 1200 x 1200 hp5 images (ms): 0.2, 1, 2: 3.49 / 4.04 / 2.86; 0.3, 1, 3:
// 3.49 / 4.10 / 2.90; 0.3, 0.75, 1.5: 3.60 / 4.30 / 2.96; layers of the full depth: 5.4 / 25 / 5.4.
constexpr double CELL_X = 0.20, CELL_Y = 1.0, CELL_Z = 2.5;

// Cells of a box of w x h x d um holding about n crystals, at most 8 n + 64 of them.  The cells of an axis
// are numbered in float arithmetic and those of the box in 32 bits, which the prefix sum over an emulsion's
// cells counts with a sign, so an axis has at most 2^24 (their numbers are exact: rounded up, the last one
// would name a cell past the row) and the box fewer than 2^31.  False when the box has no volume.
constexpr double CELLS_AXIS_MAX = 16777216.0, CELLS_BOX_MAX = 2147483000.0;
inline bool cells_layout(double w, double h, double d, double n, CellGrid& g) {
  if (!(w > 0 && h > 0 && d > 0 && n > 0) || !std::isfinite(w * h * d)) return false;
  double a = std::cbrt(w * h * d / n);
  double cx, cy, cz;
  for (;; a *= 1.25) {
    cx = std::fmax(std::floor(w / (CELL_X * a)), 1.0);
    cy = std::fmax(std::floor(h / (CELL_Y * a)), 1.0);
    cz = std::fmax(std::floor(d / (CELL_Z * a) + 0.5), 1.0);
    if (cx * cy * cz <= std::fmin(8.0 * n + 64.0, CELLS_BOX_MAX) &&
        std::fmax(std::fmax(cx, cy), cz) <= CELLS_AXIS_MAX)
      break;
  }
  auto axis = [](CellAxis& x, double len, double cells) {
    x.n = static_cast<uint32_t>(cells);
    x.last = static_cast<float>(cells - 1.0);
    x.edge = static_cast<float>(len / cells);
    x.inv = static_cast<float>(cells / len);
  };
  axis(g.x, w, cx);
  axis(g.y, h, cy);
  axis(g.z, d, cz);
  g.hx = static_cast<float>(w);
  g.hy = static_cast<float>(h);
  g.hz = static_cast<float>(d);
  g.slack = static_cast<float>(2e-3 + 2e-6 * std::fmax(std::fmax(w, h), d));
  return true;
}
inline unsigned long long cells_of(const CellGrid& g) {
  return static_cast<unsigned long long>(g.x.n) * g.y.n * g.z.n;
}

// Cell of coordinate v along an axis, clamped to its cells: monotone in v, so a query over [lo, hi]
// finds every centre in [lo, hi].
__device__ __forceinline__ int cell_coord(float v, float inv, float last) {
  return __float2int_rz(fminf(fmaxf(v * inv, 0.0f), last));
}

// Squared radius of the ball around the centre that holds the crystal (a cube lies in the ball of
// radius sqrt(3) m, the ellipsoid shapes in that of radius m), with a margin far above rounding.
__device__ __forceinline__ float cell_ball2(const float4& d) {
  const float m = fmaxf(fmaxf(d.x, d.y), d.z);
  const float R = (morph_of(d) == 0 ? 1.7320509f * m : m) * 1.001f + 1e-3f;
  return R * R;
}

// The row-by-row visit of the cells near a segment [0, step] of a ray: layers of cells along z,
// in each the rows along y that the part of the segment within reach of the layer comes near, in
// each row the x span of the part within reach of the row.
struct CellVisit {
  float step;
  float ta, tb;           // part of the segment within reach of the layer
  int iz, iz1, iy, iy1;   // layer and its last, next row and its last
  uint32_t c, cend;       // positions of the row still to test
};

// The grid must lie in device memory (the read goes through the read-only path).
__device__ __forceinline__ CellAxis cell_axis(const CellAxis& a) {
  const float4 v = __ldg(reinterpret_cast<const float4*>(&a));
  return CellAxis{v.x, v.y, v.z, __float_as_uint(v.w)};
}

__device__ __forceinline__ void cells_begin(const CellGrid& g, float3 o, float3 dir, float step, CellVisit& v) {
  const CellAxis az = cell_axis(g.z);
  const float R = g.reach;
  const float z1 = fmaf(dir.z, step, o.z);
  v.step = step;
  v.iz = cell_coord(fminf(o.z, z1) - R, az.inv, az.last) - 1;
  v.iz1 = cell_coord(fmaxf(o.z, z1) + R, az.inv, az.last);
  v.iy = 1;
  v.iy1 = 0;
  v.c = v.cend = 0;
}

__device__ __forceinline__ bool cells_done(const CellVisit& v) {
  return v.c >= v.cend && v.iy > v.iy1 && v.iz >= v.iz1;
}

// The part of [t0, t1] in which o + t d lies within R of cell k's extent along an axis.
__device__ __forceinline__ void cell_clip(float o, float inv, int k, float edge, float R, float& t0, float& t1) {
  const float lo = fmaf(static_cast<float>(k), edge, -R), hi = fmaf(static_cast<float>(k + 1), edge, R);
  const float a = (lo - o) * inv, b = (hi - o) * inv;
  t0 = fmaxf(t0, fminf(a, b));
  t1 = fminf(t1, fmaxf(a, b));
}

// Goes to the next row (the next layer first when this one is done) and its range of positions.
// Only for a visit that is not done.  inv_y, inv_z: 1 / dir (kept finite).
__device__ __forceinline__ void cells_advance(const CellGrid& g, float3 o, float3 dir, float inv_y, float inv_z,
                                              CellVisit& v, uint32_t* err) {
  const CellAxis ay = cell_axis(g.y), ax = cell_axis(g.x);
  const float R = g.reach;
  if (v.iy > v.iy1) {
    const CellAxis az = cell_axis(g.z);
    ++v.iz;
    v.ta = 0.0f;
    v.tb = v.step;
    cell_clip(o.z, inv_z, v.iz, az.edge, R, v.ta, v.tb);
    if (!(v.ta <= v.tb)) return;
    const float ya = fmaf(dir.y, v.ta, o.y), yb = fmaf(dir.y, v.tb, o.y);
    v.iy = cell_coord(fminf(ya, yb) - R, ay.inv, ay.last);
    v.iy1 = cell_coord(fmaxf(ya, yb) + R, ay.inv, ay.last);
  }
  const int y = v.iy++;
  float t0 = v.ta, t1 = v.tb;
  cell_clip(o.y, inv_y, y, ay.edge, R, t0, t1);
  if (!(t0 <= t1)) return;
  const float xa = fmaf(dir.x, t0, o.x), xb = fmaf(dir.x, t1, o.x);
  const uint32_t* row = g.off + (static_cast<uint32_t>(y) * g.z.n + static_cast<uint32_t>(v.iz)) * ax.n;
  const uint32_t c0 = __ldg(row + cell_coord(fminf(xa, xb) - R, ax.inv, ax.last));
  const uint32_t c1 = __ldg(row + cell_coord(fmaxf(xa, xb) + R, ax.inv, ax.last) + 1);
  if (!index_ok(c0 <= c1 && c1 <= g.npos, err, SITE_CELL, c0, c1)) return;
  v.c = c0;
  v.cend = c1;
}

// Every crystal after position p whose centre lies within R of p's centre a in each axis (fn(position,
// squared distance)): the rows from p's own on, so each pair is seen once, from its first crystal.
template <class F>
__device__ __forceinline__ void cells_around(const CellGrid& g, float3 a, float R, uint32_t p, uint32_t* err, F&& fn) {
  const CellAxis ax = cell_axis(g.x), ay = cell_axis(g.y), az = cell_axis(g.z);
  const float Rs = R + g.slack;
  const int x0 = cell_coord(a.x - Rs, ax.inv, ax.last), x1 = cell_coord(a.x + Rs, ax.inv, ax.last);
  const int z0 = cell_coord(a.z - Rs, az.inv, az.last), z1 = cell_coord(a.z + Rs, az.inv, az.last);
  const int yc = cell_coord(a.y, ay.inv, ay.last), y1 = cell_coord(a.y + Rs, ay.inv, ay.last);
  const int zc = cell_coord(a.z, az.inv, az.last);
  for (int y = yc; y <= y1; ++y)
    for (int z = y == yc ? zc : z0; z <= z1; ++z) {
      const uint32_t* row = g.off + (static_cast<uint32_t>(y) * az.n + static_cast<uint32_t>(z)) * ax.n;
      const uint32_t c0 = y == yc && z == zc ? p + 1 : __ldg(row + x0), c1 = __ldg(row + x1 + 1);
      if (!index_ok(c1 <= g.npos, err, SITE_CELL, c0, c1)) continue;
      for (uint32_t c = c0; c < c1; ++c) {
        const float4 b = __ldg(&g.pos[c]);
        const float dx = b.x - a.x, dy = b.y - a.y, dz = b.z - a.z;
        fn(c, dx * dx + dy * dy + dz * dz);
      }
    }
}

// Crystal slot at a position.
__device__ __forceinline__ uint32_t cell_slot(const CellGrid& g, uint32_t p) {
  return __float_as_uint(__ldg(&g.leaf[2ull * p + 1].w));
}

}  // namespace fg
